// bfloat16 products of at most 8 rows of x with the RMSNorm before them: out[m][n] = (norm(x)[m] . w[n]) (+ bias[n]) (+
// residual[m][n]), or the gated form act(.) * (.) over [gate; up] rows. norm(x) = x * g * rsqrt(mean(x^2) + eps): x * g is
// rounded to bfloat16 as the operand, the root joins the float32 sum, as in the norm that gemm_tcgen05.cu spreads over two
// products; without g, x itself is the operand.
//
// A decode step is a chain of such products of a few megabytes, each waiting for the one before, so what counts is the time from
// the wait to the last output. Against the 128-row tiles of gemm_tcgen05.cu (tensor maps, tensor memory, partial sums through
// L2 and a last arrival) this form has little to set up and nothing to hand over: a block streams 16 or 32 rows of w in
// 16-byte pieces straight from global memory into mma.sync fragments (m16n8k16: weights on the 16, tokens on the 8; k is
// permuted alike in both operands so that a lane's 16 bytes are whole fragments), its 8 warps take alternate runs of 128 k,
// and a cluster of up to 4 blocks shares the k range where the rows alone give too few blocks; parts meet in shared memory, in
// a fixed order. Every block squares the rows of x it reads anyway, so no kernel before has to leave sums for it. The first
// weights are asked for before the wait for the kernels ahead.
// The 5th-generation tensor cores would not help: the arithmetic is 2 % of what mma.sync can do, the weights' way from HBM is
// the bound.
// A layer of 31 MB (hidden size 1024): 5.0 us a product against 7.9, a step of 28 layers 1036 -> 916 us with one token, 1105 -> 1023
// with 8. Where a product takes more than a wave of blocks it loses: the blocks of the kernel behind it, started early, wait in
// the places that its own last blocks want. A layer of 101 MB (hidden size 2048): 1325 us the other way, 1371 this; of 386 MB 3173 and
// 4198. Fewer, larger or pinned blocks that walk over the rows did not mend that (1681 us and more for the layer of 101 MB).
#pragma once
#include "common.cuh"
#include <cooperative_groups.h>

namespace few {

constexpr int WARPS = 8, THREADS = WARPS * 32;
constexpr int STEP = 32, STEPS = 4, RUN = STEP * STEPS;      // k of one lane's 16 bytes over four lanes; of a warp's turn
constexpr int MAX_ROWS = 8;

struct Args {
    __nv_bfloat16* out;
    const __nv_bfloat16 *x, *w, *residual;
    const float *g, *bias;
    float eps;
    int M, N, K;                                             // gated: w has 2N rows
};

__device__ __forceinline__ uint4 load_weights(const __nv_bfloat16* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
// x may have been written by a kernel that this one overlaps with: no read-only path.
__device__ __forceinline__ uint4 load_rows(const __nv_bfloat16* p) {
    uint4 v;
    asm volatile("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// Multiplies two neighbouring x by g, rounds, and adds their squares up.
__device__ __forceinline__ uint32_t scaled(uint32_t u, float g0, float g1, float& squares) {
    const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u));
    squares = fmaf(f.x, f.x, squares);
    squares = fmaf(f.y, f.y, squares);
    const __nv_bfloat162 r = __floats2bfloat162_rn(f.x * g0, f.y * g1);
    return *reinterpret_cast<const uint32_t*>(&r);
}

// TILES: 16-row tiles of w a block holds (gated: the first half gate rows, the second the up rows of the same outputs).
// GATED: 0 no, 1 silu, 2 the tanh form of gelu.
template <int TILES, bool NORM, int GATED>
__global__ void __launch_bounds__(THREADS) gemm_few_kernel(const Args a) {
    constexpr int ROWS = 16 * TILES, OUTS = GATED ? ROWS / 2 : ROWS;
    __shared__ float part[WARPS][MAX_ROWS][ROWS];
    __shared__ float part_sq[WARPS][MAX_ROWS];
    __shared__ float sums[MAX_ROWS][ROWS], squares_sh[MAX_ROWS];
    ti_grid_launch_dependents();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t4 = lane & 3;
    const int splits = (int)gridDim.x, rank = (int)blockIdx.x;           // the cluster spans gridDim.x
    const int n0 = (int)blockIdx.y * OUTS;
    const __nv_bfloat16* row[TILES][2];
#pragma unroll
    for (int i = 0; i < TILES; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int r = 16 * i + 8 * h + g, o = min(n0 + (GATED ? r % OUTS : r), a.N - 1);
            row[i][h] = a.w + (size_t)(GATED && r >= OUTS ? a.N + o : o) * a.K + t4 * 8;
        }
    const __nv_bfloat16* xrow = a.x + (size_t)min(g, a.M - 1) * a.K + t4 * 8;
    float c[TILES][4] = {};
    float sq = 0.f;
    bool waited = false;
    for (int k0 = (rank * WARPS + warp) * RUN; k0 < a.K || !waited; k0 += splits * WARPS * RUN) {
        uint4 wv[TILES][STEPS][2];
#pragma unroll
        for (int s = 0; s < STEPS; ++s) {
            const bool in = k0 + s * STEP + t4 * 8 < a.K;
#pragma unroll
            for (int i = 0; i < TILES; ++i)
#pragma unroll
                for (int h = 0; h < 2; ++h) wv[i][s][h] = in ? load_weights(row[i][h] + k0 + s * STEP) : make_uint4(0, 0, 0, 0);
        }
        if (!waited) {
            ti_grid_wait();
            waited = true;
        }
        uint4 xv[STEPS];
#pragma unroll
        for (int s = 0; s < STEPS; ++s) xv[s] = k0 + s * STEP + t4 * 8 < a.K ? load_rows(xrow + k0 + s * STEP) : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int s = 0; s < STEPS; ++s) {
            uint4 b = xv[s];
            if constexpr (NORM) {
                const int k = min(k0 + s * STEP + t4 * 8, a.K - 8);
                const float4 g0 = __ldg(reinterpret_cast<const float4*>(a.g + k)), g1 = __ldg(reinterpret_cast<const float4*>(a.g + k + 4));
                b = make_uint4(scaled(b.x, g0.x, g0.y, sq), scaled(b.y, g0.z, g0.w, sq), scaled(b.z, g1.x, g1.y, sq), scaled(b.w, g1.z, g1.w, sq));
            }
#pragma unroll
            for (int i = 0; i < TILES; ++i) {
                mma(c[i], wv[i][s][0].x, wv[i][s][1].x, wv[i][s][0].y, wv[i][s][1].y, b.x, b.y);
                mma(c[i], wv[i][s][0].z, wv[i][s][1].z, wv[i][s][0].w, wv[i][s][1].w, b.z, b.w);
            }
        }
    }
    // c: rows g (0, 1) and g + 8 (2, 3) of a tile, tokens 2 t4 and 2 t4 + 1
#pragma unroll
    for (int i = 0; i < TILES; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) part[warp][2 * t4 + (e & 1)][16 * i + 8 * (e >> 1) + g] = c[i][e];
    if constexpr (NORM) {
        sq += __shfl_xor_sync(0xffffffffu, sq, 1);
        sq += __shfl_xor_sync(0xffffffffu, sq, 2);
        if (t4 == 0) part_sq[warp][g] = sq;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < a.M * ROWS; i += THREADS) {
        const int m = i / ROWS, r = i % ROWS;
        float v = 0.f;
#pragma unroll
        for (int q = 0; q < WARPS; ++q) v += part[q][m][r];
        sums[m][r] = v;
    }
    if (NORM && threadIdx.x >= THREADS - MAX_ROWS) {
        const int m = threadIdx.x - (THREADS - MAX_ROWS);
        float v = 0.f;
#pragma unroll
        for (int q = 0; q < WARPS; ++q) v += part_sq[q][m];
        squares_sh[m] = v;
    }
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    if (splits > 1) cluster.sync();
    else __syncthreads();
    // the blocks of a cluster share out the tokens
    for (int i = threadIdx.x; i < a.M * OUTS; i += THREADS) {
        const int m = i / OUTS, r = i % OUTS, n = n0 + r;
        if (m % splits != rank || n >= a.N) continue;
        float v = 0.f, up = 0.f, squares = 0.f;
        for (int q = 0; q < splits; ++q) {
            v += *cluster.map_shared_rank(&sums[m][r], q);
            if (GATED) up += *cluster.map_shared_rank(&sums[m][OUTS % ROWS + r], q);
            if (NORM) squares += *cluster.map_shared_rank(&squares_sh[m], q);
        }
        if (NORM) {
            const float root = rsqrtf(squares / (float)a.K + a.eps);
            v *= root;
            up *= root;
        }
        if (a.bias) v += a.bias[n];
        if constexpr (GATED != 0) {
            if (a.bias) up += a.bias[a.N + n];
            const float e = GATED == 2 ? v * fmaf(0.0713548162726f, v * v, 1.5957691216057308f) : v;
            v = v / (1.f + __expf(-e)) * up;
        } else if (a.residual) {
            v += __bfloat162float(a.residual[(size_t)m * a.N + n]);
        }
        a.out[(size_t)m * a.N + n] = __float2bfloat16_rn(v);
    }
    if (splits > 1) cluster.sync();                          // nobody leaves while its sums may be read
}

template <int TILES, bool NORM, int GATED>
cudaError_t launch(const Args& a, cudaStream_t stream) {
    constexpr int OUTS = 16 * TILES / (GATED ? 2 : 1);
    const int groups = (a.N + OUTS - 1) / OUTS;
    // enough blocks for the machine, as long as every warp of a cluster has a run of its own
    int splits = 1;
    while (splits < 4 && groups * splits < 148 && a.K >= 2 * splits * WARPS * RUN) splits *= 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(splits, groups);
    cfg.blockDim = THREADS;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = splits;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = ti_pdl_enabled() ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, gemm_few_kernel<TILES, NORM, GATED>, a);
}

// 1 <= M <= 8, K a multiple of 8, rows on 16-byte boundaries. g null: no norm. Two tiles a block where that leaves two blocks an SM.
inline cudaError_t product(const Args& a, int gated, cudaStream_t stream) {
    const bool wide = a.N >= 32 * 296;
#define FEW_GO(T, G) return a.g ? launch<T, true, G>(a, stream) : launch<T, false, G>(a, stream)
    if (gated == 2) { FEW_GO(2, 2); }
    if (gated) { FEW_GO(2, 1); }
    if (wide) { FEW_GO(2, 0); }
    FEW_GO(1, 0);
#undef FEW_GO
}

}  // namespace few
