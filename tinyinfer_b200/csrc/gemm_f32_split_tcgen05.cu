// y[M,N] = x[M,K] . w[N,K]^T of float32 operands on the 5th-generation tensor cores, with float32's precision: every operand
// is the sum of three bfloat16 numbers (8 + 8 + 8 bits: a = a1 + a2 + a3 up to 2^-26 |a|), and of the nine products of such
// parts the six down to 2^-18 of the largest are taken: a1 b1 + (a1 b2 + a2 b1) + (a2 b2 + a1 b3 + a3 b1). Each is exact in
// the multiplier; what is left out is below 2^-25 |a b|, half of what one float32 rounding of the product may cost.
//
// The sums decide the precision. The tensor core cuts bits off when it adds to its accumulator, always towards zero, so a
// long run in one accumulator would drift. Here a run is CHUNK = 2 k blocks of 64, the small parts of a block before the
// large ones; then the accumulator is added, rounded to nearest, to float32 registers and starts again from zero.
//
//   weights on the 128 accumulator lanes (gated form: 64 gate rows and the 64 up rows of the same outputs), up to 128 tokens
//   on the columns; a cluster of S CTAs cuts the k range of a tile where the tiles alone would leave SMs idle, and adds its
//   parts up in a fixed order through distributed shared memory, each CTA finishing a share of the tokens.
//   warps 8..15   read the float32 weights (32 bytes a lane, a k block ahead in registers), split them, and write three
//                 swizzled bfloat16 planes into the stage
//   warp 16       TMA: the three planes of x, which a small kernel has laid out before ([3][M][Kp])
//   warp 17       one thread issues the MMAs, 24 of 128 x BN x 16 a k block
//   warps 0..7    drain finished chunks into their registers, at the end into shared memory
// A weight is read from HBM once per 128 tokens and never stored in another form, so the 32-bit model stays as large as it is.
// An output that comes out infinite or NaN (an infinite operand has no finite parts) is computed again by plain
// multiply-adds in k order, so that such operands give what they give in float32.
// MEASURED
#include "sm100_ptx.cuh"
#include <cooperative_groups.h>

namespace {

constexpr int BK = 64;                           // bf16 elements of a 128-byte swizzled row
constexpr int CHUNK = 2;                         // k blocks a run of the accumulator
constexpr int MAX_BN = 128;
constexpr int PLANE_A = 128 * BK * 2;            // 16 KB
constexpr int MAX_STAGES = 4;
constexpr int DRAIN_WARPS = 8, SPLIT_WARPS = 8;
constexpr int NUM_THREADS = (DRAIN_WARPS + SPLIT_WARPS + 2) * 32;
constexpr int SMEM_BYTES = 227 * 1024;
constexpr int STAGE_ROOM = SMEM_BYTES - 1024 - 256;          // alignment slack, barriers

struct SplitParams {
    float* out;
    const float *x, *w, *bias, *residual;
    int M, N, K, gated;                          // gated: 0 no, 1 silu, 2 the tanh form of gelu; then w has 2N rows
    int bn, stages;
    int* status;
};

// Three bfloat16 parts of two floats each, every part the nearest to what the parts before leave.
__device__ __forceinline__ void split2(float a, float b, uint32_t& p1, uint32_t& p2, uint32_t& p3) {
    auto pack = [](float lo, float hi) {
        uint32_t r;
        asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
        return r;
    };
    p1 = pack(a, b);
    a -= __uint_as_float(p1 << 16);
    b -= __uint_as_float(p1 & 0xffff0000u);
    p2 = pack(a, b);
    a -= __uint_as_float(p2 << 16);
    b -= __uint_as_float(p2 & 0xffff0000u);
    p3 = pack(a, b);
}

// x [M, K] -> planes [3][M][Kp], zeros behind K.
__global__ void __launch_bounds__(256) split_rows_kernel(__nv_bfloat16* planes, const float* x, int M, int K, int Kp) {
    ti_grid_launch_dependents();
    ti_grid_wait();
    const long long i = ((long long)blockIdx.x * 256 + threadIdx.x) * 4;
    const long long total = (long long)M * Kp;
    if (i >= total) return;
    const int row = (int)(i / Kp), k = (int)(i - (long long)row * Kp);
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (k < K) v = *reinterpret_cast<const float4*>(x + (size_t)row * K + k);
    uint2 p1, p2, p3;
    split2(v.x, v.y, p1.x, p2.x, p3.x);
    split2(v.z, v.w, p1.y, p2.y, p3.y);
    *reinterpret_cast<uint2*>(planes + i) = p1;
    *reinterpret_cast<uint2*>(planes + total + i) = p2;
    *reinterpret_cast<uint2*>(planes + 2 * total + i) = p3;
}

__device__ __noinline__ float plain_dot(const float* x, const float* w, int K) {
    float v = 0.f;
    for (int k = 0; k < K; ++k) v = fmaf(x[k], w[k], v);
    return v;
}

__global__ void __launch_bounds__(NUM_THREADS, 1) gemm_f32_split_kernel(const __grid_constant__ CUtensorMap map_x, const SplitParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ uint64_t bars[2 * MAX_STAGES + 4];
    __shared__ uint32_t tmem_base_sh;
    __shared__ int abort_sh;
    volatile int* abort_flag = &abort_sh;
    const uint32_t bar0 = smem_u32(bars);
    auto full_bar = [&](int s) { return bar0 + 8u * s; };
    auto empty_bar = [&](int s) { return bar0 + 8u * (MAX_STAGES + s); };
    auto acc_full_bar = [&](int a) { return bar0 + 8u * (2 * MAX_STAGES + a); };
    auto acc_empty_bar = [&](int a) { return bar0 + 8u * (2 * MAX_STAGES + 2 + a); };

    ti_grid_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int splits = (int)gridDim.x, part = (int)blockIdx.x;           // the cluster spans gridDim.x
    const int outs = p.gated ? 64 : 128;
    const int m0 = (int)blockIdx.y * p.bn, n0 = (int)blockIdx.z * outs;
    const int num_kb = (p.K + BK - 1) / BK;
    const int kb0 = num_kb * part / splits, kb1 = num_kb * (part + 1) / splits;      // at least one each: splits <= num_kb
    const int blocks = kb1 - kb0, chunks = (blocks + CHUNK - 1) / CHUNK;
    const int plane_b = p.bn * BK * 2, stage_bytes = 3 * (PLANE_A + plane_b);

    if (threadIdx.x == 0) {
        abort_sh = 0;
        for (int s = 0; s < MAX_STAGES; ++s) { mbar_init(full_bar(s), 1 + SPLIT_WARPS); mbar_init(empty_bar(s), 1); }
        for (int a = 0; a < 2; ++a) { mbar_init(acc_full_bar(a), 1); mbar_init(acc_empty_bar(a), DRAIN_WARPS); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == DRAIN_WARPS + SPLIT_WARPS + 1) tmem_alloc(&tmem_base_sh, 2 * MAX_BN);
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    const uint32_t tmem_base = tmem_base_sh;
    float* sums = reinterpret_cast<float*>(smem);            // [bn][128], once the stages are done with

    if (warp < DRAIN_WARPS) {
        // ------------------------------------------------------------ drain: chunks into registers
        const int group = warp & 3, half = warp >> 2;        // the 32 lanes this warp may read; its part of the columns
        const int units = p.bn / 16, unit0 = half ? (units + 1) / 2 : 0, count = half ? units / 2 : (units + 1) / 2;
        float acc[4][16] = {};
        bool ok = true;
        for (int c = 0; c < chunks && ok; ++c) {
            const int a = c & 1;
            // the whole warp goes on or leaves: what follows is for all 32 lanes
            if (!__all_sync(0xffffffffu, mbar_wait(acc_full_bar(a), (c >> 1) & 1u, abort_flag, p.status, 81))) { ok = false; break; }
            tmem_fence_after();
            const uint32_t t = tmem_base + a * MAX_BN + unit0 * 16 + ((uint32_t)(group * 32) << 16);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (u < count) {
                    float v[16];
                    tmem_ld16(t + 16 * u, v);
#pragma unroll
                    for (int i = 0; i < 16; ++i) acc[u][i] += v[i];
                }
            }
            tmem_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(acc_empty_bar(a));
        }
        ti_grid_wait();                                      // this CTA's outputs are written behind the kernels ahead
        // the last chunk's barrier says that every MMA has read its stage: shared memory is free
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (u < count) {
#pragma unroll
                for (int i = 0; i < 16; ++i) sums[((unit0 + u) * 16 + i) * 128 + group * 32 + lane] = acc[u][i];
            }
        }
    } else if (warp < DRAIN_WARPS + SPLIT_WARPS) {
        // ------------------------------------------------------------ weights: float32 -> three planes
        const int t = (int)threadIdx.x - DRAIN_WARPS * 32;
        const int c = t & 7, row0 = t >> 3;                  // 8 lanes a row of 64 floats, 32 rows at a time
        const float* src[4];
        bool there[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = row0 + 32 * i;
            const int o = n0 + (p.gated ? r & 63 : r);
            there[i] = o < p.N;
            src[i] = p.w + (size_t)(there[i] ? (p.gated && r >= 64 ? p.N + o : o) : 0) * p.K;
        }
        auto load = [&](int kb, float4 (&v)[4][2]) {
            const int k = kb * BK + c * 8;
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    v[i][h] = there[i] && kb < kb1 && k + 4 * h < p.K ? __ldg(reinterpret_cast<const float4*>(src[i] + k + 4 * h))
                                                                      : make_float4(0.f, 0.f, 0.f, 0.f);
        };
        float4 cur[4][2], nxt[4][2];
        load(kb0, cur);
        int s = 0;
        uint32_t phase = 0;
        for (int kb = kb0; kb < kb1; ++kb) {
            load(kb + 1, nxt);
            if (!__all_sync(0xffffffffu, mbar_wait(empty_bar(s), phase ^ 1u, abort_flag, p.status, 82))) break;
            uint8_t* a = smem + s * stage_bytes;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int r = row0 + 32 * i;
                uint4 q1, q2, q3;
                split2(cur[i][0].x, cur[i][0].y, q1.x, q2.x, q3.x);
                split2(cur[i][0].z, cur[i][0].w, q1.y, q2.y, q3.y);
                split2(cur[i][1].x, cur[i][1].y, q1.z, q2.z, q3.z);
                split2(cur[i][1].z, cur[i][1].w, q1.w, q2.w, q3.w);
                uint8_t* d = a + r * 128 + ((c ^ (r & 7)) << 4);
                *reinterpret_cast<uint4*>(d) = q1;
                *reinterpret_cast<uint4*>(d + PLANE_A) = q2;
                *reinterpret_cast<uint4*>(d + 2 * PLANE_A) = q3;
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(full_bar(s));
#pragma unroll
            for (int i = 0; i < 4; ++i) { cur[i][0] = nxt[i][0]; cur[i][1] = nxt[i][1]; }
            if (++s == p.stages) { s = 0; phase ^= 1u; }
        }
    } else if (warp == DRAIN_WARPS + SPLIT_WARPS) {
        // ------------------------------------------------------------ TMA: the planes of x
        if (lane == 0) {
            ti_grid_wait();
            int s = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int kb = kb0; kb < kb1; ++kb) {
                if (!mbar_wait(empty_bar(s), phase ^ 1u, abort_flag, p.status, 83)) { ok = false; break; }
                mbar_expect_tx(full_bar(s), 3 * plane_b);
                const uint32_t b = smem_u32(smem + s * stage_bytes) + 3 * PLANE_A;
                // rows past M of a plane are the next plane's, or zeros: columns that nothing reads
                for (int q = 0; q < 3; ++q) tma_load_2d(b + q * plane_b, &map_x, full_bar(s), kb * BK, q * p.M + m0);
                if (++s == p.stages) { s = 0; phase ^= 1u; }
            }
            if (!ok) {       // give the copies still in flight time to land before shared memory is given up
                const unsigned long long t0 = global_ns();
                while (global_ns() - t0 < 1000000ull) {}
            }
        }
    } else if (lane == 0) {
        // ------------------------------------------------------------ MMA issuer
        const uint32_t idesc = make_idesc(128, p.bn);
        int s = 0, kb = 0;
        uint32_t phase = 0;
        bool ok = true;
        for (int c = 0; c < chunks && ok; ++c) {
            const int a = c & 1;
            if (!mbar_wait(acc_empty_bar(a), ((c >> 1) & 1u) ^ 1u, abort_flag, p.status, 84)) { ok = false; break; }
            tmem_fence_after();
            const uint32_t d = tmem_base + a * MAX_BN;
            uint32_t accumulate = 0;
            for (int j = 0; j < CHUNK && kb < blocks; ++j, ++kb) {
                if (!mbar_wait(full_bar(s), phase, abort_flag, p.status, 85)) { ok = false; break; }
                tmem_fence_after();
                const uint32_t addr = smem_u32(smem + s * stage_bytes);
                uint64_t A[3], B[3];
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    A[q] = make_sw128_desc(addr + q * PLANE_A);
                    B[q] = make_sw128_desc(addr + 3 * PLANE_A + q * plane_b);
                }
                auto products = [&](int qa, int qb) {
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k) {
                        umma_bf16(d, A[qa] + 2u * k, B[qb] + 2u * k, idesc, accumulate);
                        accumulate = 1;
                    }
                };
                products(1, 1); products(0, 2); products(2, 0);          // the small ones first
                products(0, 1); products(1, 0);
                products(0, 0);
                umma_commit(empty_bar(s));
                if (++s == p.stages) { s = 0; phase ^= 1u; }
            }
            if (ok) umma_commit(acc_full_bar(a));
        }
    }

    // ---------------------------------------------------------------- the cluster's parts meet; epilogue and store
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    __syncwarp();
    if (splits > 1) cluster.sync();
    else __syncthreads();
    const int c0 = p.bn * part / splits, c1 = p.bn * (part + 1) / splits;
    if (!*abort_flag) {
        ti_grid_wait();
        for (int i = threadIdx.x; i < (c1 - c0) * outs; i += NUM_THREADS) {
            const int col = c0 + i / outs, o = i % outs, m = m0 + col, n = n0 + o;
            if (m >= p.M || n >= p.N) continue;
            auto total = [&](int row, int w_row) {
                float v = 0.f;
                for (int r = 0; r < splits; ++r) v += *cluster.map_shared_rank(sums + col * 128 + row, r);
                return isfinite(v) ? v : plain_dot(p.x + (size_t)m * p.K, p.w + (size_t)w_row * p.K, p.K);
            };
            float v = total(o, n);
            if (p.bias) v += p.bias[n];
            if (p.gated) {
                float up = total(64 + o, p.N + n);
                if (p.bias) up += p.bias[p.N + n];
                if (p.gated == 1) v = v / (1.f + expf(-v));
                else v = 0.5f * v * (1.f + tanhf(0.7978845608028654f * (v + 0.044715f * v * v * v)));
                v *= up;
            } else if (p.residual) {
                v += p.residual[(size_t)m * p.N + n];
            }
            p.out[(size_t)m * p.N + n] = v;
        }
    }
    tmem_fence_before();
    if (splits > 1) cluster.sync();                          // nobody leaves while its sums may be read
    else __syncthreads();
    if (warp == DRAIN_WARPS + SPLIT_WARPS + 1) {
        tmem_fence_after();
        tmem_dealloc(tmem_base, 2 * MAX_BN);
    }
}

// How many CTAs share a tile's k range: the count with the least time, in k blocks and with some for the start and the end
// of a CTA, over the waves it makes. A cluster lies within a GPC of 18 SMs at most, so some counts leave SMs unused.
int choose_splits(int tiles, int num_kb) {
    int best = 1;
    double least = 1e30;
    for (int s = 1; s <= 8 && s <= num_kb; ++s) {
        const int sms = s <= 2 ? ti_sm_count() / s * s : 18 / s * s * 8;
        const int waves = (tiles * s + sms - 1) / sms;
        const double cost = waves * ((double)((num_kb + s - 1) / s) + 4.0);
        if (cost < least * 0.999) { least = cost; best = s; }
    }
    return best;
}

}  // namespace

// As ti_gemm_simt for float32 operands with K a multiple of 4 and x and w on 16-byte boundaries. ``planes``: room for
// 3 * M * Kp bfloat16 on a 16-byte boundary, Kp = K rounded up to a multiple of 64.
TI_API int ti_gemm_f32_split(float* out, const float* x, const float* w, const float* bias, const float* residual, void* planes,
                             int M, int N, int K, int gated, int* status, cudaStream_t stream) {
    TI_REQUIRE(M >= 1 && N > 0 && K > 0 && K % 4 == 0, "gemm_f32_split: bad sizes M=%d N=%d K=%d", M, N, K);
    TI_REQUIRE(((uintptr_t)x | (uintptr_t)w | (uintptr_t)planes) % 16 == 0, "gemm_f32_split: operands must lie on 16-byte boundaries");
    TI_REQUIRE(!(gated && residual), "gemm: the gated form takes no residual");
    const int Kp = (K + BK - 1) / BK * BK;
    SplitParams p{out, x, w, bias, residual, M, N, K, gated, 0, 0, status};
    const int row_tiles = (M + MAX_BN - 1) / MAX_BN;
    p.bn = ((M + row_tiles - 1) / row_tiles + 15) / 16 * 16;
    const int outs = gated ? 64 : 128, col_tiles = (N + outs - 1) / outs;
    TI_REQUIRE(row_tiles <= 65535 && col_tiles <= 65535, "gemm_f32_split: too many tiles");
    const int stage_bytes = 3 * (PLANE_A + p.bn * BK * 2);
    p.stages = STAGE_ROOM / stage_bytes < MAX_STAGES ? STAGE_ROOM / stage_bytes : MAX_STAGES;
    CUtensorMap map;
    if (!ti_get_bf16_map(planes, 3ll * M, Kp, p.bn, &map)) return -1;
    static const cudaError_t set = cudaFuncSetAttribute(gemm_f32_split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
    TI_REQUIRE(set == cudaSuccess, "gemm_f32_split: %s", cudaGetErrorString(set));
    const long long quads = (long long)M * Kp / 4;
    ti_launch(split_rows_kernel, dim3((unsigned)((quads + 255) / 256)), 256, 0, stream, (__nv_bfloat16*)planes, x, M, K, Kp);
    TI_CHECK_LAUNCH("gemm_f32_split rows");
    cudaLaunchConfig_t cfg = {};
    const int splits = choose_splits(row_tiles * col_tiles, (K + BK - 1) / BK);
    cfg.gridDim = dim3(splits, row_tiles, col_tiles);
    cfg.blockDim = NUM_THREADS;
    cfg.dynamicSmemBytes = SMEM_BYTES;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = splits;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = ti_pdl_enabled() ? 2 : 1;
    cudaLaunchKernelEx(&cfg, gemm_f32_split_kernel, map, p);
    TI_CHECK_LAUNCH("gemm_f32_split");
    return 0;
}
