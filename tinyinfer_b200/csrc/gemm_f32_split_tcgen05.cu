// y[M,N] = x[M,K] . w[N,K]^T of float32 operands on the 5th-generation tensor cores, with float32's precision: every operand,
// times 2^24, is the sum of three bfloat16 numbers (8 + 8 + 8 bits: a = a1 + a2 + a3), and of the nine products of such
// parts the six down to 2^-18 of the largest are taken: a1 b1 + (a1 b2 + a2 b1) + (a2 b2 + a1 b3 + a3 b1). Each is exact in
// the multiplier; what is left out is below 2^-25 |a b|, half of what one float32 rounding of the product may cost.
// The factor keeps the last bits of small operands: bfloat16's normal numbers end where float32's do, so the second and third
// part of a number below 2^-109 would lose bits (rows of 1e-36 came out 2.6e-5 off, now 3.2e-7); times 2^24 every part of every float32 number,
// subnormal ones included, is a normal bfloat16 number. What grows past float32's range by it (operands from 2^104,
// sums from 2^80 on) comes out infinite and is computed again as below. In packed arithmetic the split costs no more with the
// factor than it did without: 333 rows by 2 x 6,144 x 2,048 121.0 -> 119.7 us, 30 rows 53.5 -> 53.4, 9 rows by 12,288 x 2,048 52.0 -> 51.4.
//
// The sums decide the precision. The tensor core cuts bits off when it adds to its accumulator, always towards zero, so a
// long run in one accumulator would drift. Here a run is CHUNK = 2 k blocks of 32, the small parts of a block before the
// large ones; then the accumulator is added, rounded to nearest, to float32 registers and starts again from zero. Against 64
// bits, at K = 320, 2048 and 6144: 3.2e-7, 3.3e-7 and 3.3e-7 of the result's norm, where multiply-adds in k order have 3.2e-7,
// 8.1e-7 and 1.4e-6 (at 256 2.9e-7: shorter rows are the general kernel's).
//
//   weights on the 128 accumulator lanes (gated form: 64 gate rows and the 64 up rows of the same outputs), up to 128 tokens
//   on the columns; a cluster of S CTAs cuts the k range of a tile where the tiles alone would leave SMs idle, and adds its
//   parts up in a fixed order through distributed shared memory, each CTA finishing a share of the tokens.
//   warp 16       TMA: the float32 weights, several k blocks ahead
//   warps 8..15   in two groups, a k block each: a thread takes a row of it into registers, splits it and writes three bfloat16 planes
//                 to tensor memory, where the MMAs read them as their A operand
//   warp 17       TMA: the three planes of x, which a small kernel has laid out before ([3][M][Kp])
//   warp 18       issues the MMAs, 12 of 128 x BN x 16 a k block
//   warps 0..7    drain finished chunks into their registers, at the end into shared memory
// Bound by the chain of a k block (copy, split, products, drain). With the weights' planes in shared memory and the MMAs issued by one
// lane of a diverged warp 333 x 12,288 x 2,048 took 113.6 us; from uniform registers (see elect_one) 103.2, with the planes in tensor
// memory as well 97.4; 64 rows 55.7, 46.1, 41.2; 16 rows 53.6, 40.7, 32.0; 333 x 2,048 x 6,144 77.1, 70.7, 65.3.
// A weight is read from HBM once per 128 tokens and never stored in another form, so the 32-bit model stays as large as it is.
// An output that comes out infinite or NaN (an infinite operand has no finite parts) is computed again by plain
// multiply-adds in k order, so that such operands give what they give in float32: the CTA that finds one makes all its outputs
// again through shared memory (finish_odd): 333 rows of NaN by 12,288 x 2,048 weights 1.24 ms, where gemm_simt.cu takes 0.89.
// Against the 64 x 64 tiles of gemm_simt.cu: 333 rows by 12,288 x 2,048 weights 882 -> 97 us (172 TFLOP/s), by 2,048 x 6,144
// 799 -> 65 us; 9 to 16 rows 306 -> 32 us; 200 rows by 1,024 x 320 weights, the shortest k that comes here, 26 -> 17 us.
#include "sm100_ptx.cuh"
#include <algorithm>
#include <array>
#include <cooperative_groups.h>

namespace {

constexpr int BK = 32;                           // bf16 elements of a 64-byte swizzled row
constexpr int CHUNK = 2;                         // k blocks a run of the accumulator
constexpr int MAX_BN = 128;
constexpr int PLANE_A = BK / 2;                  // columns of tensor memory: two bf16 each
constexpr int SLOT = 128 * BK * 4;               // float32 weights of a k block
constexpr int A_STAGES = 4;                      // planes of the weights
constexpr int A_COL = 2 * MAX_BN, TMEM_COLS = 512;
constexpr int MAX_B_STAGES = 6;                  // planes of x: a copy takes about a microsecond to come
constexpr int DRAIN_WARPS = 8, SPLIT_WARPS = 8, GROUPS = SPLIT_WARPS / 4;       // a group: a warp for each 32 lanes
constexpr int MAX_SLOTS = 6;                     // fetched weights; like A_STAGES a multiple of GROUPS, so that a slot and a stage are
                                                 // one group's: it sees every phase of the barriers it waits on
constexpr int W_WARP = DRAIN_WARPS + SPLIT_WARPS, X_WARP = W_WARP + 1, MMA_WARP = W_WARP + 2;
constexpr int NUM_THREADS = (MMA_WARP + 1) * 32;
constexpr int SMEM_BYTES = 226 * 1024;           // beside the barriers, of 227 KB
static_assert(tmem_shares_sm(TMEM_COLS, SMEM_BYTES), "all of tensor memory");

struct SplitParams {
    float* out;
    const float *x, *w, *bias, *residual;
    int M, N, K, gated;                          // gated: 0 no, 1 silu, 2 the tanh form of gelu; then w has 2N rows
    int bn, b_stages, slots, early;
    int* status;
};

constexpr float OPERAND_SCALE = 16777216.f;               // 2^24
constexpr float RESULT_SCALE = 0x1p-48f;

// Three bfloat16 parts of two scaled floats each, every part the nearest to what the parts before leave.
__device__ __forceinline__ void split2(float a, float b, uint32_t& p1, uint32_t& p2, uint32_t& p3) {
    uint64_t v, scale;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
    asm("mov.b64 %0, {%1, %1};" : "=l"(scale) : "f"(OPERAND_SCALE));
    asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(v) : "l"(scale));
    auto part = [&] {                                        // of both
        float lo, hi;
        uint32_t r;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
        asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
        return r;
    };
    auto leave = [&](uint32_t r) {
        uint64_t taken;
        asm("mov.b64 %0, {%1, %2};" : "=l"(taken) : "r"(r << 16), "r"(r & 0xffff0000u));
        asm("sub.rn.f32x2 %0, %0, %1;" : "+l"(v) : "l"(taken));
    };
    p1 = part();
    leave(p1);
    p2 = part();
    leave(p2);
    p3 = part();
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

// Shared-memory operand descriptor: K-major tile of rows x 32 bf16, 64-byte swizzle; groups of 8 rows 512 bytes apart.
__device__ __forceinline__ uint64_t make_sw64_desc(uint32_t smem_addr) {
    return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | (uint64_t)1 << 16 | (uint64_t)(512 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)4 << 61;
}


// The CTA's share of the outputs by multiply-adds in k order, one accumulator an output: out[col][row] for `cols` tokens from
// m on and the 128 rows of w that the tile has on its lanes. A thread has one row and every fourth token; operands come 32 k at a
// time, the next piece while this one is multiplied.
constexpr int REDO_K = 32, REDO_LD = REDO_K + 4, REDO_THREADS = 512, REDO_PIECE = 2 * 128 * REDO_LD;
__device__ __forceinline__ void redo_plain(float* out, float* pieces, const SplitParams& p, int m, int cols, int n0, int outs) {
    const int row = threadIdx.x & 127, group = threadIdx.x >> 7;
    auto fetch = [&](int k0) {                               // 128 rows of w, then up to 128 of x
        float* to = pieces + k0 / REDO_K % 2 * REDO_PIECE;
        for (int i = threadIdx.x; i < (128 + cols) * (REDO_K / 4); i += NUM_THREADS) {
            const int r = i / (REDO_K / 4), k = k0 + i % (REDO_K / 4) * 4;
            const int w_row = (r < outs ? 0 : p.N) + min(n0 + r % outs, p.N - 1);
            const float* src = r < 128 ? p.w + (size_t)w_row * p.K : p.x + (size_t)min(m + r - 128, p.M - 1) * p.K;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(to + r * REDO_LD + k - k0)), "l"(src + min(k, p.K - 4)),
                         "r"(k < p.K ? 16 : 0) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float acc[MAX_BN / 4] = {};
    fetch(0);
    for (int k0 = 0; k0 < p.K; k0 += REDO_K) {
        if (k0 + REDO_K < p.K) {
            fetch(k0 + REDO_K);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();                                     // the piece is there
        const float* ws = pieces + k0 / REDO_K % 2 * REDO_PIECE + row * REDO_LD;
        const float* xs = pieces + k0 / REDO_K % 2 * REDO_PIECE + (128 + group) * REDO_LD;
        if (threadIdx.x < REDO_THREADS) {
#pragma unroll 1
            for (int k = 0; k < REDO_K; k += 4) {
                const float4 w = *reinterpret_cast<const float4*>(ws + k);
#pragma unroll
                for (int j0 = 0; j0 < MAX_BN / 4; j0 += 4) {
                    if (4 * j0 >= cols) break;
#pragma unroll
                    for (int j = j0; j < j0 + 4; ++j) {      // rows past cols hold what they hold, and are not stored
                        const float4 x = *reinterpret_cast<const float4*>(xs + 4 * j * REDO_LD + k);
                        acc[j] = fmaf(x.x, w.x, acc[j]);
                        acc[j] = fmaf(x.y, w.y, acc[j]);
                        acc[j] = fmaf(x.z, w.z, acc[j]);
                        acc[j] = fmaf(x.w, w.w, acc[j]);
                    }
                }
            }
        }
        __syncthreads();                                     // everyone is done with the piece
    }
    if (threadIdx.x < REDO_THREADS) {
#pragma unroll
        for (int j = 0; j < MAX_BN / 4; ++j)
            if (group + 4 * j < cols) out[(group + 4 * j) * 128 + row] = acc[j];
    }
    __syncthreads();
}

// Bias, activation or residual, and the store of four neighbouring outputs of token m (gated: of the gates and the ups).
__device__ __forceinline__ void store_quad(const SplitParams& p, int m, int n, const float (&total)[2][4]) {
    float res[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        if (n + e >= p.N) { res[e] = 0.f; continue; }
        float v = total[0][e];
        if (p.bias) v += p.bias[n + e];
        if (p.gated) {
            float up = total[1][e];
            if (p.bias) up += p.bias[p.N + n + e];
            if (p.gated == 1) v = v / (1.f + expf(-v));
            else v = 0.5f * v * (1.f + tanhf(0.7978845608028654f * (v + 0.044715f * v * v * v)));
            v *= up;
        } else if (p.residual) {
            v += p.residual[(size_t)m * p.N + n + e];
        }
        res[e] = v;
    }
    float* dst = p.out + (size_t)m * p.N + n;
    if (p.N % 4 == 0 && ((uintptr_t)p.out & 15) == 0) *reinterpret_cast<float4*>(dst) = make_float4(res[0], res[1], res[2], res[3]);
    else
        for (int e = 0; e < 4 && n + e < p.N; ++e) dst[e] = res[e];
}

// The kernel's last act where sums were not finite: `odd` names the calling thread's quads that have some, which are stored from
// what is made again. A function of its own, so that the kernel holds nothing for it: what it would hold goes to local memory, and a
// few spilled registers cost the products 2 %.
__device__ __noinline__ void finish_odd(const SplitParams& p, float* sums, uint32_t odd) {
    const int splits = (int)gridDim.x, part = (int)blockIdx.x, outs = p.gated ? 64 : 128, shift = p.gated ? 4 : 5;
    const int c0 = p.bn * part / splits, c1 = p.bn * (part + 1) / splits;
    const int m = (int)blockIdx.y * p.bn + c0, n0 = (int)blockIdx.z * outs;
    redo_plain(sums, sums + MAX_BN * 128, p, m, c1 - c0, n0, outs);
    for (int i = threadIdx.x; odd; i += NUM_THREADS, odd >>= 1) {
        if (!(odd & 1)) continue;
        const int col = i >> shift, o = (i & ((1 << shift) - 1)) * 4;
        float total[2][4] = {};
#pragma unroll
        for (int g = 0; g < 2; ++g) {
            if (g && !p.gated) break;
#pragma unroll
            for (int e = 0; e < 4; ++e) total[g][e] = sums[col * 128 + o + 64 * g + e];
        }
        store_quad(p, m + col, n0 + o, total);
    }
}

__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_f32_split_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const __grid_constant__ SplitParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ uint64_t bars[2 * (A_STAGES + MAX_B_STAGES + MAX_SLOTS) + 4];
    __shared__ uint32_t tmem_base_sh;
    __shared__ int abort_sh, odd_sh;                         // a wait ran out; an output that is not finite
    volatile int* abort_flag = &abort_sh;
    const uint32_t bar0 = smem_u32(bars);
    auto acc_full_bar = [&](int a) { return bar0 + 8u * a; };
    auto acc_empty_bar = [&](int a) { return bar0 + 8u * (2 + a); };
    auto a_full_bar = [&](int s) { return bar0 + 8u * (4 + s); };
    auto a_empty_bar = [&](int s) { return bar0 + 8u * (4 + A_STAGES + s); };
    auto b_full_bar = [&](int s) { return bar0 + 8u * (4 + 2 * A_STAGES + s); };
    auto b_empty_bar = [&](int s) { return bar0 + 8u * (4 + 2 * A_STAGES + MAX_B_STAGES + s); };
    auto w_full_bar = [&](int s) { return bar0 + 8u * (4 + 2 * A_STAGES + 2 * MAX_B_STAGES + s); };
    auto w_empty_bar = [&](int s) { return bar0 + 8u * (4 + 2 * A_STAGES + 2 * MAX_B_STAGES + MAX_SLOTS + s); };

    ti_grid_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int splits = (int)gridDim.x, part = (int)blockIdx.x;           // the cluster spans gridDim.x
    const int outs = p.gated ? 64 : 128;
    const int m0 = (int)blockIdx.y * p.bn, n0 = (int)blockIdx.z * outs;
    const int num_kb = (p.K + BK - 1) / BK;
    const int kb0 = num_kb * part / splits, kb1 = num_kb * (part + 1) / splits;      // at least one each: splits <= num_kb
    const int blocks = kb1 - kb0, chunks = (blocks + CHUNK - 1) / CHUNK;
    const int plane_b = p.bn * BK * 2;
    uint8_t* b_ring = smem;
    uint8_t* slot_ring = b_ring + p.b_stages * 3 * plane_b;

    if (threadIdx.x == 0) {
        abort_sh = odd_sh = 0;
        for (int s = 0; s < A_STAGES; ++s) { mbar_init(a_full_bar(s), 4); mbar_init(a_empty_bar(s), 1); }
        for (int s = 0; s < MAX_SLOTS; ++s) { mbar_init(w_full_bar(s), 1); mbar_init(w_empty_bar(s), 4); }
        for (int s = 0; s < MAX_B_STAGES; ++s) { mbar_init(b_full_bar(s), 1); mbar_init(b_empty_bar(s), 1); }
        for (int a = 0; a < 2; ++a) { mbar_init(acc_full_bar(a), 1); mbar_init(acc_empty_bar(a), DRAIN_WARPS); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == MMA_WARP) tmem_alloc(&tmem_base_sh, TMEM_COLS);
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
        for (int c = 0; c < chunks; ++c) {
            const int a = c & 1;
            // the whole warp goes on or leaves: what follows is for all 32 lanes
            if (!__all_sync(0xffffffffu, mbar_wait(acc_full_bar(a), (c >> 1) & 1u, abort_flag, p.status, 81))) break;
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
        // the last chunk's barrier says that every MMA has read its stage: shared memory is free
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (u < count) {
#pragma unroll
                for (int i = 0; i < 16; ++i) sums[((unit0 + u) * 16 + i) * 128 + group * 32 + lane] = acc[u][i];
            }
        }
    } else if (warp < W_WARP) {
        // ------------------------------------------------------------ weights: float32 -> three planes
        const int group = (warp - DRAIN_WARPS) >> 2;         // this group takes k blocks group, group + GROUPS, ...
        const int row = (warp & 3) * 32 + lane;              // the thread's row of the tile = lane of tensor memory
        int slot = group, stage = group;
        uint32_t slot_phase = 0, phase = 0;
        for (int i = group; i < blocks; i += GROUPS) {
            if (!__all_sync(0xffffffffu, mbar_wait(w_full_bar(slot), slot_phase, abort_flag, p.status, 87))) break;
            const uint8_t* d = slot_ring + slot * SLOT + row * 128;      // rows of 128 bytes, 128-byte swizzle
            float4 v[BK / 4];
#pragma unroll
            for (int c = 0; c < BK / 4; ++c) v[c] = *reinterpret_cast<const float4*>(d + ((c ^ (row & 7)) << 4));
            // the copy that refills the slot is the async proxy's: without this fence the loads above may be put off past it
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(w_empty_bar(slot));
            if ((slot += GROUPS) >= p.slots) { slot = group; slot_phase ^= 1u; }
            if (!__all_sync(0xffffffffu, mbar_wait(a_empty_bar(stage), phase ^ 1u, abort_flag, p.status, 82))) break;
            tmem_fence_after();
            const uint32_t to = tmem_base + A_COL + stage * (3 * PLANE_A) + ((uint32_t)((warp & 3) * 32) << 16);
#pragma unroll
            for (int h = 0; h < 2; ++h) {                    // 16 k: 8 columns of each plane
                uint32_t q[3][8];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    split2(v[4 * h + c].x, v[4 * h + c].y, q[0][2 * c], q[1][2 * c], q[2][2 * c]);
                    split2(v[4 * h + c].z, v[4 * h + c].w, q[0][2 * c + 1], q[1][2 * c + 1], q[2][2 * c + 1]);
                }
#pragma unroll
                for (int plane = 0; plane < 3; ++plane) tmem_st8(to + plane * PLANE_A + 8 * h, q[plane]);
            }
            tmem_wait_st();
            tmem_fence_before();                             // the MMAs read what was written
            __syncwarp();
            if (lane == 0) mbar_arrive(a_full_bar(stage));
            if ((stage += GROUPS) >= A_STAGES) { stage = group; phase ^= 1u; }
        }
    } else if (warp == X_WARP) {
        // ------------------------------------------------------------ TMA: the planes of x
        if (lane == 0) {
            ti_grid_wait();
            int s = 0;
            uint32_t phase = 0;
            for (int kb = kb0; kb < kb1; ++kb) {
                if (!mbar_wait(b_empty_bar(s), phase ^ 1u, abort_flag, p.status, 83)) break;
                mbar_expect_tx(b_full_bar(s), 3 * plane_b);
                const uint32_t b = smem_u32(b_ring) + s * 3 * plane_b;
                // rows past M of a plane are the next plane's, or zeros: columns that nothing reads
                for (int q = 0; q < 3; ++q) tma_load_2d(b + q * plane_b, &map_x, b_full_bar(s), kb * BK, q * p.M + m0);
                if (++s == p.b_stages) { s = 0; phase ^= 1u; }
            }
        }
    } else if (warp == W_WARP) {
        // ------------------------------------------------------------ TMA: the weights; `early`: no earlier kernel writes them
        if (lane == 0) {
            if (!p.early) ti_grid_wait();
            int slot = 0;
            uint32_t phase = 0;
            for (int kb = kb0; kb < kb1; ++kb) {
                if (!mbar_wait(w_empty_bar(slot), phase ^ 1u, abort_flag, p.status, 88)) break;
                mbar_expect_tx(w_full_bar(slot), SLOT);
                const uint32_t d = smem_u32(slot_ring) + slot * SLOT;
                // rows past N are the other half's, or zeros: outputs that nothing stores
                tma_load_2d(d, &map_w, w_full_bar(slot), kb * BK, n0);
                tma_load_2d(d + SLOT / 2, &map_w, w_full_bar(slot), kb * BK, p.gated ? p.N + n0 : n0 + 64);
                if (++slot == p.slots) { slot = 0; phase ^= 1u; }
            }
        }
    } else {
        // ------------------------------------------------------------ MMA issuer
        const bool leader = elect_one();
        const uint32_t idesc = make_idesc(128, p.bn);
        int sa = 0, sb = 0, kb = 0;
        uint32_t phase_a = 0, phase_b = 0;
        bool ok = true;
        for (int c = 0; c < chunks && ok; ++c) {
            const int a = c & 1;
            if (!mbar_wait_warp(acc_empty_bar(a), ((c >> 1) & 1u) ^ 1u, abort_flag, p.status, 84)) { ok = false; break; }
            tmem_fence_after();
            const uint32_t d = tmem_base + a * MAX_BN;
            uint32_t accumulate = 0;
            for (int j = 0; j < CHUNK && kb < blocks; ++j, ++kb) {
                if (!mbar_wait_warp(b_full_bar(sb), phase_b, abort_flag, p.status, 85) ||
                    !mbar_wait_warp(a_full_bar(sa), phase_a, abort_flag, p.status, 86)) { ok = false; break; }
                tmem_fence_after();
                const uint32_t A = tmem_base + A_COL + sa * (3 * PLANE_A), addr_b = smem_u32(b_ring) + sb * 3 * plane_b;
                uint64_t B[3];
#pragma unroll
                for (int q = 0; q < 3; ++q) B[q] = make_sw64_desc(addr_b + q * plane_b);
                auto products = [&](int qa, int qb) {
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k) {
                        if (leader) umma_bf16_ts(d, A + qa * PLANE_A + 8 * k, B[qb] + 2u * k, idesc, accumulate);
                        accumulate = 1;
                    }
                };
                products(1, 1); products(0, 2); products(2, 0);          // the small ones first
                products(0, 1); products(1, 0);
                products(0, 0);
                if (leader) {
                    umma_commit(a_empty_bar(sa));
                    umma_commit(b_empty_bar(sb));
                }
                if (++sa == A_STAGES) { sa = 0; phase_a ^= 1u; }
                if (++sb == p.b_stages) { sb = 0; phase_b ^= 1u; }
            }
            if (ok && leader) umma_commit(acc_full_bar(a));
        }
        if (!ok) land_copies(abort_flag);
    }

    // ---------------------------------------------------------------- the cluster's parts meet; epilogue and store
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    __syncwarp();
    if (splits > 1) cluster.sync();
    else __syncthreads();
    uint32_t odd = 0;                                        // this thread's quads that are not finite
    if (!*abort_flag) {
        ti_grid_wait();                                      // out and residual belong to the kernels ahead until now
        const int c0 = p.bn * part / splits, c1 = p.bn * (part + 1) / splits;
        const int shift = p.gated ? 4 : 5, kinds = p.gated ? 2 : 1;
        for (int i = threadIdx.x, q = 0; i < (c1 - c0) << shift; i += NUM_THREADS, ++q) {       // four neighbouring outputs a thread
            const int col = c0 + (i >> shift), o = (i & ((1 << shift) - 1)) * 4, m = m0 + col, n = n0 + o;
            if (m >= p.M || n >= p.N) continue;
            float total[2][4] = {};
            bool finite = true;
            for (int g = 0; g < kinds; ++g) {
#pragma unroll
                for (int r0 = 0; r0 < 8; r0 += 4) {          // four at a time: the registers of eight would spill
                    float4 f[4];
#pragma unroll
                    for (int r = 0; r < 4; ++r)
                        if (r0 + r < splits) f[r] = *reinterpret_cast<const float4*>(cluster.map_shared_rank(sums + col * 128 + o + 64 * g, r0 + r));
#pragma unroll
                    for (int r = 0; r < 4; ++r)
                        if (r0 + r < splits) {
                            total[g][0] += f[r].x; total[g][1] += f[r].y; total[g][2] += f[r].z; total[g][3] += f[r].w;
                        }
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    finite = finite && (n + e >= p.N || isfinite(total[g][e]));
                    total[g][e] *= RESULT_SCALE;
                }
            }
            if (finite) store_quad(p, m, n, total);
            else odd |= 1u << q;
        }
        if (odd) odd_sh = 1;
    }
    tmem_fence_before();
    if (splits > 1) cluster.sync();                          // nobody leaves, or writes over its sums, while they may be read
    else __syncthreads();
    if (warp == MMA_WARP) {
        tmem_fence_after();
        tmem_dealloc(tmem_base, TMEM_COLS);
    }
    if (odd_sh) finish_odd(p, sums, odd);
}

// How many clusters of s CTAs the device holds at a time (a cluster lies within one GPC, so some sizes leave SMs unused).
int resident_clusters(int s) {
    static const std::array<int, 9> counts = [] {
        std::array<int, 9> n{};
        for (int c = 1; c <= 8; ++c) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(c);
            cfg.blockDim = NUM_THREADS;
            cfg.dynamicSmemBytes = SMEM_BYTES;
            cudaLaunchAttribute attr;
            attr.id = cudaLaunchAttributeClusterDimension;
            attr.val.clusterDim.x = c;
            attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
            cfg.attrs = &attr;
            cfg.numAttrs = 1;
            int got = 0;
            n[c] = cudaOccupancyMaxActiveClusters(&got, gemm_f32_split_kernel, &cfg) == cudaSuccess && got > 0 ? got : std::max(1, ti_sm_count() / (2 * c));
        }
        cudaGetLastError();
        return n;
    }();
    return counts[s];
}
// How many CTAs share a tile's k range: the count with the least time, in k blocks and with some for the start and the end
// of a CTA, over the waves it makes.
int choose_splits(int tiles, int num_kb) {
    int best = 1;
    double least = 1e30;
    for (int s = 1; s <= 8 && s <= num_kb; ++s) {
        const int waves = (tiles + resident_clusters(s) - 1) / resident_clusters(s);
        const double cost = waves * ((double)((num_kb + s - 1) / s) + 12.0);
        if (cost < least * 0.999) { least = cost; best = s; }
    }
    return best;
}

}  // namespace

// As ti_gemm_simt for float32 operands with K a multiple of 4 and x and w on 16-byte boundaries. ``planes``: room for
// 3 * M * Kp bfloat16 on a 16-byte boundary, Kp = K rounded up to a multiple of 64. early: no kernel that may still run writes w.
TI_API int ti_gemm_f32_split(float* out, const float* x, const float* w, const float* bias, const float* residual, void* planes,
                             int M, int N, int K, int gated, int early, int* status, cudaStream_t stream) {
    TI_REQUIRE(M >= 1 && N > 0 && K > 0 && K % 4 == 0, "gemm_f32_split: bad sizes M=%d N=%d K=%d", M, N, K);
    TI_REQUIRE(((uintptr_t)x | (uintptr_t)w | (uintptr_t)planes) % 16 == 0, "gemm_f32_split: operands must lie on 16-byte boundaries");
    TI_REQUIRE(!(gated && residual), "gemm: the gated form takes no residual");
    const int Kp = (K + 63) / 64 * 64;
    SplitParams p{out, x, w, bias, residual, M, N, K, gated, 0, 0, 0, early, status};
    const int row_tiles = (M + MAX_BN - 1) / MAX_BN;
    p.bn = ((M + row_tiles - 1) / row_tiles + 15) / 16 * 16;
    const int outs = gated ? 64 : 128, col_tiles = (N + outs - 1) / outs;
    TI_REQUIRE(row_tiles <= 65535 && col_tiles <= 65535, "gemm_f32_split: too many tiles");
    // shared memory: the slots, and as many copies of x as leave room for them
    const int b_bytes = 3 * p.bn * BK * 2, room = SMEM_BYTES - 1024;
    p.b_stages = std::min(MAX_B_STAGES, (room - MAX_SLOTS * SLOT) / b_bytes);       // at least five
    p.slots = MAX_SLOTS;
    static_assert(4 * (MAX_BN * 128 + 2 * REDO_PIECE) <= SMEM_BYTES - 1024, "the outputs made again and their operands");
    static_assert(MAX_BN * 32 <= 32 * NUM_THREADS, "a thread's quads have a bit each");
    static_assert(5 * 3 * MAX_BN * BK * 2 + MAX_SLOTS * SLOT <= SMEM_BYTES - 1024, "128 columns: five copies of x");
    static_assert(MAX_SLOTS % GROUPS == 0 && A_STAGES % GROUPS == 0 && A_COL + A_STAGES * 3 * PLANE_A <= TMEM_COLS, "stages and slots");
    TiEncodeTiledFn encode = ti_encode_tiled_fn();
    TI_REQUIRE(encode, "cuTensorMapEncodeTiled is not available from this driver");
    CUtensorMap map, map_w;
    const cuuint64_t dims[2] = {(cuuint64_t)Kp, (cuuint64_t)M * 3}, strides[1] = {(cuuint64_t)Kp * 2};
    const cuuint32_t box[2] = {BK, (cuuint32_t)p.bn}, elem[2] = {1, 1};
    const CUresult r = encode(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, planes, dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    const cuuint64_t w_dims[2] = {(cuuint64_t)K, (cuuint64_t)N * (gated ? 2 : 1)}, w_strides[1] = {(cuuint64_t)K * 4};
    const cuuint32_t w_box[2] = {BK, 64};
    const CUresult rw = encode(&map_w, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(w), w_dims, w_strides, w_box, elem,
                               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    TI_REQUIRE(r == CUDA_SUCCESS && rw == CUDA_SUCCESS, "cuTensorMapEncodeTiled failed (%d, %d) for M=%d N=%d K=%d", (int)r, (int)rw, M, N, K);
    const cudaError_t set = ti_allow_shared<gemm_f32_split_kernel>(SMEM_BYTES);
    TI_REQUIRE(set == cudaSuccess, "gemm_f32_split: %s", cudaGetErrorString(set));
    const int splits = choose_splits(row_tiles * col_tiles, (K + BK - 1) / BK);
    const long long quads = (long long)M * Kp / 4;
    ti_launch(split_rows_kernel, dim3((unsigned)((quads + 255) / 256)), 256, 0, stream, (__nv_bfloat16*)planes, x, M, K, Kp);
    TI_CHECK_LAUNCH("gemm_f32_split rows");
    cudaLaunchConfig_t cfg = {};
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
    cudaLaunchKernelEx(&cfg, gemm_f32_split_kernel, map, map_w, p);
    TI_CHECK_LAUNCH("gemm_f32_split");
    return 0;
}
