// The batched product of gemm_batched.cu on the tcgen05 tensor cores, for many rows (prompt portions): a CTA makes 128 rows by 128
// outputs of one batch in tensor memory, operands by TMA. A piece of x is found by its column in the rows, so that its first column
// and K are whole 16 bytes and whole k blocks of 64; rows of w past a batch's are the next batch's: computed and not stored.
//   warp 0 TMA, warp 1 issues the MMAs, warps 2..5 store, a thread a row
// Bound by its few k blocks' latency (K is 128 to 512) and the store of the outputs: two CTAs share an SM, one's copies under the
// other's store. 16 heads, against the warp-level form: 2,048 rows of K 128 by 512 outputs 54.7 -> 21.0 us, of K 512 by 128 30.9 -> 8.9; 333
// rows 11.9 -> 6.0 and 16.0 -> 6.1, 128 rows 9.1 -> 4.9 and 8.5 -> 5.0. Bias and sigmoid stay with that form: 10 blocks of 256 by 512 outputs in
// float32 took 61.7 us here for its 58.3, and 19.1 for 14.2 at 128 rows, four warps making all the exponentials.
#include "sm100_ptx.cuh"

namespace gbt {
constexpr int BM = 128, BN = 128, BK = 64, STAGES = 3, THREADS = 192;
constexpr int STAGE_BYTES = (BM + BN) * BK * 2, SMEM = 1024 + STAGES * STAGE_BYTES;
static_assert(tmem_shares_sm(BN, SMEM), "one accumulator");

struct Args {
    void* out;
    int M, N, K, sx;
    long long ldo, so;
    int* status;
};

template <typename OutT>
__global__ void __launch_bounds__(THREADS, 2)
kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const Args p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* stages = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ uint64_t bars[2 * STAGES + 1];
    __shared__ uint32_t tmem_base_sh;
    __shared__ int abort_sh;
    volatile int* abort_flag = &abort_sh;
    const uint32_t bar0 = smem_u32(bars), done = bar0 + 16u * STAGES;
    auto full = [&](int s) { return bar0 + 8u * s; };
    auto empty = [&](int s) { return bar0 + 8u * (STAGES + s); };
    ti_grid_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        abort_sh = 0;
        for (int s = 0; s < STAGES; ++s) { mbar_init(full(s), 1); mbar_init(empty(s), 1); }
        mbar_init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tmem_alloc(&tmem_base_sh, BN);
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    const uint32_t tmem_base = tmem_base_sh;
    const int n0 = blockIdx.x * BN, m0 = blockIdx.y * BM, b = blockIdx.z, blocks = p.K / BK;
    ti_grid_wait();
    if (warp == 0) {
        if (lane == 0) {
            for (int kb = 0; kb < blocks; ++kb) {
                const int s = kb % STAGES;
                if (!mbar_wait(empty(s), ((kb / STAGES) & 1u) ^ 1u, abort_flag, p.status, 94)) break;
                mbar_expect_tx(full(s), STAGE_BYTES);
                const uint32_t dst = smem_u32(stages + s * STAGE_BYTES);
                tma_load_2d(dst, &map_x, full(s), b * p.sx + kb * BK, m0);
                tma_load_2d(dst + BM * BK * 2, &map_w, full(s), kb * BK, b * p.N + n0);
            }
        }
    } else if (warp == 1) {
        const bool leader = elect_one();
        constexpr uint32_t idesc = make_idesc(BM, BN);
        bool ok = true;
        for (int kb = 0; kb < blocks; ++kb) {
            const int s = kb % STAGES;
            if (!mbar_wait_warp(full(s), (kb / STAGES) & 1u, abort_flag, p.status, 95)) { ok = false; break; }
            tmem_fence_after();
            const uint32_t at = smem_u32(stages + s * STAGE_BYTES);
            const uint64_t adesc = make_sw128_desc(at), bdesc = make_sw128_desc(at + BM * BK * 2);
#pragma unroll
            for (int k = 0; k < BK / 16; ++k)
                if (leader) umma_bf16(tmem_base, adesc + 2u * k, bdesc + 2u * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
            if (leader) umma_commit(empty(s));
        }
        if (ok && leader) umma_commit(done);
        if (!ok) land_copies(abort_flag);
    } else if (mbar_wait_warp(done, 0, abort_flag, p.status, 96)) {
        tmem_fence_after();
        const int lane_group = warp & 3, m = m0 + lane_group * 32 + lane;
        const bool live = m < p.M;
#pragma unroll 1
        for (int c = 0; c < BN; c += 32) {
            if (n0 + c >= p.N) break;                            // N is whole 32s: the same for the warp
            float v[32];
            tmem_ld32(tmem_base + ((uint32_t)(lane_group * 32) << 16) + c, v);
            if (!live) continue;
            OutT* dst = (OutT*)p.out + (size_t)b * p.so + (size_t)m * p.ldo + n0 + c;
            if constexpr (sizeof(OutT) == 4) {
#pragma unroll
                for (int i = 0; i < 32; i += 4) *reinterpret_cast<float4*>(dst + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
            } else {
#pragma unroll
                for (int i = 0; i < 32; i += 8) {
                    uint4 q;
                    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&q);
#pragma unroll
                    for (int j = 0; j < 4; ++j) h[j] = __floats2bfloat162_rn(v[i + 2 * j], v[i + 2 * j + 1]);
                    *reinterpret_cast<uint4*>(dst + i) = q;
                }
            }
        }
    }
    tmem_fence_before();
    __syncthreads();
    if (warp == 1) {
        tmem_fence_after();
        tmem_dealloc(tmem_base, BN);
    }
}
}  // namespace gbt

// Whether this form takes the product: no bias, activation or gate; rows for a whole tile; K in whole blocks, as a box of x past a piece
// would bring the next one's columns (times zeros, which NaN survive); outputs in whole stores.
bool gbt_takes(const void* out, const void* x, const void* w, int batch, int M, int N, int K, long long ldx, long long sx, long long ldw,
               long long sw, long long ldo, long long so, int out_f32) {
    const long long whole = out_f32 ? 4 : 8;                 // outputs of a 16-byte store
    return M >= gbt::BM && K % gbt::BK == 0 && N % 32 == 0 && ldw == K && sw == (long long)N * K && ldx % 8 == 0 && sx % 8 == 0 && sx >= 0 &&
           ldx >= (batch - 1) * sx + K && ldx < (1ll << 30) && ldo % whole == 0 && so % whole == 0 && (long long)batch * N < (1ll << 31) - 128 &&
           (((uintptr_t)x | (uintptr_t)w | (uintptr_t)out) & 15) == 0;
}

int gbt_launch(void* out, const void* x, const void* w, int batch, int M, int N, int K, long long ldx, long long sx, long long ldo, long long so,
               int out_f32, int* status, cudaStream_t stream) {
    CUtensorMap map_x, map_w;
    if (!ti_get_bf16_map(x, M, (int)ldx, gbt::BM, &map_x)) return -1;
    if (!ti_get_bf16_map(w, (long long)batch * N, K, gbt::BN, &map_w)) return -1;
    const gbt::Args a = {out, M, N, K, (int)sx, ldo, so, status};
    const dim3 grid((N + gbt::BN - 1) / gbt::BN, (M + gbt::BM - 1) / gbt::BM, batch);
    TI_REQUIRE(grid.y <= 65535, "gemm_batched: too many rows");
    cudaError_t e = out_f32 ? ti_allow_shared<gbt::kernel<float>>(gbt::SMEM) : ti_allow_shared<gbt::kernel<__nv_bfloat16>>(gbt::SMEM);
    if (e == cudaSuccess)
        e = out_f32 ? ti_launch(gbt::kernel<float>, grid, gbt::THREADS, gbt::SMEM, stream, map_x, map_w, a)
                    : ti_launch(gbt::kernel<__nv_bfloat16>, grid, gbt::THREADS, gbt::SMEM, stream, map_x, map_w, a);
    TI_REQUIRE(e == cudaSuccess, "gemm_batched: %s", cudaGetErrorString(e));
    TI_CHECK_LAUNCH("gemm_batched");
    return 0;
}
