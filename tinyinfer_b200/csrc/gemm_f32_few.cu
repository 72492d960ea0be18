// y[M,N] = x[M,K] . w[N,K]^T in float32 for at most 8 rows of x (a decode step of the 32-bit path, the head of a prompt):
// every weight is read once, at 16 bytes a lane, and meets all rows of x in registers.
//
// Bound by the weights' way from HBM. A block of 8 warps takes ROWS rows of w; the warps share out the k range in
// interleaved pieces of 128 (4 floats a lane), so that a block asks for 8 x ROWS x 512 contiguous bytes at a time, and add
// their sums up through shared memory. ROWS x M accumulators a lane: 4 rows of w up to M = 4 (64 bytes a lane in flight an
// unrolled step, twice), 8 rows for M = 5..8, where the x that a lane reads from L1/L2 would otherwise cost more than the
// weights. With `early` the first weights are asked for before the wait for the kernels ahead in the stream, which none of those
// may write then.
// The order of the sums does not depend on M: a lane's k pieces in rising order, a tree over the lanes, the warps in order.
// In place of the 64 x 64 tiles of gemm_simt.cu, which used 4 of their 64 rows and 16 to 96 blocks: a decode step of 4
// requests over a 1.7B model (28 layers, hidden size 2048), 69.0 -> 2.1 ms together with attention_f32.cu. Alone, 12,288 x 2,048 weights: 15.8 us
// for one row (6.4 TB/s), 17.6 for 4, 25.9 for 8; 2,048 x 2,048: 4.4 us against 225.
#include "common.cuh"

namespace {

constexpr int WARPS = 8;
constexpr int PIECE = 128;                       // k elements of a warp's step: a float4 a lane

__device__ __forceinline__ float4 load_w(const float* p) {
    float4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}
// x may have been written by a kernel that this one overlaps with: no read-only path.
__device__ __forceinline__ float4 load_x(const float* p) {
    float4 v;
    asm volatile("ld.global.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
    return v;
}

// Sums V values over the 32 lanes in the order of the tree 16, 8, 4, 2, 1; value i ends up in v[i % (V / 32)] of the lanes
// that `lane_of(i)` names. While there are several values, each exchange halves them.
template <int V, int OFF> __device__ __forceinline__ void fold(float* v, int lane) {
    if constexpr (OFF > 0) {
        if constexpr (V > 1) {
            const bool upper = lane & OFF;
#pragma unroll
            for (int i = 0; i < V / 2; ++i) {
                const float give = upper ? v[i] : v[i + V / 2];
                const float keep = upper ? v[i + V / 2] : v[i];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, give, OFF);
            }
            fold<V / 2, OFF / 2>(v, lane);
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], OFF);
            fold<1, OFF / 2>(v, lane);
        }
    }
}

// GATED: 0 no, 1 silu, 2 the tanh form of gelu; then half of a block's ROWS streams are gate rows and half the up rows of the
// same outputs.
template <int MT, int ROWS, int GATED>
__global__ void __launch_bounds__(WARPS * 32) gemm_f32_few_kernel(
    float* out, const float* x, const float* w, const float* bias, const float* residual, int M, int N, int K, bool early) {
    constexpr int V = MT * ROWS;                 // sums a block makes
    constexpr int OUTS = GATED ? ROWS / 2 : ROWS;
    constexpr int U = ROWS <= 4 ? 2 : 1;         // steps whose weights are asked for together
    constexpr int LEFT = V > 32 ? V / 32 : 1;    // sums a lane holds after the exchange
    __shared__ float part[WARPS][V];
    ti_grid_launch_dependents();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n0 = blockIdx.x * OUTS;
    const float* wrow[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
        const int o = min(n0 + r % OUTS, N - 1);
        wrow[r] = w + (size_t)(r < OUTS ? o : N + o) * K;
    }
    float acc[V] = {};
    if (!early) ti_grid_wait();
    bool waited = false;
    for (int k0 = warp * PIECE; k0 < K || !waited; k0 += U * WARPS * PIECE) {
        float4 wv[U][ROWS];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int k = k0 + u * WARPS * PIECE + lane * 4;
#pragma unroll
            for (int r = 0; r < ROWS; ++r) wv[u][r] = k < K ? load_w(wrow[r] + k) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        if (!waited) {
            ti_grid_wait();
            waited = true;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int k = k0 + u * WARPS * PIECE + lane * 4;
            if (k < K) {
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    const float4 xv = load_x(x + (size_t)min(m, M - 1) * K + k);
#pragma unroll
                    for (int r = 0; r < ROWS; ++r) {
                        float a = acc[m * ROWS + r];
                        a = fmaf(xv.x, wv[u][r].x, a);
                        a = fmaf(xv.y, wv[u][r].y, a);
                        a = fmaf(xv.z, wv[u][r].z, a);
                        acc[m * ROWS + r] = fmaf(xv.w, wv[u][r].w, a);
                    }
                }
            }
        }
    }
    fold<V, 16>(acc, lane);
    // After the exchanges lane l holds the values whose index has, from its top bit on, the bits of l from bit 4 on: value
    // (l >> SHIFT) * LEFT + i, in every lane with the same l >> SHIFT.
    constexpr int HELD = V > 32 ? 32 : V;        // groups of lanes with different values
    constexpr int GROUP = 32 / HELD;
    if (lane % GROUP == 0) {
#pragma unroll
        for (int i = 0; i < LEFT; ++i) part[warp][(lane / GROUP) * LEFT + i] = acc[i];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < MT * OUTS; i += WARPS * 32) {
        const int m = i / OUTS, r = i % OUTS, n = n0 + r;
        if (m >= M || n >= N) continue;
        float v = 0.f;
#pragma unroll
        for (int q = 0; q < WARPS; ++q) v += part[q][m * ROWS + r];
        if (bias) v += bias[n];
        if constexpr (GATED != 0) {
            float up = 0.f;
#pragma unroll
            for (int q = 0; q < WARPS; ++q) up += part[q][m * ROWS + OUTS + r];
            if (bias) up += bias[N + n];
            if constexpr (GATED == 1) v = v / (1.f + expf(-v));
            else v = 0.5f * v * (1.f + tanhf(0.7978845608028654f * (v + 0.044715f * v * v * v)));
            v *= up;
        } else if (residual) {
            v += residual[(size_t)m * N + n];
        }
        out[(size_t)m * N + n] = v;
    }
}

template <int MT, int ROWS>
void launch_few(float* out, const float* x, const float* w, const float* bias, const float* residual, int M, int N, int K,
                int gated, bool early, cudaStream_t stream) {
    const int outs = gated ? ROWS / 2 : ROWS;
    const dim3 grid((N + outs - 1) / outs);
    if (gated == 2) ti_launch(gemm_f32_few_kernel<MT, ROWS, 2>, grid, WARPS * 32, 0, stream, out, x, w, bias, residual, M, N, K, early);
    else if (gated) ti_launch(gemm_f32_few_kernel<MT, ROWS, 1>, grid, WARPS * 32, 0, stream, out, x, w, bias, residual, M, N, K, early);
    else ti_launch(gemm_f32_few_kernel<MT, ROWS, 0>, grid, WARPS * 32, 0, stream, out, x, w, bias, residual, M, N, K, early);
}

}  // namespace

// As ti_gemm_simt for float32 operands with 1 <= M <= 8, K a multiple of 4 and x and w on 16-byte boundaries. early: no kernel that
// may still run writes w (a model's weights).
TI_API int ti_gemm_f32_few(float* out, const float* x, const float* w, const float* bias, const float* residual,
                           int M, int N, int K, int gated, int early, cudaStream_t stream) {
    TI_REQUIRE(M >= 1 && M <= 8 && N > 0 && K > 0 && K % 4 == 0, "gemm_f32_few: bad sizes M=%d N=%d K=%d", M, N, K);
    TI_REQUIRE(((uintptr_t)x | (uintptr_t)w) % 16 == 0, "gemm_f32_few: operands must lie on 16-byte boundaries");
    TI_REQUIRE(!(gated && residual), "gemm: the gated form takes no residual");
    if (M == 1) launch_few<1, 4>(out, x, w, bias, residual, M, N, K, gated, early, stream);
    else if (M == 2) launch_few<2, 4>(out, x, w, bias, residual, M, N, K, gated, early, stream);
    else if (M <= 4) launch_few<4, 4>(out, x, w, bias, residual, M, N, K, gated, early, stream);
    else launch_few<8, 8>(out, x, w, bias, residual, M, N, K, gated, early, stream);
    TI_CHECK_LAUNCH("gemm_f32_few");
    return 0;
}
