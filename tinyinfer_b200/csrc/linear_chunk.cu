// Linear attention with one decay per head and token (see linear_scan.cu for the recurrence S_t = a_t S_(t-1) + k_t v_t^T,
// o_t = S_t^T q_t) over long portions, in chunks of 64 tokens. Inside a chunk the recurrence is three matrix products, which a
// block holds in registers as tiles: an operand read from shared memory serves 4 to 8 multiply-adds, where the walk token by token
// reads three rows for two. All in float32.
//   state kernel  B = K'^T V with K'_s = k_s (a_(s+1) ... a_last), A = the product of all decays; then linear_scan.cu's fold makes
//                 of every chunk's B the state that it starts from
//   out kernel    o_t = D_t (q_t^T S) + sum_(s <= t) (q_t . k_s) R_ts v_s (+ skip v_t), D_t the product of the decays up to t, R_ts that
//                 of those behind s up to t (made as products, never as quotients: decays may be tiny)
// Chunks lie at cu_seqlens[i] / 64 + i and behind for request i, so num_tokens / 64 + num_seqs of them hold any division of the tokens among
// the requests; those that no request reaches end at once.
// Products of decays are made in 64 bits and rounded once, and sums over 128 channels in pieces of 32: without, 2,000 tokens of decays
// of 0.999 came out 1.0e-6 from 64 bits, where the walk has 6.1e-7.
// 2,000 tokens of 16 heads of 128 x 128 are 1.4 G multiply-adds a layer, 39 us of the chip's float32 rate, of 130. The rest is the fold, a
// third of the time (its threads wait for loads), and operands on their way: the state and out kernels fill the FMA pipe to 46 and 33 %.
// Measured, three kernels, against the walk in stretches: 2,000 tokens 552 -> 130 us (out 1.7e-7 to 2.8e-7 from 64 bits, the walk
// 2.0e-7 to 6.1e-7), 1,000 284 -> 68, 333 108 -> 58, 128 75 -> 48. Decoded tokens and many short portions stay with the walk: see
// ops.linear_chunks.
#include "common.cuh"

namespace lc {
constexpr int C = 64, THREADS = 256, MAXD = 128;
constexpr int LD = MAXD + 4, PLD = C + 4, SK = 32, SLD = SK + 4;      // rows in shared memory: 16-byte reads of 8 rows fall into different banks

struct Args {
    float* y;                 // [T][H * dv]
    const void *q, *k, *v;
    int ld_q, q_off, ld_k, k_off, ld_v, v_off;
    const float* decay;       // rows of ld_decay, first column decay_off: [H]
    int ld_decay, decay_off;
    const float* kscale;      // [T][H] or null
    const float* skip;        // [H] or null
    float q_scale;
    const int* cu_seqlens;
    int heads, groups, dk, dv;
    int num_seqs;
    float *part_b, *part_a;   // [chunk][H][dv][dk], [chunk][H][dk]
};

// The tokens of a chunk: t0 .. t0 + n - 1 (n 0: nobody's chunk).
__device__ __forceinline__ int2 chunk_tokens(const Args& a, int chunk) {
    int low = 0, high = a.num_seqs - 1;                  // the last request that begins at or before the chunk
    while (low < high) {
        const int mid = (low + high + 1) >> 1;
        if (a.cu_seqlens[mid] / C + mid <= chunk) low = mid;
        else high = mid - 1;
    }
    const int begin = a.cu_seqlens[low], t0 = begin + (chunk - begin / C - low) * C;
    return make_int2(t0, max(0, min(C, a.cu_seqlens[low + 1] - t0)));
}

__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
}

// Rows t0 .. t0 + n - 1 of x (first column `at`), `width` columns, times factor[t] * scale, into rows of `ld` floats; zeros past both.
template <typename T>
__device__ __forceinline__ void stage(float* dst, int ld, const void* x, int row, int at, int t0, int n, int width, float scale, const float* factor) {
#pragma unroll 4
    for (int e = threadIdx.x; e < C * (MAXD / 4); e += THREADS) {
        const int t = e / (MAXD / 4), c = e % (MAXD / 4) * 4;
        float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t < n && c < width) {
            f = load4((const T*)x + (size_t)(t0 + t) * row + at + c);
            const float m = factor ? scale * factor[t] : scale;
            f.x *= m; f.y *= m; f.z *= m; f.w *= m;
        }
        *reinterpret_cast<float4*>(dst + t * ld + c) = f;
    }
}

template <typename T>
__global__ void __launch_bounds__(THREADS, 2) state_kernel(Args a) {
    extern __shared__ float smem[];
    float *ks = smem, *vs = smem + C * MAXD;             // [C][MAXD] each
    __shared__ float decay[C], factor[C], whole;
    ti_grid_launch_dependents();
    ti_grid_wait();
    const int h = blockIdx.x, chunk = blockIdx.y, tid = threadIdx.x, g = h / (a.heads / a.groups);
    const int2 tokens = chunk_tokens(a, chunk);
    const int t0 = tokens.x, n = tokens.y;
    if (n == 0) return;
    if (tid < C) decay[tid] = tid < n ? a.decay[(size_t)(t0 + tid) * a.ld_decay + a.decay_off + h] : 1.f;
    __syncthreads();
    if (tid < C) {                                       // the decays behind a token
        double f = 1.;
        for (int s = n - 1; s > tid; --s) f *= decay[s];
        if (tid == 0) whole = (float)(f * decay[0]);
        if (a.kscale && tid < n) f *= a.kscale[(size_t)(t0 + tid) * a.heads + h];
        factor[tid] = (float)f;
    }
    stage<T>(vs, MAXD, a.v, a.ld_v, a.v_off + h * a.dv, t0, n, a.dv, 1.f, nullptr);
    __syncthreads();
    stage<T>(ks, MAXD, a.k, a.ld_k, a.k_off + g * a.dk, t0, n, a.dk, 1.f, factor);
    __syncthreads();
    // 8 key channels (4 tx .. and 64 + 4 tx ..) by 8 value columns (4 ty .. and 64 + 4 ty ..) a thread
    const int tx = tid & 15, ty = tid >> 4;
    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
#pragma unroll 4
    for (int s = 0; s < n; ++s) {
        const float4 k0 = load4(ks + s * MAXD + tx * 4), k1 = load4(ks + s * MAXD + 64 + tx * 4);
        const float4 v0 = load4(vs + s * MAXD + ty * 4), v1 = load4(vs + s * MAXD + 64 + ty * 4);
        const float kk[8] = {k0.x, k0.y, k0.z, k0.w, k1.x, k1.y, k1.z, k1.w}, vv[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(vv[i], kk[j], acc[i][j]);
    }
    float* out = a.part_b + ((size_t)chunk * a.heads + h) * a.dv * a.dk;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int e = (i >> 2) * 64 + ty * 4 + (i & 3);
        if (e >= a.dv) continue;
#pragma unroll
        for (int j = 0; j < 2; ++j)
            if (j * 64 + tx * 4 < a.dk)
                *reinterpret_cast<float4*>(out + (size_t)e * a.dk + j * 64 + tx * 4) = make_float4(acc[i][4 * j], acc[i][4 * j + 1], acc[i][4 * j + 2], acc[i][4 * j + 3]);
    }
    if (tid < a.dk) a.part_a[((size_t)chunk * a.heads + h) * a.dk + tid] = whole;
}

constexpr int OUT_FLOATS = 2 * C * LD + C * PLD + MAXD * SLD;

template <typename T>
__global__ void __launch_bounds__(THREADS, 2) out_kernel(Args a) {
    extern __shared__ float smem[];
    float* qs = smem;                                    // [C][LD]
    float* kv = qs + C * LD;                             // [C][LD]: k, then v
    float* ps = kv + C * LD;                             // [C][PLD]: R_ts, then the products of q and k times it
    float* st = ps + C * PLD;                            // [MAXD][SLD]: 32 key channels of the state, a value column a row
    __shared__ float decay[C], upto[C], factor[C];
    ti_grid_launch_dependents();
    ti_grid_wait();
    const int h = blockIdx.x, chunk = blockIdx.y, tid = threadIdx.x, g = h / (a.heads / a.groups);
    const int2 tokens = chunk_tokens(a, chunk);
    const int t0 = tokens.x, n = tokens.y;
    if (n == 0) return;
    if (tid < C) {
        decay[tid] = tid < n ? a.decay[(size_t)(t0 + tid) * a.ld_decay + a.decay_off + h] : 1.f;
        factor[tid] = a.kscale && tid < n ? a.kscale[(size_t)(t0 + tid) * a.heads + h] : 1.f;
    }
    __syncthreads();
    if (tid < C) {                                       // column s of R; and the product of the decays up to a token
        double f = 1.;
        for (int t = 0; t < tid; ++t) ps[t * PLD + tid] = 0.f;
        for (int t = tid; t < C; ++t) {
            if (t > tid) f *= decay[t];
            ps[t * PLD + tid] = (float)f;
        }
        f = 1.;
        for (int t = 0; t <= tid; ++t) f *= decay[t];
        upto[tid] = (float)f;
    }
    stage<T>(qs, LD, a.q, a.ld_q, a.q_off + g * a.dk, t0, n, a.dk, a.q_scale, nullptr);
    stage<T>(kv, LD, a.k, a.ld_k, a.k_off + g * a.dk, t0, n, a.dk, 1.f, factor);
    __syncthreads();
    {   // q . k: tokens ty + 16 j by keys tx + 16 i, i <= j
        const int tx = tid & 15, ty = tid >> 4;
        float acc[4][4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[j][i] = 0.f;
        float sum[4][4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) sum[j][i] = 0.f;
#pragma unroll 2
        for (int d = 0; d < MAXD; d += 4) {
            float4 q[4], k[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                q[j] = load4(qs + (ty + 16 * j) * LD + d);
                k[j] = load4(kv + (tx + 16 * j) * LD + d);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int i = 0; i <= j; ++i) {
                    acc[j][i] = fmaf(q[j].x, k[i].x, acc[j][i]);
                    acc[j][i] = fmaf(q[j].y, k[i].y, acc[j][i]);
                    acc[j][i] = fmaf(q[j].z, k[i].z, acc[j][i]);
                    acc[j][i] = fmaf(q[j].w, k[i].w, acc[j][i]);
                }
            if ((d & 28) == 28) {                        // a piece has ended
#pragma unroll
                for (int j = 0; j < 4; ++j)
#pragma unroll
                    for (int i = 0; i <= j; ++i) { sum[j][i] += acc[j][i]; acc[j][i] = 0.f; }
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int i = 0; i <= j; ++i)                 // R is zero above the diagonal, and the other tiles stay so
                if (tx + 16 * i <= ty + 16 * j) ps[(ty + 16 * j) * PLD + tx + 16 * i] *= sum[j][i];
    }
    __syncthreads();
    // outputs: tokens 8 ty .. 8 ty + 7 by value columns tx + 32 i; first what the state at the chunk's start gives
    const int tx = tid & 31, ty = tid >> 5;
    float o[8][4], past[8][4];
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) o[j][i] = past[j][i] = 0.f;
    const float* state = a.part_b + ((size_t)chunk * a.heads + h) * a.dv * a.dk;
    stage<T>(kv, LD, a.v, a.ld_v, a.v_off + h * a.dv, t0, n, a.dv, 1.f, nullptr);
    for (int d0 = 0; d0 < a.dk; d0 += SK) {
        __syncthreads();                                 // the piece before has been read
#pragma unroll
        for (int e = tid; e < MAXD * (SK / 4); e += THREADS) {
            const int col = e / (SK / 4), d = e % (SK / 4) * 4;
            float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
            if (col < a.dv && d0 + d < a.dk) f = load4(state + (size_t)col * a.dk + d0 + d);
            *reinterpret_cast<float4*>(st + col * SLD + d) = f;
        }
        __syncthreads();
#pragma unroll 2
        for (int d = 0; d < SK; d += 4) {
            float4 s[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) s[i] = load4(st + (tx + 32 * i) * SLD + d);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float4 q = load4(qs + (8 * ty + j) * LD + d0 + d);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    o[j][i] = fmaf(q.x, s[i].x, o[j][i]);
                    o[j][i] = fmaf(q.y, s[i].y, o[j][i]);
                    o[j][i] = fmaf(q.z, s[i].z, o[j][i]);
                    o[j][i] = fmaf(q.w, s[i].w, o[j][i]);
                }
            }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) { past[j][i] += o[j][i]; o[j][i] = 0.f; }
    }
#pragma unroll 1
    for (int s = 0; s < 8 * ty; s += 4) {                // keys before the thread's tokens
        float4 w[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) w[j] = load4(ps + (8 * ty + j) * PLD + s);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            float v[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = kv[(s + e) * LD + tx + 32 * i];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float p = e == 0 ? w[j].x : e == 1 ? w[j].y : e == 2 ? w[j].z : w[j].w;
#pragma unroll
                for (int i = 0; i < 4; ++i) o[j][i] = fmaf(p, v[i], o[j][i]);
            }
        }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) {                        // and those among them: a token takes in none behind it, not even times 0
        float v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = kv[(8 * ty + e) * LD + tx + 32 * i];
#pragma unroll
        for (int j = e; j < 8; ++j) {
            const float p = ps[(8 * ty + j) * PLD + 8 * ty + e];
#pragma unroll
            for (int i = 0; i < 4; ++i) o[j][i] = fmaf(p, v[i], o[j][i]);
        }
    }
    const float skip = a.skip ? a.skip[h] : 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int t = 8 * ty + j;
        const float reach = upto[t];
        if (t >= n) break;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int e = tx + 32 * i;
            if (e < a.dv) a.y[(size_t)(t0 + t) * a.heads * a.dv + h * a.dv + e] = fmaf(skip, kv[t * LD + e], fmaf(past[j][i], reach, o[j][i]));
        }
    }
}
}  // namespace lc

// Whether the chunked form takes the operands: heads of at most 128 x 128, rows read four neighbouring elements at a time.
bool lc_takes(const void* q, int ld_q, int q_off, const void* k, int ld_k, int k_off, const void* v, int ld_v, int v_off, const float* scratch,
              int dk, int dv, int esize) {
    const int shape = dk | dv | ld_q | q_off | ld_k | k_off | ld_v | v_off;
    return dk <= lc::MAXD && dv <= lc::MAXD && shape % 4 == 0 && ((uintptr_t)q | (uintptr_t)k | (uintptr_t)v) % (4 * esize) == 0 && (uintptr_t)scratch % 16 == 0;
}

// The state kernel (part 0) or the out kernel (part 1) over `chunks` chunks of 64 tokens.
int lc_launch(int part, float* y, const void* q, int ld_q, int q_off, const void* k, int ld_k, int k_off, const void* v, int ld_v, int v_off,
              const float* decay, int ld_decay, int decay_off, const float* kscale, const float* skip, float q_scale, const int* cu_seqlens,
              int num_seqs, int heads, int groups, int dk, int dv, int chunks, float* part_b, float* part_a, int dtype,
              cudaStream_t stream) {
    typedef __nv_bfloat16 B;
    lc::Args a = {y, q, k, v, ld_q, q_off, ld_k, k_off, ld_v, v_off, decay, ld_decay, decay_off, kscale, skip, q_scale, cu_seqlens, heads, groups,
                  dk, dv, num_seqs, part_b, part_a};
    const dim3 grid(heads, chunks);
    constexpr int state_bytes = 2 * lc::C * lc::MAXD * 4, out_bytes = lc::OUT_FLOATS * 4;
    cudaError_t e;
    if (part == 0) {
        e = dtype == TI_F32 ? ti_allow_shared<lc::state_kernel<float>>(state_bytes) : ti_allow_shared<lc::state_kernel<B>>(state_bytes);
        if (e == cudaSuccess)
            e = dtype == TI_F32 ? ti_launch(lc::state_kernel<float>, grid, lc::THREADS, state_bytes, stream, a) : ti_launch(lc::state_kernel<B>, grid, lc::THREADS, state_bytes, stream, a);
    } else {
        e = dtype == TI_F32 ? ti_allow_shared<lc::out_kernel<float>>(out_bytes) : ti_allow_shared<lc::out_kernel<B>>(out_bytes);
        if (e == cudaSuccess)
            e = dtype == TI_F32 ? ti_launch(lc::out_kernel<float>, grid, lc::THREADS, out_bytes, stream, a) : ti_launch(lc::out_kernel<B>, grid, lc::THREADS, out_bytes, stream, a);
    }
    TI_REQUIRE(e == cudaSuccess, "linear_chunk: %s", cudaGetErrorString(e));
    TI_CHECK_LAUNCH("linear_chunk");
    return 0;
}
