// The gated delta rule of delta_scan.cu over long portions, four tokens at a time. The walk token by token is a chain: a token's sums
// over the key channels (D^T k), their round of shuffles, and only then the state that the next token reads. With the decays between
// them multiplied in before, the sums of four tokens read one state, and meet in one round of shuffles. Per head, for the tokens
// 0 .. 3 behind a state S, g_i their decays per channel, P_i = g_0 ... g_i:
//     s_i = S^T (P_i k_i)        u_i = beta_i (v_i - s_i - sum_(j < i) c_ij u_j)             c_ij = sum_c k_j (g_(j+1) ... g_i) k_i
//     r_i = S^T (P_i q_i)        o_i = r_i + sum_(j <= i) d_ij u_j                           d_ij = sum_c k_j (g_(j+1) ... g_i) q_i
//     S  <- P_3 S + sum_j (g_(j+1) ... g_3 k_j) u_j^T
// Decays are only ever multiplied, never divided, so that none of them is too small. All in float32, two rows an instruction.
//   prepare_kernel, a warp a quad and head, makes what no column of S changes: 13 rows of channels and the coefficients, as one
//   record that a walking block fetches with one bulk copy, and the values, four tokens of a column side by side
//   walk_kernel: a block walks a request x head x some columns of S; a lane holds 8 rows of two columns, KP lanes a column. Its 16
//   sums a quad go through a reduce-scatter (15 shuffles for 16 lanes, where every token took 16), each lane ending with one of
//   them; all lanes fetch the s_i and solve for their two columns' u.
// Bound by the chain of a quad, 0.72 us of it (sums, five rounds of shuffles, the solve, the update) on one warp a scheduler, beside 26
// reads of 16 bytes a lane from shared memory. Measured with the prepare kernel, 16 heads of 128 x 128, against the walk: 2,000 tokens
// 572 -> 405 us, 1,000 285 -> 205, 333 102 -> 76, 128 46 -> 37, 64 30 -> 31, 16 36 -> 41 (host included); 1 to 4 % closer to 64 bits. More
// blocks than run at a time lose: ops.delta_quads_pay.
// Quads lie at cu_seqlens[i] / 4 + i and behind for request i, so num_tokens / 4 + num_seqs of them hold any division of the tokens
// among the requests. A request's last quad may be short: rows of zeros, and u_i = 0 by choice, not by product.
#include "sm100_ptx.cuh"

namespace dq {
constexpr int ROWS = 13, COEFS = 32, MAX_WARPS = 4, STAGES = 6;      // rows: P_i k_i, P_i q_i, what is left of k_j, P_3
constexpr int C_AT = 0, D_AT = 8, BETA_AT = 24;                      // of the coefficients: c_10 c_20 c_21 c_30 c_31 c_32, d 4 x 4, beta

struct Args {
    float *y, *state;
    long long slot_stride;
    const void *q, *k, *v;        // rows of ld_* elements, first column *_off; q and k: [groups][dk], v: [H][dv]
    int ld_q, q_off, ld_k, k_off, ld_v, v_off;
    const float* a;               // float32 rows of ld_a, first column a_off: [H][dk]
    int ld_a, a_off;
    const float* b;               // float32 rows of ld_b, first column b_off: [H]
    int ld_b, b_off;
    const float *a_log, *dt_bias; // [H], [H * dk] or null
    float q_scale, unit_eps;
    const int *cu_seqlens, *state_slots;
    int num_seqs, heads, groups, dk, dv, quads, dvp;                 // dvp: dv in whole blocks of columns
    float *records, *values;      // [quad][H][ROWS * 8 KP + COEFS], [quad][H][dvp][4]
    int* status;
};

__device__ __forceinline__ float softplus(float x) { return fmaxf(x, 0.f) + log1pf(expf(-fabsf(x))); }
__device__ __forceinline__ uint64_t pack(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ float2 unpack(uint64_t a) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
    return r;
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const float* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

template <typename T, int KP>
__global__ void __launch_bounds__(128) prepare_kernel(Args a) {
    constexpr int DKP = 8 * KP, CH = DKP / 32;
    ti_grid_launch_dependents();
    ti_grid_wait();
    const int lane = threadIdx.x & 31;
    const size_t item = (size_t)blockIdx.x * 4 + (threadIdx.x >> 5);
    const int quad = (int)(item / a.heads), h = (int)(item % a.heads), g = h / (a.heads / a.groups);
    if (quad >= a.quads) return;
    int low = 0, high = a.num_seqs - 1;                  // the last request that begins at or before the quad
    while (low < high) {
        const int mid = (low + high + 1) >> 1;
        if (a.cu_seqlens[mid] / 4 + mid <= quad) low = mid;
        else high = mid - 1;
    }
    const int begin = a.cu_seqlens[low], t0 = begin + (quad - begin / 4 - low) * 4, n = min(4, a.cu_seqlens[low + 1] - t0);
    if (n <= 0) return;                                  // nobody's quad
    const float rate = expf(a.a_log[h]);
    float q[4][CH], k[4][CH], z[4][CH];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const T* qr = (const T*)a.q + (size_t)(t0 + i) * a.ld_q + a.q_off + g * a.dk;
        const T* kr = (const T*)a.k + (size_t)(t0 + i) * a.ld_k + a.k_off + g * a.dk;
        const float* ar = a.a + (size_t)(t0 + i) * a.ld_a + a.a_off + h * a.dk;
#pragma unroll
        for (int j = 0; j < CH; ++j) {
            const int c = lane + 32 * j;
            const bool ok = i < n && c < a.dk;
            q[i][j] = ok ? to_f32(qr[c]) : 0.f;
            k[i][j] = ok ? to_f32(kr[c]) : 0.f;
            z[i][j] = ok ? ar[c] : 0.f;
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float ssq = 0.f, ssk = 0.f;
#pragma unroll
        for (int j = 0; j < CH; ++j) {
            ssq = fmaf(q[i][j], q[i][j], ssq);
            ssk = fmaf(k[i][j], k[i][j], ssk);
        }
        ssq = warp_sum(ssq);
        ssk = warp_sum(ssk);
        const float fq = a.q_scale / sqrtf(ssq + a.unit_eps), fk = 1.f / sqrtf(ssk + a.unit_eps);
#pragma unroll
        for (int j = 0; j < CH; ++j) {
            const int c = lane + 32 * j;
            q[i][j] = i < n ? q[i][j] * fq : 0.f;
            k[i][j] = i < n ? k[i][j] * fk : 0.f;
            z[i][j] = i < n && c < a.dk ? expf(-rate * softplus(z[i][j] + (a.dt_bias ? a.dt_bias[h * a.dk + c] : 0.f))) : 1.f;
        }
    }
    float* rec = a.records + item * (ROWS * DKP + COEFS);
    float cs[4][4], ds[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) cs[i][j] = ds[i][j] = 0.f;
#pragma unroll
    for (int x = 0; x < CH; ++x) {
        const int c = lane + 32 * x;
        float left[4], p = 1.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float gi = z[i][x], ki = k[i][x], qi = q[i][x];
            p *= gi;
#pragma unroll
            for (int j = 0; j < i; ++j) {
                left[j] *= gi;
                cs[i][j] = fmaf(left[j], ki, cs[i][j]);
                ds[i][j] = fmaf(left[j], qi, ds[i][j]);
            }
            left[i] = ki;
            ds[i][i] = fmaf(ki, qi, ds[i][i]);
            rec[i * DKP + c] = ki * p;
            rec[(4 + i) * DKP + c] = qi * p;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) rec[(8 + j) * DKP + c] = left[j];
        rec[12 * DKP + c] = p;
    }
    float mine = 0.f;                                    // lane l: coefficient l
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int j = 0; j <= i; ++j) {
            const float d = warp_sum(ds[i][j]);
            if (lane == D_AT + 4 * i + j) mine = d;
            if (j < i) {
                const float c = warp_sum(cs[i][j]);
                if (lane == C_AT + i * (i - 1) / 2 + j) mine = c;
            }
        }
    }
    if (lane >= BETA_AT && lane - BETA_AT < n) mine = 1.f / (1.f + expf(-a.b[(size_t)(t0 + lane - BETA_AT) * a.ld_b + a.b_off + h]));
    rec[ROWS * DKP + lane] = mine;
    for (int c = lane; c < a.dvp; c += 32) {
        float v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = i < n && c < a.dv ? to_f32(((const T*)a.v)[(size_t)(t0 + i) * a.ld_v + a.v_off + h * a.dv + c]) : 0.f;
        *reinterpret_cast<float4*>(a.values + (item * a.dvp + c) * 4) = make_float4(v[0], v[1], v[2], v[3]);
    }
}

template <int KP>
__global__ void __launch_bounds__((MAX_WARPS + 1) * 32) walk_kernel(Args a) {
    constexpr int DKP = 8 * KP, REC = ROWS * DKP + COEFS, LANE_COLS = 32 / KP * 2;
    extern __shared__ __align__(128) float smem[];
    __shared__ uint64_t bars[2 * STAGES];
    __shared__ int abort_sh;
    volatile int* abort_flag = &abort_sh;
    const int warps = (blockDim.x >> 5) - 1, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int cpb = warps * LANE_COLS, stage_floats = REC + cpb * 4, col_blocks = a.dvp / cpb;
    const uint32_t bar0 = smem_u32(bars);
    auto full = [&](int s) { return bar0 + 8u * s; };
    auto empty = [&](int s) { return bar0 + 8u * (STAGES + s); };
    if (threadIdx.x == 0) {
        abort_sh = 0;
        for (int s = 0; s < STAGES; ++s) { mbar_init(full(s), 1); mbar_init(empty(s), warps); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    ti_grid_wait();
    const int h = blockIdx.x / col_blocks, cb = blockIdx.x % col_blocks, seq = blockIdx.y;
    const int row0 = a.cu_seqlens[seq], row1 = a.cu_seqlens[seq + 1], first = row0 / 4 + seq, nq = (row1 - row0 + 3) / 4;

    if (warp == warps) {                                 // the copies
        if (lane == 0) {
            for (int j = 0; j < nq; ++j) {
                const int s = j % STAGES;
                if (!mbar_wait(empty(s), ((j / STAGES) & 1u) ^ 1u, abort_flag, a.status, 91)) break;
                const size_t item = (size_t)(first + j) * a.heads + h;
                const uint32_t dst = smem_u32(smem + (size_t)s * stage_floats);
                mbar_expect_tx(full(s), (uint32_t)stage_floats * 4u);
                bulk_load(dst, a.records + item * REC, REC * 4, full(s));
                bulk_load(dst + REC * 4, a.values + (item * a.dvp + cb * cpb) * 4, cpb * 16, full(s));
            }
        }
    } else {
        const int kpart = lane % KP, base = lane - kpart, lcol = warp * LANE_COLS + (lane / KP) * 2, col0 = cb * cpb + lcol;
        // rows 4 kpart .. + 3 and DKP / 2 + 4 kpart .. + 3: the lanes of a column read neighbouring 16 bytes
        auto channel = [&](int e) { return (e >> 2) * (DKP / 2) + kpart * 4 + (e & 3); };
        float* shead = a.state + (size_t)a.state_slots[seq] * a.slot_stride + (size_t)h * a.dv * a.dk;
        uint64_t S[2][4];
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                float s[2];
#pragma unroll
                for (int e = 0; e < 2; ++e)
                    s[e] = col0 + c < a.dv && channel(2 * r + e) < a.dk ? shead[(size_t)(col0 + c) * a.dk + channel(2 * r + e)] : 0.f;
                S[c][r] = pack(s[0], s[1]);
            }
        auto read = [&](const float* at, uint64_t (&x)[4]) {
            const ulonglong2 u = *reinterpret_cast<const ulonglong2*>(at + kpart * 4), w = *reinterpret_cast<const ulonglong2*>(at + DKP / 2 + kpart * 4);
            x[0] = u.x; x[1] = u.y; x[2] = w.x; x[3] = w.y;
        };
        uint64_t ahead[8][4];                            // P_i k_i and P_i q_i of the next quad
        bool ok = nq == 0 || mbar_wait(full(0), 0, abort_flag, a.status, 92);
        ok = __all_sync(0xffffffffu, ok);
        if (ok && nq > 0)
#pragma unroll
            for (int i = 0; i < 8; ++i) read(smem + i * DKP, ahead[i]);
        for (int j = 0; j < nq && ok; ++j) {
            const int s = j % STAGES, next = (j + 1) % STAGES, t = row0 + 4 * j, n = min(4, row1 - t);
            const float* st = smem + (size_t)s * stage_floats;
            float val[16];                               // [s or r][token][column]
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    uint64_t x = mul2(ahead[i][0], S[c][0]);
#pragma unroll
                    for (int r = 1; r < 4; ++r) x = fma2(ahead[i][r], S[c][r], x);
                    const float2 f = unpack(x);
                    val[2 * i + c] = f.x + f.y;
                }
            uint64_t left[4][4], p[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) read(st + (8 + i) * DKP, left[i]);
            read(st + 12 * DKP, p);
            const float* coef = st + ROWS * DKP;
            const int mi = (kpart / (KP / 8)) & 3;       // the token of the lane's own sum
            const float4 ca = *reinterpret_cast<const float4*>(coef + C_AT), cd = *reinterpret_cast<const float4*>(coef + C_AT + 4);
            const float4 beta = *reinterpret_cast<const float4*>(coef + BETA_AT), drow = *reinterpret_cast<const float4*>(coef + D_AT + 4 * mi);
            float4 v[2];
#pragma unroll
            for (int c = 0; c < 2; ++c) v[c] = *reinterpret_cast<const float4*>(st + REC + (lcol + c) * 4);
            if (j + 1 < nq) {
                ok = __all_sync(0xffffffffu, mbar_wait(full(next), ((j + 1) / STAGES) & 1u, abort_flag, a.status, 92));
                if (!ok) break;
#pragma unroll
                for (int i = 0; i < 8; ++i) read(smem + (size_t)next * stage_floats + i * DKP, ahead[i]);
            }
#pragma unroll
            for (int half = 8, off = KP / 2; half >= 1; half >>= 1, off >>= 1) {
                if (off == 0) break;                     // 8 lanes a column: two sums a lane
                const bool upper = kpart & off;
#pragma unroll
                for (int e = 0; e < half; ++e) {
                    const float give = upper ? val[e] : val[e + half], keep = upper ? val[e + half] : val[e];
                    val[e] = keep + __shfl_xor_sync(0xffffffffu, give, off);
                }
            }
            if (KP == 32) val[0] += __shfl_xor_sync(0xffffffffu, val[0], 1);
            float u[2][4];
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                float d[4];
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    d[i] = KP == 8 ? __shfl_sync(0xffffffffu, val[c], base + i) : __shfl_sync(0xffffffffu, val[0], base + i * (KP / 8) + c * (KP / 16));
                u[c][0] = beta.x * (v[c].x - d[0]);
                u[c][1] = n > 1 ? beta.y * fmaf(-ca.x, u[c][0], v[c].y - d[1]) : 0.f;
                u[c][2] = n > 2 ? beta.z * fmaf(-ca.z, u[c][1], fmaf(-ca.y, u[c][0], v[c].z - d[2])) : 0.f;
                u[c][3] = n > 3 ? beta.w * fmaf(-cd.y, u[c][2], fmaf(-cd.x, u[c][1], fmaf(-ca.w, u[c][0], v[c].w - d[3]))) : 0.f;
            }
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                uint64_t uu[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) uu[i] = pack(u[c][i], u[c][i]);
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    uint64_t x = mul2(p[r], S[c][r]);
#pragma unroll
                    for (int i = 0; i < 4; ++i) x = fma2(left[i][r], uu[i], x);
                    S[c][r] = x;
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty(s));        // everything of this quad is in registers
            if ((kpart & (KP / 2)) && mi < n && (KP < 32 || !(kpart & 1))) {
                // a token takes in none behind it, not even times 0
                auto out = [&](int col, float o, float u0, float u1, float u2, float u3) {
                    o = fmaf(drow.x, u0, o);
                    o = mi > 0 ? fmaf(drow.y, u1, o) : o;
                    o = mi > 1 ? fmaf(drow.z, u2, o) : o;
                    o = mi > 2 ? fmaf(drow.w, u3, o) : o;
                    if (col < a.dv) a.y[(size_t)(t + mi) * a.heads * a.dv + h * a.dv + col] = o;
                };
                if (KP == 8) {
                    out(col0, val[0], u[0][0], u[0][1], u[0][2], u[0][3]);
                    out(col0 + 1, val[1], u[1][0], u[1][1], u[1][2], u[1][3]);
                } else {
                    const bool second = kpart & (KP / 16);
                    out(col0 + second, val[0], second ? u[1][0] : u[0][0], second ? u[1][1] : u[0][1], second ? u[1][2] : u[0][2],
                        second ? u[1][3] : u[0][3]);
                }
            }
        }
        if (ok)
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const float2 f = unpack(S[c][r]);
                    const float x[2] = {f.x, f.y};
#pragma unroll
                    for (int e = 0; e < 2; ++e)
                        if (col0 + c < a.dv && channel(2 * r + e) < a.dk) shead[(size_t)(col0 + c) * a.dk + channel(2 * r + e)] = x[e];
                }
    }
    __syncthreads();
    if (warp == warps) land_copies(abort_flag);
    ti_grid_launch_dependents();                         // only now (a block's first thread speaks for it): the walk is long, and the next
}                                                        // kernel's blocks would sit on the SMs through it

// Lanes a column, and the columns of a block of `warps` warps.
static int lanes(int dk) { return dk <= 64 ? 8 : dk <= 128 ? 16 : 32; }
static int block_warps(int num_seqs, int heads, int dk, int dv) {
    int warps = MAX_WARPS;                               // few columns a block when there are few (request, head) pairs
    const int cols = 32 / lanes(dk) * 2;
    while (warps > 1 && (long long)num_seqs * heads * ((dv + warps * cols - 1) / (warps * cols)) < 100) warps >>= 1;
    return warps;
}
static long long padded_dv(int num_seqs, int heads, int dk, int dv) {
    const int cpb = block_warps(num_seqs, heads, dk, dv) * (32 / lanes(dk) * 2);
    return (long long)((dv + cpb - 1) / cpb) * cpb;
}

template <int KP> static cudaError_t launch(const Args& a, int warps, int dtype, cudaStream_t stream) {
    const unsigned blocks = (unsigned)(((size_t)a.quads * a.heads + 3) / 4);
    cudaError_t e = dtype == TI_F32 ? ti_launch(prepare_kernel<float, KP>, blocks, 128, 0, stream, a)
                                    : ti_launch(prepare_kernel<__nv_bfloat16, KP>, blocks, 128, 0, stream, a);
    const int cpb = warps * (32 / KP * 2), smem = STAGES * (ROWS * 8 * KP + COEFS + cpb * 4) * 4;
    if (e == cudaSuccess) e = ti_allow_shared<walk_kernel<KP>>(smem);
    if (e == cudaSuccess) e = ti_launch_alone(walk_kernel<KP>, dim3(a.heads * (a.dvp / cpb), a.num_seqs), (warps + 1) * 32, smem, stream, a);
    return e;
}
}  // namespace dq

// Floats of workspace that ti_delta_quads needs, or 0 where the walk token by token should be taken: key channels beyond 256, and
// steps of few tokens (one request of 64: 31 us against 30, of 128: 37 against 46), where a request counts for its 4 at least, as a
// lone token costs a whole quad.
TI_API long long ti_delta_quads_floats(int num_seqs, int num_tokens, int heads, int dk, int dv) {
    if (num_seqs <= 0 || num_seqs > 65535 || heads <= 0 || dk <= 0 || dk > 256 || dv <= 0 || num_tokens < 64 + 4ll * num_seqs) return 0;
    const long long items = (num_tokens / 4 + (long long)num_seqs) * heads;
    if (items > (1ll << 31) - 8) return 0;
    return items * (dq::ROWS * 8ll * dq::lanes(dk) + dq::COEFS + 4 * dq::padded_dv(num_seqs, heads, dk, dv));
}

// As ti_delta_scan (delta_scan.cu), four tokens at a time. work: ti_delta_quads_floats floats, 16-byte aligned.
TI_API int ti_delta_quads(float* y, float* state, long long slot_stride, const void* q, int ld_q, int q_off, const void* k, int ld_k,
                          int k_off, const void* v, int ld_v, int v_off, const float* a, int ld_a, int a_off, const float* b, int ld_b,
                          int b_off, const float* a_log, const float* dt_bias, float q_scale, float unit_eps, const int* cu_seqlens,
                          const int* state_slots, int num_seqs, int num_tokens, int heads, int groups, int dk, int dv, float* work,
                          long long work_floats, int* status, int dtype, cudaStream_t stream) {
    TI_REQUIRE(groups > 0 && heads % groups == 0, "delta_quads: bad sizes");
    const long long floats = ti_delta_quads_floats(num_seqs, num_tokens, heads, dk, dv);
    TI_REQUIRE(floats > 0, "delta_quads: %d requests of %d tokens, %d key channels are not taken", num_seqs, num_tokens, dk);
    TI_REQUIRE(a && b && a_log, "delta_quads: the decay's and the step's tensors are needed");
    TI_REQUIRE(dtype == TI_F32 || dtype == TI_BF16, "delta_quads: unknown dtype %d", dtype);
    TI_REQUIRE(work && ((uintptr_t)work & 15) == 0 && work_floats >= floats, "delta_quads: the workspace is too small or not 16-byte aligned");
    const int kp = dq::lanes(dk), quads = num_tokens / 4 + num_seqs;
    const size_t items = (size_t)quads * heads;
    dq::Args args = {y, state, slot_stride, q, k, v, ld_q, q_off, ld_k, k_off, ld_v, v_off, a, ld_a, a_off, b, ld_b, b_off, a_log, dt_bias,
                     q_scale, unit_eps, cu_seqlens, state_slots, num_seqs, heads, groups, dk, dv, quads,
                     (int)dq::padded_dv(num_seqs, heads, dk, dv), work, work + items * (dq::ROWS * 8 * kp + dq::COEFS), status};
    const int warps = dq::block_warps(num_seqs, heads, dk, dv);
    const cudaError_t e = kp == 8 ? dq::launch<8>(args, warps, dtype, stream) : kp == 16 ? dq::launch<16>(args, warps, dtype, stream)
                                                                                      : dq::launch<32>(args, warps, dtype, stream);
    TI_REQUIRE(e == cudaSuccess, "delta_quads: %s", cudaGetErrorString(e));
    TI_CHECK_LAUNCH("delta_quads");
    return 0;
}
