// Paged causal attention of the 32-bit path for head sizes 64 and 128, in float32 arithmetic throughout. Masks, pages, the
// softmax and the map from query to kv heads are those of attention_generic.cu, which stays for every other shape.
//
// Single decoded tokens: a cluster of 8 blocks serves up to 4 query heads of one kv head of one token; the blocks share the
// keys out, so that every key and value is read once per such group and a batch of few requests still spreads over the
// machine. 8 lanes hold a key (16 bytes a lane and load, 128 contiguous bytes a key), every such group of lanes keeps a
// running maximum, sum and output of its own; they meet by shuffles, then in shared memory, then across the cluster through
// distributed shared memory, where every block finishes an eighth of the output. Bound by the keys' and values' way from HBM: 4 tokens
// behind 1,024 keys 13 us, where their bytes need 5.
//
// Portions of prompts: a block takes 16 or 32 query rows, which are the query heads of one kv head for neighbouring tokens,
// over tiles of 64 keys: keys and values come in by cp.async, the values' copy runs under the scores. A thread makes 2 x 4
// scores and 2 x (D / 16) outputs. Bound by shared-memory reads beside the multiply-adds on the SMs with the most keys (58 % of the cycles there,
// 41 % on the average, for 333 tokens).
// A layer of 16 over 8 heads of 128: 333 prompt tokens 0.8 ms with a block a (token, head) -> 53 us with
// 32 rows a block -> some 30 us with 16, the longest ranges first (a step of 28 layers 11.0 -> 10.4 ms); 4 tokens behind 1,024 keys
// 32 us with the queries in registers and one block an SM -> 13 us with them in shared memory and two.
#include "common.cuh"
#include <cooperative_groups.h>
#include <type_traits>

namespace {

struct AfArgs {
    float* out;
    const float *q, *k, *v;
    const int *positions, *token_seq, *block_table;
    const int *rows;            // decode: the flat row of each single token; portions: tiles [entry, first row, rows, first position]
    int max_blocks, hq, hkv, page_size, num_pages, window;
    float scale;
    int* status;
};

// Offset of key j's row in the key (and value) planes, or -1 where the request holds no page for it.
__device__ __forceinline__ long long key_row(const AfArgs& a, const int* table, int kvh, int j, int d) {
    const int logical = j / a.page_size;
    const int page = logical < a.max_blocks ? table[logical] : -1;
    if (page < 0 || page >= a.num_pages) return -1;
    return (((long long)page * a.hkv + kvh) * a.page_size + (j - logical * a.page_size)) * d;
}

constexpr int DEC_CTAS = 8, DEC_WARPS = 8;

template <int D, int GT>
__global__ void __cluster_dims__(DEC_CTAS, 1, 1) __launch_bounds__(DEC_WARPS * 32, GT <= 2 ? 2 : 1) decode_f32_kernel(const AfArgs a) {
    constexpr int E4 = D / 32;                   // float4s of a head that a lane holds
    constexpr int U = 2;                         // keys of a lane group asked for together
    __shared__ float wm[DEC_WARPS][GT], wl[DEC_WARPS][GT];
    __shared__ __align__(16) float wacc[DEC_WARPS][GT][D];
    __shared__ float cm[GT], cl[GT], cacc[GT][D];
    __shared__ __align__(16) float qs[GT][D];        // read anew for every key: registers for it would cost the second block of an SM
    ti_grid_launch_dependents();
    ti_grid_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane & 7, grp = lane >> 3;
    const int G = a.hq / a.hkv, chunks = (G + GT - 1) / GT;
    const int kvh = blockIdx.y / chunks, g0 = (blockIdx.y % chunks) * GT;
    const int t = a.rows[blockIdx.z];
    const int pos = a.positions[t];
    const int lo = ti_first_key(pos, a.window);
    const int* table = a.block_table + (size_t)a.token_seq[t] * a.max_blocks;
    const int share = ((pos + 1 - lo + DEC_CTAS - 1) / DEC_CTAS + 31) & ~31;
    const int begin = lo + (int)blockIdx.x * share, end = min(pos + 1, begin + share);

    for (int i = threadIdx.x; i < GT * D; i += DEC_WARPS * 32)
        qs[i / D][i % D] = a.q[((size_t)t * a.hq + kvh * G + min(g0 + i / D, G - 1)) * D + i % D];
    __syncthreads();
    float acc[GT][4 * E4], m[GT], l[GT];
#pragma unroll
    for (int g = 0; g < GT; ++g) {
#pragma unroll
        for (int i = 0; i < 4 * E4; ++i) acc[g][i] = 0.f;
        m[g] = -INFINITY;
        l[g] = 0.f;
    }
    for (int base = begin + warp * 4; base < end; base += U * DEC_WARPS * 4) {
        float4 kf[U][E4], vf[U][E4];
        bool there[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int j = base + u * DEC_WARPS * 4 + grp;
            long long off = -1;
            if (j < end) {
                off = key_row(a, table, kvh, j, D);
                if (off < 0 && a.status) atomicExch(a.status, 2);      // a visible key without a page
            }
            there[u] = off >= 0;
#pragma unroll
            for (int i = 0; i < E4; ++i) {
                kf[u][i] = there[u] ? reinterpret_cast<const float4*>(a.k + off)[sub + 8 * i] : make_float4(0.f, 0.f, 0.f, 0.f);
                vf[u][i] = there[u] ? reinterpret_cast<const float4*>(a.v + off)[sub + 8 * i] : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
#pragma unroll
        for (int g = 0; g < GT; ++g) {
            float s[U] = {}, top = m[g];
#pragma unroll
            for (int i = 0; i < E4; ++i) {
                const float4 q = *reinterpret_cast<const float4*>(&qs[g][4 * (sub + 8 * i)]);
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    s[u] = fmaf(q.x, kf[u][i].x, s[u]);
                    s[u] = fmaf(q.y, kf[u][i].y, s[u]);
                    s[u] = fmaf(q.z, kf[u][i].z, s[u]);
                    s[u] = fmaf(q.w, kf[u][i].w, s[u]);
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                float dot = s[u];
#pragma unroll
                for (int o = 4; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
                s[u] = there[u] ? dot * a.scale : -INFINITY;
                top = fmaxf(top, s[u]);
            }
            const float corr = m[g] == -INFINITY ? 0.f : expf(m[g] - top);
            m[g] = top;
            l[g] *= corr;
#pragma unroll
            for (int i = 0; i < 4 * E4; ++i) acc[g][i] *= corr;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const float p = s[u] == -INFINITY ? 0.f : expf(s[u] - top);
                l[g] += p;
                if (!there[u]) continue;
#pragma unroll
                for (int i = 0; i < E4; ++i) {
                    acc[g][4 * i] = fmaf(p, vf[u][i].x, acc[g][4 * i]);
                    acc[g][4 * i + 1] = fmaf(p, vf[u][i].y, acc[g][4 * i + 1]);
                    acc[g][4 * i + 2] = fmaf(p, vf[u][i].z, acc[g][4 * i + 2]);
                    acc[g][4 * i + 3] = fmaf(p, vf[u][i].w, acc[g][4 * i + 3]);
                }
            }
        }
    }
    // the four lane groups of a warp
#pragma unroll
    for (int g = 0; g < GT; ++g) {
#pragma unroll
        for (int o = 8; o < 32; o <<= 1) {
            const float mo = __shfl_xor_sync(0xffffffffu, m[g], o), lo_ = __shfl_xor_sync(0xffffffffu, l[g], o);
            const float top = fmaxf(m[g], mo);
            const float c0 = m[g] == -INFINITY ? 0.f : expf(m[g] - top), c1 = mo == -INFINITY ? 0.f : expf(mo - top);
            l[g] = l[g] * c0 + lo_ * c1;
            m[g] = top;
#pragma unroll
            for (int i = 0; i < 4 * E4; ++i) acc[g][i] = acc[g][i] * c0 + __shfl_xor_sync(0xffffffffu, acc[g][i], o) * c1;
        }
        if (grp == 0) {
            if (sub == 0) { wm[warp][g] = m[g]; wl[warp][g] = l[g]; }
#pragma unroll
            for (int i = 0; i < E4; ++i)
                *reinterpret_cast<float4*>(&wacc[warp][g][4 * (sub + 8 * i)]) =
                    make_float4(acc[g][4 * i], acc[g][4 * i + 1], acc[g][4 * i + 2], acc[g][4 * i + 3]);
        }
    }
    __syncthreads();
    // the warps of a block
    for (int i = threadIdx.x; i < GT * D; i += DEC_WARPS * 32) {
        const int g = i / D, f = i % D;
        float top = -INFINITY;
#pragma unroll
        for (int w = 0; w < DEC_WARPS; ++w) top = fmaxf(top, wm[w][g]);
        float sum = 0.f, o = 0.f;
#pragma unroll
        for (int w = 0; w < DEC_WARPS; ++w) {
            const float c = wm[w][g] == -INFINITY ? 0.f : expf(wm[w][g] - top);
            sum += wl[w][g] * c;
            o += wacc[w][g][f] * c;
        }
        cacc[g][f] = o;
        if (f == 0) { cm[g] = top; cl[g] = sum; }
    }
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    cluster.sync();
    // the blocks of the cluster: each finishes its eighth of the outputs
    constexpr int PART = GT * D / DEC_CTAS;
    for (int i = threadIdx.x; i < PART; i += DEC_WARPS * 32) {
        const int e = (int)blockIdx.x * PART + i, g = e / D, f = e % D;
        float top = -INFINITY, ms[DEC_CTAS];
#pragma unroll
        for (int c = 0; c < DEC_CTAS; ++c) {
            ms[c] = *cluster.map_shared_rank(&cm[g], c);
            top = fmaxf(top, ms[c]);
        }
        float sum = 0.f, o = 0.f;
#pragma unroll
        for (int c = 0; c < DEC_CTAS; ++c) {
            const float w = ms[c] == -INFINITY ? 0.f : expf(ms[c] - top);
            sum += *cluster.map_shared_rank(&cl[g], c) * w;
            o += *cluster.map_shared_rank(&cacc[g][f], c) * w;
        }
        if (g0 + g < G) a.out[((size_t)t * a.hq + kvh * G + g0 + g) * D + f] = sum > 0.f ? o / sum : 0.f * o;
    }
    cluster.sync();                              // nobody leaves while its shared memory may be read
}

constexpr int PR_KEYS = 64, PR_MAX_ROWS = 32;

template <int D, int PR_ROWS> constexpr int portion_smem() {
    return 4 * (PR_ROWS * (D + 4) + PR_KEYS * (D + 4) + PR_KEYS * D + PR_ROWS * (PR_KEYS + 4)) + 8 * PR_KEYS;
}
__device__ __forceinline__ void copy16(void* dst, const void* src, bool there) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(there ? 16 : 0) : "memory");
}

template <int D, int PR_ROWS>
__global__ void __launch_bounds__(PR_ROWS * 8) portion_f32_kernel(const AfArgs a) {
    constexpr int PR_THREADS = PR_ROWS * 8;
    extern __shared__ float4 smem4[];
    float* qs = reinterpret_cast<float*>(smem4);             // [PR_ROWS][D + 4]: rows 16 bytes askew, so that 8 lanes meet 32 banks
    float* ks = qs + PR_ROWS * (D + 4);                      // [64][D + 4]
    float* vs = ks + PR_KEYS * (D + 4);                      // [64][D]
    float* ps = vs + PR_KEYS * D;                            // [PR_ROWS][64 + 4]
    long long* off = reinterpret_cast<long long*>(ps + PR_ROWS * (PR_KEYS + 4));
    ti_grid_launch_dependents();
    ti_grid_wait();
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int kvh = blockIdx.x, G = a.hq / a.hkv, per = PR_ROWS / G;
    const int* tile = a.rows + 4 * blockIdx.z;
    const int first = ((int)gridDim.y - 1 - (int)blockIdx.y) * per;    // the block's first token within the tile, the longest ranges first
    const int tokens = min(per, tile[2] - first);
    if (tokens <= 0) return;
    const int row0 = tile[1] + first, pos0 = tile[3] + first, last = pos0 + tokens - 1;
    const int* table = a.block_table + (size_t)tile[0] * a.max_blocks;

    for (int i = tid; i < PR_ROWS * (D / 4); i += PR_THREADS) {
        const int r = i / (D / 4), c = i % (D / 4), tok = r / G;
        const float* src = a.q + ((size_t)(row0 + min(tok, tokens - 1)) * a.hq + kvh * G + r % G) * D + 4 * c;
        *reinterpret_cast<float4*>(qs + r * (D + 4) + 4 * c) = *reinterpret_cast<const float4*>(src);
    }
    int pos[2], lo[2];
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f}, acc[2][D / 16];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        pos[r] = pos0 + min((ty * 2 + r) / G, tokens - 1);
        lo[r] = ti_first_key(pos[r], a.window);
#pragma unroll
        for (int i = 0; i < D / 16; ++i) acc[r][i] = 0.f;
    }
    for (int key0 = ti_first_key(pos0, a.window); key0 <= last; key0 += PR_KEYS) {
        __syncthreads();                                     // everyone is done with the tile before
        if (tid < PR_KEYS) {
            const int j = key0 + tid;
            long long o = -1;
            if (j <= last) {
                o = key_row(a, table, kvh, j, D);
                if (o < 0 && a.status) atomicExch(a.status, 2);
            }
            off[tid] = o;
        }
        __syncthreads();
#pragma unroll 4
        for (int i = tid; i < PR_KEYS * (D / 4); i += PR_THREADS) {
            const int j = i / (D / 4), c = i % (D / 4);
            const long long o = off[j];
            copy16(ks + j * (D + 4) + 4 * c, a.k + (o < 0 ? 0 : o) + 4 * c, o >= 0);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
#pragma unroll 4
        for (int i = tid; i < PR_KEYS * (D / 4); i += PR_THREADS) {
            const int j = i / (D / 4), c = i % (D / 4);
            const long long o = off[j];
            copy16(vs + j * D + 4 * c, a.v + (o < 0 ? 0 : o) + 4 * c, o >= 0);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();                                     // the keys are there
        float s[2][4] = {};
#pragma unroll 4
        for (int f = 0; f < D; f += 4) {
            float4 qv[2];
#pragma unroll
            for (int r = 0; r < 2; ++r) qv[r] = *reinterpret_cast<const float4*>(qs + (ty * 2 + r) * (D + 4) + f);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float4 kv = *reinterpret_cast<const float4*>(ks + (tx + 16 * i) * (D + 4) + f);
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    s[r][i] = fmaf(qv[r].x, kv.x, s[r][i]);
                    s[r][i] = fmaf(qv[r].y, kv.y, s[r][i]);
                    s[r][i] = fmaf(qv[r].z, kv.z, s[r][i]);
                    s[r][i] = fmaf(qv[r].w, kv.w, s[r][i]);
                }
            }
        }
        // A key that a row does not see must not reach it even as 0 x infinity: its probability says so by its sign. Only tiles with
        // such keys pay for the test.
        const bool all_see = key0 + PR_KEYS - 1 <= pos0 && key0 >= ti_first_key(last, a.window);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            float top = m[r];
            bool seen[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int j = key0 + tx + 16 * i;
                seen[i] = j >= lo[r] && j <= pos[r] && off[tx + 16 * i] >= 0;
                s[r][i] = seen[i] ? s[r][i] * a.scale : -INFINITY;
                top = fmaxf(top, s[r][i]);
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
            const float corr = m[r] == -INFINITY ? 0.f : expf(m[r] - top);
            float sum = 0.f;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float p = s[r][i] == -INFINITY ? 0.f : expf(s[r][i] - top);
                sum += p;
                ps[(ty * 2 + r) * (PR_KEYS + 4) + tx + 16 * i] = seen[i] || all_see ? p : -1.f;
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            l[r] = l[r] * corr + sum;
            m[r] = top;
#pragma unroll
            for (int i = 0; i < D / 16; ++i) acc[r][i] *= corr;
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                                     // the values and everyone's probabilities are there
        auto add = [&](auto guarded) {
#pragma unroll 2
            for (int j = 0; j < PR_KEYS; j += 4) {
                float pr[2][4];
#pragma unroll
                for (int r = 0; r < 2; ++r)
                    *reinterpret_cast<float4*>(pr[r]) = *reinterpret_cast<const float4*>(ps + (ty * 2 + r) * (PR_KEYS + 4) + j);
#pragma unroll
                for (int jj = 0; jj < 4; ++jj)
#pragma unroll
                    for (int i = 0; i < D / 64; ++i) {
                        const float4 vv = *reinterpret_cast<const float4*>(vs + (j + jj) * D + tx * 4 + 64 * i);
#pragma unroll
                        for (int r = 0; r < 2; ++r) {
                            if constexpr (decltype(guarded)::value) { if (pr[r][jj] < 0.f) continue; }
                            acc[r][4 * i] = fmaf(pr[r][jj], vv.x, acc[r][4 * i]);
                            acc[r][4 * i + 1] = fmaf(pr[r][jj], vv.y, acc[r][4 * i + 1]);
                            acc[r][4 * i + 2] = fmaf(pr[r][jj], vv.z, acc[r][4 * i + 2]);
                            acc[r][4 * i + 3] = fmaf(pr[r][jj], vv.w, acc[r][4 * i + 3]);
                        }
                    }
            }
        };
        if (all_see) add(std::false_type{});
        else add(std::true_type{});
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int row = ty * 2 + r, tok = row / G;
        if (tok >= tokens) continue;
        const float inv = l[r] > 0.f ? 1.f / l[r] : 0.f;
        float* o = a.out + ((size_t)(row0 + tok) * a.hq + kvh * G + row % G) * D;
#pragma unroll
        for (int i = 0; i < D / 64; ++i)
            *reinterpret_cast<float4*>(o + tx * 4 + 64 * i) =
                make_float4(acc[r][4 * i] * inv, acc[r][4 * i + 1] * inv, acc[r][4 * i + 2] * inv, acc[r][4 * i + 3] * inv);
    }
}

template <int D, int PR_ROWS>
int launch_portions(const AfArgs& a, int tiles, int tile_rows, cudaStream_t stream) {
    const cudaError_t set = ti_allow_shared<portion_f32_kernel<D, PR_ROWS>>(portion_smem<D, PR_ROWS>());
    TI_REQUIRE(set == cudaSuccess, "attention_f32: %s", cudaGetErrorString(set));
    const int per = PR_ROWS / (a.hq / a.hkv);
    ti_launch(portion_f32_kernel<D, PR_ROWS>, dim3(a.hkv, (tile_rows + per - 1) / per, tiles), PR_ROWS * 8, portion_smem<D, PR_ROWS>(), stream, a);
    return 0;
}
template <int D>
void launch_decode(const AfArgs& a, int rows, cudaStream_t stream) {
    const int G = a.hq / a.hkv, gt = G == 1 ? 1 : G == 2 ? 2 : 4;
    const dim3 grid(DEC_CTAS, a.hkv * ((G + gt - 1) / gt), rows);
    if (gt == 1) ti_launch(decode_f32_kernel<D, 1>, grid, DEC_WARPS * 32, 0, stream, a);
    else if (gt == 2) ti_launch(decode_f32_kernel<D, 2>, grid, DEC_WARPS * 32, 0, stream, a);
    else ti_launch(decode_f32_kernel<D, 4>, grid, DEC_WARPS * 32, 0, stream, a);
}

}  // namespace

// float32 q [T, hq, d], cache [2, pages, hkv, page, d], d 64 or 128, at most 32 query heads a kv head, everything on 16-byte
// boundaries. ``decode_rows`` [num_decode]: flat rows of single tokens; ``tiles`` [num_tiles, 4]: portions of at most
// ``tile_rows`` consecutive tokens of one request: its row of the block table, first flat row, rows, first position.
TI_API int ti_attention_f32(float* out, const float* q, const float* kv_cache, const int* positions, const int* token_seq,
                            const int* decode_rows, int num_decode, const int* tiles, int num_tiles, int tile_rows,
                            const int* block_table, int max_blocks, int hq, int hkv, int d, int page_size, int num_pages,
                            float scale, int window, int* status, cudaStream_t stream) {
    TI_REQUIRE(d == 64 || d == 128, "attention_f32: head_dim %d is neither 64 nor 128", d);
    TI_REQUIRE(hq > 0 && hkv > 0 && hq % hkv == 0 && hq / hkv <= PR_MAX_ROWS, "attention_f32: %d query heads over %d kv heads", hq, hkv);
    TI_REQUIRE(page_size > 0 && num_decode >= 0 && num_tiles >= 0 && tile_rows > 0 && num_decode <= 65535 && num_tiles <= 65535 &&
                   tile_rows <= 65535, "attention_f32: bad sizes");
    TI_REQUIRE(((uintptr_t)out | (uintptr_t)q | (uintptr_t)kv_cache) % 16 == 0, "attention_f32: operands must lie on 16-byte boundaries");
    AfArgs a{out, q, kv_cache, kv_cache + (size_t)num_pages * hkv * page_size * d, positions, token_seq, block_table, nullptr,
             max_blocks, hq, hkv, page_size, num_pages, window, scale, status};
    if (num_decode) {
        a.rows = decode_rows;
        if (d == 128) launch_decode<128>(a, num_decode, stream);
        else launch_decode<64>(a, num_decode, stream);
        TI_CHECK_LAUNCH("attention_f32 decode");
    }
    if (num_tiles) {
        a.rows = tiles;
        // 16 rows a block until blocks of 32 would fill the machine four times over: 333 tokens make 168 of those, and the step
        // waits for the one with the most keys
        const int G = hq / hkv;
        const bool small = G <= 16 && (long long)num_tiles * tile_rows * G / 32 * hkv < 4 * 148;
        const int rc = d == 128 ? (small ? launch_portions<128, 16>(a, num_tiles, tile_rows, stream) : launch_portions<128, 32>(a, num_tiles, tile_rows, stream))
                                : (small ? launch_portions<64, 16>(a, num_tiles, tile_rows, stream) : launch_portions<64, 32>(a, num_tiles, tile_rows, stream));
        if (rc) return rc;
        TI_CHECK_LAUNCH("attention_f32 portions");
    }
    return 0;
}
