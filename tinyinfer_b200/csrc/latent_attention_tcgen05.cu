// The attention over a cached latent (see latent_attention.cu for the mechanism) for prompt portions on the tcgen05 tensor
// cores, bfloat16. The 128 accumulator lanes are (token, head) rows (8 tokens of 16 heads): every head reads the same cached
// rows [c | k_rot], so one tile of cached rows serves as keys (all features) and as values (the first `rank`).
//
//   warp 0      TMA: tiles of 32 cached rows through the block table, 64 features a copy, into a ring of four
//   warp 1      issues S = Q K^T (128 x 32, two buffers in tensor memory) and O += P V, P from tensor memory, V the
//               first features of the same shared-memory tile read as an MN-major operand
//   warps 2..9  the rows, brought as bfloat16 by TMA, their last features into tensor memory; then the softmax: two threads a row, each
//               16 of a tile's keys and half of O's columns. O stays in tensor memory and is multiplied there when a row of the warp has
//               a new maximum. (Rows of float32, which a caller with rows of its own may have, these warps fetch and round; the model's
//               kernels leave bfloat16.)
//
// The rows' last features, up to 320 of them, are read by the MMAs from tensor memory: with all 576 in shared memory it would hold a
// ring of two tiles alone, each refilled only when its products with P are through. 2,048 tokens over 16 heads of rank 512, a
// layer: 420 us with a ring of two, 354 with four, 285 with the MMAs issued from uniform registers as well (see elect_one), 218 with
// rows that the kernels before leave as bfloat16: TMA brings these, where 110 us were the CTAs' beginnings, rounding rows of float32.
// What is left is the softmax's chain of a tile.
// O of 512 value features would fill tensor memory and leave no room for scores: above 256 a row tile goes to two CTAs, which
// both make the scores and take half of the value features each.
// The products, their operands' roundings and the softmax's steps of 32 keys are those of the warp-level form
// (latent_attention_mma.cu), which stays for decoded tokens, windows and sizes not taken here: a probability is rounded against the
// running maximum after its own 32 keys. So the two forms differ by the order of float32 sums alone; larger tiles would round
// every probability anew, and a model with routers turns that into other choices of experts near a tie.
#include "sm100_ptx.cuh"
#include <algorithm>

namespace lt {
constexpr int QM = 128, KT = 32, STAGES = 4, THREADS = 320, SOFTMAX_THREADS = 256;
constexpr int S_COL = 256, P_COL = S_COL + 2 * KT, Q_COL = P_COL + KT, TMEM_COLS = 512;
constexpr int MAX_TMEM_CHUNKS = (TMEM_COLS - Q_COL) / 32;             // 64 features: 32 columns

struct Args {
    __nv_bfloat16* out;
    float* parts;
    const float* q;                                               // null: the rows come as bfloat16, by TMA
    const __nv_bfloat16* cache;
    const float* sink;
    const int *positions, *cu_seqlens, *block_table;
    int max_blocks, num_seqs, heads, rank, rot, page_size, num_pages, piece_rows;
    float scale;
    int splits, tpb, hpb, chunks, value_halves;
    int smem_chunks;                                              // of the rows' features in shared memory, the others in tensor memory
    int *status, *page_status;                                    // a wait that ran out, a key without a page; either may be null
};

__device__ __forceinline__ void tmem_st32(uint32_t taddr, const float* v) {
    const uint32_t* r = reinterpret_cast<const uint32_t*>(v);
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
          "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
          "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}
// 8 bfloat16 without those that are infinite or NaN; says whether there were any.
__device__ __forceinline__ bool drop_odd(uint4& u) {
    uint32_t* w = &u.x;
    bool odd = false;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const bool lo = (w[i] & 0x7f80u) == 0x7f80u, hi = (w[i] & 0x7f800000u) == 0x7f800000u;
        w[i] &= (lo ? 0xffff0000u : ~0u) & (hi ? 0xffffu : ~0u);
        odd |= lo || hi;
    }
    return odd;
}
// Which of 32 value features, the first of them at `values` of a row of dk, are infinite or NaN in any of the keys key0 .. key1 - 1 of the
// request whose pages `table` holds.
__device__ __noinline__ uint32_t odd_features(const __nv_bfloat16* values, int dk, const int* table, int max_blocks, int page_size, int num_pages,
                                              int key0, int key1) {
    uint32_t odd = 0;
    for (int key = key0; key < key1; ++key) {
        const int logical = key / page_size, page = logical < max_blocks ? table[logical] : -1;
        if (page < 0 || page >= num_pages) continue;
        const uint32_t* row = reinterpret_cast<const uint32_t*>(values + ((size_t)page * page_size + key % page_size) * dk);
        for (int i = 0; i < 16; ++i)
            odd |= ((row[i] & 0x7f80u) == 0x7f80u ? 1u : 0u) << (2 * i) | ((row[i] & 0x7f800000u) == 0x7f800000u ? 2u : 0u) << (2 * i);
    }
    return odd;
}
// The rows' chunks on their way to tensor memory wait in the ring behind its first tile.
int tmem_chunks(int chunks) { return std::min(MAX_TMEM_CHUNKS, (STAGES - 1) * chunks * KT / QM); }
int smem_bytes(int chunks) {                                          // small ranks use less than all of tensor memory asks for
    return std::max(TMEM_SHARED_ALONE, 1024 + (chunks - tmem_chunks(chunks)) * (QM * 128) + STAGES * chunks * (KT * 128) + 128);
}
static_assert(tmem_shares_sm(TMEM_COLS, TMEM_SHARED_ALONE), "smem_bytes");

// NV: value features of a CTA.
template <int NV>
__global__ void __launch_bounds__(THREADS, 1) latent_attend_tc_kernel(const __grid_constant__ CUtensorMap map, const __grid_constant__ CUtensorMap map_q, const Args a) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* q_tile = smem;                                       // [chunk of 64 features][row][128 bytes, swizzled]
    uint8_t* ring = smem + a.smem_chunks * (QM * 128);            // [stage][chunk][key][128 bytes, swizzled]
    const int stage_bytes = a.chunks * (KT * 128);
    const uint32_t bar0 = smem_u32(ring + STAGES * stage_bytes);
    const uint32_t q_full = bar0, p_full = bar0 + 8u, o_full = bar0 + 16u;
    auto s_full = [&](int b) { return bar0 + 8u * (3 + b); };
    auto s_empty = [&](int b) { return bar0 + 8u * (5 + b); };
    const uint32_t q_landed = bar0 + 8u * (7 + 2 * STAGES);
    auto kv_full = [&](int s) { return bar0 + 8u * (7 + s); };
    auto kv_empty = [&](int s) { return bar0 + 8u * (7 + STAGES + s); };
    __shared__ uint32_t tmem_base_sh;
    __shared__ float sum_xch[2][QM];
    __shared__ int abort_sh, odd_sh, tile_sh[3];
    volatile int* abort_flag = &abort_sh;

    ti_grid_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        abort_sh = odd_sh = 0;
        mbar_init(q_full, 8);
        mbar_init(q_landed, 1);
        for (int s = 0; s < STAGES; ++s) { mbar_init(kv_full(s), 1); mbar_init(kv_empty(s), 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(s_full(b), 1); mbar_init(s_empty(b), 8); }
        mbar_init(p_full, 8);
        mbar_init(o_full, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tmem_alloc(&tmem_base_sh, TMEM_COLS);
    ti_grid_wait();
    // the tokens of this CTA: row tiles are dealt request by request, the last to the first CTAs (a prompt's longest key ranges; decoded
    // tokens, which a step has before its portions and whose ranges may be longer still, start last, and have a form of their own then)
    const int place = (int)gridDim.x - 1 - (int)blockIdx.x;
    if (threadIdx.x == 64) {
        const int tile = place / a.value_halves;
        int at = 0, seq = -1, first = 0, n = 0;
        const int base = a.cu_seqlens[0];                          // requests before these may lie ahead of the rows
        for (int s = 0; s < a.num_seqs; ++s) {
            const int r0 = a.cu_seqlens[s] - base, len = a.cu_seqlens[s + 1] - base - r0, nb = (len + a.tpb - 1) / a.tpb;
            if (tile < at + nb) {
                seq = s;
                first = r0 + (tile - at) * a.tpb;
                n = min(a.tpb, r0 + len - first);
                break;
            }
            at += nb;
        }
        tile_sh[0] = seq; tile_sh[1] = first; tile_sh[2] = n;
    }
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    const uint32_t tmem_base = tmem_base_sh;
    const int seq = tile_sh[0], tok0 = tile_sh[1], ntok = tile_sh[2];
    const int vhalf = place % a.value_halves;
    const int dk = a.rank + a.rot, h0 = blockIdx.y * a.hpb;
    int first_key = 0, last_key = 0, common = 0;                  // keys below `common` are seen by every row
    if (seq >= 0) {
        common = a.positions[tok0] + 1;
        last_key = a.positions[tok0 + ntok - 1] + 1;
        if (a.splits > 1) {
            const int per = ((last_key + a.splits - 1) / a.splits + KT - 1) / KT * KT;
            first_key = blockIdx.z * per;
            last_key = min(last_key, first_key + per);
        }
    }
    const int num_tiles = max(0, (last_key - first_key + KT - 1) / KT);
    // of the softmax warps: the row, which half of a tile's keys and of O's columns, the row's maximum and the half's sum
    const int lane_group = warp & 3, half = warp >= 6 ? 1 : 0, r = lane_group * 32 + lane;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(lane_group * 32) << 16);
    const int tl = r / a.hpb, head = h0 + r % a.hpb;
    const bool live = warp >= 2 && tl < ntok && head < a.heads;
    const int pos = live ? a.positions[tok0 + tl] : -1;
    constexpr int KH = KT / 2, VH = NV / 2;
    float m_run = -INFINITY, l_run = 0.f;
    bool ok = warp >= 2 && seq >= 0;

    if (seq < 0) {
        // more CTAs than row tiles
    } else if (warp == 0) {
        // ------------------------------------------------------------ TMA producer: a lane a copy
        const int* table = a.block_table + (size_t)seq * a.max_blocks;
        const int pieces = KT / a.piece_rows, copies = pieces * a.chunks;
        if (a.q == nullptr) {                                      // rows of (token, head) lie one behind the other
            if (lane == 0) mbar_expect_tx(q_landed, (uint32_t)a.chunks * (QM * 128));
            __syncwarp();
            if (lane < a.chunks) {
                const int behind = lane - a.smem_chunks;
                uint8_t* dst = behind < 0 ? q_tile + lane * (QM * 128) : ring + stage_bytes + behind * (QM * 128);
                tma_load_2d(smem_u32(dst), &map_q, q_landed, lane * 64, tok0 * a.heads + h0);
            }
        }
        for (int j = 0; j < num_tiles; ++j) {
            const int s = j % STAGES;
            int go = 1;
            if (lane == 0) {
                go = mbar_wait(kv_empty(s), ((j / STAGES) & 1u) ^ 1u, abort_flag, a.status, 71) ? 1 : 0;
                if (j == 1 && go) go = mbar_wait(q_full, 0, abort_flag, a.status, 72) ? 1 : 0;      // the rows' chunks have left the ring
                if (go) mbar_expect_tx(kv_full(s), (uint32_t)stage_bytes);
            }
            if (!__shfl_sync(0xffffffffu, go, 0)) break;
            for (int c = lane; c < copies; c += 32) {
                const int piece = c % pieces, chunk = c / pieces, key = first_key + j * KT + piece * a.piece_rows;
                const int logical = key / a.page_size;
                const int page = logical < a.max_blocks ? table[logical] : -1;
                int row = a.num_pages * a.page_size;               // outside the map: zeros
                if (page >= 0 && page < a.num_pages) row = page * a.page_size + key % a.page_size;
                else if (key < last_key && a.page_status) atomicExch(a.page_status, 2);     // a visible key without a page
                tma_load_2d(smem_u32(ring + s * stage_bytes + chunk * (KT * 128) + piece * a.piece_rows * 128), &map, kv_full(s), chunk * 64, row);
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer
        if (num_tiles > 0) {
            const bool leader = elect_one();
            constexpr uint32_t idesc_s = make_idesc(QM, KT), idesc_o = make_idesc(QM, NV, true);
            const uint64_t q_desc = make_sw128_desc(smem_u32(q_tile));
            const uint64_t k_desc = make_sw128_desc(smem_u32(ring));
            const uint64_t v_desc = make_sw128_desc_mn(smem_u32(ring) + vhalf * (NV / 64) * (KT * 128), KT * 128, 1024);
            bool go = mbar_wait_warp(q_full, 0, abort_flag, a.status, 72);
            tmem_fence_after();
            auto issue_s = [&](int j) {                            // scores of tile j into buffer j % 2
                const int s = j % STAGES, b = j & 1;
                if (!mbar_wait_warp(kv_full(s), (j / STAGES) & 1u, abort_flag, a.status, 73)) return false;
                if (!mbar_wait_warp(s_empty(b), ((j >> 1) & 1u) ^ 1u, abort_flag, a.status, 74)) return false;
                tmem_fence_after();
                const uint64_t kd = k_desc + (uint64_t)((s * stage_bytes) >> 4);
                const uint32_t d = tmem_base + S_COL + b * KT;
                uint64_t qd = q_desc, kk = kd;
                for (int c = 0; c < a.smem_chunks; ++c, qd += (QM * 128) >> 4, kk += (KT * 128) >> 4)
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (leader) umma_bf16(d, qd + 2 * k, kk + 2 * k, idesc_s, (c > 0 || k > 0) ? 1u : 0u);
                uint32_t qt = tmem_base + Q_COL;
                for (int c = a.smem_chunks; c < a.chunks; ++c, qt += 32, kk += (KT * 128) >> 4)
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (leader) umma_bf16_ts(d, qt + 8 * k, kk + 2 * k, idesc_s, (c > 0 || k > 0) ? 1u : 0u);
                if (leader) umma_commit(s_full(b));
                return true;
            };
            if (go) go = issue_s(0);
            for (int j = 0; j < num_tiles && go; ++j) {
                if (j + 1 < num_tiles) go = issue_s(j + 1);
                if (!go || !mbar_wait_warp(p_full, j & 1u, abort_flag, a.status, 75)) break;
                tmem_fence_after();
                const uint64_t vd = v_desc + (uint64_t)(((j % STAGES) * stage_bytes) >> 4);
#pragma unroll
                for (int ks = 0; ks < KT / 16; ++ks)
                    if (leader) umma_bf16_ts(tmem_base, tmem_base + P_COL + ks * 8, vd + (uint64_t)(ks * 128), idesc_o, (j > 0 || ks > 0) ? 1u : 0u);
                if (leader) { umma_commit(o_full); umma_commit(kv_empty(j % STAGES)); }
            }
        }
    } else {
        // ------------------------------------------------------------ rows and softmax (warps 2..9)
        const int etid = threadIdx.x - 64;
        if (a.q == nullptr) {
            ok = mbar_wait_warp(q_landed, 0, abort_flag, a.status, 79);
        } else {
            const int chunks8 = a.chunks * 8, total = QM * chunks8;
#pragma unroll 12
            for (int i = etid; i < total; i += 256) {              // 8 features: two 16-byte loads, one store
                const int row = i / chunks8, c = i % chunks8, rt = row / a.hpb, hl = row % a.hpb;
                uint4 w = make_uint4(0, 0, 0, 0);
                if (rt < ntok && h0 + hl < a.heads && c * 8 < dk) {
                    const float4* src = reinterpret_cast<const float4*>(a.q + ((size_t)(tok0 + rt) * a.heads + h0 + hl) * dk + c * 8);
                    const float4 u = src[0], v = src[1];
                    w = make_uint4(pack2(u.x, u.y), pack2(u.z, u.w), pack2(v.x, v.y), pack2(v.z, v.w));
                }
                const int chunk = c >> 3, behind = chunk - a.smem_chunks;
                uint8_t* dst = behind < 0 ? q_tile + chunk * (QM * 128) : ring + stage_bytes + behind * (QM * 128);
                *reinterpret_cast<uint4*>(dst + row * 128 + (((c & 7) ^ (row & 7)) << 4)) = w;
            }
            asm volatile("bar.sync 1, %0;" ::"n"(SOFTMAX_THREADS) : "memory");
        }
        if (ok) {
            for (int t = 0; t < a.chunks - a.smem_chunks; ++t) {   // a thread's half of its row's chunk: 32 features, 16 columns
                const uint8_t* src = ring + stage_bytes + t * (QM * 128) + r * 128;
#pragma unroll
                for (int i = 0; i < 4; i += 2) {
                    const uint4 u = *reinterpret_cast<const uint4*>(src + (((half * 4 + i) ^ (r & 7)) << 4));
                    const uint4 w = *reinterpret_cast<const uint4*>(src + (((half * 4 + i + 1) ^ (r & 7)) << 4));
                    const uint32_t words[8] = {u.x, u.y, u.z, u.w, w.x, w.y, w.z, w.w};
                    tmem_st8(lane_addr + Q_COL + t * 32 + half * 16 + i * 4, words);
                }
            }
            tmem_wait_st();
            tmem_fence_before();
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(q_full);
        }
        for (int j = 0; j < num_tiles && ok; ++j) {
            const int b = j & 1, key0 = first_key + j * KT;
            // a warp's threads stay together: tensor memory is read and written by whole warps
            ok = __all_sync(0xffffffffu, mbar_wait(s_full(b), (j >> 1) & 1u, abort_flag, a.status, 76));
            if (!ok) break;
            tmem_fence_after();
            float v[KT], e[KH];
            tmem_ld32(lane_addr + S_COL + b * KT, v);
            tmem_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(s_empty(b));
            const int seen = min(pos + 1, last_key) - key0;
            float mx = -INFINITY;                                  // of the whole row: nothing to exchange with its other thread
#pragma unroll
            for (int i = 0; i < KT; ++i) {
                v[i] = i < seen ? v[i] * a.scale : -INFINITY;
                mx = fmaxf(mx, v[i]);
            }
            const float m_new = fmaxf(m_run, mx);
            const float corr = m_run == -INFINITY ? 1.f : expf(m_run - m_new);   // nothing summed yet: O's row is zero
            float sum = 0.f;
#pragma unroll
            for (int i = 0; i < KH; ++i) {
                e[i] = m_new == -INFINITY ? 0.f : expf((half ? v[KH + i] : v[i]) - m_new);
                sum += e[i];
            }
            l_run = l_run * corr + sum;
            m_run = m_new;
            uint32_t pk[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) pk[i] = pack2(e[2 * i], e[2 * i + 1]);
            if (j > 0) {                                           // O and P are free when the product before has ended
                ok = __all_sync(0xffffffffu, mbar_wait(o_full, (j - 1) & 1u, abort_flag, a.status, 77));
                if (!ok) break;
                tmem_fence_after();
                if (__any_sync(0xffffffffu, corr != 1.f)) {
#pragma unroll
                    for (int c = 0; c < VH; c += 32) {
                        float o[32];
                        tmem_ld32(lane_addr + half * VH + c, o);
#pragma unroll
                        for (int i = 0; i < 32; ++i) o[i] *= corr;
                        tmem_st32(lane_addr + half * VH + c, o);
                    }
                }
            }
            tmem_st8(lane_addr + P_COL + half * 8, pk);
            // Values that not every row sees must not meet a probability of zero: those past the last key, whatever the page holds
            // there, become zero, and so do infinities and NaN among those that only some rows see. These rows get them at the end.
            if (key0 + KT > common) {
                uint8_t* v_tile = ring + (j % STAGES) * stage_bytes + vhalf * (NV / 64) * (KT * 128);
                for (int i = etid; i < KT * (NV / 8); i += 256) {
                    const int row = i / (NV / 8), c = i % (NV / 8);
                    if (row < common - key0) continue;
                    uint4* at = reinterpret_cast<uint4*>(v_tile + (c >> 3) * (KT * 128) + row * 128 + (((c & 7) ^ (row & 7)) << 4));
                    if (row >= last_key - key0) {
                        *at = make_uint4(0, 0, 0, 0);
                    } else {
                        uint4 u = *at;
                        if (drop_odd(u)) { *at = u; odd_sh = 1; }
                    }
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            }
            tmem_wait_st();
            tmem_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(p_full);
        }
        if (ok && num_tiles > 0) ok = __all_sync(0xffffffffu, mbar_wait(o_full, (num_tiles - 1) & 1u, abort_flag, a.status, 78));
        sum_xch[half][r] = l_run;
    }
    __syncthreads();                                               // every role has ended, well or not
    if (ok) {                                                      // the same for a whole warp
        tmem_fence_after();
        float l = l_run + sum_xch[half ^ 1][r], c = 1.f;
        const size_t at = live ? (size_t)(tok0 + tl) * a.heads + head : 0;
        float* part = a.splits > 1 ? a.parts + (at * a.splits + blockIdx.z) * (a.rank + 2) : nullptr;
        if (part && live && half == 0 && vhalf == 0) { part[0] = m_run; part[1] = l; }
        if (!part && a.sink != nullptr && live) {
            const float sk = a.sink[head], m_new = fmaxf(m_run, sk);
            c = m_run == -INFINITY ? 0.f : expf(m_run - m_new);
            l = l * c + expf(sk - m_new);
        }
        const float inv = l > 0.f ? c / l : 0.f;
        const int col0 = vhalf * NV + half * VH;
#pragma unroll
        for (int cc = 0; cc < VH; cc += 32) {
            float o[32];
            if (num_tiles > 0) {
                tmem_ld32(lane_addr + half * VH + cc, o);
            } else {
#pragma unroll
                for (int i = 0; i < 32; ++i) o[i] = 0.f;
            }
            if (odd_sh && live) {
                // a seen value of infinity makes its sum NaN whatever its probability: its key's score is infinite or NaN, so that
                // is 0 or NaN
                const uint32_t odd = odd_features(a.cache + col0 + cc, dk, a.block_table + (size_t)seq * a.max_blocks, a.max_blocks, a.page_size,
                                                  a.num_pages, max(first_key, common), min(pos + 1, last_key));
#pragma unroll
                for (int i = 0; i < 32; ++i) if (odd >> i & 1u) o[i] = NAN;
            }
            if (a.splits > 1) {
                // Through shared memory, so that a row of a part is stored by the whole warp: four bytes a lane into 32 rows made 8 tokens
                // behind 4,096 take 59 us, longer than at warp level (51); now 35.
                float* turn = reinterpret_cast<float*>(smem) + (warp - 2) * (32 * 33);
#pragma unroll
                for (int i = 0; i < 32; ++i) turn[lane * 33 + i] = o[i];
                __syncwarp();
                const uint32_t lives = __ballot_sync(0xffffffffu, live);
#pragma unroll 4
                for (int row = 0; row < 32; ++row) {
                    float* to = reinterpret_cast<float*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(part), row));
                    if (lives >> row & 1u) to[2 + col0 + cc + lane] = turn[row * 33 + lane];
                }
            } else if (live) {
                uint4* dst = reinterpret_cast<uint4*>(a.out + at * a.rank + col0 + cc);
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    dst[i] = make_uint4(pack2(o[8 * i] * inv, o[8 * i + 1] * inv), pack2(o[8 * i + 2] * inv, o[8 * i + 3] * inv),
                                        pack2(o[8 * i + 4] * inv, o[8 * i + 5] * inv), pack2(o[8 * i + 6] * inv, o[8 * i + 7] * inv));
            }
            __syncwarp();
        }
    }
    tmem_fence_before();
    __syncthreads();
    if (warp == 1) {
        tmem_fence_after();
        land_copies(abort_flag);
        tmem_dealloc(tmem_base, TMEM_COLS);
    }
}

template <int NV> static cudaError_t launch(const CUtensorMap& map, const CUtensorMap& map_q, const Args& a, dim3 grid, int smem, cudaStream_t stream) {
    const cudaError_t e = ti_allow_shared<latent_attend_tc_kernel<NV>>(smem);
    return e != cudaSuccess ? e : ti_launch(latent_attend_tc_kernel<NV>, grid, THREADS, smem, stream, map, map_q, a);
}
}  // namespace lt

// CTAs that this form needs for a step, or 0 if it does not take the sizes: value features in whole swizzled chunks of 64,
// rows that TMA can copy and shared memory holds, pages of a multiple of 16 keys.
TI_API int ti_latent_attend_tc_ctas(int num_tokens, int num_seqs, int heads, int rank, int rot, int page_size) {
    const bool taken = rot >= 0 && (rank + rot) % 8 == 0 && rank + rot <= 576 && page_size % 16 == 0 &&
                       (rank == 64 || rank == 128 || rank == 256 || rank == 512);
    if (!taken || heads <= 0) return 0;
    const int hpb = heads < lt::QM ? heads : lt::QM, tpb = lt::QM / hpb;
    return ((num_tokens + tpb - 1) / tpb + num_seqs - 1) * ((heads + hpb - 1) / hpb) * (rank > 256 ? 2 : 1);
}

// Every token's keys 0 .. its position (no window). cu_seqlens counts from its first entry on. q [T, heads, rank + rot] float32 or, q_bf16, bfloat16; out bfloat16 [T, heads, rank]; splits > 1:
// the keys are shared out over grid z and the parts are left for ti_latent_merge. status (may be null): set if a wait runs out; page_status (may be null): if a visible key has no page.
TI_API int ti_latent_attend_tc(void* out, float* parts, long long parts_floats, const void* q, int q_bf16, const void* cache, const float* sink,
                               const int* positions, const int* cu_seqlens, const int* block_table, int max_blocks, int num_seqs,
                               int num_tokens, int heads, int rank, int rot, int page_size, int num_pages, float scale, int splits,
                               int* status, int* page_status, cudaStream_t stream) {
    TI_REQUIRE(num_tokens >= 0 && num_seqs > 0 && num_pages > 0, "latent_attend_tc: bad sizes");
    if (num_tokens == 0) return 0;
    const int ctas = ti_latent_attend_tc_ctas(num_tokens, num_seqs, heads, rank, rot, page_size);
    TI_REQUIRE(ctas > 0, "latent_attend_tc: %d heads, rows of %d + %d features, pages of %d are not taken", heads, rank, rot, page_size);
    TI_REQUIRE((((uintptr_t)cache | (uintptr_t)q | (uintptr_t)out) & 15) == 0, "latent_attend_tc: operands start on 16-byte boundaries");
    TI_REQUIRE(splits >= 1 && splits <= 65535, "latent_attend_tc: bad number of splits");
    TI_REQUIRE(splits == 1 || (parts != nullptr && parts_floats >= (long long)num_tokens * heads * splits * (rank + 2)),
               "latent_attend_tc: scratch too small for %d splits", splits);
    TI_REQUIRE((long long)num_pages * page_size < (1ll << 31) - 65536, "latent_attend_tc: too many cached rows");
    lt::Args a;
    a.out = (__nv_bfloat16*)out; a.parts = parts; a.q = q_bf16 ? nullptr : (const float*)q; a.cache = (const __nv_bfloat16*)cache; a.sink = sink; a.positions = positions; a.cu_seqlens = cu_seqlens;
    a.block_table = block_table; a.max_blocks = max_blocks; a.num_seqs = num_seqs; a.heads = heads; a.rank = rank; a.rot = rot;
    a.page_size = page_size; a.num_pages = num_pages; a.scale = scale; a.splits = splits; a.status = status; a.page_status = page_status;
    a.hpb = heads < lt::QM ? heads : lt::QM;
    a.tpb = lt::QM / a.hpb;
    a.chunks = (rank + rot + 63) / 64;
    a.smem_chunks = a.chunks - lt::tmem_chunks(a.chunks);
    a.value_halves = rank > 256 ? 2 : 1;
    a.piece_rows = page_size % 32 == 0 ? 32 : 16;
    TI_REQUIRE((long long)num_tokens * heads < (1ll << 31) - 65536, "latent_attend_tc: too many query rows");
    CUtensorMap map, map_q;
    if (!ti_get_bf16_map(cache, (long long)num_pages * page_size, rank + rot, a.piece_rows, &map)) return -1;
    map_q = map;
    if (q_bf16 && !ti_get_bf16_map(q, (long long)num_tokens * heads, rank + rot, lt::QM, &map_q)) return -1;
    const int groups = (heads + a.hpb - 1) / a.hpb, smem = lt::smem_bytes(a.chunks);
    TI_REQUIRE(groups <= 65535, "latent_attend_tc: too many heads");
    const dim3 grid(ctas / groups, groups, splits);
    const int nv = rank / a.value_halves;
    const cudaError_t e = nv == 64 ? lt::launch<64>(map, map_q, a, grid, smem, stream) : nv == 128 ? lt::launch<128>(map, map_q, a, grid, smem, stream)
                                                                                         : lt::launch<256>(map, map_q, a, grid, smem, stream);
    TI_REQUIRE(e == cudaSuccess, "latent_attend_tc: %s", cudaGetErrorString(e));
    TI_CHECK_LAUNCH("latent_attend_tc");
    return 0;
}
