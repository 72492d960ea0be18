// The blocks of a dense pre-norm decoder (grouped-query attention, gated feed-forward) from ONE call: every launch of a step's
// layers is made here, through the launchers of the other libraries, on buffers that one workspace holds.
//
// Bound by the host in steps of some hundred tokens: a launch through Python cost 16 to 21 us (three output tensors,
// 20 arguments, checks), 172 of them a step of 37 tokens over 28 layers, whose kernels need 0.9 ms; from here it costs what
// the launch costs. The kernels and their operands are what the layers' parts would launch, in their order, and the outputs the
// same bit for bit; only the two attention kernels of a step that brings portions and decoded tokens run on two streams.
// 37 tokens, 28 layers of hidden size 1024: 3.66 -> 1.31 ms a step.
#include "common.cuh"
#include <algorithm>

struct TiStackLayer {
    const void* w_qkv; const float* b_qkv; const void* w_o; const float* b_o; const float *q_norm, *k_norm, *inv_freq, *cos_sin;
    const float *norm1, *norm2; const void *w_gate_up, *w_down; void* kv; const int* block_table;
    long long max_blocks, num_pages, window, writes;
};

typedef int (*RmsnormFn)(void*, const void*, const float*, const int*, int, int, float, int, cudaStream_t);
typedef int (*AppendFn)(void*, const void*, void*, const float*, const float*, float, const float*, const float*, int, int, int,
                        const int*, const int*, const int*, int, int, int, int, int, int, int, int*, int, cudaStream_t);
typedef int (*GemmFn)(void*, const void*, const void*, const float*, const void*, int, int, int, int, int, float*, long long, int*,
                      int, int*, cudaStream_t);
typedef int (*LinkedFn)(void*, const void*, const void*, const float*, const void*, int, int, int, int, float*, long long, int*, int,
                        const float*, int, int, float, const float*, void*, float*, int*, int*, cudaStream_t);
typedef int (*DecodeFn)(void*, const void*, const void*, float*, long long, const int*, int, const int*, const int*, const int*, int,
                        int, int, int, int, int, float, int, int, int*, cudaStream_t);
typedef int (*OneTileFn)(void*, const void*, const void*, const int*, int, int, const int*, int, int, int, int, int, int, float, int,
                         int, int, int, float*, long long, int*, cudaStream_t);
typedef int (*TwoTileFn)(void*, const void*, const void*, const int*, int, int, const int*, int, int, int, int, int, int, float, int,
                         int*, cudaStream_t);
typedef int (*SimtFn)(void*, const void*, const void*, const float*, const void*, int, int, int, int, int, int, cudaStream_t);
typedef int (*FewFn)(float*, const float*, const float*, const float*, const float*, int, int, int, int, int, cudaStream_t);
typedef int (*SplitFn)(float*, const float*, const float*, const float*, const float*, void*, int, int, int, int, int, int*, cudaStream_t);
typedef int (*Attention32Fn)(float*, const float*, const float*, const int*, const int*, const int*, int, const int*, int, int,
                             const int*, int, int, int, int, int, int, float, int, int*, cudaStream_t);

struct TiStackCall {
    RmsnormFn rmsnorm; AppendFn append; GemmFn gemm; LinkedFn linked; DecodeFn decode; OneTileFn one_tile; TwoTileFn two_tile;
    void (*plain_next)();                          // sm100's: the next launch waits for all that its stream waits for
    SimtFn simt; FewFn few; SplitFn split; Attention32Fn attention32;
    const TiStackLayer* layer;
    const void* x; void* out;                      // [T, hidden]: the embedding's output, the last block's
    void* workspace; long long workspace_bytes;
    const int *positions, *token_seq, *decode_rows, *tiles;
    float* gemm_ws; long long gemm_ws_floats; int* counters;
    float* attn_scratch; long long attn_floats, decode_floats;
    int *wait_status, *page_status;
    cudaStream_t stream, side;
    int layers, tokens, hidden, heads, kv_heads, head_dim, inter, act, page_size, dtype;
    int num_decode, num_tiles, num_pairs, max_context;
    int table_positions, interleaved, rotary_dim, num_counters;
    int link_max_tokens, pair_min_ctas, split_max_ctas, few_rows, min_k, split_min_k, tile_rows;
    float eps1, eps2, qk_eps, scale;
    int failed;                                    // out: which library's launcher failed (0 core, 1 sm100, 2 f32)
};

namespace {

struct Buffers {
    char *x1, *x2, *h, *qkv, *q, *att, *hid, *planes;
    float* sums;
    long long bytes;
};
Buffers lay_out(char* base, int tokens, int hidden, int q_size, int kv_size, int inter, int esize) {
    Buffers b;
    long long at = 0;
    auto take = [&](long long bytes) {
        char* p = base + at;
        at += (bytes + 255) / 256 * 256;
        return p;
    };
    const long long t = tokens;
    b.x1 = take(t * hidden * esize);
    b.x2 = take(t * hidden * esize);
    b.h = take(t * hidden * esize);
    b.qkv = take(t * (q_size + 2 * kv_size) * esize);
    b.q = take(t * q_size * esize);
    b.att = take(t * q_size * esize);
    b.hid = take(t * inter * esize);
    b.sums = reinterpret_cast<float*>(take(t * ((hidden + 127) / 128) * 4));
    const long long widest = std::max(std::max(hidden, q_size), inter);
    b.planes = esize == 4 ? take(6 * t * ((widest + 63) / 64 * 64)) : nullptr;
    b.bytes = at;
    return b;
}

// The two events of a call that runs on two streams. An event may be given up while work still waits for it.
struct Fork {
    bool on, open = false;
    cudaStream_t main, side;
    cudaEvent_t begin = nullptr, end = nullptr;
    Fork(bool wanted, cudaStream_t main, cudaStream_t side) : on(wanted), main(main), side(side) {
        if (on && (cudaEventCreateWithFlags(&begin, cudaEventDisableTiming) != cudaSuccess ||
                   cudaEventCreateWithFlags(&end, cudaEventDisableTiming) != cudaSuccess)) on = false;      // one stream, then
    }
    ~Fork() {
        if (open) {                                 // a launch was refused in between: nobody frees what the second stream uses
            cudaEventRecord(end, side);
            cudaStreamWaitEvent(main, end, 0);
        }
        if (begin) cudaEventDestroy(begin);
        if (end) cudaEventDestroy(end);
    }
};

// Floats of scratch that a one-tile attention launch over `count` tiles needs, and its split of the keys: with few query tiles
// behind a long prefix the keys are shared out over CTAs too (at least 1,024 to a CTA), so that most SMs have one.
long long one_tile_plan(const TiStackCall& c, int count, int halves, int& splits, int& split_keys) {
    const int ctas = count * (halves ? 2 : 1) * c.heads;
    splits = 1;
    if (ctas * 2 <= c.split_max_ctas && c.max_context >= 2048) splits = std::max(1, std::min(c.split_max_ctas / ctas, c.max_context / 1024));
    split_keys = splits > 1 ? ((c.max_context + splits - 1) / splits + 127) / 128 * 128 : 0;
    return splits > 1 ? (long long)count * (halves ? 2 : 1) * splits * c.heads * 128 * (c.head_dim + 2) : 0;
}

}  // namespace

TI_API long long ti_dense_stack_bytes(int tokens, int hidden, int q_size, int kv_size, int inter, int dtype) {
    return lay_out(nullptr, tokens, hidden, q_size, kv_size, inter, dtype == TI_F32 ? 4 : 2).bytes;
}

// Floats of attn_scratch that the prompt portions of the call need (the decoded tokens' are the decode kernel's to say).
TI_API long long ti_dense_stack_portion_floats(const TiStackCall* call) {
    const TiStackCall& c = *call;
    if (c.dtype == TI_F32) return 0;
    int s, k;
    long long need = 0;
    if (c.num_pairs && c.num_pairs * c.heads < c.pair_min_ctas) need = one_tile_plan(c, c.num_pairs, 1, s, k);
    if (c.num_tiles > c.num_pairs) need = std::max(need, one_tile_plan(c, c.num_tiles - c.num_pairs, 0, s, k));
    return need;
}

TI_API int ti_dense_stack(TiStackCall* call) {
    TiStackCall& c = *call;
    const int T = c.tokens, H = c.hidden, qs = c.heads * c.head_dim, kvs = c.kv_heads * c.head_dim;
    const bool f32 = c.dtype == TI_F32;
    TI_REQUIRE(T > 0 && c.layers > 0, "dense_stack: nothing to run");
    const Buffers b = lay_out((char*)c.workspace, T, H, qs, kvs, c.inter, f32 ? 4 : 2);
    TI_REQUIRE(c.workspace_bytes >= b.bytes, "dense_stack: a workspace of %lld bytes, %lld are needed", c.workspace_bytes, b.bytes);
    ti_set_error("%s", "");
    const bool links = !f32 && T <= c.link_max_tokens;
    int parts = 0;                                  // > 0: the product before left x * g in b.h and its sums of squares
#define STACK_RUN(lib, ...)                       \
    do {                                          \
        c.failed = lib;                           \
        const int rc__ = (__VA_ARGS__);           \
        if (rc__) return rc__;                    \
    } while (0)
    // out = x . w^T (+ bias) (+ residual) or the gated form; `scaled`: x is b.h of a norm shared with the product before;
    // `emit`: the weight of the norm that follows, which a product of few tokens can prepare
    auto product = [&](void* out, const void* x, const void* w, const float* bias, const void* residual, int n, int k, int gated,
                       bool scaled, float eps, const float* emit) -> int {
        if (f32) {
            const bool fits = k % 4 == 0 && k >= (T <= c.few_rows ? c.min_k : c.split_min_k) && ((uintptr_t)x | (uintptr_t)w) % 16 == 0;
            const int early = 1;                    // the weights are the model's: no kernel of a step writes them
            if (!fits) STACK_RUN(0, c.simt(out, x, w, bias, residual, T, n, k, gated, 0, c.dtype, c.stream));
            else if (T <= c.few_rows)
                STACK_RUN(2, c.few((float*)out, (const float*)x, (const float*)w, bias, (const float*)residual, T, n, k, gated, early, c.stream));
            else
                STACK_RUN(2, c.split((float*)out, (const float*)x, (const float*)w, bias, (const float*)residual, b.planes, T, n, k, gated,
                                     early, c.wait_status, c.stream));
            return 0;
        }
        if (scaled || emit) {
            int written = 0;
            STACK_RUN(1, c.linked(out, x, w, bias, residual, T, n, k, gated, c.gemm_ws, c.gemm_ws_floats, c.counters, c.num_counters,
                                  scaled ? b.sums : nullptr, scaled ? parts : 0, scaled ? k : 0, scaled ? eps : 0.f, emit,
                                  emit ? b.h : nullptr, emit ? b.sums : nullptr, &written, c.wait_status, c.stream));
            if (emit) parts = written;
            return 0;
        }
        STACK_RUN(1, c.gemm(out, x, w, bias, residual, T, n, k, gated, 0, c.gemm_ws, c.gemm_ws_floats, c.counters, c.num_counters,
                            c.wait_status, c.stream));
        return 0;
    };
#define STACK_PRODUCT(...)                        \
    do {                                          \
        const int rc__ = product(__VA_ARGS__);    \
        if (rc__) return rc__;                    \
    } while (0)
    Fork fork(!f32 && c.side != nullptr && c.num_decode > 0 && c.num_tiles > 0, c.stream, c.side);
    const void* x = c.x;
    for (int i = 0; i < c.layers; ++i) {
        const TiStackLayer& l = c.layer[i];
        const bool last = i + 1 == c.layers;
        const bool from_link = parts > 0;
        if (!from_link) STACK_RUN(0, c.rmsnorm(b.h, x, l.norm1, nullptr, T, H, c.eps1, c.dtype, c.stream));
        STACK_PRODUCT(b.qkv, b.h, l.w_qkv, l.b_qkv, nullptr, qs + 2 * kvs, H, 0, from_link, c.eps1, nullptr);
        STACK_RUN(0, c.append(b.q, b.qkv, l.writes ? l.kv : nullptr, l.q_norm, l.k_norm, c.qk_eps, l.inv_freq, l.cos_sin, c.table_positions,
                              c.interleaved, c.rotary_dim, c.positions, c.token_seq, l.block_table, (int)l.max_blocks, T, c.heads,
                              c.kv_heads, c.head_dim, l.writes ? c.page_size : 1, l.writes ? (int)l.num_pages : 1, c.page_status, c.dtype,
                              c.stream));
        const int mb = (int)l.max_blocks, pages = (int)l.num_pages, window = (int)l.window;
        if (f32) {
            STACK_RUN(2, c.attention32((float*)b.att, (const float*)b.q, (const float*)l.kv, c.positions, c.token_seq, c.decode_rows,
                                       c.num_decode, c.tiles, c.num_tiles, std::min(T, c.tile_rows), l.block_table, mb, c.heads, c.kv_heads,
                                       c.head_dim, c.page_size, pages, c.scale, window, c.page_status, c.stream));
        } else {
            // Portions beside decoded tokens: two sets of rows, two kernels that each leave half the machine idle. The decoded
            // tokens' runs on the second stream, on scratch of its own, and the output projection waits for both: a portion of 512
            // tokens beside 27 decoded ones over 28 layers, 4.67 -> 4.49 ms.
            if (fork.on) {
                TI_REQUIRE(cudaEventRecord(fork.begin, c.stream) == cudaSuccess && cudaStreamWaitEvent(c.side, fork.begin, 0) == cudaSuccess,
                           "dense_stack: the second stream cannot wait for the first");
                fork.open = true;
                c.plain_next();
            }
            if (c.num_decode)
                STACK_RUN(1, c.decode(b.att, b.q, l.kv, c.attn_scratch, c.decode_floats, c.decode_rows, c.num_decode, c.positions, c.token_seq,
                                      l.block_table, mb, c.heads, c.kv_heads, c.head_dim, c.page_size, pages, c.scale, window, c.max_context,
                                      c.wait_status, fork.on ? c.side : c.stream));
            if (fork.on) TI_REQUIRE(cudaEventRecord(fork.end, c.side) == cudaSuccess, "dense_stack: the second stream takes no event");
            float* portion_scratch = c.attn_scratch + (fork.on ? c.decode_floats : 0);
            const long long portion_floats = c.attn_floats - (fork.on ? c.decode_floats : 0);
            for (int kind = 0; kind < 2; ++kind) {  // tiles of more than 128 rows, then the ends of portions
                const int first = kind ? c.num_pairs : 0, count = kind ? c.num_tiles - c.num_pairs : c.num_pairs;
                if (!count) continue;
                if (!kind && count * c.heads >= c.pair_min_ctas) {
                    STACK_RUN(1, c.two_tile(b.att, b.q, l.kv, c.tiles, count, T, l.block_table, mb, c.heads, c.kv_heads, c.head_dim,
                                            c.page_size, pages, c.scale, window, c.wait_status, c.stream));
                    continue;
                }
                int splits, split_keys;
                const long long need = one_tile_plan(c, count, !kind, splits, split_keys);
                TI_REQUIRE(need <= portion_floats, "dense_stack: %lld floats of attention scratch, %lld are needed", portion_floats, need);
                STACK_RUN(1, c.one_tile(b.att, b.q, l.kv, c.tiles + 4 * first, count, T, l.block_table, mb, c.heads, c.kv_heads, c.head_dim,
                                        c.page_size, pages, c.scale, window, !kind, splits, split_keys, splits > 1 ? portion_scratch : nullptr,
                                        splits > 1 ? portion_floats : 0, c.wait_status, c.stream));
            }
            if (fork.on) {
                TI_REQUIRE(cudaStreamWaitEvent(c.stream, fork.end, 0) == cudaSuccess, "dense_stack: the first stream cannot wait for the second");
                fork.open = false;
                c.plain_next();
            }
        }
        void* out = last ? c.out : (void*)b.x2;
        parts = 0;
        STACK_PRODUCT(b.x1, b.att, l.w_o, l.b_o, x, H, qs, 0, false, 0.f, links ? l.norm2 : nullptr);
        const bool mlp_link = parts > 0;
        if (!mlp_link) STACK_RUN(0, c.rmsnorm(b.h, b.x1, l.norm2, nullptr, T, H, c.eps2, c.dtype, c.stream));
        STACK_PRODUCT(b.hid, b.h, l.w_gate_up, nullptr, nullptr, c.inter, H, c.act, mlp_link, c.eps2, nullptr);
        parts = 0;
        STACK_PRODUCT(out, b.hid, l.w_down, nullptr, b.x1, H, c.inter, 0, false, 0.f, links && !last ? c.layer[i + 1].norm1 : nullptr);
        x = out;
    }
#undef STACK_PRODUCT
#undef STACK_RUN
    return 0;
}
