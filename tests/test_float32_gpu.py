"""Kernels of the 32-bit path on the GPU against 64-bit references, with bounds that follow from the number of roundings."""
from types import SimpleNamespace

import pytest
import torch

from test_kernels_gpu import ops, fill_cache, paged_setup, rnd  # noqa: F401  (the fixture and the paged caches)

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -24


def dev():
    return torch.device("cuda:0")


def gated(z, act):
    g, u = z.chunk(2, dim=1)
    return (torch.nn.functional.silu(g) if act == "silu" else torch.nn.functional.gelu(g, approximate="tanh")) * u


def check_product(ops, m, n, k, roundings, seed=0):
    """Every form of the product: within ``roundings`` roundings of sum |x||w| of the 64-bit result, and a few more of the
    result itself for the epilogue."""
    x, w = rnd(m, k, dtype=torch.float32, seed=seed), rnd(n, k, dtype=torch.float32, seed=seed + 1)
    b, r = rnd(n, dtype=torch.float32, seed=seed + 2), rnd(m, n, dtype=torch.float32, seed=seed + 3)
    mass, z = x.double().abs() @ w.double().abs().T, x.double() @ w.double().T
    for got, want in ((ops.linear(x, w), z), (ops.linear(x, w, out_float32=True), z), (ops.linear(x, w, bias=b), z + b),
                      (ops.linear(x, w, bias=b, residual=r), z + b + r)):
        assert ((got - want).abs() <= EPS * (roundings * mass + 4 * (want.abs() + mass + 4))).all()
    if n % 2 == 0:
        for act in ("silu", "gelu_tanh"):
            got = ops.gated_linear(x, w, activation=act, bias=b)
            want = gated(z + b, act)
            g, u = (z + b).chunk(2, dim=1)
            mg, mu = (EPS * (roundings + 4) * (mass + b.abs())).chunk(2, dim=1)
            # |act'| <= 1.13; the activation itself is right to some 10 roundings
            assert ((got - want).abs() <= 1.13 * mg * (u.abs() + mu) + mu * g.abs() + 12 * EPS * (want.abs() + 1e-3)).all()


@pytest.mark.parametrize("m", [1, 2, 3, 4, 5, 8])
@pytest.mark.parametrize("n,k", [(2, 256), (7, 260), (130, 1020), (514, 2048), (96, 6148)])
def test_product_of_few_rows(ops, m, n, k):
    # a lane adds its products in runs of ceil(k / 1024) * 4, then come 5 + 8 sums
    check_product(ops, m, n, k, (k + 1023) // 1024 * 4 + 13)


def test_product_of_few_rows_does_not_depend_on_the_rows(ops):
    x, w = rnd(8, 2052, dtype=torch.float32, seed=1), rnd(77, 2052, dtype=torch.float32, seed=2)
    whole = ops.linear(x, w)
    for m in (1, 2, 3, 4, 6):
        assert torch.equal(ops.linear(x[:m].contiguous(), w), whole[:m])


@pytest.mark.parametrize("m,n,k", [(9, 2, 256), (16, 130, 260), (17, 514, 2048), (48, 96, 6148), (64, 4096, 1024), (127, 64, 320),
                                   (128, 1000, 2048), (129, 130, 516), (333, 2048, 6144), (300, 12000, 256), (1000, 388, 1100)])
def test_product_on_the_tensor_cores(ops, m, n, k):
    # what is cut off of 16 products at a time, in runs of 64 that are added up: fewer roundings than k / 16
    check_product(ops, m, n, k, k / 16 + 8)


@pytest.mark.parametrize("m", [1, 5, 8, 9, 200])
def test_product_by_what_the_kernel_before_makes(ops, m):
    """The second operand of a product may be the output of a kernel that has just been launched, in memory that held another."""
    x, a = rnd(m, 2048, dtype=torch.float32, seed=1), rnd(3000, 2048, dtype=torch.float32, seed=2)
    bs = [rnd(2048, 2048, dtype=torch.float32, seed=3 + i) for i in range(4)]
    for i in range(8):
        w = ops.linear(a, bs[i % 4])                          # long
        y = ops.linear(x, w)
        z = ops.gated_linear(x, w)
        torch.cuda.synchronize()
        assert torch.equal(ops.linear(x, w), y) and torch.equal(ops.gated_linear(x, w), z)
        del w


def test_split_products_back_to_back(ops):
    """Products that start while the one before still runs (their weights are on their way long before x is there)."""
    x, w = rnd(333, 6144, dtype=torch.float32, seed=1), rnd(2048, 6144, dtype=torch.float32, seed=2)
    outs = [ops.linear(x, w) for _ in range(12)]
    want = x.double() @ w.double().T
    assert ((outs[0] - want).norm() / want.norm()).item() < 1e-6
    assert all(torch.equal(o, outs[0]) for o in outs[1:])


def test_split_product_is_no_less_exact_than_multiply_adds(ops):
    """Sizes of the 1.7B model against 64 bits, beside the general kernel's sums in k order."""
    for m, n, k, std in ((333, 2048, 6144, 1.0), (37, 4096, 2048, 0.02), (200, 6144, 2048, 30.0)):
        x, w = rnd(m, k, dtype=torch.float32, seed=1), rnd(n, k, dtype=torch.float32, seed=2, std=std)
        want = x.double() @ w.double().T
        plain = torch.empty((m, n), dtype=torch.float32, device=dev())
        ops._run("core", "ti_gemm_simt", plain.data_ptr(), x.data_ptr(), w.data_ptr(), None, None, m, n, k, 0, 0, 0, ops._stream())
        errors = [((y - want).norm() / want.norm()).item() for y in (ops.linear(x, w), plain)]
        assert errors[0] <= errors[1], errors


@pytest.mark.parametrize("draw", ["normal", "positive"])
@pytest.mark.parametrize("m,n,k", [(1500, 4096, 256), (1500, 4096, 320), (200, 512, 320), (1500, 4096, 384), (40, 512, 512), (333, 1024, 1024)])
def test_product_of_a_short_row_is_no_less_exact_than_multiply_adds(ops, m, n, k, draw):
    """Where k is short the general kernel's sums are few, and the split products must not be further off."""
    x, w = rnd(m, k, dtype=torch.float32, seed=1), rnd(n, k, dtype=torch.float32, seed=2)
    if draw == "positive":
        x, w = x.abs(), w.abs()
    want = x.double() @ w.double().T
    plain = torch.empty((m, n), dtype=torch.float32, device=dev())
    ops._run("core", "ti_gemm_simt", plain.data_ptr(), x.data_ptr(), w.data_ptr(), None, None, m, n, k, 0, 0, 0, ops._stream())
    errors = [((y - want).norm() / want.norm()).item() for y in (ops.linear(x, w), plain)]
    assert errors[0] <= errors[1], errors


def test_split_product_takes_infinite_and_tiny_operands_as_multiply_adds_do(ops):
    m, n, k = 40, 200, 512
    x, w = rnd(m, k, dtype=torch.float32, seed=1), rnd(n, k, dtype=torch.float32, seed=2)
    x[3, 7], x[5, 9], w[11, 100], x[20], x[21] = float("inf"), float("nan"), -float("inf"), 0.0, 1e-30
    w[12] = 3.4e38                                     # rounds to infinity in bfloat16
    x[22] = 0.0
    x[22, 0] = 0.5
    want = (x.double() @ w.double().T)
    got = ops.linear(x, w)
    judged = torch.ones_like(want, dtype=torch.bool)
    judged[:, 12] = False                              # products that overflow on the way, in any order of the sums ...
    judged[20:23, 12] = True                           # ... but for these rows
    assert torch.equal(torch.isnan(got)[judged], torch.isnan(want)[judged])
    assert torch.equal(torch.isinf(got)[judged], torch.isinf(want)[judged])
    fine = judged & torch.isfinite(want)
    mass = x.double().abs() @ w.double().abs().T
    assert ((got - want).abs()[fine] <= EPS * (k / 16 + 8) * mass[fine]).all()


ATTENTION = [
    # hq, hkv, d, page, window, [(context, q_len)]
    (16, 8, 128, 64, None, [(333, 333), (1025, 1), (1, 1), (64, 1), (257, 1)]),
    (4, 4, 64, 16, None, [(130, 130), (129, 1), (200, 2), (2300, 1)]),
    (12, 4, 128, 48, 40, [(300, 44), (65, 1), (64, 1), (700, 301)]),
    (32, 1, 64, 64, -50, [(149, 99), (150, 1), (151, 1), (333, 17)]),
    (6, 1, 128, 5, None, [(91, 1), (64, 64), (65, 64)]),
    (16, 16, 64, 64, None, [(1300, 1300), (77, 70)]),             # enough rows for 32 a block
    (20, 4, 128, 64, None, [(700, 700), (1200, 513), (300, 300)]),
]


@pytest.mark.parametrize("hq,hkv,d,page,window,work", ATTENTION)
def test_attention(ops, hq, hkv, d, page, window, work):
    lens = [c for c, _ in work]
    bt, kv = paged_setup(torch.float32, lens, hq, hkv, d, page, seed=1)
    ks, vs = fill_cache(kv, bt, lens, hkv, d, page, torch.float32)
    q_lens, starts = [n for _, n in work], [c - n for c, n in work]
    rows, tiles, pairs = ops.plan_attention(q_lens, starts)
    step = SimpleNamespace(decode_rows=torch.tensor(rows or [0], dtype=torch.int32, device=dev()), num_decode=len(rows),
                           prefill_tiles=torch.tensor(tiles or [0], dtype=torch.int32, device=dev()),
                           num_prefill_tiles=len(tiles) // 4, num_pair_tiles=pairs, max_context=max(lens))
    pos = torch.tensor([p for c, n in work for p in range(c - n, c)], dtype=torch.int32, device=dev())
    seq = torch.tensor([i for i, (c, n) in enumerate(work) for _ in range(n)], dtype=torch.int32, device=dev())
    q = rnd(pos.shape[0], hq, d, dtype=torch.float32, seed=7)
    status = torch.zeros(1, dtype=torch.int32, device=dev())
    mask = dict(window=window) if (window or 0) >= 0 else dict(chunk=-window)
    out = ops.paged_attention(q, kv, positions=pos, token_seq=seq, block_table=bt, scale=d ** -0.5, step=step, status=status,
                              **mask)
    assert int(status.item()) == 0
    got, row = out.view(-1, hq, d).double(), 0
    for i, (c, n) in enumerate(work):
        k, v = (x[i].double().repeat_interleave(hq // hkv, dim=1) for x in (ks, vs))
        p, j = torch.arange(c - n, c, device=dev())[:, None], torch.arange(c, device=dev())[None]
        lo = torch.zeros_like(p) if not window else p - window + 1 if window > 0 else p - p % -window
        z = torch.einsum("nhd,lhd->hnl", q[row:row + n].double(), k) * d ** -0.5
        a = torch.softmax(z.masked_fill((j > p) | (j < lo), float("-inf")), dim=-1)
        want = torch.einsum("hnl,lhd->nhd", a, v)
        # a score is off by at most d roundings of sum |q||k| (some 0.7 d^1/2 here), a probability by that factor, and the
        # sums over the keys, of at most |v| = 5, by c / 8 roundings
        assert (got[row:row + n] - want).abs().max() <= EPS * 5 * (2 * d + c / 8 + 16)
        row += n


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_attention_multiplies_every_value_that_a_row_sees(ops, value):
    """A seen key whose probability underflows still brings 0 x its value, as in the general kernel: in a tile that all rows see
    whole, in one that some do not, and for single tokens."""
    hq, hkv, d, page = 4, 2, 64, 16
    work = [(200, 200), (170, 1)]
    bt, kv = paged_setup(torch.float32, [c for c, _ in work], hq, hkv, d, page, seed=1)
    fill_cache(kv, bt, [c for c, _ in work], hkv, d, page, torch.float32)
    rows, tiles, pairs = ops.plan_attention([n for _, n in work], [c - n for c, n in work])
    step = SimpleNamespace(decode_rows=torch.tensor(rows, dtype=torch.int32, device=dev()), num_decode=1,
                           prefill_tiles=torch.tensor(tiles, dtype=torch.int32, device=dev()), num_prefill_tiles=len(tiles) // 4,
                           num_pair_tiles=pairs, max_context=200)
    q = rnd(201, hq, d, dtype=torch.float32, seed=3).abs() + 0.1
    args = dict(positions=torch.tensor(list(range(200)) + [169], dtype=torch.int32, device=dev()),
                token_seq=torch.tensor([0] * 200 + [1], dtype=torch.int32, device=dev()), block_table=bt, scale=0.125)
    for request, key in ((0, 3), (0, 150), (1, 20)):
        at = (0, int(bt[request, key // page]), slice(None), key % page)
        kv[at] = -1e4                                   # a score far below every other
        kv[(1,) + at[1:]] = value
    got, want = ops.paged_attention(q, kv, step=step, **args), ops.paged_attention(q, kv, **args)
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.isnan(got[160]).all() and not torch.isnan(got[2]).any()


def test_attention_reports_a_key_without_a_page_and_keeps_rows_apart(ops):
    """A missing page is reported and its keys are left out; infinities of a later token of the portion do not reach the
    tokens before it."""
    hq, hkv, d, page = 4, 2, 64, 16
    bt, kv = paged_setup(torch.float32, [40, 40], hq, hkv, d, page, seed=1)
    fill_cache(kv, bt, [40, 40], hkv, d, page, torch.float32)
    q = rnd(21, hq, d, dtype=torch.float32, seed=3)
    rows, tiles, pairs = ops.plan_attention([20, 1], [20, 39])
    step = SimpleNamespace(decode_rows=torch.tensor(rows, dtype=torch.int32, device=dev()), num_decode=1,
                           prefill_tiles=torch.tensor(tiles, dtype=torch.int32, device=dev()), num_prefill_tiles=1,
                           num_pair_tiles=pairs, max_context=40)
    args = dict(positions=torch.tensor(list(range(20, 40)) + [39], dtype=torch.int32, device=dev()),
                token_seq=torch.tensor([0] * 20 + [1], dtype=torch.int32, device=dev()), scale=0.125, step=step)
    status = torch.zeros(1, dtype=torch.int32, device=dev())
    want = ops.paged_attention(q, kv, block_table=bt, status=status, **args)
    assert int(status.item()) == 0
    kv[:, int(bt[0, 38 // page]), :, 38 % page] = float("inf")
    got = ops.paged_attention(q, kv, block_table=bt, status=status, **args)
    assert torch.equal(got[:18], want[:18]) and torch.equal(got[20], want[20]) and not torch.isfinite(got[18:20]).all()
    bt[1, 0] = -1
    got = ops.paged_attention(q, kv, block_table=bt, status=status, **args)
    assert int(status.item()) == 2 and torch.isfinite(got[20]).all() and torch.equal(got[:18], want[:18])


@pytest.mark.parametrize("size", [1e-30, 1e-33, 1e-35, 1e-37, 1e-38, 1e-42, 1e30])
def test_split_product_keeps_the_bits_of_small_operands(ops, size):
    """Operands down to float32's subnormal numbers against large partners: as exact as multiply-adds. The sums are judged as
    float32 holds the operands."""
    for m, n, k in ((40, 200, 512), (150, 130, 2052)):
        small, large = rnd(m, k, dtype=torch.float32, seed=1) * size, rnd(n, k, dtype=torch.float32, seed=2) * min(1e10, 1e36 / size)
        for x, w in ((small, large), (large, small)):
            want, mass = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
            assert ((ops.linear(x, w) - want).abs() <= EPS * (k / 16 + 8) * mass + 2.0 ** -149).all()


@pytest.mark.parametrize("m,n,k,act", [(9, 514, 2048, None), (130, 259, 516, None), (333, 1000, 1028, None), (140, 130, 6144, "gelu_tanh"), (333, 6000, 512, "silu")])
def test_split_product_makes_infinite_and_nan_outputs_again(ops, m, n, k, act):
    """Outputs that are not finite in parts are the general kernel's bit for bit, whatever share of a tile they are, and the rest
    of the tile keeps its precision; a product of NaN alone costs no more than a few of the general kernel's."""
    rows = n * (2 if act else 1)
    x, w, b = (rnd(*s, dtype=torch.float32, seed=i) for i, s in enumerate(((m, k), (rows, k), (rows,))))
    x[1], x[m - 1, k - 1], x[m // 2, 3], w[rows - 2, 5] = float("nan"), float("inf"), -float("inf"), float("nan")
    w[3] = 0.0
    w[3, ::7] = 3.4e38                                  # rounds to infinity in bfloat16: finite outputs of rows that are small enough
    x[4:6] *= 1e-9

    def product(x):
        return ops.gated_linear(x, w, activation=act, bias=b) if act else ops.linear(x, w, bias=b)

    def plain(x):
        out = torch.empty((m, n), dtype=torch.float32, device=dev())
        ops._run("core", "ti_gemm_simt", out.data_ptr(), x.data_ptr(), w.data_ptr(), b.data_ptr(), None, m, n, k,
                 ops.GATED_ACTIVATIONS[act] if act else 0, 0, 0, ops._stream())
        return out
    got, want = product(x), plain(x)
    same = torch.zeros((m, n), dtype=torch.bool, device=dev())
    same[[1, m // 2, m - 1]] = True                     # made again whole
    same[:, (rows - 2) % n] = True
    same[:, 3] = True
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    fine = same & ~torch.isnan(want)
    if not act:
        assert torch.equal(got[fine], want[fine])
    z = x.double() @ w.double().T + b
    rest = ~same
    exact = gated(z, act) if act else z
    assert (got - exact)[rest].norm() <= 2e-6 * exact[rest].norm()

    def best(run):
        times = []
        for _ in range(4):
            begin, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            begin.record()
            run()
            end.record()
            torch.cuda.synchronize()
            times.append(begin.elapsed_time(end))
        return min(times)
    x[:] = float("nan")
    assert torch.isnan(product(x)).all()
    assert best(lambda: product(x)) <= 4 * best(lambda: plain(x)) + 0.1
    ops.check_kernel_status()
