"""Kernels of the 32-bit path on the GPU against 64-bit references, with bounds that follow from the number of roundings."""
import pytest
import torch

from test_kernels_gpu import ops, rnd  # noqa: F401  (the fixture)

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -24


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
