"""The grouped products on tcgen05 with units of 256 features, which only steps of many rows take, beside units of 128."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu


# rows of every expert: none, one, a row tile, a row tile and one row more, the rest in between
@pytest.mark.parametrize("n,k,features", [(1408, 256, 256), (1100, 128, 256), (1026, 192, 256), (999, 64, 256), (130, 128, 128)])
@pytest.mark.parametrize("form", ["up", "linear", "down"])
def test_grouped_product_against_64_bits(n, k, features, form):
    from tinyinfer_b200 import ops
    counts = [0, 1, 128, 129, 0, 257, 2000, 1, 3300, 127, 4000, 129]
    slots, experts = sum(counts), len(counts)
    assert ops._fn("sm100", "ti_moe_tcgen05_unit_features")(slots, n) == features
    gen = torch.Generator().manual_seed(n)
    x = torch.randn(slots, k, generator=gen).to(torch.bfloat16).cuda()
    w = (torch.randn(experts, n, k, generator=gen) * k ** -0.5).to(torch.bfloat16).cuda()
    tiles, starts = [], [0]
    for e, c in enumerate(counts):
        tiles += [(e, starts[-1] + r, min(128, c - r)) for r in range(0, c, 128)]
        starts.append(starts[-1] + c)
    order = torch.randperm(slots, generator=gen)              # the token of every sorted row
    routing = SimpleNamespace(tile_rows=128, token_of=order.int().cuda(), max_tiles=len(tiles) + experts,
                              tiles=torch.tensor(tiles + [(0, 0, 0)] * experts, dtype=torch.int32).cuda(),
                              num_tiles=torch.tensor([len(tiles)], dtype=torch.int32).cuda())
    got = ops.expert_linear(x, w, routing, up=form != "down", activation=form == "up")
    rows = x if form == "down" else x[order.cuda()]
    for e, c in enumerate(counts):
        at = slice(starts[e], starts[e + 1])
        want = rows[at].double() @ w[e].double().T
        mass = rows[at].double().abs() @ w[e].double().abs().T
        # bfloat16 products are exact; the sums lose up to a bit of float32 every 16 products
        slack = 2.0 ** -23 * (k / 16 + 2) * mass
        if form == "up":
            slack, want = slack * (2 * want.clamp(min=0) + slack), want.clamp(min=0) ** 2
        if form != "down":
            slack = slack + 2.0 ** -8 * want.abs()
        assert got[at].shape == want.shape and ((got[at].double() - want).abs() <= slack).all(), (e, c)
    ops.check_kernel_status()
