"""The grouped products of experts in the pair form (row tiles of 256) against the form of 128, whose bits they have."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu


# rows of every expert: none, one, around 128 and 256, many; features in whole units, past one, not a multiple of 8
@pytest.mark.parametrize("n,k", [(1408, 256), (256, 64), (1026, 192), (999, 128)])
@pytest.mark.parametrize("form", ["up", "linear", "down"])
def test_pair_form_has_the_bits_of_the_other(n, k, form):
    from tinyinfer_b200 import ops
    counts = [0, 1, 128, 129, 0, 255, 256, 257, 2000, 1, 700, 127]
    slots, experts = sum(counts), len(counts)
    gen = torch.Generator().manual_seed(n)
    x = torch.randn(slots, k, generator=gen).to(torch.bfloat16).cuda()
    w = (torch.randn(experts, n, k, generator=gen) * k ** -0.5).to(torch.bfloat16).cuda()
    order = torch.randperm(slots, generator=gen).int().cuda()
    got = []
    for rows in (128, 256):
        tiles, start = [], 0
        for e, c in enumerate(counts):
            tiles += [(e, start + r, min(rows, c - r)) for r in range(0, c, rows)]
            start += c
        routing = SimpleNamespace(tile_rows=rows, token_of=order, max_tiles=len(tiles) + experts, num_tiles=torch.tensor([len(tiles)], dtype=torch.int32).cuda(),
                                  tiles=torch.tensor(tiles + [(0, 0, 0)] * experts, dtype=torch.int32).cuda())
        got.append(ops.expert_linear(x, w, routing, up=form != "down", activation=form == "up"))
    ops.check_kernel_status()
    source = x if form == "down" else x[order.long()]
    e, at = 8, slice(sum(counts[:8]), sum(counts[:9]))
    want = source[at].double() @ w[e].double().T
    want = want.clamp(min=0) ** 2 if form == "up" else want
    assert ((got[1][at].double() - want).norm() <= 2.0 ** -8 * want.norm()) and torch.equal(got[0], got[1])


def test_which_steps_take_pairs():
    from tinyinfer_b200 import ops
    rows = lambda t, hidden, ff: ops.expert_tile_rows_of(t, hidden, torch.bfloat16, 64, 6, ff)
    least = -(-ops.EXPERT_PAIR_MIN_ROWS * 64 // 6)
    assert [rows(least, 2048, 1408), rows(least - 1, 2048, 1408), rows(least, 2048, 192), rows(least, 128, 1408)] == [256, 128, 128, 128]
