"""The router's and the plan's forms at their edges: one block or many place the choices, one token or eight share a block."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# 1,024 choices are the most one block places; 1,184 tokens the fewest that go eight a block
@pytest.mark.parametrize("tokens,experts,identity,top,hidden", [
    (1, 3, 0, 1, 40), (256, 33, 2, 4, 64), (257, 64, 0, 4, 72), (1183, 40, 1, 2, 128), (1184, 256, 0, 2, 96), (1201, 70, 6, 6, 2048),
    (2048, 5, 0, 1, 64)])
@pytest.mark.parametrize("router,rows", [(torch.float32, torch.float32), (torch.bfloat16, torch.float32), (torch.bfloat16, torch.bfloat16)])
def test_routing(tokens, experts, identity, top, hidden, router, rows):
    from tinyinfer_b200 import ops
    gen = torch.Generator().manual_seed(tokens + experts)
    x = torch.randn(tokens, hidden, generator=gen).to(rows)
    w = (torch.randn(experts + identity, hidden, generator=gen) * hidden ** -0.5 * 2).to(router)
    got = ops.route_experts(x.cuda(), w.cuda(), top, 1e-20, real_experts=experts)
    scores = torch.softmax(x.double() @ w.double().T, dim=-1)
    best, want = torch.topk(scores, min(top + 1, experts + identity))
    chosen, weight = got.chosen.cpu().long(), got.weight.cpu().double()
    # float32 sums of `hidden` products: scores apart by more than their rounding are chosen alike
    clear = (best[:, :-1] - best[:, 1:]).min(dim=1).values > 1e-5 if best.shape[1] > top else torch.ones(tokens, dtype=torch.bool)
    assert torch.equal(chosen[clear], want[:, :top][clear]) and clear.float().mean() > 0.9
    of_chosen = scores.gather(1, chosen)
    assert (weight - of_chosen / of_chosen.sum(1, keepdim=True)).abs().max() <= 1e-5
    counts = torch.bincount(chosen.flatten(), minlength=experts + identity)
    assert torch.equal(got.counts.cpu().long(), counts)
    slots = got.slot_of.cpu().long()
    assert torch.equal(slots.flatten().sort().values, torch.arange(tokens * top))
    starts = counts.cumsum(0) - counts
    assert ((slots >= starts[chosen]) & (slots < (starts + counts)[chosen])).all()
    assert torch.equal(got.token_of.cpu().long()[slots], torch.arange(tokens)[:, None].expand(-1, top))
    assert torch.equal(got.slot_weight.cpu()[slots], got.weight.cpu())
    tiles = [(e, int(starts[e]) + r, min(got.tile_rows, int(counts[e]) - r)) for e in range(experts) for r in range(0, int(counts[e]), got.tile_rows)]
    assert int(got.num_tiles.item()) == len(tiles) and [tuple(t) for t in got.tiles[:len(tiles)].tolist()] == tiles
