"""The gated delta rule four tokens at a time against 64 bits and against the walk token by token: requests that end inside, at and
behind a quad, one token long, heads smaller than the lanes' rows, shared groups, decays that vanish, states carried on."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,groups,dk,dv,lens", [
    (16, 16, 128, 128, [333]),
    (4, 2, 128, 100, [4, 1, 90, 7]),
    (3, 3, 64, 7, [2, 141]),
    (2, 1, 10, 33, [71]),
    (2, 2, 200, 64, [8, 1, 90]),
])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_quads_against_plain(monkeypatch, heads, groups, dk, dv, lens, dtype):
    from tinyinfer_b200 import ops
    gen = torch.Generator().manual_seed(heads * dk + dv)
    T, n, pad = sum(lens), len(lens), 3
    row = torch.randn(T, pad + 2 * groups * dk + heads * dv, generator=gen).to(dtype)
    decay, beta = torch.randn(T, heads * dk, generator=gen), torch.randn(T, 1 + heads, generator=gen)
    decay[:, ::7] = 90.0                                 # forgets everything at once
    a_log, dt_bias = torch.randn(heads, generator=gen) * 0.5, torch.randn(heads * dk, generator=gen) - 3
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32)
    start = torch.randn(n + 1, heads, dv, dk, generator=gen)

    def run(quads, rows=row):
        monkeypatch.setattr(ops, "DELTA_QUADS", quads)
        state, d = start.cuda(), rows.cuda()
        out = ops.delta_scan(d, d, d, decay.cuda(), beta.cuda(), a_log=a_log.cuda(), dt_bias=dt_bias.cuda(), state=state, heads=heads,
                             groups=groups, key_dim=dk, value_dim=dv, q_offset=pad, k_offset=pad + groups * dk, v_offset=pad + 2 * groups * dk,
                             beta_offset=1, q_scale=0.5, cu_seqlens=cu.cuda(), state_slots=torch.arange(n, 0, -1, dtype=torch.int32).cuda(), num_seqs=n)
        return out.cpu().double().view(T, heads, dv), state.cpu().double()

    quads = lambda requests, tokens: ops._fn("hybrid", "ti_delta_quads_floats")(requests, tokens, heads, dk, dv) > 0
    assert quads(n, T) and not quads(1, 67) and not quads(8, 95) and not ops._fn("hybrid", "ti_delta_quads_floats")(1, 500, heads, 257, dv)
    got, state = run(True)
    walk, walk_state = run(False)
    ops.check_kernel_status()
    r = row.double()
    q, k = (r[:, pad + i * groups * dk:pad + (i + 1) * groups * dk].reshape(T, groups, dk).repeat_interleave(heads // groups, 1) for i in (0, 1))
    q, k = (x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6) for x in (q, k))
    q = 0.5 * q
    v = r[:, pad + 2 * groups * dk:].reshape(T, heads, dv)
    g = torch.exp(-torch.exp(a_log.double())[:, None] * torch.nn.functional.softplus((decay + dt_bias).double(), threshold=1e9).view(T, heads, dk))
    b = torch.sigmoid(beta[:, 1:].double())
    want, want_state = torch.empty_like(got), start.double().clone()
    for i in range(n):
        S = start[n - i].double()
        for t in range(cu[i], cu[i + 1]):
            S = S * g[t][:, None, :]
            u = b[t][:, None] * (v[t] - torch.einsum("hvk,hk->hv", S, k[t]))
            S = S + u[:, :, None] * k[t][:, None, :]
            want[t] = torch.einsum("hvk,hk->hv", S, q[t])
        want_state[n - i] = S
    # float32: roundings of 2^-24 over the channels' sums and the tokens that a decay remembers; no worse than token by token
    for x, y, z in ((got, walk, want), (state, walk_state, want_state)):
        err, err_walk = ((w - z).norm() / z.norm() for w in (x, y))
        assert torch.isfinite(x).all() and err <= 2e-6 and err <= 1.5 * err_walk + 1e-7, (err, err_walk)
    assert torch.equal(state[0], start[0].double())
    # a value that is no number reaches no token before its own, and no other request
    at = int(cu[1]) - 2
    spoiled = row.clone()
    spoiled[at, pad + 2 * groups * dk:] = float("nan")
    out, after = run(True, spoiled)
    assert torch.equal(out[:at], got[:at]) and torch.equal(out[cu[1]:], got[cu[1]:]) and torch.equal(after[:n], state[:n])
    assert out[at:cu[1]].isnan().all()
