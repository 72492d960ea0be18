"""Long portions of linear attention with one decay a head, in chunks of 64 tokens, against 64 bits and against the walk: portions
that end inside, at and behind a chunk, heads smaller than the tiles, shared groups, decays that vanish, all gates, states carried on."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,groups,dk,dv,gate,lens", [
    (16, 16, 128, 128, "constant", [1000]),
    (3, 3, 128, 128, "raw", [129, 64, 1, 193]),
    (4, 2, 64, 100, "step_size", [128, 65]),
    (2, 1, 20, 8, "step_size", [191, 192, 63]),
    (2, 2, 124, 128, "raw", [320]),
])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_chunks_against_plain(monkeypatch, heads, groups, dk, dv, gate, lens, dtype):
    from tinyinfer_b200 import ops
    gen = torch.Generator().manual_seed(heads * dk + dv + len(lens))
    T, n, pad = sum(lens), len(lens), 8
    row = torch.randn(T, pad + 2 * groups * dk + heads * dv, generator=gen).to(dtype)
    g = torch.randn(1 if gate == "constant" else T, heads, generator=gen)
    if gate in ("raw", "constant"):
        g = torch.sigmoid(3 * g + 2)
        g[..., 0] = 1e-30 if gate == "raw" else g[..., 0]          # forgets everything: no quotient of products of decays survives this
    a_log, dt_bias, skip = (torch.randn(heads, generator=gen) for _ in range(3))
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32)
    start = torch.randn(n + 1, heads, dv, dk, generator=gen)
    sg = ops.ScanGate(gate, g.cuda(), per_channel=False, a_log=a_log.cuda(), dt_bias=dt_bias.cuda())

    def run(chunks):
        monkeypatch.setattr(ops, "LINEAR_CHUNKS", chunks)
        state = start.cuda()
        d = row.cuda()
        out = ops.linear_scan(d, d, d, sg, state=state, heads=heads, groups=groups, key_dim=dk, value_dim=dv, q_offset=pad,
                              k_offset=pad + groups * dk, v_offset=pad + 2 * groups * dk, q_scale=0.5, skip=skip.cuda(), cu_seqlens=cu.cuda(),
                              state_slots=torch.arange(n, 0, -1, dtype=torch.int32).cuda(), num_seqs=n, max_q_len=max(lens))
        return out.cpu().double().view(T, heads, dv), state.cpu().double()

    from tinyinfer_b200.ops import _dtype_code, _fn
    at = [x for offset in (pad, pad + groups * dk, pad + 2 * groups * dk) for x in (0, row.shape[1], offset)]       # address (any on 16 bytes), row, offset
    assert ops.linear_chunks(T, n, max(lens), heads, dk, dv) and _fn("hybrid", "ti_linear_scan_chunks_ok")(*at, dk, dv, _dtype_code(row))
    got, state = run(True)
    walk, walk_state = run(False)
    ops.check_kernel_status()
    r = row.double()
    q, k = (r[:, pad + i * groups * dk:pad + (i + 1) * groups * dk].reshape(T, groups, dk).repeat_interleave(heads // groups, 1) for i in (0, 1))
    v = r[:, pad + 2 * groups * dk:].reshape(T, heads, dv)
    if gate == "step_size":
        dt = torch.nn.functional.softplus(g.double() + dt_bias.double(), threshold=1e9)
        a, k = torch.exp(-torch.exp(a_log.double()) * dt), k * dt[:, :, None]
    else:
        a = g.double().expand(T, heads)
    want, want_state = torch.empty_like(got), start.double().clone()
    for i in range(n):
        S = start[n - i].double().transpose(1, 2)
        for t in range(cu[i], cu[i + 1]):
            S = a[t][:, None, None] * S + k[t][:, :, None] * v[t][:, None, :]
            want[t] = torch.einsum("hkv,hk->hv", S, 0.5 * q[t]) + skip.double()[:, None] * v[t]
        want_state[n - i] = S.transpose(1, 2)
    # float32 sums: 2^-24 a step, over 128 channels and the tokens that a decay remembers; no worse than the walk's order of them
    for x, y, z in ((got, walk, want), (state, walk_state, want_state)):
        err, err_walk = ((u - z).norm() / z.norm() for u in (x, y))
        assert torch.isfinite(x).all() and err <= 2e-6 and err <= 1.5 * err_walk + 1e-7, (err, err_walk)
    assert torch.equal(state[0], start[0].double())


def test_chunks_hold_any_division_and_look_at_no_later_token():
    """``max_q_len`` is a hint: one too small gives the same outputs. And a value that is no number reaches no token before its own."""
    from tinyinfer_b200 import ops
    lens, heads, dk = [3, 700, 1, 66], 2, 64
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32).cuda()
    gen = torch.Generator().manual_seed(7)
    row = torch.randn(sum(lens), 3 * heads * dk, generator=gen).cuda()
    decay = ops.ScanGate("constant", torch.tensor([[0.9, 0.99]]).cuda(), per_channel=False)

    def run(rows, longest):
        state = torch.zeros(len(lens), heads, dk, dk, device="cuda")
        out = ops.linear_scan(rows, rows, rows, decay, state=state, heads=heads, groups=heads, key_dim=dk, value_dim=dk, k_offset=heads * dk,
                              v_offset=2 * heads * dk, cu_seqlens=cu, state_slots=torch.arange(len(lens), dtype=torch.int32).cuda(),
                              num_seqs=len(lens), max_q_len=longest)
        return out, state

    assert all(ops.linear_chunks(sum(lens), len(lens), longest, heads, dk, dk) for longest in (128, 700))
    out, state = run(row, 700)
    again, state_again = run(row, 128)
    assert torch.equal(out, again) and torch.equal(state, state_again)
    for at in (3 + 77, 3 + 64, 3 + 127):
        spoiled = row.clone()
        spoiled[at, 2 * heads * dk:] = float("nan")
        got, _ = run(spoiled, 700)
        assert torch.equal(got[:at], out[:at]) and got[at:703].isnan().all() and torch.equal(got[703:], out[703:])
