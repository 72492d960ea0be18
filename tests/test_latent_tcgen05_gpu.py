"""The attention over cached latent rows on tcgen05 (prompt portions) against 64 bits, and against the warp-level form, whose
probabilities it rounds alike: edges of its tiles of 32 keys and of its row tiles, pages of 16 keys, rows past a chunk of 64
features, sinks, shared-out keys, portions beside decoded tokens, pages that hold NaN behind the last key."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,rank,rot,page,sink,work", [
    (16, 512, 64, 64, True, [(75, 75), (900, 1), (300, 9)]),         # two CTAs a row tile; a decoded token among portions
    (16, 512, 64, 16, False, [(33, 33), (64, 31), (65, 2)]),
    (16, 512, 64, 64, True, [(1500, 16)]),                           # keys shared out over CTAs
    (5, 256, 32, 32, False, [(130, 130), (31, 31), (32, 32)]),       # heads that do not divide the 128 rows
    (3, 64, 8, 48, True, [(700, 600)]),                              # features past a chunk; pages of 48
    (130, 128, 0, 128, False, [(40, 3)]),                            # more heads than rows
])
def test_portions_on_tcgen05(monkeypatch, heads, rank, rot, page, sink, work):
    from tinyinfer_b200 import ops
    from tinyinfer_b200.engine.batch import BatchBuffers, StepEntry
    gen = torch.Generator().manual_seed(heads * rank)
    dk, lens = rank + rot, [c for c, _ in work]
    pages_of = [-(-n // page) for n in lens]
    perm = torch.randperm(sum(pages_of) + 2, generator=gen).tolist()
    tables = [[perm.pop() for _ in range(nb)] for nb in pages_of]
    cache = torch.full((1, sum(pages_of) + 2, 1, page, dk), float("nan"), dtype=torch.bfloat16)
    rows = [torch.randn(n, dk, generator=gen).to(torch.bfloat16) for n in lens]
    for i, n in enumerate(lens):
        for p in range(n):
            cache[0, tables[i][p // page], 0, p % page] = rows[i][p]
    buffers = BatchBuffers(torch.device("cuda"), sum(n for _, n in work), len(work), max(pages_of), 1)
    step = buffers.build([StepEntry(i, [0] * n, []) for i, (_, n) in enumerate(work)], [c - n for c, n in work], [0] * len(work), [tables])
    T = step.num_tokens
    q = 2.0 * torch.randn(T, heads * dk, generator=gen)
    scale = dk ** -0.5
    sinks = torch.randn(heads, generator=gen) if sink else None
    args = dict(heads=heads, rank=rank, rot=rot, scale=scale, sink=sinks.cuda() if sink else None, positions=step.positions,
                token_seq=step.token_seq, block_table=step.block_tables[0], max_context=max(lens), step=step)
    assert ops._fn("latent", "ti_latent_attend_tc_ctas")(T, len(work), heads, rank, rot, page) > 0
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    new = ops.latent_attention(q.cuda(), cache.cuda(), status=status, **args).cpu().double()
    assert ops.latent_rows_dtype(T, cache.cuda(), heads=heads, rank=rank, rot=rot, step=step) == torch.bfloat16
    assert torch.equal(new, ops.latent_attention(q.cuda().bfloat16(), cache.cuda(), status=status, **args).cpu().double())    # rounded before
    monkeypatch.setattr(ops, "LATENT_TCGEN05", False)
    old = ops.latent_attention(q.cuda(), cache.cuda(), status=status, **args).cpu().double()
    ops.check_kernel_status()
    pos, seq = step.positions.cpu().tolist(), step.token_seq.cpu().tolist()
    want = torch.empty_like(new)
    for t in range(T):
        keys = rows[seq[t]][:pos[t] + 1].double()
        z = (q[t].view(heads, dk).to(torch.bfloat16).double() @ keys.T) * scale
        if sink:
            z = torch.cat([z, sinks.double()[:, None]], dim=1)
        want[t] = (torch.softmax(z, dim=1)[:, :pos[t] + 1] @ keys[:, :rank]).reshape(-1)
    # two roundings to 8 bits, of the probabilities and of the result: at most 2^-9 of the result's norm each
    err, err_old = ((x - want).norm() / want.norm() for x in (new, old))
    assert err <= 2.0 ** -8 and err <= 1.02 * err_old + 1e-5, (err, err_old)


@pytest.mark.parametrize("heads,rank,rot,page,work,at", [
    (16, 512, 64, 64, [(75, 75), (33, 9)], 42),                      # 8 tokens a row tile, two CTAs
    (16, 512, 64, 64, [(1500, 16)], 1491),                           # keys shared out over CTAs
    (3, 64, 8, 48, [(300, 100), (64, 1)], 231),                      # 42 tokens a row tile, whose keys lie in three tiles
    (1, 128, 0, 16, [(160, 160)], 64),
])
@pytest.mark.parametrize("value,feature", [(float("nan"), 3), (float("inf"), 40), (float("-inf"), 63), (float("inf"), -1)])
def test_a_value_that_is_no_number_reaches_no_token_before_its_own(monkeypatch, heads, rank, rot, page, work, at, value, feature):
    from tinyinfer_b200 import ops
    from tinyinfer_b200.engine.batch import BatchBuffers, StepEntry
    gen = torch.Generator().manual_seed(heads + at)
    dk, pages = rank + rot, [-(-c // page) for c, _ in work]
    tables = [list(range(sum(pages[:i]), sum(pages[:i + 1]))) for i in range(len(work))]
    cache = torch.randn(1, sum(pages), 1, page, dk, generator=gen).bfloat16()
    buffers = BatchBuffers(torch.device("cuda"), sum(n for _, n in work), len(work), max(pages), 1)
    step = buffers.build([StepEntry(i, [0] * n, []) for i, (_, n) in enumerate(work)], [c - n for c, n in work], [0] * len(work), [tables])
    q = torch.randn(step.num_tokens, heads * dk, generator=gen).bfloat16()

    def run(rows):
        return ops.latent_attention(q.cuda() if ops.LATENT_TCGEN05 else q.float().cuda(), rows.cuda(), heads=heads, rank=rank, rot=rot,
                                    scale=dk ** -0.5, sink=None, positions=step.positions, token_seq=step.token_seq,
                                    block_table=step.block_tables[0], max_context=max(c for c, _ in work), step=step).cpu()

    spoiled = cache.clone()
    spoiled[0, at // page, 0, at % page, feature] = value             # of the first request's token at position `at`
    clean, got = run(cache), run(spoiled)
    monkeypatch.setattr(ops, "LATENT_TCGEN05", False)
    warp_level = run(spoiled)
    ops.check_kernel_status()
    row, end = at - (work[0][0] - work[0][1]), work[0][1]             # the token's place in the step
    assert torch.equal(got[:row], clean[:row]) and torch.equal(got[end:], clean[end:])
    assert torch.equal(got[row:end].isnan(), warp_level[row:end].isnan()) and got[row:end].isnan().any()


@pytest.mark.parametrize("tc", [True, False])
def test_a_key_without_a_page_is_reported_to_the_caller_s_word_alone(monkeypatch, tc):
    from tinyinfer_b200 import ops
    from tinyinfer_b200.engine.batch import BatchBuffers, StepEntry
    monkeypatch.setattr(ops, "LATENT_TCGEN05", tc)
    heads, rank, rot, page = 16, 512, 64, 64
    buffers = BatchBuffers(torch.device("cuda"), 100, 1, 4, 1)
    step = buffers.build([StepEntry(0, [0] * 100, [])], [100], [0], [[[0, 1, -1, 3]]])     # keys 128 .. 191 have no page
    cache = torch.zeros(1, 4, 1, page, rank + rot, dtype=torch.bfloat16, device="cuda")
    q = torch.zeros(100, heads * (rank + rot), device="cuda")
    word = torch.zeros(2, dtype=torch.int32, device="cuda")
    for status in (word[:1], None):
        ops.latent_attention(q, cache, heads=heads, rank=rank, rot=rot, scale=0.1, sink=None, positions=step.positions,
                             token_seq=step.token_seq, block_table=step.block_tables[0], max_context=200, step=step, status=status)
    assert word.tolist() == [2, 0]
    ops.check_kernel_status()                            # nothing in the device's own words


@pytest.mark.parametrize("heads,rank,rot,decoded,portion", [(16, 512, 64, [4200] + [70] * 8, (70, 70)), (4, 128, 32, [33, 5000], (300, 100))])
def test_decoded_tokens_behind_many_keys_take_their_own_form(heads, rank, rot, decoded, portion):
    """Beside a portion they come out as in a step of their own, and so does the portion."""
    from tinyinfer_b200 import ops
    from tinyinfer_b200.engine.batch import BatchBuffers, StepEntry
    gen = torch.Generator().manual_seed(heads)
    dk, page, work = rank + rot, 64, [(c, 1) for c in decoded] + [portion]
    pages = [-(-c // page) for c, _ in work]
    tables = [list(range(sum(pages[:i]), sum(pages[:i + 1]))) for i in range(len(work))]
    cache = torch.randn(1, sum(pages), 1, page, dk, generator=gen).bfloat16().cuda()
    q = torch.randn(sum(n for _, n in work), heads * dk, generator=gen).bfloat16().cuda()

    def run(some):
        mine = work[some]
        buffers = BatchBuffers(torch.device("cuda"), 400, len(mine), max(pages), 1)
        step = buffers.build([StepEntry(i, [0] * n, []) for i, (_, n) in enumerate(mine)], [c - n for c, n in mine], [0] * len(mine), [tables[some]])
        first = sum(n for _, n in work[:some.start or 0])
        rows = q[first:first + step.num_tokens]
        kind = ops.latent_rows_dtype(step.num_tokens, cache, heads=heads, rank=rank, rot=rot, step=step)
        out = ops.latent_attention(rows.to(kind), cache, heads=heads, rank=rank, rot=rot, scale=dk ** -0.5, sink=None, positions=step.positions,
                                   token_seq=step.token_seq, block_table=step.block_tables[0], max_context=max(c for c, _ in mine), step=step)
        return out, ops.latent_decoded_apart(step.q_lens, step.starts)

    n = len(decoded)
    both, apart = run(slice(0, n + 1))
    alone, portion_alone = run(slice(0, n)), run(slice(n, n + 1))
    ops.check_kernel_status()
    assert apart == n and alone[1] == portion_alone[1] == 0
    assert torch.equal(both[:n], alone[0]) and torch.equal(both[n:], portion_alone[0])
