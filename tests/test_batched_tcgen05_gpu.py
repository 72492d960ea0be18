"""Batched products of many rows on tcgen05 against 64 bits and the warp-level form: rows past a tile, outputs past a tile and less than
one, one and several k blocks, pieces side by side at an offset, both output types; and what stays with the others."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def takes(x, w, x_offset, x_batch_stride, out, out_offset, out_batch_stride):
    """Whether the tcgen05 form takes a product without bias, sigmoid or gate."""
    from tinyinfer_b200 import ops
    batch, n, k = w.shape
    return bool(ops._fn("latent", "ti_gemm_batched_tc_ok")(
        out.data_ptr() + out_offset * out.element_size(), x.data_ptr() + x_offset * x.element_size(), w.data_ptr(), batch, x.shape[0], n, k,
        x.shape[1], x_batch_stride, out.shape[1], out_batch_stride, int(out.dtype == torch.float32)))


@pytest.mark.parametrize("m,batch,n,k,extra", [(128, 3, 512, 128, 64), (300, 2, 32, 64, 8), (257, 5, 160, 512, 0), (129, 1, 256, 320, 16)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_many_rows_on_tcgen05(monkeypatch, m, batch, n, k, extra, out_dtype):
    from tinyinfer_b200 import ops
    gen = torch.Generator().manual_seed(m * n + k)
    x = torch.randn(m, 8 + batch * (k + extra), generator=gen).bfloat16()
    x[:, :8] = float("nan")                              # beside the pieces
    w = (torch.randn(batch, n, k, generator=gen) * k ** -0.5).bfloat16()
    outs = []
    for on in (True, False):
        monkeypatch.setattr(ops, "BATCHED_TCGEN05", on)
        out = torch.full((m, 8 + batch * (n + 8)), 7.0, dtype=out_dtype, device="cuda")
        assert takes(x.cuda(), w.cuda(), 8, k + extra, out, 8, n + 8)
        ops.batched_linear(x.cuda(), w.cuda(), x_offset=8, x_batch_stride=k + extra, k=k, out=out, out_offset=8, out_batch_stride=n + 8)
        outs.append(out.cpu().double())
    ops.check_kernel_status()
    pieces = torch.stack([x[:, 8 + b * (k + extra):8 + b * (k + extra) + k] for b in range(batch)]).double()
    want = torch.einsum("bmk,bnk->mbn", pieces, w.double())
    for out in outs:
        got = out[:, 8:].view(m, batch, n + 8)
        assert (out[:, :8] == 7).all() and (got[:, :, n:] == 7).all()             # nothing beside the pieces is written
        err = (got[:, :, :n] - want).norm() / want.norm()
        assert err <= (2e-6 if out_dtype == torch.float32 else 2.0 ** -8), err             # float32 sums; one rounding to 8 bits


def test_what_other_forms_keep(monkeypatch):
    """A row length or an offset that TMA cannot start at, K of less than whole k blocks, bias, sigmoid and gate: as without the tcgen05 form, bit for bit."""
    from tinyinfer_b200 import ops
    gen = torch.Generator().manual_seed(3)
    for cols, offset, k, n in ((2 * 64 + 4, 0, 64, 64), (2 * 64 + 8, 4, 64, 64), (2 * 72, 0, 72, 64), (2 * 64, 0, 64, 20)):
        x, w = torch.randn(130, cols, generator=gen).bfloat16().cuda(), torch.randn(2, n, k, generator=gen).bfloat16().cuda()
        assert not takes(x, w, offset, k, torch.empty(130, 2 * n, dtype=x.dtype, device="cuda"), 0, n)
        outs = []
        for on in (True, False):
            monkeypatch.setattr(ops, "BATCHED_TCGEN05", on)
            outs.append(ops.batched_linear(x, w, x_offset=offset, x_batch_stride=k, k=k))
        assert torch.equal(*outs)
    gate, bias = torch.randn(130, 128, generator=gen).bfloat16().cuda(), torch.randn(2, 64, generator=gen).cuda()
    x, w = torch.randn(130, 128, generator=gen).bfloat16().cuda(), torch.randn(2, 64, 64, generator=gen).bfloat16().cuda()
    assert takes(x, w, 0, 64, torch.empty_like(x), 0, 64)                # without what follows
    for extra in (dict(bias=bias), dict(sigmoid=True), dict(gate=gate)):
        outs = []
        for on in (True, False):
            monkeypatch.setattr(ops, "BATCHED_TCGEN05", on)
            outs.append(ops.batched_linear(x, w, x_batch_stride=64, k=64, **extra))
        assert torch.equal(*outs)
