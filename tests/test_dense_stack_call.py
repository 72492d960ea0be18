"""What ``ops.dense_stack`` hands to the native call, with the libraries replaced by ones that only look."""
from types import SimpleNamespace

import pytest
import torch

from tinyinfer_b200 import ops


@pytest.fixture
def calls(monkeypatch):
    """The arguments of every native call that ``ops.dense_stack`` makes on CPU tensors."""
    seen = []

    def fn(lib, name):
        if name == "ti_dense_stack":
            return lambda address: seen.append(bytes(ops._StackCall.from_address(address))) or 0
        return lambda *a: 4096
    monkeypatch.setattr(ops, "_fn", lambda lib, name: type("F", (), {"__call__": staticmethod(fn(lib, name))})())
    monkeypatch.setattr(ops, "_stack_launchers", {torch.bfloat16: [None] * len(ops._STACK_LAUNCHERS)})
    monkeypatch.setattr(ops, "_check", lambda t, *a: t)
    monkeypatch.setattr(ops, "status_words", lambda device: torch.zeros(2, dtype=torch.int32))
    monkeypatch.setattr(ops, "_gemm_scratch", lambda device: (torch.zeros(4), torch.zeros(4, dtype=torch.int32)))
    monkeypatch.setattr(ops, "_decode_scratch", lambda device, floats: torch.empty(floats))
    monkeypatch.setattr(ops, "_stream", lambda: 0)
    monkeypatch.setattr(ops, "_side_stream", lambda device: SimpleNamespace(cuda_stream=1))
    return lambda: [ops._StackCall.from_buffer_copy(b) for b in seen]


@pytest.mark.parametrize("heads,kv_heads,dim", [(40, 8, 128), (28, 4, 128), (24, 8, 64), (16, 16, 64), (7, 1, 128), (16, 8, 128)])
def test_scratch_of_portions_beside_decoded_tokens_is_aligned(calls, monkeypatch, heads, kv_heads, dim):
    """The portions' part of the scratch begins behind the decoded tokens', whatever size that has, on a 16-byte boundary (its
    partial outputs are stored as float4), and both fit."""
    need = []
    monkeypatch.setattr(ops, "decode_scratch_floats",
                        lambda rows, hq, hkv, d, context, window: need.append((ctas + rows * hkv) * (hq // hkv) * (d + 2)) or need[-1])
    for rows in (1, 2, 3, 8, 27):
        for ctas in (1, 2, 37, 148, 259):
            t = rows + 64
            step = SimpleNamespace(positions=torch.zeros(t), token_seq=torch.zeros(t), decode_rows=torch.zeros(rows),
                                   prefill_tiles=torch.zeros(4), status=None, num_decode=rows, num_prefill_tiles=1, num_pair_tiles=0,
                                   max_context=3000)
            row = [0] * 18
            row[14:17] = [8, 32, 0]
            ops.dense_stack(torch.zeros(t, 64, dtype=torch.bfloat16), [row], step, heads=heads, kv_heads=kv_heads, head_dim=dim, inter=64,
                            activation="silu", page_size=64, eps=(1e-6, 1e-6, 1e-6), scale=1.0, rotation=None)
            call = calls()[-1]
            assert call.side == 1 and call.decode_floats >= need[-1]
            assert (call.attn_scratch + 4 * call.decode_floats) % 16 == 0
            assert call.attn_floats >= call.decode_floats + 4096


@pytest.mark.parametrize("heads,dim", [(1, 64), (7, 64), (16, 128), (40, 128)])
def test_the_native_call_shares_keys_out_as_the_part_does(heads, dim):
    """The scratch that the native call asks for is what ``key_split``'s shares need, whatever tiles and contexts there are."""
    floats = ops._fn("stack", "ti_dense_stack_portion_floats")
    floats.restype = ops.c_ll
    call = ops._StackCall()
    call.dtype, call.heads, call.head_dim = 1, heads, dim
    call.pair_min_ctas, call.split_max_ctas = ops.PAIR_MIN_CTAS, ops.KEY_SPLIT_MAX_CTAS
    for pairs in (0, 1, 2, 5, 37, 148):
        for singles in (0, 1, 3, 30, 75):
            for context in (1, 1000, 2047, 2048, 2049, 3000, 4096, 9999, 32768, 40960):
                call.num_pairs, call.num_tiles, call.max_context = pairs, pairs + singles, context
                need = [0]
                for count, halves in ((pairs if pairs * heads < ops.PAIR_MIN_CTAS else 0, 2), (singles, 1)):
                    if count:
                        splits, keys = ops.key_split(count * halves * heads, context)
                        assert splits == 1 or (keys % 128 == 0 and splits * keys >= context)
                        need.append(count * halves * splits * heads * 128 * (dim + 2) if splits > 1 else 0)
                assert floats(ops.ctypes.addressof(call)) == max(need), (pairs, singles, context)
