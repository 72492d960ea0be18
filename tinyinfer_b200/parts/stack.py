"""The blocks of a dense pre-norm decoder (the reference's model: tinyinfer/models/qwen3.py:192-288) run by one native call.

Part by part, every kernel of a step is checked, given its output and launched from Python, which costs several times what a
kernel of a short step runs for. A model whose blocks are all pre-norm blocks of plain attention and a gated feed-forward, of
the same sizes, is recognised here once; its steps then hand the native side their layers' addresses and make the launches of
all layers in one call. The kernels are the parts' own, on the same operands in the same order, but for the two attention kernels of a
step that brings portions and decoded tokens: these run beside each other, on two streams. Operands that the parts' calls would
refuse are left to them."""
from __future__ import annotations

from typing import Optional

import torch

from .. import ops
from .attention import Attention
from .block import PreNormBlock
from .feedforward import GatedMLP
from .norm import RMSNorm


class DenseStack:
    def __init__(self, blocks, execution):
        self.blocks, self.execution = blocks, execution

    @classmethod
    def of(cls, blocks, execution) -> Optional["DenseStack"]:
        """The stack of these blocks run in this order, or None if one of them asks for something else."""
        def shape(block):
            mixer, ff = block.mixer, block.feed_forward
            s, r = mixer.spec, mixer._rotation
            turn = None if r is None else (r.rotary_dim, r.interleaved, r.factor, None if r.cos_sin is None else r.cos_sin.shape[0])
            return (s.num_heads, s.num_kv_heads, s.head_dim, s.hidden_size, s.scale, s.qk_norm.eps if s.qk_norm is not None else 0.0, turn,
                    ff.spec.intermediate_size, ff.spec.activation, block.mixer_norm.spec.eps, block.feed_forward_norm.spec.eps,
                    mixer.dtype)

        for b in blocks:
            if (type(b) is not PreNormBlock or type(b.mixer) is not Attention or type(b.feed_forward) is not GatedMLP
                    or type(b.mixer_norm) is not RMSNorm or type(b.feed_forward_norm) is not RMSNorm or b.mixer._general
                    or b.feed_forward.spec.bias):
                return None
        if any(e.adds_embedding or e.projects_embedding or e.adds_vector is not None for e in execution):
            return None
        if not blocks or any(shape(b) != shape(blocks[0]) for b in blocks[1:]):
            return None
        turn = shape(blocks[0])[6]
        return cls(blocks, execution) if turn is None or (turn[2] == 1.0 and turn[0] <= blocks[0].mixer.spec.head_dim) else None

    def run(self, x: torch.Tensor, step) -> Optional[torch.Tensor]:
        """The last block's output, or None where the parts have to run themselves (shapes that take other kernels)."""
        first = self.blocks[0]
        s, ff = first.mixer.spec, first.feed_forward.spec
        if x.dim() != 2 or x.shape[0] == 0 or not _lies(x, x.dtype, (x.shape[0], s.hidden_size)) or x.data_ptr() % 16:
            return None
        if s.hidden_size % 8 or s.q_size % 8 or ff.intermediate_size % 8:
            return None
        if not all(_lies(t, torch.int32, (t.numel(),)) for t in (step.positions, step.token_seq)):
            return None
        # what the parts' own calls look at: an operand that is not as the kernels read it is left to them to refuse
        kind, real = x.dtype, torch.float32
        hidden, inter, packed = s.hidden_size, ff.intermediate_size, s.q_size + 2 * s.kv_size
        of_qkv, of_o, of_gate_up, of_down = (packed, hidden), (hidden, s.q_size), (2 * inter, hidden), (hidden, inter)
        rows, page = [], 0
        for entry in self.execution:
            block, view = self.blocks[entry.layer], step.cache_view(entry)
            m, f, kv, table, r = block.mixer, block.feed_forward, view.kv, view.block_table, block.mixer._rotation
            if kv is None or kv.dim() != 5 or table is None or table.dim() != 2:
                return None
            page = page or kv.shape[3]
            if not (_lies(m.w_qkv, kind, of_qkv) and _lies(m.w_o, kind, of_o) and _lies(f.w_gate_up, kind, of_gate_up)
                    and _lies(f.w_down, kind, of_down) and _lies(block.mixer_norm.weight, real, (hidden,))
                    and _lies(block.feed_forward_norm.weight, real, (hidden,)) and _lies(table, torch.int32, table.shape)
                    and _lies(kv, kind, (2, kv.shape[1], s.num_kv_heads, page, s.head_dim))
                    and (m.b_qkv is None or _lies(m.b_qkv, real, (packed,))) and (m.b_o is None or _lies(m.b_o, real, (hidden,)))
                    and (m.q_norm is None or _lies(m.q_norm, real, (s.head_dim,)))
                    and (m.k_norm is None or _lies(m.k_norm, real, (s.head_dim,)))):
                return None
            if r is not None:
                t = r.inv_freq if r.inv_freq is not None else r.cos_sin
                if not _lies(t, real, t.shape):
                    return None
            row = (m.w_qkv.data_ptr(), _at(m.b_qkv), m.w_o.data_ptr(), _at(m.b_o), _at(m.q_norm), _at(m.k_norm),
                   _at(r.inv_freq) if r is not None else 0, _at(r.cos_sin) if r is not None else 0, block.mixer_norm.weight.data_ptr(),
                   block.feed_forward_norm.weight.data_ptr(), f.w_gate_up.data_ptr(), f.w_down.data_ptr(), kv.data_ptr(),
                   table.data_ptr(), table.shape[1], kv.shape[1], int(m.spec.window or 0), int(view.writes))
            if (row[0] | row[2] | row[8] | row[9] | row[10] | row[11] | row[12]) % 16:
                return None
            rows.append(row)
        if not ops.attention_shape_ok(x.dtype, s.num_heads, s.num_kv_heads, s.head_dim, page):
            return None
        return ops.dense_stack(
            x, rows, step, heads=s.num_heads, kv_heads=s.num_kv_heads, head_dim=s.head_dim, inter=ff.intermediate_size,
            activation=ff.activation, page_size=page, scale=s.scale, rotation=first.mixer._rotation,
            eps=(first.mixer_norm.spec.eps, first.feed_forward_norm.spec.eps, s.qk_norm.eps if s.qk_norm is not None else 0.0))


def _lies(t: torch.Tensor, kind: torch.dtype, shape) -> bool:
    """Whether the kernels can read ``t`` as it lies: on the GPU, of this type and shape, without gaps."""
    return t.is_cuda and t.dtype is kind and t.is_contiguous() and t.shape == shape


def _at(t: Optional[torch.Tensor]) -> int:
    return 0 if t is None else t.data_ptr()
