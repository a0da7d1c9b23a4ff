"""All layers of a small decode step as one persistent kernel.

A decode step of up to eight requests (one token each) through a stack of
pre-norm layers - grouped-query attention over pages, rotation of whole heads,
a silu-gated feed-forward - runs in ``ops.decode_stack``: one CTA per SM works
through all layers, weights streaming ahead of the phases that wait for one
another.  :meth:`DecodeStack.build` says whether a model's layers may be of that
form, :meth:`DecodeStack.takes` whether a step is; every other model and step
goes layer by layer.  (The order of a layer:
src/alofa/model/arch/qwen.mojo:1367-1510.)"""
from __future__ import annotations

from dataclasses import dataclass
from typing import Optional

import torch

from ..cache.storage import LayerCache
from ..csrc import ops
from . import fast_linear
from .attention import GQAttention
from .block import PrenormResidual
from .feed_forward import GatedMLP
from .linear import GATED, RESIDUAL, STORE
from .norm import RMSNorm
from .position import RotaryNeox


@dataclass(frozen=True)
class Form:
    """All that the kernel's table and launch go by, as numbers: two equal
    ones describe the same step.  Nothing of a model is kept alive by it."""

    sizes: tuple  # hidden, heads, kv heads, head size, intermediate
    scale: float
    group: int
    rope: int  # the rotary table's address
    layers: tuple  # per run entry the addresses of its weights, vectors and caches, and the norms' eps


GRANULE, WARPS = 16, 16  # keys a warp takes at a time, warps of a CTA


def keys_per_cta_fit(lengths: list, kv_heads: int, ctas: int, most: int) -> bool:
    """Whether requests of these lengths leave no CTA a split of more than
    ``most`` granules, and, where a warp takes more than one, none of more than
    five fourths of what even shares would be.  The kernel's own division: the
    smallest splits of which all are resident together, a granule a warp at least."""
    granules = [-(-n // GRANULE) for n in lengths]
    total = sum(granules) * kv_heads
    per = max(WARPS, -(-total // ctas))
    while per <= most and sum(-(-g // per) for g in granules) * kv_heads > ctas:
        per += 1
    return per <= most and (per == WARPS or 4 * per * ctas <= 5 * total)


class DecodeStack:
    # Steps this kernel is the faster way for: as many numbers of the stream as every SM can read before each product (us a decode step at
    # 128 tokens of context, layer by layer and here: hidden 896, 1 token 590 and 542, 8 tokens 664 and 616; hidden 1,536, 1 token 1,112 and
    # 1,054, 8 tokens 1,201 and 1,186; hidden 3,584, 4 tokens 2,959 and 2,744, 5 tokens 2,975 and 2,933, 6 tokens more than layer by layer; hidden
    # 2,560, 6 tokens 695 and 684, 8 tokens 695 and 735) ...
    MOST_NUMBERS = 16384
    # ... and as many keys as the SMs get through in a few trips.  A CTA has one split of one (request, KV head) pair's keys, a warp of it 16
    # keys at a time with none on their way behind them: up to 16 granules of 16 keys a split one trip, with twice that two.  Beyond, the
    # kernels of a layer read faster (6 TB/s; 3.6 here with heads of 64, 4.4 with 128): hidden 896 (2 KV heads), 8 requests of 4,096 tokens
    # (29 granules) 742 and 711, of 8,192 (57) 805 and 822, of 32,768 1,198 and 1,515; hidden 1,536, 4 of 8,192 (29) 1,379 and 1,354, 8 of
    # 8,192 (57) 1,522 and 1,661.  A model whose layers are many rings of weights gains more by the rest: hidden 3,584, 1 of 32,768 (56) 3,465
    # and 3,159, 4 of 8,192 (57) 3,367 and 3,299, 4 of 32,768 (228) 4,207 and 4,506.
    MOST_GRANULES, MOST_GRANULES_WIDE, WIDE_BYTES = 32, 64, 1 << 28
    # More than one trip only where the splits keep the SMs busy, a quarter more than with keys dealt evenly at most: 16 KV heads of 64,
    # 8 requests of 512 tokens (128 CTAs of 32 granules where 28 would be even) 381 and 370, 5 of 512 (80 CTAs, 17) 366 and 383.

    def __init__(self, model, caches: dict, block_size: int):
        self.model = model
        self.caches = caches
        self.page = block_size
        self.form = None  # what the table and the scratch below were made for
        self.ctas = [0] * (ops.DECODE_STACK_TOKENS + 1)  # by tokens, 0 where the kernel does not take a step
        self.sms = torch.cuda.get_device_properties(model.rt.device).multi_processor_count if model.rt.device.type == "cuda" else fast_linear.SMS

    def look(self) -> Optional[Form]:
        """The model as it is loaded now, None where its layers are not of the
        form the kernel has (or not loaded).  Looked at anew for every step
        that is not a replay: a model may be loaded again."""
        model, caches = self.model, self.caches
        if model.rt.dtype != torch.bfloat16 or model.stream_copies or model.keeps_embedding or model.shared_value_width:
            return None
        shapes, layers, bf16, fp32, cuda = set(), [], torch.bfloat16, torch.float32, model.rt.device.type == "cuda"
        for i, (layer, cache) in enumerate(model.run):
            block = model.layers[layer]
            if type(block) is not PrenormResidual or type(block.mixer) is not GQAttention or type(block.feed_forward) is not GatedMLP or type(block.mixer.position) is not RotaryNeox:
                return None
            mixer, ff, norm_a, norm_b, kv = block.mixer, block.feed_forward, block.mixer_norm, block.feed_forward_norm, caches.get(cache)
            if cache != i or type(kv) is not LayerCache or mixer.window or type(norm_a) is not RMSNorm or type(norm_b) is not RMSNorm or norm_a.shift is not None or norm_b.shift is not None:
                return None
            table, rot = mixer.position.rotary_table()
            qkv, out, gate_up, down = mixer.qkv, mixer.out, ff.gate_up, ff.down
            if qkv is None or out is None or gate_up is None or down is None or table is None or norm_a.weight is None or norm_b.weight is None:
                return None  # not loaded yet
            if (qkv.epi, out.epi, gate_up.epi, down.epi) != (STORE, RESIDUAL, GATED, RESIDUAL) or qkv.act or gate_up.gate != ops.SILU_GATE:
                return None
            if out.bias is not None or gate_up.bias is not None or down.bias is not None or rot != mixer.hd:
                return None
            hidden, rows, q_dim, inter = mixer.hidden, mixer.q_dim + 2 * mixer.kv_dim, mixer.q_dim, ff.inter
            bias, k, v = qkv.bias, kv.k, kv.v
            tensors = (qkv.weight, out.weight, gate_up.weight, down.weight, k, v, norm_a.weight, norm_b.weight) + (() if bias is None else (bias,))
            if v is None or [t.shape for t in tensors] != [(rows, hidden), (hidden, q_dim), (2 * inter, hidden), (hidden, inter), *[(k.shape[0], mixer.nkv, mixer.hd)] * 2, (hidden,), (hidden,), (rows,)][: len(tensors)]:
                return None
            at = [t.data_ptr() for t in tensors if t.dtype == (bf16 if t.dim() > 1 else fp32) and t.is_contiguous() and t.is_cuda == cuda]
            if len(at) != len(tensors) or any(a % 16 for a in at):
                return None
            shapes.add((hidden, mixer.nh, mixer.nkv, mixer.hd, inter, mixer.scale, table.data_ptr(), kv.group, k.shape[0]))
            layers.append((*at, norm_a.eps, norm_b.eps))
        if len(shapes) != 1:
            return None
        *sizes, scale, rope, group, _ = shapes.pop()
        return Form(tuple(sizes), scale, group, rope, tuple(layers)) if sizes[0] == model.spec.hidden_size else None

    def _open(self, form: Form) -> None:
        """Asks the kernel what it takes, makes its scratch and its table of
        layers (a runner that never decodes a few tokens loads no library for it)."""
        device, before = self.model.rt.device, self.form
        self.form = None
        if before is None or before.sizes != form.sizes:
            self.ctas = [0] + [ops.decode_stack_ctas(n, *form.sizes, self.page) for n in range(1, ops.DECODE_STACK_TOKENS + 1)]
            if any(self.ctas):
                # the kernel's own scratch: rotated queries, the key splits' outputs, the activation; and its barrier word
                _, heads, _, hd, inter = form.sizes
                most, ctas = max(n for n, c in enumerate(self.ctas) if c), max(self.ctas)
                self.q = torch.empty((most, heads * hd), dtype=torch.bfloat16, device=device)
                self.act = torch.empty(ops.decode_stack_act_numbers(most, inter, ctas), dtype=torch.bfloat16, device=device)
                self.part_o = torch.empty((ctas, 8, hd), dtype=torch.float32, device=device)
                self.part_ml = torch.empty((ctas, 8, 2), dtype=torch.float32, device=device)
                self.barrier = torch.zeros(32, dtype=torch.int32, device=device)
        if any(self.ctas):
            entries = []
            for layer, cache in self.model.run:
                block, kv = self.model.layers[layer], self.caches[cache]
                mixer, ff = block.mixer, block.feed_forward
                entries.append(ops.decode_stack_layer(mixer.qkv.weight, mixer.out.weight, ff.gate_up.weight, ff.down.weight, block.mixer_norm.weight, block.feed_forward_norm.weight, mixer.qkv.bias,
                                                      kv.k, kv.v, block.mixer_norm.eps, block.feed_forward_norm.eps, *form.sizes))
            self.table = b"".join(entries)
        self.form = form

    @classmethod
    def build(cls, model, caches: dict, block_size: int) -> Optional["DecodeStack"]:
        """The stack of a model over one runner's caches, or None where the
        model's blocks are not ones the kernel could take.  (Whether they are is
        seen at a step: the model may be loaded, or loaded again, after this.)"""
        if model.rt.device.type != "cuda" or model.rt.dtype != torch.bfloat16 or not model.run or any(type(block) is not PrenormResidual for block in model.layers):
            return None
        return cls(model, caches, block_size)

    def reaches(self, ctx) -> bool:
        """Whether a step's tokens and keys are as few as this kernel is the
        faster way for: from its lengths alone, for recorded steps too (which
        are recorded apart by it)."""
        n = ctx.n_tokens
        if not ctx.decode_only or n > ops.DECODE_STACK_TOKENS or n * self.model.spec.hidden_size > self.MOST_NUMBERS:
            return False
        block = self.model.layers[self.model.run[0][0]]
        pairs, inter = getattr(block.mixer, "nkv", 0), getattr(block.feed_forward, "inter", 0)
        if not pairs or not inter:
            return False
        wide = 6 * self.model.spec.hidden_size * inter >= self.WIDE_BYTES  # the gate, up and down weights' bytes
        return keys_per_cta_fit(ctx.host_field("kv_len").tolist(), pairs, self.sms, self.MOST_GRANULES_WIDE if wide else self.MOST_GRANULES)

    def takes(self, ctx, h) -> bool:
        n = ctx.n_tokens
        if ctx.stream_of(h) is None or not self.reaches(ctx):
            return False
        form = self.look()
        if form is None:
            return False
        if form != self.form:
            self._open(form)
        return self.ctas[n] > 0

    def forward(self, ctx, h) -> None:
        """The step's rows through all layers (a step that :meth:`takes` has
        just said yes to): what the last product added to ``h`` is left in the
        stream's accumulator."""
        form = self.form
        alt, acc, other = ctx.stream_buffers(h)
        group = ctx.groups[form.group]
        rope = self.model.layers[self.model.run[0][0]].mixer.position.rotary_table()[0]
        ops.decode_stack(self.table, len(form.layers), self.ctas[ctx.n_tokens], form.sizes, self.page, form.scale, h, alt, acc, other, ctx.positions, group.block_table, group.slot_map, rope,
                         self.q, self.part_o, self.part_ml, self.act, self.barrier, ctx.status)
        ctx.owe_accumulator(h)
        ctx.keep += [rope, self.q, self.part_o, self.part_ml, self.act, self.barrier]  # a recording of this launch reads them at its replays

    def reset(self) -> None:
        """After a kernel gave up: its barrier may stand half way."""
        if any(self.ctas):
            self.barrier.zero_()
