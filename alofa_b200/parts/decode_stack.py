"""All layers of a small decode step as one persistent kernel.

A decode step of up to eight requests (one token each) through a stack of
pre-norm layers - grouped-query attention over pages, rotation of whole heads,
a silu-gated feed-forward - runs in ``ops.decode_stack``: one CTA per SM works
through all layers, weights streaming ahead of the phases that wait for one
another.  :meth:`DecodeStack.build` says whether a model's layers are of that
form, :meth:`DecodeStack.takes` whether a step is; every other model and step
goes layer by layer.  (The order of a layer:
src/alofa/model/arch/qwen.mojo:1367-1510.)"""
from __future__ import annotations

from typing import Optional

import torch

from ..cache.storage import LayerCache
from ..csrc import ops
from .attention import GQAttention
from .block import PrenormResidual
from .feed_forward import GatedMLP
from .norm import RMSNorm
from .position import RotaryNeox


class DecodeStack:
    # Steps this kernel is the faster way for: as many numbers of the stream as every SM can read before each product.  us a pass of four
    # steps, layer by layer and here: hidden 896, 3 tokens 2,748 and 2,535; hidden 1,536, 1 token 4,955 and 4,602, 4 tokens 5,207 and
    # 4,855, 8 tokens 5,414 and 5,387; hidden 3,584, 1 token 12,682 and 11,118, 4 tokens 12,890 and 11,836, 6 tokens 12,974 and 13,015.
    MOST_NUMBERS = 16384

    def __init__(self, model, caches: dict, block_size: int):
        self.model = model
        block = model.layers[model.run[0][0]]
        mixer = block.mixer
        self.sizes = (block.mixer_norm.size, mixer.nh, mixer.nkv, mixer.hd, block.feed_forward.inter)
        self.page = block_size
        self.scale = mixer.scale
        self.group = caches[model.run[0][1]].group
        self.caches = caches
        self.ctas = None  # by tokens, 0 where the kernel does not take a step; worked out at the first step it may be for
        self.described = None  # the tensors whose addresses the table holds

    def _open(self) -> None:
        """Asks the kernel what it takes and makes its scratch (a runner that never decodes a few tokens loads no library for it)."""
        block, device = self.model.layers[self.model.run[0][0]], self.model.rt.device
        mixer = block.mixer
        self.ctas = [0] + [ops.decode_stack_ctas(n, *self.sizes, self.page) for n in range(1, ops.DECODE_STACK_TOKENS + 1)]
        if not any(self.ctas):
            return
        # the kernel's own scratch: rotated queries, the key splits' outputs, the activation; and its barrier word
        most = max(n for n, c in enumerate(self.ctas) if c)
        ctas = max(self.ctas)
        self.q = torch.empty((most, mixer.q_dim), dtype=torch.bfloat16, device=device)
        self.act = torch.empty(ops.decode_stack_act_numbers(most, block.feed_forward.inter, ctas), dtype=torch.bfloat16, device=device)
        self.part_o = torch.empty((ctas, 8, mixer.hd), dtype=torch.float32, device=device)
        self.part_ml = torch.empty((ctas, 8, 2), dtype=torch.float32, device=device)
        self.barrier = torch.zeros(32, dtype=torch.int32, device=device)

    def _tensors(self) -> list:
        """Per run entry the tensors that the kernel reads and writes in place."""
        out = []
        for layer, cache in self.model.run:
            block, kv = self.model.layers[layer], self.caches[cache]
            out.append((block.mixer.qkv.weight, block.mixer.out.weight, block.feed_forward.gate_up.weight, block.feed_forward.down.weight, block.mixer_norm.weight, block.feed_forward_norm.weight,
                        block.mixer.qkv.bias, kv.k, kv.v))
        return out

    def _describe(self) -> None:
        """The kernel's table of layers, made again if the model was loaded again."""
        now = self._tensors()
        if self.described is not None and all(a is b for old, new in zip(self.described, now) for a, b in zip(old, new)):
            return
        blocks = [self.model.layers[layer] for layer, _ in self.model.run]
        entries = [ops.decode_stack_layer(*tensors, block.mixer_norm.eps, block.feed_forward_norm.eps, *self.sizes) for tensors, block in zip(now, blocks)]
        self.table = torch.frombuffer(bytearray(b"".join(entries)), dtype=torch.uint8).to(self.model.rt.device)
        self.rope = blocks[0].mixer.position.rotary_table()[0]
        self.described = now

    @staticmethod
    def fits(model, caches: dict) -> bool:
        """Whether the model's layers are of the form the kernel has."""
        if model.rt.dtype != torch.bfloat16 or model.stream_copies or model.keeps_embedding or model.shared_value_width:
            return False
        shapes = set()
        for i, (layer, cache) in enumerate(model.run):
            block = model.layers[layer]
            if type(block) is not PrenormResidual or type(block.mixer) is not GQAttention or type(block.feed_forward) is not GatedMLP:
                return False
            mixer, ff = block.mixer, block.feed_forward
            if mixer.qkv is None or ff.gate_up is None:
                return False  # not loaded yet
            norms = (block.mixer_norm, block.feed_forward_norm)
            if any(type(n) is not RMSNorm or n.spec.kind != "rmsnorm" or n.shift is not None for n in norms) or type(mixer.position) is not RotaryNeox:
                return False
            if cache != i or not isinstance(caches.get(cache), LayerCache) or mixer.window or mixer.out.bias is not None or ff.down.bias is not None or ff.gate_up.bias is not None:
                return False
            table, rot = mixer.position.rotary_table()
            if rot != mixer.hd or ff.gate_up.gate != ops.SILU_GATE:
                return False
            weights = (mixer.qkv.weight, mixer.out.weight, ff.gate_up.weight, ff.down.weight)
            if any(w.dtype != torch.bfloat16 or w.data_ptr() % 16 for w in weights):
                return False
            shapes.add((norms[0].size, norms[1].size, mixer.hidden, ff.hidden, mixer.nh, mixer.nkv, mixer.hd, ff.inter, mixer.scale, table.data_ptr(), caches[cache].group, tuple(caches[cache].k.shape)))
        return len(shapes) == 1 and model.spec.hidden_size == next(iter(shapes))[0]

    @classmethod
    def build(cls, model, caches: dict, block_size: int) -> Optional["DecodeStack"]:
        """The stack of a loaded model over one runner's caches, or None where
        the model's layers or sizes are not ones the kernel takes."""
        if model.rt.device.type != "cuda" or not cls.fits(model, caches):
            return None
        return cls(model, caches, block_size)

    def takes(self, ctx, h) -> bool:
        n = ctx.n_tokens
        if not ctx.decode_only or n > ops.DECODE_STACK_TOKENS or n * self.sizes[0] > self.MOST_NUMBERS or ctx.stream_of(h) is None:
            return False
        if self.ctas is None:
            self._open()
        return self.ctas[n] > 0

    def forward(self, ctx, h) -> None:
        """The step's rows through all layers: what the last product added to
        ``h`` is left in the stream's accumulator."""
        self._describe()
        alt, acc, other = ctx.stream_buffers(h)
        group = ctx.groups[self.group]
        ops.decode_stack(self.table, len(self.model.run), self.ctas[ctx.n_tokens], self.sizes, self.page, self.scale, h, alt, acc, other, ctx.positions, group.block_table, group.slot_map, self.rope,
                         self.q, self.part_o, self.part_ml, self.act, self.barrier, ctx.status)
        ctx.owe_accumulator(h)

    def reset(self) -> None:
        """After a kernel gave up: its barrier may stand half way."""
        if self.ctas is not None and any(self.ctas):
            self.barrier.zero_()
