"""Choice of the tensor-core matrix product for bfloat16 operands.

``plan(linear)`` returns a callable ``(out, x, defer) -> True | Partial | False``
that runs the tcgen05 kernel, or returns False, having launched nothing, when
the call's sizes are ones that kernel refuses (the caller then uses the generic
kernel), or None when the weight can never go that way (depth not a multiple
of 8: a TMA row must start on a 16-byte boundary).

Tokens per CTA and the number of k-splits are chosen from the token count and
the weight's shape so that even a handful of decode tokens pulls the weight
through most of the 148 SMs; the split partial sums are added in a fixed
order, so a given (tokens, weight) pair always sums the same way."""
from __future__ import annotations

import os
from functools import lru_cache

import torch

from ..csrc import ops
from ..errors import AlofaError

SMS = 148  # streaming multiprocessors the grids are sized for: a B200's, replaced by the device's own count at first use
K_SLICE = 64
_asked_device = False


def _sms_of_device(device) -> None:
    """The tile and split choices below fill the GPU once: they go by the
    number of SMs the device reports."""
    global SMS, _asked_device
    if not _asked_device and device.type == "cuda":
        _asked_device = True
        SMS = torch.cuda.get_device_properties(device).multi_processor_count


def _tile(tokens: int, features: int, gated: bool) -> int:
    """The kernel's tile argument.  Positive: weights on the M side of the MMA
    with that many tokens per CTA (decode: few tokens, weights streamed).
    Negative: tokens on the M side (128 per CTA) with that many weight rows
    per MMA (prompt portions: an MMA of M = 128 costs the same for any N up to
    256, so wide feature tiles are what pays)."""
    for bn in (16, 32, 64):
        if tokens <= bn:
            # a very tall weight (an output head) fills the GPU several times over
            # either way; wide tiles with the tokens on the M side stream it faster
            if not gated and -(-features // 128) > 4 * SMS:
                return -256
            return bn
    if gated:
        return -256  # 128 gate rows and their 128 up rows
    # narrow outputs: 128-wide tiles keep more SMs busy
    return -128 if -(-features // 256) * -(-tokens // 128) < SMS else -256


def _ctas(tokens: int, features: int, tile: int, gated: bool) -> int:
    if tile > 0:
        return -(-features // 128) * -(-tokens // tile)
    per_cta = -tile // 2 if gated else -tile
    return -(-features // per_cta) * -(-tokens // 128)


def _splits(ctas: int, depth: int, deferrable: bool = False) -> int:
    slices = -(-depth // K_SLICE)
    if slices < 2:
        return 1
    if ctas >= SMS // 2:
        # a deep product that does not fill the GPU once: two halves of the depth
        # side by side, when the consumer adds the halves up for free
        return 2 if deferrable and ctas < SMS and slices >= DEEP_SLICES else 1
    return max(1, min(slices, SMS // ctas))


PAIR_ROWS = 256  # tokens and weight rows of a tile of the kernel on pairs of CTAs
SLICE_PAYS_FOR = 135_000  # sums written and read again for a k-slice less of the busiest SM's work
MOST_PARTS = 4   # of the depth that such a product may leave to its consumer
DEEP_SLICES = 32  # k-slices from which a product's depth goes in halves, or on pairs in parts, for a consumer that adds them up
PAIRS_ALLOWED = os.environ.get("ALOFA_GEMM_PAIR", "1") != "0"


def _pair_splits(tokens: int, features: int, depth: int, gated: bool, deferrable: bool) -> int:
    """Into how many parts the depth of a prompt portion's product goes on the
    kernel that runs on pairs of CTAs; 0: it runs on another kernel.

    Undivided: wide products with more tiles than SMs even of one CTA each,
    and deep: 2,048 tokens, depth 3,584 x 37,888 weight rows 477 against 540 us
    on single CTAs, depth 1,536 x 17,920 rows 85 against 92 us; at depth 896 the
    pair's epilogue is not hidden behind its shorter MMA phase (9,728 rows: 33.9
    against 32.7 us).  In up to four parts, added up by the consumer: deep, narrow
    products, whose tiles of 256 x 256 leave most of the pairs idle or a last
    round nearly empty, where that takes a quarter off the busiest pair's work
    and seven of ten pairs have some.  Depth 8,960 x 1,536 rows, us on single
    CTAs (with their own splits) and in parts on pairs: 532 tokens 34.1 and 20.4,
    905 tokens 36.3 and 24.4, 2,048 tokens 68.1 and 46.5; depth 4,864 x 896 rows,
    905 tokens 21.2 and 14.7, 2,048 tokens 23.4 and 21.0, but 532 tokens, 48
    tiles on 74 pairs, 13.1 and 13.8; depth 18,944 x 3,584 rows, 1,400 tokens
    216 and 172 - at 2,048 tokens a sixth less work for the busiest pair (242
    and 218) goes into writing and reading the parts.  A part more than the kernel
    that would run otherwise leaves has to save the busiest SM a k-slice for every
    135,000 sums: with the norm after it, us otherwise and in parts, depth 3,584 x
    3,584 rows 532 tokens 33.3 and 37.5, 1,400 tokens 65.6 and 92.5; depth 2,048 x
    2,048 rows 257 tokens 20.7 and 22.5, 1,400 tokens 29.6 and 30.4; depth 18,944 x
    3,584 rows 532 tokens 93.1 and 101.1, but 700 tokens 152 and 102; with the
    rotate-and-store after it, depth 2,048 x 2,560 rows, 2,048 tokens 38.4 and 55.1."""
    if not PAIRS_ALLOWED or tokens <= 128 or features % 4:
        return 0
    undivided = 1 if depth >= 1024 and -(-features // (128 if gated else 256)) * -(-tokens // 128) > SMS else 0
    slices = -(-depth // K_SLICE)
    if gated or not deferrable or tokens <= 256 or slices < DEEP_SLICES:
        return undivided
    return _depth_parts(tokens, features, depth, undivided, SMS)


def owed_row_bytes(features: int, depth: int) -> int:
    """Scratch a token that a product called with ``defer`` may leave as fp32
    planes for its consumer, in steps whose rows alone fill the GPU (fewer rows
    in more parts are a few megabytes in all)."""
    return 4 * features * (MOST_PARTS if -(-depth // K_SLICE) >= DEEP_SLICES else 2)


@lru_cache(maxsize=1024)  # microseconds to work out, twice a layer of a step that is issued launch by launch
def _depth_parts(tokens: int, features: int, depth: int, undivided: int, sms: int) -> int:
    """The parts of a deferrable product's depth by :func:`_pair_splits`'s rule;
    ``undivided`` where none pay."""
    slices, pairs = -(-depth // K_SLICE), sms // 2
    tiles = -(-features // PAIR_ROWS) * -(-tokens // PAIR_ROWS)
    rounds = lambda s: -(-tiles * s // pairs) * -(-slices // s)  # k-slices that the busiest pair works through  # noqa: E731
    s = min(range(1, MOST_PARTS + 1), key=lambda s: (rounds(s), s))
    if 4 * rounds(s) > 3 * rounds(1) or 10 * tiles * s < 7 * pairs:
        return undivided
    # what it runs on otherwise: k-slices of the busiest pair, or of the busiest SM with up to two CTAs, and the planes left
    work, planes = rounds(1), 1
    if not undivided:
        ctas = _ctas(tokens, features, _tile(tokens, features, False), False)
        planes = _splits(ctas, depth, True)
        work = -(-slices // planes) * -(-ctas * planes // (2 * sms)) * (1.3 if ctas * planes > sms else 1.0)  # a slice of two CTAs takes 1.3 of one's
    return s if (work - rounds(s)) * SLICE_PAYS_FOR >= (s - planes) * tokens * features else undivided


def plan(linear):
    """The tensor-core product of ``linear``'s weight, or None."""
    w = linear.weight
    if linear.in_features % 8 or w.data_ptr() % 16:
        return None
    _sms_of_device(w.device)
    return TensorCoreProduct(linear)


class TensorCoreProduct:
    """What :func:`plan` returns.  It holds the weight and the numbers it goes
    by, not the :class:`~alofa_b200.parts.linear.Linear` that holds it: a
    dropped layer gives its weight back at once, not when the cycle collector
    next runs."""

    __slots__ = ("weight", "bias", "epi", "act", "gate", "depth", "out_features")

    def __init__(self, linear):
        self.weight, self.bias, self.epi, self.act, self.gate = linear.weight, linear.bias, linear.epi, linear.act, linear.gate
        self.depth, self.out_features = linear.in_features, linear.out_features

    def weights_on_m(self, tokens: int) -> bool:
        return _tile(tokens, self.out_features, self.epi == ops.EPI_GATED) > 0

    def __call__(self, out, x, defer: bool = False, buf=None, acc=None):
        from .linear import ACCUMULATED, Partial

        w, depth, features = self.weight, self.depth, self.out_features
        gated = self.epi == ops.EPI_GATED
        n_acc = 2 if gated else 1
        tokens = x.shape[0]
        if tokens == 0:
            return True
        bn = _tile(tokens, features, gated)
        lazy = None if isinstance(x, torch.Tensor) else x
        if lazy is not None:
            x = None
        deferrable = defer and n_acc == 1 and not self.act
        pair = _pair_splits(tokens, features, depth, gated, deferrable) if bn < 0 else 0
        bn = -PAIR_ROWS if pair else bn
        splits = ops.gemm_tc_splits(depth, pair or _splits(_ctas(tokens, features, bn, gated), depth, deferrable))
        computed = None
        if lazy is not None:
            # Rows still to be made.  The weights-on-M kernel makes them as it loads, a k-slice at a
            # time and each a trip to L2: worth it while a CTA has a few slices, else they are made first.
            per_cta = -(-(-(-depth // K_SLICE)) // splits)
            kind = getattr(lazy, "kind", "merged")
            if kind == "merged" and bn == 16 and self.epi == ops.EPI_RESIDUAL and per_cta <= 2 and lazy.fits_kernel():
                computed = lazy.computed()
            elif kind == "normed" and bn == 16 and gated and splits <= 8 and per_cta <= 6 and lazy.fits_kernel():
                computed = lazy.computed()  # the norm folded into a gated product whose splits are one cluster
            else:
                x = lazy.rows()
        if x is not None and (x.data_ptr() % 16 or not x.is_contiguous()):
            return False
        normed = computed is not None and computed[0] == ops.B_NORMED
        partial = None
        if splits > 1 and acc is None and not normed:
            shape = (splits * n_acc, tokens, features)
            partial = buf(shape, torch.float32) if buf is not None else torch.empty(shape, dtype=torch.float32, device=w.device)
        deferred = defer and splits > 1 and n_acc == 1 and acc is None and not self.act  # whoever adds deferred sums up applies no activation
        dst = partial[0] if deferred else out  # a deferred product writes partial sums only
        if not ops.gemm_tc(dst, x, w, self.bias, self.epi, bn, splits, partial, reduce=not deferred, computed=computed, acc=acc, act=self.act, gate=self.gate, pair=pair > 0):
            if normed:
                lazy.undo()
                return self(out, lazy.rows(), defer, buf)
            if computed is not None or acc is not None:
                raise AlofaError("state", "the tensor-core product refused an operand it had accepted")
            return False
        if normed:
            lazy.done(computed)
        if acc is not None:
            return ACCUMULATED
        return Partial(partial, splits, self.bias) if deferred else True
