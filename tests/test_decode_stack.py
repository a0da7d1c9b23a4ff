"""How the one-kernel decode step divides a layer's products: every weight row and column by exactly one warp, within the
matrices and within shared memory, over shapes with odd and even chunk counts, groups of one to eight and one to eight
tokens."""
import ctypes

import pytest

SHAPES = {
    "0.5b": (896, 14, 2, 64, 4864), "1.5b": (1536, 12, 2, 128, 8960), "7b": (3584, 28, 4, 128, 18944),
    "one_chunk": (64, 2, 1, 64, 64), "odd": (192, 3, 3, 64, 576), "wide_ff": (256, 8, 1, 64, 16384), "group7": (896, 7, 1, 128, 2432),
}
WARPS, LIMIT, MAX_TILES = 16, 232448, 64


def plan(tokens, shape, ctas):
    from alofa_b200.csrc import ops

    out = (ctypes.c_int * 23)()
    taken = ops._decode_stack().alofa_decode_stack_plan(tokens, *shape, ctas, out)
    return bool(taken), list(out)


def share(phase, tiles, slices, kg, rg, cta, ctas):
    """(tiles, slices) of a CTA, as the kernel deals them."""
    if kg == 0:
        c = ctas - 1 - cta if phase == 2 else cta
        return list(range(c, tiles, ctas)), list(range(slices))
    if cta >= kg * rg:
        return [], []
    k, g = cta % kg, cta // kg
    return list(range(g * tiles // rg, (g + 1) * tiles // rg)), list(range(k * slices // kg, (k + 1) * slices // kg))


@pytest.mark.parametrize("name", list(SHAPES))
@pytest.mark.parametrize("tokens", [1, 3, 4, 7, 8])
@pytest.mark.parametrize("ctas", [148, 132])
def test_products_are_covered_once(name, tokens, ctas):
    hidden, heads, kv_heads, hd, inter = SHAPES[name]
    taken, p = plan(tokens, SHAPES[name], ctas)
    if not taken:
        assert name == "7b" and tokens > 4, "only wide operands of many tokens leave no room"
        return
    chunks, slots, x_stride, x_bytes, work_bytes, smem = p[16:22]
    assert slots >= 2 and smem <= LIMIT and x_bytes >= tokens * x_stride
    sizes = [((heads + 2 * kv_heads) * hd, hidden), (hidden, heads * hd), (2 * inter, hidden), (hidden, inter)]
    for phase, (rows, cols) in enumerate(sizes):
        tiles, slices, kg, rg = p[4 * phase : 4 * phase + 4]
        assert slices * chunks * 64 == cols and tiles * 16 == rows
        seen, covered = set(), set()
        for cta in range(ctas):
            own, part = share(phase, tiles, slices, kg, rg, cta, ctas)
            if not own or not part:
                continue
            assert len(own) <= MAX_TILES and 2 * len(part) * chunks * 64 + 16 <= x_stride
            pieces = [(t, s) for t in own for s in part]
            warps = min(WARPS, len(pieces))
            entries = []
            for w in range(warps):
                for u in range(w * len(pieces) // warps, (w + 1) * len(pieces) // warps):
                    assert (warps * (u + 1) - 1) // len(pieces) == w  # how an epilogue finds the warps of a tile
                    entry = w + u // len(part)
                    if (w, u // len(part)) not in entries:
                        entries.append((w, u // len(part)))
                    assert (entry + 1) * 16 * 8 * 4 + x_bytes <= work_bytes
            assert len({w + t for w, t in entries}) == len(entries)
            assert not seen & set(pieces)
            seen |= set(pieces)
            for t in own:  # two groups of eight rows: halves of a rotated head, gate and up, or neighbours
                if phase == 0:
                    first, second = t // (hd // 16) * hd + t % (hd // 16) * 8, hd // 2
                else:
                    first, second = (8 * t, inter) if phase == 2 else (16 * t, 8)
                covered |= set(range(first, first + 8)) | set(range(first + second, first + second + 8))
        assert len(seen) == tiles * slices and covered == set(range(rows))
