"""CPU: the happens-before order that protects the small rings in shared memory (gather modes of csrc/attn_sm100.cu, score CTA, and of
csrc/attn_rows64.cu): the tokens' validity bits, written by the copy warps and read by the softmax warps, and in FP8 decode
on pairs of SMs the tokens' scales, read by the converting warps.  Nobody arrives on a barrier of their own for these rings, so an entry may
only be overwritten where the chain of the other barriers already orders its last reader before the writer.

The roles' program order and the barriers between them are written down as a graph; the ring depths, and on which side of
the arrival that gives the S accumulator back the softmax warps read the mask, come from the source."""
import os
import re

import pytest

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flashmla_b200", "csrc", "attn_sm100.cu")


def _plan():
    text = open(SOURCE).read()
    narrow = {name: int(re.search(name + r" = WIDE \? \d+ : (\d+);", text).group(1)) for name in ("NKS", "S_BUFS")}
    masks = [int(m) + 1 for m in re.findall(r"kmask\)?\[\(g & (\d)\)", text)] + [int(m) + 1 for m in re.findall(r"SC_MASK\) \+ \(g & (\d)\)", text)]
    scales = [int(m) + 1 for m in re.findall(r"SC_SCALES\)\[\(g & (\d)\)", text)]
    assert len(masks) == 3 and len(set(masks)) == 1 and len(scales) == 2 and len(set(scales)) == 1, (masks, scales)
    read = re.search(r"m0 = km\[0\]", text).start()
    give_back = text.index("mbar_arrive(smem_addr(&sm.s_empty[sb]))")
    return narrow["NKS"], narrow["S_BUFS"], masks[0], scales[0], read < give_back


def _graph(tiles, nks, s_bufs, convert, read_first):
    """edges[event] = the events that directly precede it; events are (role, what, tile, group)."""
    edges = {}

    def program(role, steps):
        for i, step in enumerate(steps):
            edges.setdefault((role,) + step, [])
            if i:
                edges[(role,) + step].append((role,) + steps[i - 1])

    groups = range(3)
    program("copy", [s for g in range(tiles) for s in [("meta", g, 0)] + [("fill", g, j) for j in groups]])
    program("mma", [s for g in range(tiles) for s in [("start", g, 0)] + [("group", g, j) for j in groups]])
    softmax = lambda g: [("mask", g, 0), ("give", g, 0)] if read_first else [("give", g, 0), ("mask", g, 0)]
    program("softmax", [s for g in range(tiles) for s in [("scores", g, 0)] + softmax(g)])
    if convert:
        program("convert", [("group", g, j) for g in range(tiles) for j in groups])
    for g in range(tiles):
        for j in groups:
            fill = 3 * g + j
            if fill >= nks:                                                                     # kv_empty: MMAs that read the slot
                edges["copy", "fill", g, j].append(("mma", "group", (fill - nks) // 3, (fill - nks) % 3))
            landed = ("copy", "fill", g, j)
            if convert:                                                                         # raw_full, then kv_full
                edges["convert", "group", g, j].append(landed)
                landed = ("convert", "group", g, j)
            edges["mma", "group", g, j].append(landed)
        if g >= s_bufs:
            edges["mma", "start", g, 0].append(("softmax", "give", g - s_bufs, 0))              # s_empty
        edges["softmax", "scores", g, 0].append(("mma", "group", g, 2))                         # s_full
    return edges


ROWS64 = os.path.join(os.path.dirname(SOURCE), "attn_rows64.cu")


def _plan64():
    """Pair slots of the gather modes' variants, depth of the ring of masks, whether the mask is read before P is handed over, and
    whether a mask is written behind the wait for the slot of its tile's first pair."""
    text = open(ROWS64).read()
    upto, narrow, wide = re.search(r"NP = NH <= (\d+) \? (\d+) : (\d+);", text).groups()
    slots = {int(narrow) if nh <= int(upto) else int(wide) for nh in (16, 64)}
    masks = {int(m) + 1 for m in re.findall(r"sm\.mask\[g & (\d)\]", text)}
    assert len(masks) == 1 and len(re.findall(r"sm\.mask\[g & ", text)) == 3
    read = text.index("(sm.mask[g & 1][wq] >> lane)")
    for write in re.finditer(r"sm\.mask\[g & 1\]\)\[fw\] = ", text):
        guard = text.rindex("if (q == 0 && lane == 0)", 0, write.start())
        wait = text.rindex("WAIT_WARP_OR_LEAVE(wt, false, &sm.k_empty[ring.slot]", 0, guard)
        assert "for (int q = 0; q < 4; ++q" in text[wait - 120:wait]
    return slots, masks.pop(), read < text.index("mbar_arrive(smem_addr(&sm.p_full))")


def _graph64(tiles, slots, read_first):
    """Roles of the kernel for up to 64 rows: pairs 0 .. 3 of a tile are filled, multiplied, and given back behind P V."""
    edges = {}

    def program(role, steps):
        for i, step in enumerate(steps):
            edges.setdefault((role,) + step, [])
            if i:
                edges[(role,) + step].append((role,) + steps[i - 1])

    pairs = range(4)
    program("feed", [s for g in range(tiles) for s in [("slot", g, 0), ("mask", g, 0)] + [("fill", g, q) for q in pairs]])
    program("mma", [s for g in range(tiles) for s in [("scores", g, q) for q in pairs] + [("values", g, q) for q in pairs]])
    mask = lambda g: [("mask", g, 0), ("p", g, 0)] if read_first else [("p", g, 0), ("mask", g, 0)]
    program("softmax", [s for g in range(tiles) for s in [("start", g, 0)] + mask(g)])
    for g in range(tiles):
        for q in pairs:
            f = 4 * g + q
            if f >= slots:                                                                      # k_empty: P V that read the slot
                edges["feed", "fill" if q else "slot", g, q].append(("mma", "values", (f - slots) // 4, (f - slots) % 4))
            edges["mma", "scores", g, q].append(("feed", "fill", g, q))                         # k_full
            edges["mma", "values", g, q].append(("softmax", "p", g, 0))                         # p_full
        edges["softmax", "start", g, 0].append(("mma", "scores", g, 3))                         # s_full
    return edges


def test_masks_of_the_kernel_for_64_rows():
    slots, masks, read_first = _plan64()
    assert slots == {4, 5}
    for n in slots:
        edges = _graph64(masks + 8, n, read_first)
        for g in range(8):
            assert _before(edges, ("feed", "mask", g, 0), ("softmax", "mask", g, 0)), "a mask is read after it was written"
            assert _before(edges, ("softmax", "mask", g, 0), ("feed", "mask", g + masks, 0)), "... and before its entry is written again"
        late = _graph64(masks + 8, n, False)
        assert not _before(late, ("softmax", "mask", 7, 0), ("feed", "mask", 8, 0))             # the check sees a missing order
    # with five slots a ring of one mask would not do
    assert not _before(_graph64(8, 5, read_first), ("softmax", "mask", 3, 0), ("feed", "mask", 4, 0))


def _before(edges, first, then):
    seen, todo = set(), [then]
    while todo:
        e = todo.pop()
        if e == first:
            return True
        if e not in seen:
            seen.add(e)
            todo.extend(edges[e])
    return False


@pytest.mark.parametrize("convert", [False, True])          # prefill, FP8 decode
def test_ring_entries_are_read_before_they_are_overwritten(convert):
    nks, s_bufs, masks, scales, read_first = _plan()
    tiles = masks + 8
    edges = _graph(tiles, nks, s_bufs, convert, read_first)
    for g in range(tiles - masks):
        assert _before(edges, ("copy", "meta", g, 0), ("softmax", "mask", g, 0)), "a mask is read after it was written"
        assert _before(edges, ("softmax", "mask", g, 0), ("copy", "meta", g + masks, 0)), "... and before its entry is written again"
    if convert:
        for g in range(tiles - scales):
            assert _before(edges, ("copy", "meta", g, 0), ("convert", "group", g, 0))
            assert _before(edges, ("convert", "group", g, 0), ("copy", "meta", g + scales, 0))


def test_the_check_sees_a_missing_order():
    """The same graph with the mask read behind the arrival, and with rings of half the depth, has no such order."""
    nks, s_bufs, masks, scales, _ = _plan()
    late = _graph(masks + 8, nks, s_bufs, True, False)
    assert not _before(late, ("softmax", "mask", 3, 0), ("copy", "meta", 3 + masks, 0))
    good = _graph(masks + 8, nks, s_bufs, True, True)
    assert not _before(good, ("softmax", "mask", 3, 0), ("copy", "meta", 3 + masks // 2, 0))
    assert not _before(good, ("convert", "group", 3, 0), ("copy", "meta", 3 + scales // 2, 0))
