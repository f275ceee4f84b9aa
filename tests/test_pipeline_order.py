"""CPU: the happens-before order that protects the small rings in shared memory (gather modes of csrc/attn_pair.cu and of
csrc/attn_rows64.cu): the tokens' validity bits, written by the copy or look-up warps and read by the softmax warps, and in FP8 decode
on pairs of SMs the tokens' addresses, read by the converting warps.  Nobody arrives on a barrier of their own for the validity bits, so an
entry may only be overwritten where the chain of the other barriers already orders its last reader before the writer.

The roles' program order and the barriers between them are written down as a graph; the ring depths, and on which side of
the arrival that gives the S accumulator back the softmax warps read the mask, come from the source."""
import os
import re

import pytest

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flashmla_b200", "csrc", "attn_pair.cu")


def _plan():
    text = open(SOURCE).read()
    slots, tables = (int(re.search(r"\b" + name + r" = (\d+)[,;]", text).group(1)) for name in ("NSLOT", "NTAB"))
    assert "uint32_t mask[2 * NTAB][4];" in text and len(re.findall(r"sm\.mask\[\(?g(?: \+ i\))? % \(2 \* NTAB\)\]", text)) == 3
    read = text.index("sm.mask[g % (2 * NTAB)][quarter]")
    return slots, 2 * tables, tables, read < text.index("mbar_arrive_remote_cta(s_empty)")


def _graph(tiles, slots, tables, convert, read_first):
    """edges[event] = the events that directly precede it; events are (role, what, tile, slot of the tile)."""
    edges = {}

    def program(role, steps):
        for i, step in enumerate(steps):
            edges.setdefault((role,) + step, [])
            if i:
                edges[(role,) + step].append((role,) + steps[i - 1])

    four = range(4)
    if convert:
        program("look-up", [("meta", g, 0) for g in range(tiles)])
    # a tile's own page, then the other page of the tile before
    meta = lambda g: [("own", g, 0)] if convert else [("meta", g, 0)]
    feed = [s for g in range(tiles) for s in meta(g) + [("fill", g, q) for q in four] + ([("other", g - 1, 0)] if g else []) + [("done", g, 0)]]
    program("feed", feed)
    # (Q K^T of a tile may come before or behind P V of the one before, not earlier)
    program("scores", [("scores", g, q) for g in range(tiles) for q in four])
    program("values", [("values", g, q) for g in range(tiles) for q in four])
    softmax = lambda g: [("mask", g, 0), ("give", g, 0)] if read_first else [("give", g, 0), ("mask", g, 0)]
    program("softmax", [s for g in range(tiles) for s in [("start", g, 0)] + softmax(g) + [("p", g, 0)]])
    for g in range(tiles):
        for q in four:
            f = 4 * g + q
            if f >= slots:                                                                      # empty: P V that read the slot
                edges["feed", "fill", g, q].append(("values", "values", (f - slots) // 4, (f - slots) % 4))
            edges["scores", "scores", g, q].append(("feed", "fill", g, q))                      # full
            edges["values", "values", g, q] += [("softmax", "p", g, 0)] + ([("feed", "other", g, 0)] if g + 1 < tiles else [])    # p_full
            edges["values", "values", g, q].append(("scores", "scores", g, 3))
        if g >= 1:
            edges["scores", "scores", g, 0].append(("softmax", "give", g - 1, 0))               # s_empty
            edges["feed", "other", g - 1, 0].append(("scores", "scores", g - 1, 3))             # k_done
        if g >= 2:
            edges["scores", "scores", g, 0].append(("values", "values", g - 2, 3))              # the issuing thread's order
        edges["softmax", "start", g, 0].append(("scores", "scores", g, 3))                      # s_full
        if convert:
            edges["feed", "own", g, 0].append(("look-up", "meta", g, 0))                        # tab_full
            if g >= tables:
                edges["look-up", "meta", g, 0].append(("feed", "done", g - tables, 0))          # tab_empty
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
    slots, masks, tables, read_first = _plan()
    tiles = masks + 8
    edges = _graph(tiles, slots, tables, convert, read_first)
    writer = "look-up" if convert else "feed"
    for g in range(tiles - masks):
        assert _before(edges, (writer, "meta", g, 0), ("softmax", "mask", g, 0)), "a mask is read after it was written"
        assert _before(edges, ("softmax", "mask", g, 0), (writer, "meta", g + masks, 0)), "... and before its entry is written again"
    if convert:
        for g in range(tiles - tables):
            assert _before(edges, ("look-up", "meta", g, 0), ("feed", "own", g, 0))
            assert _before(edges, ("feed", "done", g, 0), ("look-up", "meta", g + tables, 0))


def test_the_check_sees_a_missing_order():
    """The same graph has no such order with rings of half the depth, nor for the table's entries where a mask of that depth would do."""
    slots, masks, tables, _ = _plan()
    good = _graph(masks + 8, slots, tables, True, True)
    assert not _before(good, ("softmax", "mask", 3, 0), ("look-up", "meta", 3 + tables // 2, 0))
    assert not _before(good, ("feed", "done", 3, 0), ("look-up", "meta", 3 + tables // 2, 0))
    assert not _before(_graph(masks + 8, slots, tables, False, True), ("softmax", "mask", 3, 0), ("feed", "meta", 3 + 2, 0))


# ---- bounded waits in the warps that meet at a named barrier ----------------------------------------------------------
def _softmax_steps(path):
    """What the softmax role of a kernel does in program order: ("wait", text), ("leave", text): a thread or warp leaves the role by itself,
    ("barrier", all leave): the 256 threads meet, and leave together where one says so."""
    text = open(path).read()
    start = max(m.start() for m in re.finditer(r"// -+ softmax", text))
    role = re.sub(r"//[^\n]*", "", text[start:text.index("wind_down:", start)])
    steps = []
    for m in re.finditer(r"BAR_OR_LEAVE\(wt\.expired\(\)\)|named_bar_red_or\(1, 256, [^;]*;|named_bar_sync\(1, 256\)|"
                         r"WAIT_(?:WARP_)?OR_LEAVE\([^;]*;|wt\.template wait\w*<\w+>\([^;]*;|goto wind_down", role):
        step = m.group()
        if "bar" in step.lower().split("(")[0]:
            steps.append(("barrier", "BAR_OR_LEAVE" in step or "goto wind_down" in step))
        elif step == "goto wind_down":
            steps.append(("leave", step))
        else:
            steps += [("wait", step)] + [("leave", step)] * step.startswith("WAIT_")
    return steps


@pytest.mark.parametrize("path", [SOURCE, ROWS64])
def test_softmax_threads_leave_together(path):
    """The 256 softmax threads meet at a named barrier that has no limit of its own.  So a thread whose wait ran out, while another one's
    did not, must walk on to the next barrier that tells them all."""
    steps = _softmax_steps(path)
    waits = [i for i, step in enumerate(steps) if step[0] == "wait"]
    assert len(waits) == (5 if path == SOURCE else 2)
    for i in waits:
        after = [step for step in (steps + steps)[i + 1:] if step != ("barrier", False)]          # (the role is a loop)
        assert after[0][0] == "wait" or after[0] == ("barrier", True), (steps[i], after[0])
