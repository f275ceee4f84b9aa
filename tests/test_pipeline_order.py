"""CPU: the happens-before order that protects the small rings in shared memory (gather modes of csrc/attn_pair.cu and of
csrc/attn_rows64.cu): the tokens' validity bits, written by the copy or look-up warps and read by the softmax warps, and in FP8 decode
on pairs of SMs the tokens' addresses, read by the converting warps.  Nobody arrives on a barrier of their own for the validity bits, so an
entry may only be overwritten where the chain of the other barriers already orders its last reader before the writer.

The roles' program order and the barriers between them are written down as a graph; the ring depths, and in attn_rows64.cu on which
side of P's arrival the softmax warps read the mask, come from the source.  (In attn_pair.cu the mask is needed for P, and P V of a tile
gives its slots back: that alone keeps the entry.)"""
import os
import re

import pytest

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flashmla_b200", "csrc", "attn_pair.cu")


def _plan():
    text = open(SOURCE).read()
    slots, tables = (int(re.search(r"\b" + name + r" = (\d+)[,;]", text).group(1)) for name in ("NSLOT", "NTAB"))
    assert "uint32_t mask[2 * NTAB][4];" in text and len(re.findall(r"sm\.mask\[\(?g(?: \+ i\))? % \(2 \* NTAB\)\]", text)) == 3
    assert text.index("sm.mask[g % (2 * NTAB)][quarter]") < text.index("mbar_arrive_remote_cta(p_full0", text.index("float* xmax"))
    return slots, 2 * tables, tables


def _graph(tiles, slots, tables, convert, rank=0):
    """edges[event] = the events that directly precede it; events are (role, what, tile, slot of the tile), those of CTA `rank` of the pair
    and the issuing thread's.  P V of page h (slots 2 h and 2 h + 1) waits for the other page's part of CTA 1 - h, which may be brought in
    when Q K^T has read the slots that it goes to: CTA 1's first half of them, CTA 0's second."""
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
    program("softmax", [(what, g, 0) for g in range(tiles) for what in ("start", "give", "mask", "p")])
    for g in range(tiles):
        for q in four:
            f = 4 * g + q
            if f >= slots:                                                                      # empty: P V that read the slot
                edges["feed", "fill", g, q].append(("values", "values", (f - slots) // 4, (f - slots) % 4))
            edges["scores", "scores", g, q].append(("feed", "fill", g, q))                      # full
            edges["values", "values", g, q].append(("softmax", "p", g, 0))                       # p_full
            if g + 1 < tiles and q // 2 == 1 - rank:
                edges["values", "values", g, q].append(("feed", "other", g, 0))
            edges["values", "values", g, q].append(("scores", "scores", g, 3))
        if g >= 1:
            edges["scores", "scores", g, 0].append(("softmax", "give", g - 1, 0))               # s_empty
            edges["feed", "other", g - 1, 0].append(("scores", "scores", g - 1, 1 if rank else 3))    # k_half, k_done
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
        wait = text.rindex("WAIT_WARP_OR_LEAVE(wt, &sm.k_empty[ring.slot]", 0, guard)
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


@pytest.mark.parametrize("rank", [0, 1])
@pytest.mark.parametrize("convert", [False, True])          # prefill, FP8 decode
def test_ring_entries_are_read_before_they_are_overwritten(convert, rank):
    slots, masks, tables = _plan()
    tiles = masks + 8
    edges = _graph(tiles, slots, tables, convert, rank)
    writer = "look-up" if convert else "feed"
    for g in range(tiles - masks):
        assert _before(edges, (writer, "meta", g, 0), ("softmax", "mask", g, 0)), "a mask is read after it was written"
        assert _before(edges, ("softmax", "mask", g, 0), (writer, "meta", g + masks, 0)), "... and before its entry is written again"
    if convert:
        for g in range(tiles - tables):
            assert _before(edges, ("look-up", "meta", g, 0), ("feed", "own", g, 0))
            assert _before(edges, ("feed", "done", g, 0), ("look-up", "meta", g + tables, 0))


def test_the_check_sees_a_missing_order():
    """The same graph has no such order with rings of half the depth, nor for the table's entries where a mask of that depth would do;
    nor for a mask that is still read when P has been handed over."""
    slots, masks, tables = _plan()
    good = _graph(masks + 8, slots, tables, True)
    assert not _before(good, ("softmax", "mask", 3, 0), ("look-up", "meta", 3 + tables // 2, 0))
    assert not _before(good, ("feed", "done", 3, 0), ("look-up", "meta", 3 + tables // 2, 0))
    assert not _before(_graph(masks + 8, slots, tables, False), ("softmax", "mask", 3, 0), ("feed", "meta", 3 + 2, 0))
    for convert in (False, True):
        late = _graph(masks + 8, slots, tables, convert)
        late["softmax", "p", 3, 0] = [("softmax", "give", 3, 0)]
        assert not _before(late, ("softmax", "mask", 3, 0), ("look-up" if convert else "feed", "meta", 3 + masks, 0))


# ---- the pair kernel's ring across requests: parity waits -------------------------------------------------------------
# A request takes three slots of the ring for its Q (filled by a thread of warp 0, given back by the softmax warps) and four a tile (filled by
# the feeding warps, given back behind P V of page 0, which reads the first two, and of page 1).  A wait for the release of a slot's fill, by parity, is right if the release before
# that one is ordered before the wait, and the wait before the release behind.

def _request_plan():
    """Whether warp 0's thread follows the releases of the feeding warps' fills itself, and whether warp 2's follows k_done in the gather modes."""
    text = open(SOURCE).read()
    loads = text[text.index("own page of every tile"):text.index("MMA issuer (CTA 0")]
    gather = loads[loads.index("} else {", loads.index("if (DENSE) {")):]
    other = text[text.index("half of the dims of the other CTA's page"):text.index("FP8 decode: index ->")]
    loop = other[:other.index("k_done[g & 1]")]
    return "sm.empty[" in gather, "if (!DENSE) continue;" not in loop


def _request_graph(requests, slots, follow, follow_k):
    """(edges, waits): waits = (the step before the wait, the wait, what must be past when it begins, what must not be past when it ends)."""
    edges, waits, before = {}, [], {}

    def program(role, steps):
        for i, step in enumerate(steps):
            before[(role,) + step] = (role,) + steps[i - 1] if i else None
            edges[(role,) + step] = [(role,) + steps[i - 1]] if i else []

    q_slots = 3
    owner, at, first, g = [], 0, [], 0                        # fill -> what gives it back; a request's first fill and first tile
    for n, t in enumerate(requests):
        first.append((at, g))
        owner += [("softmax", "take", n)] * q_slots + [("issue", "values", g + i if k >= 2 else ("half", g + i)) for i in range(t) for k in range(4)]
        at, g = at + q_slots + 4 * t, g + t
    release = lambda f: owner[f] if f >= 0 else None
    load, feed, issue, soft, copy = [], [], [], [], []
    for n, t in enumerate(requests):
        f0, g0 = first[n]
        if n:
            load += [("next", n)] * (not follow and requests[n - 1] > 1) + [("taken", n)]
            copy += [("free", n)] * (not follow_k)
        load += [("q wait", f0 + k) for k in range(q_slots)] + [("q load", n)] + [("follow", f) for f in range(f0 + q_slots, f0 + q_slots + 4 * t)] * follow
        copy += [("q rest", n)] + [("k_done", i) for i in range(g0, g0 + t)] * follow_k
        for i in range(t):
            f = f0 + q_slots + 4 * i
            feed += [("wait", f + k) for k in range(4)] + [("filled", g0 + i)]
            soft += [("start", g0 + i), ("p", g0 + i)]
        soft = soft[:len(soft) - 2 * t] + [("take", n)] + soft[len(soft) - 2 * t:]
        issue += [("begin", n)] + [("scores", g0)] + [x for i in range(1, t) for x in (("scores", g0 + i), ("values", g0 + i - 1))] + [("values", g0 + t - 1)]
    for role, steps in (("load", load), ("feed", feed), ("softmax", soft), ("copy", copy)):
        program(role, steps)
    # Q K^T of a tile comes before or behind P V of the one before: two chains, joined where the issuing thread takes a request
    for i, (what, x) in enumerate(issue):
        edges.setdefault(("issue", what, x), [])
        if what == "begin" and i:
            edges["issue", what, x].append(("issue",) + issue[i - 1])
    for n, t in enumerate(requests):
        f0, g0 = first[n]
        edges["issue", "begin", n] += [("softmax", "take", n), ("copy", "q rest", n)]                   # q_ready, q_full
        edges["softmax", "take", n].append(("load", "q load", n))                                       # q_staged
        if n:
            edges["load", "taken", n].append(("softmax", "take", n - 1))
            if not follow and requests[n - 1] > 1:
                edges["load", "next", n].append(("issue", "scores", first[n - 1][1] + requests[n - 1] - 2))
            if not follow_k:
                edges["copy", "free", n].append(("issue", "scores", g0 - 1))
        for k in range(q_slots):
            if release(f0 + k - slots):
                edges["load", "q wait", f0 + k].append(release(f0 + k - slots))
        for i in range(g0, g0 + t):
            f = f0 + q_slots + 4 * (i - g0)
            edges["issue", "scores", i] += [("issue", "begin", n), ("feed", "filled", i)]               # full
            edges["issue", "values", ("half", i)] = [("issue", "scores", i), ("softmax", "p", i)]       # p_full of page 0 (page 1: below)
            edges["issue", "values", i] += [("issue", "values", ("half", i)), ("softmax", "p", i)]
            edges["softmax", "start", i].append(("issue", "scores", i))                                 # s_full
            if i > g0:
                edges["issue", "scores", i] += [("issue", "scores", i - 1), ("softmax", "start", i - 1)]    # s_empty
                edges["issue", "values", ("half", i)].append(("issue", "values", i - 1))
            if i > g0 + 1:
                edges["issue", "scores", i].append(("issue", "values", i - 2))                          # at most one tile ahead
            for k in range(4):
                if release(f + k - slots):
                    edges["feed", "wait", f + k].append(release(f + k - slots))
                    if follow:
                        edges["load", "follow", f + k].append(release(f + k - slots))
            if follow_k:
                edges["copy", "k_done", i].append(("issue", "scores", i))
    for role, what, f in [e for e in edges if e[1] in ("q wait", "wait", "follow")]:
        waits.append((before[role, what, f], (role, what, f), release(f - 2 * slots), release(f) if release(f - slots) else None))
    total = sum(requests)
    for role, what, i in [e for e in edges if e[1] == "k_done"]:                                        # (two barriers, tiles in turn)
        waits.append((before[role, what, i], (role, what, i), ("issue", "scores", i - 2) if i >= 2 else None, ("issue", "scores", i + 2) if i + 2 < total else None))
    return edges, waits


def _misread(requests, follow, follow_k, slots=None):
    edges, waits = _request_graph(requests, slots or _plan()[0], follow, follow_k)
    return [w for step, w, past, behind in waits
            if (past and not (step and _before(edges, past, step))) or (behind and not _before(edges, w, behind))]


MANY = [[1] * 9, [2] * 8, [3] * 7, [1, 2] * 4, [2, 1, 1, 3, 1, 2, 2, 1], [6, 1, 2, 1, 5], [1, 4, 1, 1, 4, 2], [2, 2, 1, 2, 3, 2, 2], [9, 2, 2, 9]]


@pytest.mark.parametrize("convert", [False, True])          # prefill, FP8 decode
def test_parity_waits_of_the_ring_across_requests(convert):
    follow, follow_k = _request_plan()
    for requests in MANY:
        assert not _misread(requests, follow, follow_k and convert), requests


def test_rope_chunks_need_no_wait():
    """A tile's RoPE chunk goes to the buffer of the tile before last's without a wait of its own: Q K^T of that tile is past when the last two
    slots of this one have been given back."""
    text = open(SOURCE).read()
    assert int(re.search(r"\bNROPE = (\d+);", text).group(1)) == 2 and "r_empty" not in text
    for requests in MANY:
        for follow in (False, True):
            edges, _ = _request_graph(requests, _plan()[0], follow, False)
            for g in range(2, sum(requests)):
                assert _before(edges, ("issue", "scores", g - 2), ("feed", "filled", g)), (requests, g)
    edges, _ = _request_graph([9], 16, False, False)            # the check sees a ring that would be too deep for that
    assert not _before(edges, ("issue", "scores", 5), ("feed", "filled", 7))


def test_the_check_sees_a_parity_that_may_be_misread():
    """A thread that watches every phase without anybody waiting for it may see one two phases late."""
    assert _misread([3] * 7, True, False) and _misread([6], False, True)
    assert _misread([2] * 8, False, False, slots=4)             # ... and a thread that skips phases nobody has ordered for it


# ---- bounded waits in the warps that meet at a named barrier ----------------------------------------------------------
def _softmax_steps(path):
    """What the softmax role of a kernel does in program order: ("wait", text), ("leave", text): a thread or warp leaves the role by itself,
    ("barrier", all leave): the 256 threads meet, and leave together where one says so."""
    text = open(path).read()
    start = max(m.start() for m in re.finditer(r"// -+ softmax", text))
    role = re.sub(r"//[^\n]*", "", text[start:text.index("wind_down:", start)])
    steps = []
    for m in re.finditer(r"BAR_OR_LEAVE\(wt\.expired\(\)\)|named_bar_red_or\(1, 256, [^;]*;|named_bar_sync\(1, 256\)|"
                         r"WAIT_(?:WARP_)?OR_LEAVE\([^;]*;|wt\.wait\w*\([^;]*;|goto wind_down", role):
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
    assert len(waits) == (6 if path == SOURCE else 2)
    for i in waits:
        after = [step for step in (steps + steps)[i + 1:] if step != ("barrier", False)]          # (the role is a loop)
        assert after[0][0] == "wait" or after[0] == ("barrier", True), (steps[i], after[0])


# ---- the pair kernel's softmax warps by page ---------------------------------------------------------------------------
def _graph_by_page(tiles, slots, tables, convert, rank):
    """`_graph` with the softmax warps of page 0 and of page 1 as roles of their own: each hands its part of P over by itself, and P V of a
    page waits for that part alone.  (The vote, which holds every warp's P back until all have read their masks, is left out.)"""
    edges = {e: list(p) for e, p in _graph(tiles, slots, tables, convert, rank).items() if e[0] != "softmax"}
    for page in range(2):
        steps = [(what, g, page) for g in range(tiles) for what in ("start", "give", "mask", "p")]
        for i, step in enumerate(steps):
            edges[("softmax",) + step] = [("softmax",) + steps[i - 1]] if i else []
        for g in range(tiles):
            edges["softmax", "start", g, page].append(("scores", "scores", g, 3))                  # s_full
    for event, before in edges.items():
        if event[0] == "values":
            edges[event] = [("softmax", "p", e[2], event[3] // 2) if e[:2] == ("softmax", "p") else e for e in before]
        elif event[0] == "scores":
            edges[event] = [f for e in before for f in ([("softmax", "give", e[2], page) for page in range(2)] if e[0] == "softmax" else [e])]
    return edges


@pytest.mark.parametrize("rank", [0, 1])
@pytest.mark.parametrize("convert", [False, True])          # prefill, FP8 decode
def test_masks_are_read_by_both_pages_before_they_are_overwritten(convert, rank):
    slots, masks, tables = _plan()
    tiles, writer = masks + 8, "look-up" if convert else "feed"
    edges = _graph_by_page(tiles, slots, tables, convert, rank)

    def kept(edges, depth, page):
        return all(_before(edges, ("softmax", "mask", g, page), (writer, "meta", g + depth, 0)) for g in range(tiles - masks))

    for page in range(2):
        assert all(_before(edges, (writer, "meta", g, 0), ("softmax", "mask", g, page)) for g in range(tiles))
        assert kept(edges, masks, page)
        assert not kept(edges, masks // 2 if convert else 2, page)      # the check sees a ring that is too shallow
        late = dict(edges)                                  # ... and a mask that is read when this page's P has been handed over
        late["softmax", "p", 3, page] = [("softmax", "give", 3, page)]
        assert not _before(late, ("softmax", "mask", 3, page), (writer, "meta", 3 + masks, 0))


# ---- the conditional barriers of the pair kernel's softmax warps -----------------------------------------------------------
def _leaves_behind_every_wait(text):
    """The barriers behind the waits of a tile stand under `if (together)`.  A warp with an expired wait must find that true, every warp must go there
    where a tail was waited for, and P is stored behind the first of them."""
    start = max(m.start() for m in re.finditer(r"// -+ softmax", text))
    role = re.sub(r"//[^\n]*", "", text[start:text.index("wind_down:", start)])
    tile = role[role.index("wt.wait(&sm.s_full"):]
    decided = re.search(r"bool together = ([^;]*);", tile)
    first = tile.index("BAR_OR_LEAVE(wt.expired());")
    second = tile.index("if (together) BAR_OR_LEAVE(wt.expired());")
    announced = tile.index("if (lane == 0 && !wt.expired())", second)
    waits = [m.start() for m in re.finditer(r"wt\.wait\(", tile[:second])]
    tails = [w for w in waits if w > first]
    return (decided is not None and "wt.expired()" in decided.group(1) and all(w < decided.start() or w in tails for w in waits)
            and tile.count("{", decided.end(), first) == 1 and "if (together) {" in tile[decided.end():first]
            and re.search(r"__any_sync\(0xffffffffu, mx > m_run \+ RESCALE_THRESHOLD \|\| wt\.expired\(\)\)", tile[:decided.start()]) is not None
            and first < tile.index("store();", decided.end()) < second < announced
            and all("together = true;" in tile[w:tile.index("ring.skip(4);", w)] and "sm.f_tail" in tile[w:w + 40] for w in tails))


def test_a_warp_with_an_expired_wait_reaches_the_conditional_barriers():
    text = open(SOURCE).read()
    assert _leaves_behind_every_wait(text)
    for there, instead in ((" || wt.expired());\n                if (together) {", ");\n                if (together) {"),
                           ("RESCALE_THRESHOLD || wt.expired())", "RESCALE_THRESHOLD)"),
                           ("together = true;", ""),
                           ("if (together) BAR_OR_LEAVE(wt.expired());", "")):
        assert text.count(there) == 1
        changed = text.replace(there, instead)
        try:
            assert not _leaves_behind_every_wait(changed), there
        except ValueError:                                  # (a piece it looks for is gone)
            pass
