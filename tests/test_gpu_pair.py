"""GPU: the kernel whose MMAs span a pair of SMs (csrc/attn_pair.cu) at the sizes where it can go wrong: rows at the edges of the two CTAs'
halves, tiles of 128 tokens and their remainders, requests of a single tile behind one another, maxima that move, Q that TMA
cannot address.  Against the CPU oracle, within the bounds of tests/helpers.py (rounding of P and of the output to 16 bits; fp32
sums)."""
import pytest
import torch

from oracle import attention
from tests import test_gpu_rows64 as small
from tests.helpers import assert_lse_close, assert_out_close

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("width", [576, 512])
@pytest.mark.parametrize("h_q,page,extra_page", [(128, 61, 2), (72, 2, 69)])
def test_sparse_decode_extra_cache(width, h_q, page, extra_page):
    small.test_sparse_decode_extra_cache(width, h_q, page, extra_page)


@pytest.mark.parametrize("width", [576, 512])
@pytest.mark.parametrize("h_q", [65, 128])
def test_sparse_decode_maxima_that_move_on_later_tiles(width, h_q):
    small.test_sparse_decode_maxima_that_move_on_later_tiles(width, h_q)


@pytest.mark.parametrize("width", [576, 512])
@pytest.mark.parametrize("h_q,most", [(96, 448), (128, 448), (128, 128)])
def test_sparse_decode_more_requests_than_partitions(width, h_q, most):
    """330 ragged lists on 74 pairs: several requests and tiles per pair, with lists of at most 128 keys a single tile each; first tiles
    without a valid key; unused records NaN; Q that several heads share (no tensor map) and of their own."""
    b, topk, gen = 330, 448, torch.Generator().manual_seed(h_q)
    idx = torch.stack([torch.randperm(1000, generator=gen)[:topk] for _ in range(b)]).view(b, 1, topk).to(torch.int32)
    idx[::3, :, :130] = -1
    idx[1::7, :, 200:] = 1 << 20
    lengths = torch.randint(0, most + 1, (b,), generator=gen, dtype=torch.int32)
    lengths[5], lengths[6], lengths[9] = 0, most, 100
    used = torch.zeros(1024, dtype=torch.bool)
    used[idx[(idx >= 0) & (idx < 1024)].long()] = True
    assert not used.all()
    kv, deq = small._records(width, torch.randn(16, 64, 1, width, generator=gen).bfloat16(), poison=~used)
    sink = torch.randn(h_q, generator=gen)
    one = torch.randn(b, 1, 1, width, generator=gen).bfloat16()
    for q in (torch.randn(b, 1, h_q, width, generator=gen).bfloat16(), one.expand(-1, -1, h_q, -1)):
        ref_out, ref_lse = attention.sparse_decode(q.contiguous(), deq, torch.where(idx < 1024, idx, -1), width ** -0.5, 512, sink, lengths)
        q_dev = q.to(DEV) if q.stride(2) else one.to(DEV).expand(-1, -1, h_q, -1)
        out, lse, sched = small._sparse(q_dev, kv, idx, width, sink=sink, lengths=lengths)
        requests, tiles = small._most_tiles(sched, [max(1, (int(n) + 63) // 64) for n in lengths])
        assert requests >= 3 and (tiles >= 4 if most > 128 else tiles == 1)
        assert_out_close("out", out, ref_out)
        assert_lse_close("lse", lse, ref_lse)


@pytest.mark.parametrize("width", [576, 512])
@pytest.mark.parametrize("s_q,h_q,topk", [(1, 128, 64), (160, 65, 64), (160, 128, 192), (90, 200, 320), (3, 64, 704)])
def test_sparse_prefill(width, s_q, h_q, topk):
    """One and several query tokens per pair, of one tile and of more; more heads than a pair has rows, half a pair of them."""
    small.test_sparse_prefill(width, s_q, h_q, topk)


@pytest.mark.parametrize("width", [576, 512])
@pytest.mark.parametrize("rows,stride", [(200, 640), (200, 576), (200, 72), (1, 576), (1, 8)])
def test_sparse_prefill_keys_in_rows_of_other_strides(width, rows, stride):
    """The row gathers' tensor map: padded rows (NaN between and behind them), rows that overlap, a single row.  Entries that are no key read zeros,
    not what lies behind the last row.  Against the same keys in rows of their own."""
    import flashmla_b200 as fm
    gen = torch.Generator().manual_seed(rows + stride)
    memory = torch.full((rows * max(stride, width) + 4 * 640,), float("nan"))
    index = (torch.arange(rows).view(-1, 1) * stride + torch.arange(width)).view(-1)
    memory[index] = torch.randn(rows * width, generator=gen)
    memory = memory.bfloat16().to(DEV)
    kv = memory.as_strided((rows, 1, width), (stride, width, 1))
    idx = torch.randint(-3, rows + 40, (90, 1, 320), generator=gen, dtype=torch.int32)
    idx[7], idx[8, :, 128:] = -1, rows
    q = torch.randn(90, 128, width, generator=gen).bfloat16().to(DEV)
    out, top, lse = fm.flash_mla_sparse_fwd(q, kv, idx.to(DEV), width ** -0.5, 512)
    ref_out, ref_top, ref_lse = fm.flash_mla_sparse_fwd(q, kv.clone(memory_format=torch.contiguous_format), idx.to(DEV), width ** -0.5, 512)
    fm.check_status()
    assert not torch.isnan(out.float()).any()
    assert_out_close("out", out.cpu(), ref_out.cpu())
    assert_lse_close("lse", lse.cpu(), ref_lse.cpu())
    assert torch.allclose(top.cpu(), ref_top.cpu(), rtol=1e-4, atol=1e-4)


@pytest.mark.parametrize("impl", [0, 2])
@pytest.mark.parametrize("width,h_q,stride", [(576, 128, 640), (512, 128, 520), (576, 128, 576), (576, 128, 504), (512, 128, 72), (512, 100, 504), (576, 200, 8)])
def test_sparse_prefill_keys_of_any_row_stride_run_on_pairs(width, h_q, stride, impl):
    """The driver makes a tensor map over rows of their own, padded or not, and over rows that overlap: none of them leaves the pair kernel, and
    overlapping rows give what the oracle gives for them."""
    import flashmla_b200 as fm
    rows, s_q, topk, gen = 300, 65, 320, torch.Generator().manual_seed(h_q + stride)
    memory = torch.randn(rows * stride + width, generator=gen).bfloat16()
    kv = memory.as_strided((rows, 1, width), (stride, width, 1))
    idx = torch.randint(-3, rows + 40, (s_q, 1, topk), generator=gen, dtype=torch.int32)
    idx[7], idx[8, :, 128:] = -1, rows
    lengths = torch.randint(0, topk + 1, (s_q,), generator=gen, dtype=torch.int32)
    q, sink = torch.randn(s_q, h_q, width, generator=gen).bfloat16(), torch.randn(h_q, generator=gen)
    ref = attention.sparse_prefill(q, kv.contiguous(), torch.where(idx < rows, idx, -1), width ** -0.5, 512, sink, lengths)
    kv_dev, got = memory.to(DEV).as_strided((rows, 1, width), (stride, width, 1)), []
    fm.set_impl(impl)
    try:
        assert small.kernels(lambda: got.append(fm.flash_mla_sparse_fwd(q.to(DEV), kv_dev, idx.to(DEV), width ** -0.5, 512, sink.to(DEV), lengths.to(DEV)))) == {"attn_pair_kernel"}
    finally:
        fm.set_impl(0)
    fm.check_status()
    assert_out_close("out", got[0][0], ref[0])
    assert_lse_close("max_logits", got[0][1], ref[1])
    assert_lse_close("lse", got[0][2], ref[2])


@pytest.mark.parametrize("width", [576, 512])
def test_sparse_prefill_maxima_and_shared_query(width):
    """Maxima that move on every tile (the true maximum is a result too); heads that share their query: Q that is no tensor map."""
    import flashmla_b200 as fm
    s_q, h_q, topk, gen = 90, 128, 640, torch.Generator().manual_seed(width)
    q, kv = torch.randn(s_q, h_q, width, generator=gen).bfloat16(), torch.randn(1024, 1, width, generator=gen).bfloat16()
    small._growing(q, kv, torch.arange(1024))
    idx = torch.stack([torch.randperm(1024, generator=gen)[:topk].sort().values for _ in range(s_q)]).view(s_q, 1, topk).to(torch.int32)
    small._assert_maxima_move(q, kv[:, 0], width ** -0.5, [(i, idx[i, 0]) for i in range(s_q)])
    for rows, rows_dev in ((q, q.to(DEV)), (q[:, :1].expand(-1, h_q, -1), q[:, :1].to(DEV).expand(-1, h_q, -1))):
        ref = attention.sparse_prefill(rows.contiguous(), kv, idx, width ** -0.5, 512)
        got = fm.flash_mla_sparse_fwd(rows_dev, kv.to(DEV), idx.to(DEV), width ** -0.5, 512)
        torch.cuda.synchronize()
        fm.check_status()
        assert_out_close("out", got[0], ref[0])
        assert_lse_close("max_logits", got[1], ref[1])
        assert_lse_close("lse", got[2], ref[2])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("s_q,h_q,h_kv", [(1, 65, 1), (1, 96, 1), (2, 48, 1), (2, 96, 1), (3, 72, 1), (2, 35, 1), (1, 200, 1), (2, 256, 2)])
def test_dense_row_counts(s_q, h_q, h_kv, dtype):
    """Heads that are one box of Q per CTA, several, and none (their number shares no 8 with the rows)."""
    small.test_dense_row_counts(s_q, h_q, h_kv, dtype)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("parts", [1, 3])
@pytest.mark.parametrize("s_q,h_q", [(1, 128), (2, 64), (2, 41)])
def test_dense_several_tiles_and_requests_per_pair(s_q, h_q, parts, dtype):
    small.test_dense_several_tiles_and_requests_per_cta(s_q, h_q, parts, dtype)


@pytest.mark.parametrize("parts", [1, 4])
def test_dense_requests_of_a_single_tile(parts):
    """Every request one tile (or none): a request's Q is staged behind the last one's before that has been multiplied."""
    lengths = [1, 128, 64, 0, 65, 127, 128, 3, 0, 0, 100, 128, 64, 90]
    q, k, bt, sl = small._dense_inputs(1, 128, 1, lengths, seed=parts)
    ref_out, ref_lse = attention.dense_decode(q, k, bt, sl, 512, True)
    out, lse, sched = small._dense_parts(q, k, bt, sl, True, parts)
    assert_out_close("out", out, ref_out)
    assert_lse_close("lse", lse, ref_lse)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_dense_maxima_that_move_on_later_tiles(dtype):
    small.test_dense_maxima_that_move_on_later_tiles(128, dtype)


def test_dense_heads_that_share_their_query():
    q, k, bt, sl = small._dense_inputs(1, 1, 1, small.LENGTHS, seed=6)
    q = q.to(DEV).expand(-1, -1, 100, -1)
    ref_out, ref_lse = attention.dense_decode(q.cpu().contiguous(), k, bt, sl, 512, False)
    out, lse = small._dense(q, k, bt, sl, False)
    assert_out_close("out", out, ref_out)
    assert_lse_close("lse", lse, ref_lse)


@pytest.mark.parametrize("h_q,topk,b,cut", [(16, 320, 4, False), (16, 384, 4, True), (64, 128, 4, False), (64, 192, 21, True), (64, 512, 37, True),
                                            (128, 448, 10, False), (128, 512, 10, True), (128, 512, 11, False)])
def test_few_requests_are_cut(h_q, topk, b, cut):
    """Few requests of equal cost (148 SMs): lists long enough are cut over all partitions, shorter ones stay whole; a stored schedule of
    the other kind, one partition per request, is still taken."""
    import flashmla_b200 as fm
    from flashmla_b200.flash_mla_interface import _make_sched_meta
    q, kv, deq, idx = small._cache(576, b, 700, topk, 1, h_q, seed=h_q + topk)
    ref_out, ref_lse = attention.sparse_decode(q, deq, idx, 576 ** -0.5, 512, None, None)
    meta, kv = fm.get_mla_metadata()[0], kv.to(DEV).contiguous()
    for stored in (False, True):
        if stored:
            meta.tile_scheduler_metadata, meta.num_splits = _make_sched_meta(b, 1, b, torch.device(DEV), topk=topk)
        out, lse = fm.flash_mla_with_kvcache(q.to(DEV), kv, None, None, 512, meta, None, 576 ** -0.5, False, True, idx.to(DEV))
        torch.cuda.synchronize()
        fm.check_status()
        assert meta.tile_scheduler_metadata.size(0) == (b if stored or not cut else 148 if h_q <= 64 else 74)
        assert_out_close("out", out, ref_out)
        assert_lse_close("lse", lse, ref_lse)


def test_schedules_of_few_long_requests():
    """Requests of many partitions each, whose starts the scheduler writes a request at a time, and both sides of that line; counts above
    the rows it makes at once."""
    from flashmla_b200.flash_mla_interface import _make_sched_meta
    from oracle import sched_meta
    gen = torch.Generator().manual_seed(0)
    for parts in (1, 2, 33, 74, 148, 255, 256, 257):
        for lengths in ([100003], [1], [64 * parts], [64 * 9 * parts + 1], [7000, 0, 1, 9000], [64, 640000], [3000] * 9,
                        torch.randint(0, 60000, (5,), generator=gen).tolist(), torch.randint(1, 4000, (12,), generator=gen).tolist()):
            got, splits = _make_sched_meta(len(lengths), 1, parts, torch.device(DEV), seqlens_k=torch.tensor(lengths, dtype=torch.int32, device=DEV))
            ref, ref_splits = sched_meta.get_sched_meta(len(lengths), parts, 64, 5, seqlens_k=lengths)
            assert torch.equal(got.cpu(), torch.as_tensor(ref, dtype=torch.int32)), (parts, lengths)
            assert splits.tolist() == list(ref_splits), (parts, lengths)


@pytest.mark.parametrize("s_q,h_q,lengths,parts", [(1, 64, [200] * 40, 74), (2, 20, [1, 900, 65, 0, 300], 74), (1, 64, [40000, 1, 300], 74), (1, 32, [900] * 4, 148),
                                                   (1, 33, [700] * 450, 148)])
def test_dense_33_to_64_rows(s_q, h_q, lengths, parts):
    """On pairs of SMs up to three thousand blocks of the table, on single SMs beyond and up to 32 rows (148 SMs); either stored schedule."""
    import flashmla_b200 as fm
    from flashmla_b200.flash_mla_interface import _make_sched_meta
    q, k, bt, sl = small._dense_inputs(s_q, h_q, 1, lengths, seed=h_q)
    bt = bt[:, :(max(lengths) + 63) // 64].contiguous()
    ref_out, ref_lse = attention.dense_decode(q, k, bt, sl, 512, True)
    meta = fm.get_mla_metadata()[0]
    for other in (False, True):
        if other:
            meta.tile_scheduler_metadata, meta.num_splits = _make_sched_meta(len(lengths), s_q, 222 - parts, torch.device(DEV), seqlens_k=sl.to(DEV))
        out, lse = small._dense(q, k, bt, sl, True, meta)
        assert meta.tile_scheduler_metadata.size(0) == (222 - parts if other else parts)
        assert_out_close("out", out, ref_out)
        assert_lse_close("lse", lse, ref_lse)


@pytest.mark.parametrize("b,width,pairs", [(34, 10, True), (35, 7, True), (35, 8, False), (49, 7, True), (49, 10, False), (50, 8, True), (62, 10, True),
                                           (63, 6, False), (74, 16, False), (80, 16, False), (128, 8, False), (160, 10, True), (192, 8, True), (193, 10, False)])
def test_dense_33_to_64_rows_in_wide_tables(b, width, pairs):
    """A table may be wider than its requests are long: one that holds short requests for which a pair of SMs per partition is slower keeps
    a partition per SM (148 SMs; 80 requests of 128 tokens in a table 16 wide took 20 us in the place of 14.5)."""
    import flashmla_b200 as fm
    lengths = [128 - i % 70 for i in range(b)]
    q, k, bt, sl = small._dense_inputs(1, 33, 1, lengths, seed=b)
    ref_out, ref_lse = attention.dense_decode(q, k, bt, sl, 512, False)
    meta = fm.get_mla_metadata()[0]
    out, lse = small._dense(q, k, torch.nn.functional.pad(bt[:, :2], (0, width - 2)), sl, False, meta)
    assert meta.tile_scheduler_metadata.size(0) == (74 if pairs else 148)
    assert_out_close("out", out, ref_out)
    assert_lse_close("lse", lse, ref_lse)


@pytest.mark.parametrize("h_kv,g,lengths,kernel", [(75, 34, [128, 60], "attn_rows64_kernel"), (74, 34, [128, 60], "attn_rows64_kernel"),
                                                   (2, 64, [70] * 8, "attn_pair_kernel"), (2, 64, [130] * 8, "attn_rows64_kernel")])
def test_dense_33_to_64_rows_with_several_kv_heads(h_kv, g, lengths, kernel):
    """As many kv heads as there are pairs and more (148 SMs) have one partition whatever the kernel, and stay on single SMs; fewer are
    on pairs where the rule for tables of two blocks says so."""
    q, k, bt, sl = small._dense_inputs(1, h_kv * g, h_kv, lengths, seed=h_kv)
    bt = bt[:, :(max(lengths) + 63) // 64].contiguous()
    ref_out, ref_lse = attention.dense_decode(q, k, bt, sl, 512, False)
    got = []
    assert small.kernels(lambda: got.append(small._dense(q, k, bt, sl, False))) == {kernel}
    assert_out_close("out", got[0][0], ref_out)
    assert_lse_close("lse", got[0][1], ref_lse)
