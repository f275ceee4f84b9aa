"""GPU: the kernel for up to 64 query rows on one SM (csrc/attn_rows64.cu) at the sizes where it can go wrong: rows at the edges
of its variants (16 / 32 / 64), tiles of 128 tokens and their remainders, scores that keep growing, Q that TMA cannot address,
schedules with another number of partitions.  (Dense calls with 33 to 64 rows run on pairs of SMs, csrc/attn_pair.cu, where the
schedule has no more partitions than there are pairs: the tests with one to three partitions or few requests among them; those of
the kernel on one SM with that many rows ask for a partition per SM.)  Against the CPU oracle, within the bounds of tests/helpers.py (element-wise
rounding of P and of the output to 16 bits; fp32 sums)."""
import pytest
import torch

from oracle import attention, quant
from tests.helpers import assert_lse_close, assert_out_close

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
LENGTHS = [0, 1, 63, 64, 65, 127, 128, 129, 255, 257, 640, 1000]


def _dense(q, k, bt, sl, causal, meta=None):
    import flashmla_b200 as fm
    out, lse = fm.flash_mla_with_kvcache(q.to(DEV), k.to(DEV), bt.to(DEV), sl.to(DEV), 512, meta or fm.get_mla_metadata()[0], None, causal=causal)
    torch.cuda.synchronize()
    fm.check_status()
    return out, lse


def _dense_inputs(s_q, h_q, h_kv, lengths, seed, dtype=torch.bfloat16):
    from tests import workloads as W
    d = W.dense_decode_inputs(torch.tensor(lengths, dtype=torch.int32), s_q, h_q, h_kv, seed=seed, device="cpu", poison_unused=True)
    return d["q"].to(dtype), d["blocked_k"].to(dtype), d["block_table"], d["cache_seqlens"]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("s_q,h_q,h_kv", [(1, 8, 1), (1, 17, 1), (1, 32, 1), (3, 11, 1), (1, 33, 1), (1, 64, 1), (2, 32, 1), (2, 64, 2)])
def test_dense_row_counts(s_q, h_q, h_kv, dtype):
    q, k, bt, sl = _dense_inputs(s_q, h_q, h_kv, LENGTHS, seed=s_q * 100 + h_q, dtype=dtype)
    ref_out, ref_lse = attention.dense_decode(q, k, bt, sl, 512, True)
    out, lse = _dense(q, k, bt, sl, True)
    assert_out_close("out", out, ref_out)
    assert_lse_close("lse", lse, ref_lse)


@pytest.mark.parametrize("h_q", [16, 32, 64])
def test_dense_scores_that_grow(h_q):
    """The RoPE part of K (not part of V) grows with the token's position.  (With a partition per SM a CTA walks one block here: scores far
    apart are combined.  test_dense_maxima_that_move_on_later_tiles has the tiles behind one another.)"""
    q, k, bt, sl = _dense_inputs(1, h_q, 1, [1500, 129, 700], seed=5)
    for b in range(3):
        for j, page in enumerate(bt[b, :(int(sl[b]) + 63) // 64].tolist()):
            k[page, :, :, 512:] *= 1.0 + 6.0 * j
    ref_out, ref_lse = attention.dense_decode(q, k, bt, sl, 512, False)
    out, lse = _dense(q, k, bt, sl, False)
    assert_out_close("out", out, ref_out)
    assert_lse_close("lse", lse, ref_lse)


def _dense_parts(q, k, bt, sl, causal, parts):
    """The C ABI, with that many partitions: a CTA walks several tiles and requests.  Returns the schedule as well."""
    from flashmla_b200 import _capi
    from flashmla_b200.flash_mla_interface import _make_sched_meta
    b, s_q, h_q, _ = q.shape
    q, k, bt, sl = (t.to(DEV) for t in (q, k, bt, sl))
    sched, num_splits = _make_sched_meta(b, s_q, parts, torch.device(DEV), seqlens_k=sl)
    out = torch.full((b, s_q, h_q, 512), float("nan"), dtype=q.dtype, device=DEV)
    lse = torch.full((b, h_q, s_q), float("nan"), device=DEV)
    status = torch.zeros(4, dtype=torch.int32, device=DEV)
    a = _capi.DenseDecodeArgs(
        b=b, s_q=s_q, h_q=h_q, h_kv=k.size(2), d_qk=576, d_v=512, num_blocks=k.size(0), page_block_size=64, is_causal=int(causal),
        softmax_scale=576 ** -0.5, q=_capi.ptr(q), q_stride_b=q.stride(0), q_stride_s=q.stride(1), q_stride_h=q.stride(2),
        k_cache=_capi.ptr(k), k_stride_block=k.stride(0), k_stride_row=k.stride(1), k_stride_head=k.stride(2),
        block_table=_capi.ptr(bt), block_table_stride_b=bt.stride(0), max_blocks_per_seq=bt.size(1), seqlens_k=_capi.ptr(sl),
        out=_capi.ptr(out), o_stride_b=out.stride(0), o_stride_s=out.stride(1), o_stride_h=out.stride(2),
        lse=_capi.ptr(lse), lse_stride_b=lse.stride(0), lse_stride_s=lse.stride(2), lse_stride_h=lse.stride(1),
        meta=_capi.ptr(sched), num_splits=_capi.ptr(num_splits), num_sm_parts=parts, status=_capi.ptr(status), impl=2,
        dtype=_capi.MLA_DTYPE_FP16 if q.dtype == torch.float16 else _capi.MLA_DTYPE_BF16, stream=torch.cuda.current_stream().cuda_stream)
    _capi.check(_capi.lib().mla_dense_decode_noalloc(a), "mla_dense_decode_noalloc")
    torch.cuda.synchronize()
    assert status.tolist() == [0, 0, 0, 0]
    return out, lse, sched.cpu()


def _most_tiles(sched, blocks):
    """Per partition: requests it walks, and the most tiles of 128 tokens it walks of one request."""
    rows = [m.tolist() for m in sched if m[0] < len(blocks)]
    tiles = [[((m[3] if r == m[1] else blocks[r]) - (m[2] if r == m[0] else 0) + 1) // 2 for r in range(m[0], m[1] + 1)] for m in rows]
    return max(len(t) for t in tiles), max(max(t) for t in tiles)


# odd and even numbers of blocks, last blocks of one token and of all, requests without keys between others
SEVERAL = [700, 0, 1023, 64, 1, 1500, 0, 257, 128, 0]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("parts", [1, 3])
@pytest.mark.parametrize("s_q,h_q", [(1, 16), (1, 32), (1, 64), (2, 32), (1, 41)])
def test_dense_several_tiles_and_requests_per_cta(s_q, h_q, parts, dtype):
    q, k, bt, sl = _dense_inputs(s_q, h_q, 1, SEVERAL, seed=h_q, dtype=dtype)
    ref_out, ref_lse = attention.dense_decode(q, k, bt, sl, 512, True)
    out, lse, sched = _dense_parts(q, k, bt, sl, True, parts)
    requests, tiles = _most_tiles(sched, [max(1, (n + 63) // 64) for n in SEVERAL])
    assert requests >= 3 and tiles >= 5
    assert_out_close("out", out, ref_out)
    assert_lse_close("lse", lse, ref_lse)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("h_q", [16, 32, 64])
def test_dense_maxima_that_move_on_later_tiles(h_q, dtype):
    """As test_dense_scores_that_grow, with one and two partitions: the maximum moves by more than the threshold on tiles behind a
    request's first, where sums and O are rescaled."""
    lengths = [1500, 129, 700]
    q, k, bt, sl = _dense_inputs(1, h_q, 1, lengths, seed=5, dtype=dtype)
    for b, n in enumerate(lengths):
        for j, page in enumerate(bt[b, :(n + 63) // 64].tolist()):
            k[page, :, :, 512:] *= 1.0 + 6.0 * j
    ref_out, ref_lse = attention.dense_decode(q, k, bt, sl, 512, False)
    for parts in (1, 2):
        out, lse, sched = _dense_parts(q, k, bt, sl, False, parts)
        assert _most_tiles(sched, [(n + 63) // 64 for n in lengths])[1] >= 6
        assert_out_close("out", out, ref_out)
        assert_lse_close("lse", lse, ref_lse)


def kernels(call):
    """Names of the attention kernels that a call launches."""
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU, torch.profiler.ProfilerActivity.CUDA], acc_events=True) as prof:
        call()
        torch.cuda.synchronize()
    return {name for e in prof.events() for name in ("attn_pair_kernel", "attn_rows64_kernel", "attn_portable_kernel") if name in e.name}


def _dense_on_single_sms(q, k, bt, sl, causal, lengths):
    """With a partition per SM (148): every CTA that walks the most requests has at least three, the longest request at least five tiles."""
    got = []
    assert kernels(lambda: got.append(_dense_parts(q, k, bt, sl, causal, 148))) == {"attn_rows64_kernel"}
    out, lse, sched = got[0]
    requests, tiles = _most_tiles(sched, [max(1, (n + 63) // 64) for n in lengths])
    assert requests >= 3 and tiles >= 5
    return out, lse


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("s_q,h_q", [(1, 64), (2, 32), (1, 41), (1, 33)])
def test_dense_33_to_64_rows_several_tiles_and_requests_per_sm(s_q, h_q, dtype):
    lengths = SEVERAL * 45
    q, k, bt, sl = _dense_inputs(s_q, h_q, 1, lengths, seed=h_q, dtype=dtype)
    ref_out, ref_lse = attention.dense_decode(q, k, bt, sl, 512, True)
    out, lse = _dense_on_single_sms(q, k, bt, sl, True, lengths)
    assert_out_close("out", out, ref_out)
    assert_lse_close("lse", lse, ref_lse)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_dense_64_rows_maxima_that_move_on_later_tiles(dtype):
    """As test_dense_maxima_that_move_on_later_tiles, with a partition per SM and requests enough for each to walk whole ones."""
    lengths = [1500, 129, 700] * 90
    q, k, bt, sl = _dense_inputs(1, 64, 1, lengths, seed=5, dtype=dtype)
    # (an output is nearly one key's value: below 4 a step of bf16 is 2^-6, within the bound of 2e-2; from 4 on it is 2^-5, and
    # 8.8 million values of N(0, 1) hold some)
    k[..., :512] *= 0.5
    for b, n in enumerate(lengths):
        for j, page in enumerate(bt[b, :(n + 63) // 64].tolist()):
            k[page, :, :, 512:] *= 1.0 + 6.0 * j
    assert k[..., :512].nan_to_num(0.0).abs().max() < 4
    ref_out, ref_lse = attention.dense_decode(q, k, bt, sl, 512, False)
    out, lse = _dense_on_single_sms(q, k, bt, sl, False, lengths)
    assert_out_close("out", out, ref_out)
    assert_lse_close("lse", lse, ref_lse)


def test_dense_heads_that_share_their_query():
    """A head stride of zero (expanded q) is no tensor map: the kernel's own threads load Q."""
    q, k, bt, sl = _dense_inputs(1, 1, 1, LENGTHS, seed=6)
    q = q.to(DEV).expand(-1, -1, 24, -1)
    assert q.stride(2) == 0
    ref_out, ref_lse = attention.dense_decode(q.cpu().contiguous(), k, bt, sl, 512, False)
    out, lse = _dense(q, k, bt, sl, False)
    assert_out_close("out", out, ref_out)
    assert_lse_close("lse", lse, ref_lse)


def test_schedule_made_for_pairs_of_sms():
    """A stored schedule with half the partitions (one per pair of SMs) gives the same results; any other count is refused."""
    import flashmla_b200 as fm
    from flashmla_b200 import _capi
    from flashmla_b200.flash_mla_interface import _make_sched_meta
    q, k, bt, sl = _dense_inputs(1, 16, 1, LENGTHS, seed=7)
    ref_out, ref_lse = _dense(q, k, bt, sl, False)
    own, pairs = (_capi.lib().mla_num_sm_parts(0, _capi.MLA_MODE_DENSE_DECODE, h, 1, 1) for h in (16, 128))
    assert pairs < own
    for parts in (pairs, pairs - 1):
        meta = fm.get_mla_metadata()[0]
        _dense(q, k, bt, sl, False, meta)
        meta.tile_scheduler_metadata, meta.num_splits = _make_sched_meta(len(LENGTHS), 1, parts, torch.device(DEV), seqlens_k=sl.to(DEV))
        if parts == pairs:
            out, lse = _dense(q, k, bt, sl, False, meta)
            assert_out_close("out", out, ref_out.cpu())
            assert_lse_close("lse", lse, ref_lse.cpu())
        else:
            with pytest.raises(RuntimeError, match="tile_scheduler_metadata must have shape"):
                _dense(q, k, bt, sl, False, meta)


@pytest.mark.parametrize("b,longest,whole", [(10, 128, False), (11, 128, True), (21, 128, True), (22, 128, False), (15, 64, False), (15, 129, False)])
@pytest.mark.parametrize("h_q", [32, 33, 64])
def test_requests_of_two_blocks_stay_whole(b, longest, whole, h_q):
    """33 to 64 rows and a table of two blocks a request (148 SMs): a new schedule has a partition per pair of SMs where that leaves the
    requests whole and one per SM does not.  A schedule with either count is taken, the table as wide as it may be."""
    import flashmla_b200 as fm
    lengths = [longest - 7 * i % 60 for i in range(b)]
    q, k, bt, sl = _dense_inputs(1, h_q, 1, lengths, seed=b)
    ref_out, ref_lse = attention.dense_decode(q, k, bt, sl, 512, False)
    meta = fm.get_mla_metadata()[0]
    assert bt.size(1) > 3
    for width in ((longest + 63) // 64, bt.size(1)):
        out, lse = _dense(q, k, bt[:, :width].contiguous(), sl, False, meta)
        assert meta.tile_scheduler_metadata.size(0) == (74 if whole and h_q > 32 else 148)
        assert_out_close("out", out, ref_out)
        assert_lse_close("lse", lse, ref_lse)
    if whole and h_q > 32:
        assert torch.equal(meta.num_splits.cpu(), torch.arange(b + 1, dtype=torch.int32))


def _records(width, k, poison=None):
    """FP8 records of k [pages, page, 1, width] on the device, and what they hold.  `poison` [pages * page]: tokens whose bytes are all
    0x7f (NaN values, scales and RoPE)."""
    from flashmla_b200.kvcache import model1_block_bytes
    from tests.helpers import model1_cache_from_bytes
    page = k.size(1)
    if width == 576:
        kv = quant.quantize_v32(k, pow2_scale=False)
        if poison is not None:
            kv.view(torch.uint8)[poison.view(-1, page)] = 0x7f
        return kv.to(DEV), quant.dequantize_v32(kv)
    kv = quant.quantize_model1(k)
    deq = quant.dequantize_model1(kv)
    data = kv.contiguous().view(torch.uint8).reshape(k.size(0), -1)
    if poison is not None:
        bad = poison.view(-1, page)
        data[:, :page * 576].view(-1, page, 576)[bad] = 0x7f
        data[:, page * 576:page * 584].view(-1, page, 8)[bad] = 0xff
        deq.view(-1, 512)[poison] = float("nan")
    return model1_cache_from_bytes(data.view(k.size(0), page, 1, 584), model1_block_bytes(page), DEV), deq


def _sparse(q, kv, indices, width, **kw):
    import flashmla_b200 as fm
    meta = fm.get_mla_metadata()[0]
    dev = lambda t: None if t is None else t.to(DEV)
    out, lse = fm.flash_mla_with_kvcache(q if q.is_cuda else q.to(DEV), kv, None, None, 512, meta, None, width ** -0.5, False, True, indices.to(DEV),
                                         dev(kw.get("sink")), kw.get("extra_kv"), dev(kw.get("extra_indices")), dev(kw.get("lengths")),
                                         dev(kw.get("extra_lengths")))
    torch.cuda.synchronize()
    fm.check_status()
    return out, lse, meta.tile_scheduler_metadata.cpu()


def _growing(q, k, where):
    """The last 64 dims of q large and those of key i proportional to where[i]: maxima move by much more than the threshold (2^6) from
    one tile of the list to the next.  V (in the 512-wide form those dims too) stays below 4, where one step of bf16 is within the bound."""
    q[..., -64:] *= 256
    k[..., :-64] *= 0.5
    k.view(-1, k.size(-1))[:, -64:] *= (0.05 * (where // 64)).view(-1, 1).to(k.dtype)


def _assert_maxima_move(q, keys, scale, lists):
    """Some row's maximum rises by more than 2^6 on every tile behind the first."""
    for row, idx in lists:
        s = (q[row].float() @ keys[idx.long()].float().T) * scale * 1.4426950408889634
        tops = torch.stack([s[:, i:i + 128].max(-1).values for i in range(0, s.size(1), 128)])
        assert ((tops[1:] - tops[:-1].cummax(0).values) > 6).any(-1).all()


@pytest.mark.parametrize("width", [576, 512])
@pytest.mark.parametrize("h_q", [16, 64])
def test_sparse_decode_maxima_that_move_on_later_tiles(width, h_q):
    """40 lists of 640 keys in the order of their scores, a CTA (of 148) each."""
    b, topk, gen = 40, 640, torch.Generator().manual_seed(h_q + width)
    q = torch.randn(b, 1, h_q, width, generator=gen).bfloat16()
    k = torch.randn(16, 64, 1, width, generator=gen).bfloat16()
    _growing(q, k, torch.arange(1024))
    kv, deq = _records(width, k)
    idx = torch.stack([torch.randperm(1024, generator=gen)[:topk].sort().values for _ in range(b)]).view(b, 1, topk).to(torch.int32)
    _assert_maxima_move(q[:, 0], deq.reshape(-1, width), width ** -0.5, [(i, idx[i, 0]) for i in range(b)])
    ref_out, ref_lse = attention.sparse_decode(q, deq, idx, width ** -0.5, 512)
    out, lse, sched = _sparse(q, kv, idx, width)
    assert sched.size(0) == b
    assert_out_close("out", out, ref_out)
    assert_lse_close("lse", lse, ref_lse)


@pytest.mark.parametrize("width", [576, 512])
def test_sparse_prefill_maxima_that_move_on_later_tiles(width):
    import flashmla_b200 as fm
    s_q, h_q, topk, gen = 100, 64, 640, torch.Generator().manual_seed(width)
    q, kv = torch.randn(s_q, h_q, width, generator=gen).bfloat16(), torch.randn(1024, 1, width, generator=gen).bfloat16()
    _growing(q, kv, torch.arange(1024))
    idx = torch.stack([torch.randperm(1024, generator=gen)[:topk].sort().values for _ in range(s_q)]).view(s_q, 1, topk).to(torch.int32)
    _assert_maxima_move(q, kv[:, 0], width ** -0.5, [(i, idx[i, 0]) for i in range(s_q)])
    ref = attention.sparse_prefill(q, kv, idx, width ** -0.5, 512)
    out, mx, lse = fm.flash_mla_sparse_fwd(q.to(DEV), kv.to(DEV), idx.to(DEV), width ** -0.5, 512)
    torch.cuda.synchronize()
    fm.check_status()
    assert_out_close("out", out, ref[0])
    assert_lse_close("max_logits", mx, ref[1])
    assert_lse_close("lse", lse, ref[2])


@pytest.mark.parametrize("width", [576, 512])
@pytest.mark.parametrize("h_q", [16, 40, 64])
def test_sparse_decode_more_requests_than_partitions(width, h_q):
    """330 ragged lists on 148 SMs: a CTA walks several requests and tiles; first tiles without a valid key; unused records NaN."""
    b, topk, gen = 330, 448, torch.Generator().manual_seed(h_q)
    q = torch.randn(b, 1, h_q, width, generator=gen).bfloat16()
    idx = torch.stack([torch.randperm(1000, generator=gen)[:topk] for _ in range(b)]).view(b, 1, topk).to(torch.int32)
    idx[::3, :, :130] = -1
    idx[1::7, :, 200:] = 1 << 20
    lengths = torch.randint(0, topk + 1, (b,), generator=gen, dtype=torch.int32)
    lengths[5], lengths[6], lengths[9] = 0, topk, 100
    used = torch.zeros(1024, dtype=torch.bool)
    used[idx[(idx >= 0) & (idx < 1024)].long()] = True
    assert not used.all()
    kv, deq = _records(width, torch.randn(16, 64, 1, width, generator=gen).bfloat16(), poison=~used)
    sink = torch.randn(h_q, generator=gen)
    ref_out, ref_lse = attention.sparse_decode(q, deq, torch.where(idx < 1024, idx, -1), width ** -0.5, 512, sink, lengths)
    out, lse, sched = _sparse(q, kv, idx, width, sink=sink, lengths=lengths)
    requests, tiles = _most_tiles(sched, [max(1, (int(n) + 63) // 64) for n in lengths])
    assert sched.size(0) == 148 and requests >= 3 and tiles >= 4
    assert_out_close("out", out, ref_out)
    assert_lse_close("lse", lse, ref_lse)


@pytest.mark.parametrize("width", [576, 512])
@pytest.mark.parametrize("h_q,page,extra_page", [(64, 61, 2), (64, 2, 69), (16, 64, 61)])
def test_sparse_decode_extra_cache(width, h_q, page, extra_page):
    """Main lists of an odd number of blocks, so that a tile holds both scopes; several tiles of each; two query tokens."""
    b, s_q, gen = 5, 2, torch.Generator().manual_seed(page)
    q = torch.randn(b, s_q, h_q, width, generator=gen).bfloat16()
    rows = lambda tokens, topk: torch.stack([torch.randperm(tokens, generator=gen)[:topk] for _ in range(b * s_q)]).view(b, s_q, topk).to(torch.int32)
    kv, deq = _records(width, torch.randn(-(-700 // page), page, 1, width, generator=gen).bfloat16())
    ekv, edeq = _records(width, torch.randn(-(-500 // extra_page), extra_page, 1, width, generator=gen).bfloat16())
    idx, eidx = rows(700, 448), rows(500, 320)
    for lengths, extra_lengths in ((None, None), (torch.tensor([448, 1, 0, 65, 192], dtype=torch.int32), torch.tensor([320, 64, 0, 65, 1], dtype=torch.int32))):
        ref_out, ref_lse = attention.sparse_decode(q, deq, idx, width ** -0.5, 512, None, lengths, edeq, eidx, extra_lengths)
        out, lse, _ = _sparse(q, kv, idx, width, lengths=lengths, extra_kv=ekv, extra_indices=eidx, extra_lengths=extra_lengths)
        assert_out_close("out", out, ref_out)
        assert_lse_close("lse", lse, ref_lse)


@pytest.mark.parametrize("width", [576, 512])
def test_gather_modes_heads_that_share_their_query(width):
    """A head stride of zero is no tensor map: the kernel's own threads load Q, several times in a CTA."""
    import flashmla_b200 as fm
    b, h_q, topk, gen = 330, 24, 192, torch.Generator().manual_seed(width)
    one = torch.randn(b, 1, 1, width, generator=gen).bfloat16()
    q = one.to(DEV).expand(-1, -1, h_q, -1)
    idx = torch.stack([torch.randperm(1000, generator=gen)[:topk] for _ in range(b)]).view(b, 1, topk).to(torch.int32)
    k = torch.randn(16, 64, 1, width, generator=gen).bfloat16()
    kv, deq = _records(width, k)
    assert q.stride(2) == 0
    ref_out, ref_lse = attention.sparse_decode(one.expand(-1, -1, h_q, -1).contiguous(), deq, idx, width ** -0.5, 512)
    out, lse, _ = _sparse(q, kv, idx, width)
    assert_out_close("out", out, ref_out)
    assert_lse_close("lse", lse, ref_lse)
    ref = attention.sparse_prefill(one[:, 0].expand(-1, h_q, -1).contiguous(), k.view(-1, 1, width), idx, width ** -0.5, 512)
    got = fm.flash_mla_sparse_fwd(q[:, 0], k.view(-1, 1, width).to(DEV), idx.to(DEV), width ** -0.5, 512)      # 330 tokens: three waves
    torch.cuda.synchronize()
    fm.check_status()
    assert_out_close("out", got[0], ref[0])
    assert_lse_close("max_logits", got[1], ref[1])
    assert_lse_close("lse", got[2], ref[2])


def _cache(width, b, s_kv, topk, s_q, h_q, seed):
    from tests import workloads as W
    d = W.sparse_decode_inputs(b, s_q, h_q, s_kv, topk, seed=seed, device="cpu")
    if width == 576:
        return d["q"], d["kv_fp8"], quant.dequantize_v32(d["kv_fp8"]), d["indices"]
    k = torch.randn(d["kv_fp8"].size(0), 64, 1, 512, generator=torch.Generator().manual_seed(seed)).bfloat16()
    kv = quant.quantize_model1(k)
    return d["q"][..., :512].contiguous(), kv, quant.dequantize_model1(kv), d["indices"]


@pytest.mark.parametrize("width", [576, 512])
@pytest.mark.parametrize("s_q,h_q,topk", [(1, 1, 64), (1, 16, 192), (2, 17, 128), (1, 48, 320), (1, 64, 640), (2, 64, 128),
                                          (1, 65, 192), (1, 128, 320)])
def test_sparse_decode(width, s_q, h_q, topk):
    """(The last two heads counts: the kernel for 128 rows.)"""
    import flashmla_b200 as fm
    b = 6
    q, kv, deq, idx = _cache(width, b, 700, topk, s_q, h_q, seed=h_q + topk)
    lengths = torch.tensor([topk, 0, 1, 65, topk - 1, 64], dtype=torch.int32)
    sink = torch.randn(h_q, generator=torch.Generator().manual_seed(1))
    kv_dev = kv.to(DEV).contiguous()
    for tl in (lengths, None):
        ref_out, ref_lse = attention.sparse_decode(q, deq, idx, width ** -0.5, 512, sink, tl)
        out, lse = fm.flash_mla_with_kvcache(q.to(DEV), kv_dev, None, None, 512, fm.get_mla_metadata()[0], None, width ** -0.5, False, True,
                                             idx.to(DEV), sink.to(DEV), None, None, None if tl is None else tl.to(DEV), None)
        torch.cuda.synchronize()
        fm.check_status()
        assert_out_close("out", out, ref_out)
        assert_lse_close("lse", lse, ref_lse)


@pytest.mark.parametrize("width", [576, 512])
@pytest.mark.parametrize("s_q,h_q,topk", [(1, 1, 64), (80, 1, 64), (90, 33, 128), (230, 64, 192), (20, 64, 704), (75, 64, 704), (100, 64, 704)])
def test_sparse_prefill(width, s_q, h_q, topk):
    """(On 148 SMs the kernel for 64 rows takes 75 to 148 and 223 to 296 tokens here, 704 keys from 76 tokens on; the one for pairs of
    SMs the others.)"""
    import flashmla_b200 as fm
    from tests import workloads as W
    d = W.sparse_prefill_inputs(s_q, h_q, 900, topk, seed=s_q)
    q, kv = d["q"].cpu()[..., :width].contiguous(), d["kv"].cpu()[..., :width].contiguous()
    idx = d["indices"].cpu().clone()
    idx[0, :, ::3] = -1
    idx[-1, :, 1::5] = 900
    lengths = torch.randint(0, topk + 1, (s_q,), generator=torch.Generator().manual_seed(3), dtype=torch.int32)
    sink = torch.randn(h_q, generator=torch.Generator().manual_seed(4))
    ref = attention.sparse_prefill(q, kv, idx, width ** -0.5, 512, sink, lengths)
    out, mx, lse = fm.flash_mla_sparse_fwd(q.to(DEV), kv.to(DEV), idx.to(DEV), width ** -0.5, 512, attn_sink=sink.to(DEV), topk_length=lengths.to(DEV))
    torch.cuda.synchronize()
    fm.check_status()
    assert_out_close("out", out, ref[0])
    assert_lse_close("max_logits", mx, ref[1])
    assert_lse_close("lse", lse, ref[2])
