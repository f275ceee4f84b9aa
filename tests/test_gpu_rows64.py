"""GPU: the kernel for up to 64 query rows on one SM (csrc/attn_rows64.cu) at the sizes where it can go wrong: rows at the edges
of its variants (16 / 32 / 64), tiles of 128 tokens and their remainders, scores that keep growing, Q that TMA cannot address,
schedules with another number of partitions.  Against the CPU oracle, within the bounds of tests/helpers.py (element-wise
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
    """Every tile raises the running maximum by more than the rescale threshold: the RoPE part of K (not part of V) grows with the
    token's position."""
    q, k, bt, sl = _dense_inputs(1, h_q, 1, [1500, 129, 700], seed=5)
    for b in range(3):
        for j, page in enumerate(bt[b, :(int(sl[b]) + 63) // 64].tolist()):
            k[page, :, :, 512:] *= 1.0 + 6.0 * j
    ref_out, ref_lse = attention.dense_decode(q, k, bt, sl, 512, False)
    out, lse = _dense(q, k, bt, sl, False)
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
