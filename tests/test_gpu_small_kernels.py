"""GPU: edges of the helper kernels' variants - the combine kernel's warps per row (chosen by the number of rows), the
scheduler's windows of 32 requests, the cache writer's division."""
import numpy as np
import pytest
import torch

from oracle import quant, sched_meta
from tests.test_gpu_sched_combine import _combine_ref, _run_meta

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("h_q,counts", [
    (3, [33]),                                    # 8 warps per row; one split beyond a block of 32 weights
    (128, [74]),
    (128, [2, 1, 9]),                             # 4 warps per row
    (101, [1, 2, 3, 4, 5]),                       # 4, last CTA of a request half full
    (128, [3, 1, 66] * 4),                        # 2 warps per row
    (96, [2, 1, 5] * 7 + [70]),                   # 1 warp per row
])
def test_combine_warps_per_row(h_q, counts):
    from flashmla_b200 import _capi
    gen = torch.Generator().manual_seed(len(counts))
    b, total = len(counts), sum(counts)
    ns = torch.tensor([0] + list(np.cumsum(counts)), dtype=torch.int32)
    lse_acc = torch.randn(total, 1, h_q, generator=gen) * 3
    lse_acc[0, 0, 0] = float("-inf")
    o_acc = torch.randn(total, 1, h_q, 512, generator=gen)
    out0, lse0 = torch.randn(b, 1, h_q, 512, generator=gen).to(torch.bfloat16), torch.randn(b, h_q, 1, generator=gen)
    ref_out, ref_lse = _combine_ref(lse_acc, o_acc, ns, b, 1, h_q, None, out0, lse0)
    out, lse, la, oa, nd = out0.to(DEV), lse0.to(DEV), lse_acc.to(DEV), o_acc.to(DEV), ns.to(DEV)
    c = _capi.CombineArgs(b=b, s_q=1, h_q=h_q, d_v=512, lse=_capi.ptr(lse), lse_stride_b=lse.stride(0), lse_stride_s=lse.stride(2),
                          lse_stride_h=lse.stride(1), out=_capi.ptr(out), o_stride_b=out.stride(0), o_stride_s=out.stride(1),
                          o_stride_h=out.stride(2), lse_accum=_capi.ptr(la), o_accum=_capi.ptr(oa), num_splits=_capi.ptr(nd),
                          attn_sink=None, stream=torch.cuda.current_stream().cuda_stream)
    _capi.check(_capi.lib().mla_combine(c), "mla_combine")
    # fp32 sums in another order, then one rounding to bf16: at most one bf16 step (2^-8 of the value, or of the terms' size)
    assert torch.allclose(out.cpu().float(), ref_out.to(torch.bfloat16).float(), rtol=2 ** -7, atol=1e-5)
    assert torch.allclose(lse.cpu(), ref_lse, rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("h_q,counts", [
    (1, [2]), (16, [64, 1, 3]), (49, [65, 63, 8]),    # a row's columns in two CTAs; 64 splits are in flight at once
    (148, [65]), (149, [64]),                         # ... up to a row per SM
])
def test_combine_columns_in_two_ctas(h_q, counts):
    test_combine_warps_per_row(h_q, counts)


@pytest.mark.parametrize("h_q,counts", [
    (49, [17, 15, 64]), (50, [65, 63, 8]),        # 147 and 150 rows: two CTAs a row up to a row per SM (148), one beyond
    (128, [2]), (128, [65]), (16, [16, 17, 2]),   # one request of 128 rows; rows of few splits beside others
])
def test_combine_up_to_a_row_per_sm(h_q, counts):
    test_combine_warps_per_row(h_q, counts)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("with_sink", [False, True])
@pytest.mark.parametrize("h_q,counts", [(24, [16, 50]), (8, [17, 3, 66])])
def test_combine_columns_in_two_ctas_two_query_tokens(h_q, counts, dtype, with_sink):
    test_combine_variants_two_query_tokens(h_q, counts, dtype, with_sink)


@pytest.mark.parametrize("b", [1, 31, 32, 33, 64, 255, 256, 257, 1000])
@pytest.mark.parametrize("parts", [1, 74, 300])
def test_schedule_window_edges(b, parts):
    gen = np.random.default_rng(b * 1000 + parts)
    seq = [int(x) for x in gen.integers(0, 3000, b)]
    seq[-1], seq[0] = 0, 40000
    meta, ns = _run_meta(b, parts, 64, 5, seqlens=seq)
    want_meta, want_ns = sched_meta.get_sched_meta(b, parts, 64, 5, seqlens_k=seq)
    assert np.array_equal(np.asarray(meta)[:, :7], want_meta[:, :7]) and np.array_equal(np.asarray(ns), want_ns)


@pytest.mark.parametrize("tokens", [1, 2, 63])
@pytest.mark.parametrize("pow2", [False, True])
def test_written_records_over_the_exponent_range(tokens, pow2):
    """Groups from the smallest to the largest bf16 magnitudes: the fast quotient and, outside its range, the division."""
    from flashmla_b200.kvcache import quantize_fp8_kvcache
    gen = torch.Generator().manual_seed(tokens)
    x = torch.randn(5, tokens, 1, 576, generator=gen)
    x[..., :512] *= torch.exp2(torch.randint(-125, 120, (5, tokens, 1, 4), generator=gen).float()).repeat_interleave(128, dim=-1)
    x[..., 7:512:16] *= 2.0 ** -21                 # far below the group's largest value
    x[0, 0, 0, 128:256] = 0
    x = x.to(torch.bfloat16)
    got = quantize_fp8_kvcache(x.to(DEV), pow2).view(torch.uint8).cpu()
    assert torch.equal(got, quant.quantize_v32(x, pow2_scale=pow2).view(torch.uint8))


def _records_by_division(x, width, pow2):
    """(value bytes [..., 512 or 448], scales [..., groups] fp32) of x [blocks, tokens, 1, width], by plain fp32 division.
    NaNs do not count towards a group's largest magnitude."""
    group, values = (128, 512) if width == 576 else (64, 448)
    f = x.squeeze(2)[..., :values].float().unflatten(-1, (-1, group))
    s = torch.where(f.isnan(), 0.0, f.abs()).amax(-1, keepdim=True) / 448
    s = torch.exp2(s.clamp_min(1e-4).log2().ceil()) if pow2 or width == 512 else s.clamp_min(1e-30)
    return (f / s).to(torch.float8_e4m3fn).view(torch.uint8).flatten(-2), s.squeeze(-1)


def _signed_zero_rows(width):
    """A block of token rows: ordinary groups, all-zero groups, and rows whose groups force the division (warps choose
    between quotient and division by all groups of their token), all with zeros of both signs."""
    gen = torch.Generator().manual_seed(width)
    group = 128 if width == 576 else 64
    x = torch.randn(3, 9, 1, width, generator=gen)
    x[:, 1, ..., :group] = 0                       # an all-zero group beside ordinary ones
    x[:, 2] = 0                                    # nothing but zeros
    x[:, 3, ..., group:2 * group] *= 2.0 ** -100   # this row divides
    x[:, 4, ..., :group] *= 2.0 ** 110
    x[:, 5, ..., :group] *= 2.0 ** -55             # the smallest of the quotient's range
    x[..., 3::7] = 0.0
    x[..., 5::11] = -0.0
    return x.to(torch.bfloat16)


@pytest.mark.parametrize("width,pow2", [(576, False), (576, True), (512, True)])
@pytest.mark.parametrize("special", [None, "nan", "inf"])
def test_written_records_signed_zeros_and_specials(width, pow2, special):
    """Byte for byte against the division: zeros keep their sign (0x80 for -0) wherever they stand, NaN stays NaN, and a group
    with an infinity has NaN in its place and signed zeros elsewhere."""
    from flashmla_b200.kvcache import quantize_fp8_kvcache, quantize_fp8_kvcache_model1
    x = _signed_zero_rows(width)
    if special == "nan":
        x[:, 6:, ..., 9:200:50] = float("nan")     # in ordinary groups, beside zeros
        x[:, 2, ..., 4] = float("nan")             # in an all-zero group
    elif special == "inf":
        x[:, 6:, ..., 9] = float("inf")
        x[:, 7, ..., 200] = float("-inf")
    got = (quantize_fp8_kvcache(x.to(DEV), pow2) if width == 576 else quantize_fp8_kvcache_model1(x.to(DEV))).view(torch.uint8).cpu()
    want, scale = _records_by_division(x, width, pow2)
    blocks, tokens = x.shape[:2]
    if width == 576:
        rows = got.squeeze(2)
        assert torch.equal(rows[..., 512:528].contiguous().view(torch.int32), scale.contiguous().view(torch.int32))
    else:
        flat = got.reshape(blocks, -1)
        rows = flat[:, :tokens * 576].view(blocks, tokens, 576)
        assert torch.equal(flat[:, tokens * 576:].view(blocks, tokens, 8)[..., :7], (scale.view(torch.int32) >> 23).to(torch.uint8))
    rows = rows[..., :want.shape[-1]]
    is_nan = (want & 0x7f) == 0x7f
    assert torch.equal((rows & 0x7f) == 0x7f, is_nan)
    assert torch.equal(rows[~is_nan], want[~is_nan])
    assert (want == 0x80).sum() > 500              # the case is not empty
    if special is None:                            # and the repository's restatement of the reference says the same
        full = quant.quantize_v32(x, pow2_scale=pow2) if width == 576 else quant.quantize_model1(x)
        assert torch.equal(got, full.view(torch.uint8).contiguous())


@pytest.mark.parametrize("blocks,page", [(39999, 1), (625, 64), (3077, 13), (40003, 1)])
def test_512_wide_writer_around_forty_thousand_tokens(blocks, page):
    """Up to 40000 tokens a warp takes one, above two (the last warp of an odd count one): 39999, 40000, 40001, 40003 tokens."""
    from flashmla_b200.kvcache import quantize_fp8_kvcache_model1
    x = (torch.randn(blocks, page, 1, 512, generator=torch.Generator().manual_seed(blocks)) * 3).to(torch.bfloat16)
    got = quantize_fp8_kvcache_model1(x.to(DEV))
    assert torch.equal(got.view(torch.uint8).cpu(), quant.quantize_model1(x).view(torch.uint8))


@pytest.mark.parametrize("h_q,counts", [
    (64, [41]),                                   # 8 warps per row
    (64, [2, 1, 9]),                              # 4
    (50, [3, 1, 34] * 4),                         # 2
    (50, [2, 1, 5, 9] * 5),                       # 1
])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("with_sink", [False, True])
def test_combine_variants_two_query_tokens(h_q, counts, dtype, with_sink):
    """Every number of warps per row with two query tokens, both output types, attention sinks (infinite ones too) and a row
    without keys."""
    from flashmla_b200 import _capi
    gen = torch.Generator().manual_seed(h_q + len(counts))
    b, s_q, total = len(counts), 2, sum(counts)
    ns = torch.tensor([0] + list(np.cumsum(counts)), dtype=torch.int32)
    lse_acc = torch.randn(total, s_q, h_q, generator=gen) * 3
    o_acc = torch.randn(total, s_q, h_q, 512, generator=gen)
    lse_acc[0, 1, 2] = float("-inf")                                       # an empty split
    lse_acc[:counts[0], 0, 3], o_acc[:counts[0], 0, 3] = float("-inf"), 0  # a row of request 0 without keys
    sink = torch.randn(h_q, generator=gen) if with_sink else None
    if with_sink:
        sink[0], sink[1], sink[3] = float("inf"), float("-inf"), float("inf")
    out0, lse0 = torch.randn(b, s_q, h_q, 512, generator=gen).to(dtype), torch.randn(b, h_q, s_q, generator=gen)
    ref_out, ref_lse = _combine_ref(lse_acc, o_acc, ns, b, s_q, h_q, sink, out0, lse0)
    out, lse, la, oa, nd = out0.to(DEV), lse0.to(DEV), lse_acc.to(DEV), o_acc.to(DEV), ns.to(DEV)
    sink_d = sink.to(DEV) if with_sink else None
    c = _capi.CombineArgs(b=b, s_q=s_q, h_q=h_q, d_v=512, lse=_capi.ptr(lse), lse_stride_b=lse.stride(0), lse_stride_s=lse.stride(2),
                          lse_stride_h=lse.stride(1), out=_capi.ptr(out), o_stride_b=out.stride(0), o_stride_s=out.stride(1),
                          o_stride_h=out.stride(2), lse_accum=_capi.ptr(la), o_accum=_capi.ptr(oa), num_splits=_capi.ptr(nd),
                          attn_sink=_capi.ptr(sink_d), dtype=_capi.MLA_DTYPE_FP16 if dtype == torch.float16 else _capi.MLA_DTYPE_BF16,
                          stream=torch.cuda.current_stream().cuda_stream)
    _capi.check(_capi.lib().mla_combine(c), "mla_combine")
    # fp32 sums in another order, then one rounding: at most one step of the output type (2^-7 / 2^-10 of the value)
    step = 2 ** -7 if dtype == torch.bfloat16 else 2 ** -10
    assert torch.allclose(out.cpu().float(), ref_out.to(dtype).float(), rtol=step, atol=1e-5, equal_nan=True)
    assert torch.allclose(lse.cpu(), ref_lse, rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("b", [1, 2, 33, 128])
@pytest.mark.parametrize("parts", [1, 31, 32, 33, 64, 65])
def test_schedule_rows_in_groups_of_32_partitions(b, parts):
    """The walk finishes 32 metadata rows at a time: the last row of a group ends where the next group starts, and the work may
    end inside a group or with it."""
    for longest in (0, 64, 5000, 90000):
        gen = np.random.default_rng(b * 100 + parts + longest)
        seq = [int(x) for x in gen.integers(0, longest + 1, b)]
        seq[-1] = longest
        meta, ns = _run_meta(b, parts, 64, 5, seqlens=seq)
        want_meta, want_ns = sched_meta.get_sched_meta(b, parts, 64, 5, seqlens_k=seq)
        assert np.array_equal(np.asarray(meta)[:, :7], want_meta[:, :7]) and np.array_equal(np.asarray(ns), want_ns)


@pytest.mark.parametrize("width,pages,h_q", [(576, 3, 64), (576, 1031, 128), (512, 3, 128), (512, 700, 64)])
def test_writer_in_a_captured_graph(width, pages, h_q):
    """The writers as links of the launch chain: in a graph behind the kernel that makes their input and in front of the decode that reads the records,
    which starts while they run.  Replayed with other inputs; bytes and results are those of single launches with the device idle between them."""
    import flashmla_b200 as fm
    from flashmla_b200.kvcache import quantize_fp8_kvcache, quantize_fp8_kvcache_model1
    write = quantize_fp8_kvcache if width == 576 else quantize_fp8_kvcache_model1
    gen = torch.Generator(device=DEV).manual_seed(pages)
    new = lambda: torch.randn(pages, 64, 1, width, generator=gen, device=DEV).bfloat16()
    q = torch.randn(2, 1, h_q, width, generator=gen, device=DEV).bfloat16()
    # the last tokens that the writers write, and some of the others
    idx = torch.randint(0, pages * 64, (2, 1, 192), generator=gen, device=DEV, dtype=torch.int32)
    idx[..., :64] = torch.arange(pages * 64 - 64, pages * 64, device=DEV, dtype=torch.int32)
    source, meta = new(), fm.get_mla_metadata()[0]

    def step(wait):
        made = source * 0.5
        wait()
        records = write(made)
        wait()
        return (records,) + fm.flash_mla_with_kvcache(q, records, None, None, 512, meta, None, width ** -0.5, False, True, idx)

    step(torch.cuda.synchronize)                   # (makes the schedule, loads the kernels)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = step(lambda: None)
    for _ in range(4):
        source.copy_(new())
        graph.replay()
        torch.cuda.synchronize()
        want = step(torch.cuda.synchronize)
        torch.cuda.synchronize()
        assert torch.equal(got[0].view(torch.uint8), want[0].view(torch.uint8))
        assert torch.equal(got[1], want[1]) and torch.equal(got[2], want[2])
    fm.check_status()
