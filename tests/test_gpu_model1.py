"""GPU parity of the 512-wide ("MODEL1") forms of the sparse paths: FP8 decode on 584-byte records with e8m0 scales
(flash_mla/flash_mla_interface.py:99-103, csrc/api/sparse_decode.h:290-296) and token-sparse prefill with d_qk = 512,
against vectors generated by the reference's own torch code and against the CPU oracle."""
import os

import pytest
import torch

from oracle import attention, quant
from tests.helpers import assert_lse_close, assert_out_close, model1_cache_from_bytes, non_contiguousify

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _dev(t):
    return None if t is None else t.to(DEV)


def _decode(q, kv, indices, sm_scale, attn_sink=None, topk_length=None, extra_kv=None, extra_indices=None,
            extra_topk_length=None):
    import flashmla_b200 as fm
    meta, _ = fm.get_mla_metadata()
    out, lse = fm.flash_mla_with_kvcache(q, kv, None, None, 512, meta, None, sm_scale, False, True, indices, attn_sink,
                                         extra_kv, extra_indices, topk_length, extra_topk_length)
    torch.cuda.synchronize()
    fm.check_status()
    return out, lse


@pytest.mark.parametrize("impl", [1, 2])
def test_model1_decode_golden(golden_dir, impl):
    """Reference-generated vectors: attn_sink with +-inf, topk_length, an extra cache, 64- and 16-token blocks; through the
    all-shape kernel (1) and the tcgen05 kernel (2)."""
    import flashmla_b200 as fm
    fm.set_impl(impl)
    try:
        _model1_decode_golden(golden_dir)
    finally:
        fm.set_impl(0)


def _model1_decode_golden(golden_dir):
    for c in torch.load(os.path.join(golden_dir, "model1.pt"), weights_only=False)["decode"]:
        kv = model1_cache_from_bytes(c["kv_bytes"], c["kv_stride0"], DEV)
        extra = model1_cache_from_bytes(c["extra_kv_bytes"], c["extra_kv_stride0"], DEV) if "extra_kv_bytes" in c else None
        out, lse = _decode(_dev(c["q"]), kv, _dev(c["indices"]), c["sm_scale"], _dev(c["attn_sink"]), _dev(c["topk_length"]),
                           extra, _dev(c.get("extra_indices")), _dev(c.get("extra_topk_length")))
        assert out.shape == c["out"].shape and lse.shape == c["lse"].shape
        assert_out_close("out", out, c["out"])
        assert_lse_close("lse", lse, c["lse"])


@pytest.mark.parametrize("impl", [1, 2])
def test_model1_prefill_golden(golden_dir, impl):
    """Both kernel families: the all-shape kernel (1) and the tcgen05 kernel (2), which treats the missing ninth 64-column
    chunk of 512-wide rows as zeros."""
    import flashmla_b200 as fm
    fm.set_impl(impl)
    try:
        _model1_prefill_golden(golden_dir)
    finally:
        fm.set_impl(0)


def _model1_prefill_golden(golden_dir):
    import flashmla_b200 as fm
    for c in torch.load(os.path.join(golden_dir, "model1.pt"), weights_only=False)["prefill"]:
        out, mx, lse = fm.flash_mla_sparse_fwd(_dev(c["q"]), _dev(c["kv"]), _dev(c["indices"]), c["sm_scale"], 512,
                                               _dev(c["attn_sink"]), _dev(c["topk_length"]))
        torch.cuda.synchronize()
        assert_out_close("out", out, c["out"])
        assert_lse_close("max_logits", mx, c["max_logits"])
        assert_lse_close("lse", lse, c["lse"])


@pytest.mark.parametrize("b,s_q,h_q,s_kv,topk,page,sink", [
    (3, 2, 128, 1024, 320, 64, True),
    (5, 1, 64, 960, 192, 48, False),       # a block size that is not a power of two: 48 * 584 bytes padded to 49 * 576
    (2, 1, 200, 512, 128, 64, False),      # more heads than one row block
    (80, 1, 16, 256, 128, 64, True),       # more requests than pairs of SMs
    (200, 1, 16, 256, 128, 64, True),      # more requests than SM partitions
    (9, 2, 128, 4096, 2048, 64, False),    # the serving top-k: 16 tiles per request
])
@pytest.mark.parametrize("impl", [1, 2])
def test_model1_decode_cases(b, s_q, h_q, s_kv, topk, page, sink, impl):
    import flashmla_b200 as fm
    if impl == 2 and h_q > 128:
        pytest.skip("the tcgen05 kernel serves up to 128 heads")
    fm.set_impl(impl)
    try:
        _model1_decode_case(b, s_q, h_q, s_kv, topk, page, sink)
    finally:
        fm.set_impl(0)


def _model1_decode_case(b, s_q, h_q, s_kv, topk, page, sink):
    g = torch.Generator().manual_seed(b * 100 + h_q)
    nblk = b * (s_kv // page)
    block_table = torch.randperm(nblk, generator=g).to(torch.int32).view(b, -1)
    blocked_k = (torch.randn(nblk, page, 1, 512, generator=g) * 1.5).to(torch.bfloat16)
    kv = quant.quantize_model1(blocked_k)
    assert kv.stride(0) == quant.model1_block_bytes(page)
    kv_deq = quant.dequantize_model1(kv)
    q = torch.randn(b, s_q, h_q, 512, generator=g).to(torch.bfloat16)
    abs_idx = torch.stack([torch.stack([torch.randperm(s_kv, generator=g)[:topk] for _ in range(s_q)]) for _ in range(b)]).to(torch.int32)
    abs_idx[:, :, -7:] = -1
    abs_idx[0, 0, ::3] = -1
    phys = quant.abs_to_physical_indices(abs_idx, block_table, page)
    attn_sink = topk_length = None
    if sink:
        attn_sink = torch.randn(h_q, generator=g)
        attn_sink[0], attn_sink[-1] = float("inf"), float("-inf")
        topk_length = torch.randint(0, topk + 1, (b,), generator=g, dtype=torch.int32)
    sm_scale = 512 ** -0.5
    ref_out, ref_lse = attention.sparse_decode(q, kv_deq, phys, sm_scale, 512, attn_sink, topk_length)
    kv_dev = model1_cache_from_bytes(kv.contiguous().view(torch.uint8), kv.stride(0), DEV)
    out, lse = _decode(non_contiguousify(q.to(DEV)), kv_dev, non_contiguousify(phys.to(DEV)), sm_scale, _dev(attn_sink), _dev(topk_length))
    assert_out_close("out", out, ref_out)
    assert_lse_close("lse", lse, ref_lse)


@pytest.mark.parametrize("impl", [1, 2])
@pytest.mark.parametrize("s_q,h_q,s_kv,topk", [(37, 128, 1500, 256), (5, 64, 90, 128), (3, 136, 400, 64), (150, 128, 4096, 512)])
def test_model1_prefill_cases(s_q, h_q, s_kv, topk, impl):
    import flashmla_b200 as fm
    fm.set_impl(impl)
    try:
        _model1_prefill_case(s_q, h_q, s_kv, topk)
    finally:
        fm.set_impl(0)


def _model1_prefill_case(s_q, h_q, s_kv, topk):
    import flashmla_b200 as fm
    g = torch.Generator().manual_seed(s_q)
    q = (torch.randn(s_q, h_q, 512, generator=g) / 2).to(torch.bfloat16)
    kv = torch.randn(s_kv, 1, 512, generator=g).to(torch.bfloat16)
    idx = torch.full((s_q, 1, topk), -1, dtype=torch.int32)
    n = min(topk, s_kv)
    for r in range(s_q):
        idx[r, 0, :n] = torch.randperm(s_kv, generator=g)[:n].to(torch.int32)
    idx[:, 0, 5] = s_kv                       # out of range: invalid
    idx[1] = 2147483647                       # a query token without any valid key
    sink = torch.randn(h_q, generator=g)
    tl = torch.randint(0, topk + 1, (s_q,), generator=g, dtype=torch.int32)
    ref = attention.sparse_prefill(q, kv, idx, 0.7 * 512 ** -0.5, 512, sink, tl)
    out, mx, lse = fm.flash_mla_sparse_fwd(non_contiguousify(q.to(DEV)), non_contiguousify(kv.to(DEV)), idx.to(DEV),
                                           0.7 * 512 ** -0.5, 512, sink.to(DEV), tl.to(DEV))
    torch.cuda.synchronize()
    assert_out_close("out", out, ref[0])
    assert_lse_close("max_logits", mx, ref[1])
    assert_lse_close("lse", lse, ref[2])


def test_model1_cache_writer_bit_exact(golden_dir):
    """The cache-writer kernel against the reference's own quantised bytes and against the oracle on further inputs
    (zero rows, huge rows, a block size that needs padding)."""
    from flashmla_b200.kvcache import model1_block_bytes, quantize_fp8_kvcache_model1

    def compare(mine, ref_bytes, nb, bs):
        a = mine.contiguous().view(torch.uint8).cpu().view(nb, -1)
        b = ref_bytes.view(nb, -1)
        assert torch.equal(a[:, :bs * 576], b[:, :bs * 576])
        assert torch.equal(a[:, bs * 576:].view(nb, bs, 8)[..., :7], b[:, bs * 576:].view(nb, bs, 8)[..., :7])

    c = torch.load(os.path.join(golden_dir, "model1.pt"), weights_only=False)["quant"]
    nb, bs = c["x"].shape[:2]
    qz = quantize_fp8_kvcache_model1(c["x"].to(DEV))
    assert qz.stride(0) == c["quant_stride0"] == model1_block_bytes(bs)
    compare(qz, c["quant_bytes"], nb, bs)
    g = torch.Generator().manual_seed(5)
    for nb, bs, mag in ((7, 48, 1.0), (3, 64, 300.0), (5, 2, 1e-3)):
        x = (torch.randn(nb, bs, 1, 512, generator=g) * mag).to(torch.bfloat16)
        x[0, 0] = 0
        x[-1, -1, 0, :64] = 3e38
        ref = quant.quantize_model1(x)
        qz = quantize_fp8_kvcache_model1(x.to(DEV))
        assert qz.stride(0) == ref.stride(0)
        compare(qz, ref.contiguous().view(torch.uint8), nb, bs)
    # and the kernel-written cache feeds the decode path
    x = torch.randn(4, 64, 1, 512, generator=g).to(torch.bfloat16)
    kv = quantize_fp8_kvcache_model1(x.to(DEV))
    q = torch.randn(1, 1, 16, 512, generator=g).to(torch.bfloat16)
    idx = torch.randperm(256, generator=g)[:128].to(torch.int32).view(1, 1, 128)
    ref_out, ref_lse = attention.sparse_decode(q, quant.dequantize_model1(quant.quantize_model1(x)), idx, 512 ** -0.5, 512)
    out, lse = _decode(q.to(DEV), kv, idx.to(DEV), 512 ** -0.5)
    assert_out_close("out", out, ref_out)
    assert_lse_close("lse", lse, ref_lse)


def test_model1_rejects_wrong_record_size():
    import flashmla_b200 as fm
    q = torch.zeros(1, 1, 8, 512, dtype=torch.bfloat16, device=DEV)
    kv = torch.zeros(2, 64, 1, 656, dtype=torch.uint8, device=DEV).view(torch.float8_e4m3fn)
    idx = torch.zeros(1, 1, 64, dtype=torch.int32, device=DEV)
    meta, _ = fm.get_mla_metadata()
    with pytest.raises(RuntimeError, match="584"):
        fm.flash_mla_with_kvcache(q, kv, None, None, 512, meta, None, None, False, True, idx)


@pytest.mark.parametrize("block_size", [64, 1, 61, 72])
def test_model1_block_padding_is_zero(block_size):
    """The bytes behind a block's records (blocks are padded to a multiple of 576 bytes) are part of what is saved or sent
    with the storage: zeros, whatever the memory held before."""
    from flashmla_b200.kvcache import model1_block_bytes, quantize_fp8_kvcache_model1
    blocks, n = 7, model1_block_bytes(block_size)
    x = torch.randn(blocks, block_size, 1, 512, generator=torch.Generator().manual_seed(block_size)).to(torch.bfloat16).to("cuda:0")
    dirty = torch.full((blocks * n,), 0xa5, dtype=torch.uint8, device="cuda:0")
    del dirty                                      # the allocator hands the same memory out again
    got = quantize_fp8_kvcache_model1(x)
    assert got.stride(0) == n
    whole = got.view(torch.uint8).as_strided((blocks, n), (n, 1))
    assert not whole[:, block_size * 584:].any()
    assert torch.equal(got.view(torch.uint8).cpu(), quant.quantize_model1(x.cpu()).view(torch.uint8))


@pytest.mark.parametrize("impl", [1, 2])
@pytest.mark.parametrize("h_q", [16, 64, 128])
def test_exponent_bytes_at_their_ends(h_q, impl):
    """Scale bytes 0 (2^-127, a subnormal), 1 and 2 in every place of a record: values are those of the format to 2^-7 (16-bit probabilities and
    outputs: 2^-9 each; values of one sign).  Byte 255 is NaN: the request that has such a key gets no number (NaN, or the zeros of a request without
    keys), the other nothing of it."""
    import flashmla_b200 as fm
    gen, tokens, topk = torch.Generator().manual_seed(h_q), 256, 128
    kv = quant.quantize_model1(torch.randn(4, 64, 1, 512, generator=gen).bfloat16())
    data = kv.contiguous().view(torch.uint8).reshape(4, -1)
    values, scales = data[:, :64 * 576].view(4, 64, 576), data[:, 64 * 576:].view(4, 64, 8)
    values[..., :448] = torch.randint(0x78, 0x7f, (4, 64, 448), generator=gen, dtype=torch.uint8)      # 256 .. 448
    scales[..., :7] = torch.randint(0, 3, (4, 64, 7), generator=gen, dtype=torch.uint8)
    e4m3 = values[..., :448].clone().view(torch.float8_e4m3fn).double().view(tokens, 7, 64)
    keys = torch.cat([(e4m3 * torch.exp2(scales[..., :7].double().view(tokens, 7, 1) - 127)).view(tokens, 448),
                      values[..., 448:].clone().view(torch.bfloat16).double().view(tokens, 64)], 1)
    scales[3, 8, 3] = 255                                                   # token 200
    idx = torch.stack([torch.randperm(200, generator=gen)[:topk], torch.randperm(256, generator=gen)[:topk]]).view(2, 1, topk).to(torch.int32)
    idx[1, 0, 77] = 200
    q = (torch.randn(2, 1, h_q, 512, generator=gen) * 0.1).bfloat16()
    fm.set_impl(impl)
    try:
        out, lse = _decode(q.to(DEV), model1_cache_from_bytes(data.view(4, 64, 1, 584), quant.model1_block_bytes(64), DEV), idx.to(DEV), 512 ** -0.5)
    finally:
        fm.set_impl(0)
    chosen = keys[idx[0, 0].long()]
    score = q[0, 0].double() @ chosen.T * 512 ** -0.5
    want = torch.softmax(score, -1) @ chosen
    got = out[0, 0].cpu().double()
    assert (want[:, :448] > 0).all() and ((got - want)[:, :448].abs() <= 2 ** -7 * want[:, :448]).all()
    assert_out_close("RoPE columns", got[:, 448:], want[:, 448:])
    assert_lse_close("lse", lse[0, :, 0], torch.logsumexp(score, -1))
    assert (out[1].isnan() | (out[1] == 0)).all() and not lse[1].isfinite().any()
