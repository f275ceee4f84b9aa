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
