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
