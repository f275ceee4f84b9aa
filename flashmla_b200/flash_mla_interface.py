"""Host-side mirror of the reference's Python API for the MLA decode / sparse-prefill path
(flash_mla/flash_mla_interface.py:8-211 of deepseek-ai/FlashMLA): same function names, parameter
order, keywords, assertion texts and return shapes, so existing call sites only change the import.

PyTorch is used for device memory and the current stream; csrc/host.cpp checks the arguments, allocates the outputs and
launches every kernel through the C ABI of libflashmla_b200.so (include/flashmla_b200.h).  There is no CPU path.
"""
import dataclasses
from typing import Optional, Tuple

import torch

from . import _capi
from ._capi import ptr

# Kernel selection for tests / benchmarks: 0 = fastest supporting kernel, 1 = portable, 2 = tcgen05
_impl_override = 0


# Optional kernel timer for benchmarks: an object with start(name) / stop(name) that records CUDA events on
# the current stream around each kernel launch.  None (the default) costs nothing.
_kernel_timer = None


def set_kernel_timer(timer) -> None:
    global _kernel_timer
    _kernel_timer = timer


def _status(device) -> torch.Tensor:
    """The device's status words, written by kernels whose bounded waits ran out: [first code, count, -, -]."""
    device = torch.device(device)
    return _capi.host().status(torch.cuda.current_device() if device.index is None else device.index)


def check_status(device=None) -> None:
    """Synchronises and raises if a kernel reported that one of its bounded waits ran out (a pipeline
    error: the results of that launch are invalid).  The status words are cleared."""
    for buf in _capi.host().known_status():
        if device is not None and buf.device != torch.device(device):
            continue
        vals = buf.cpu().tolist()
        if vals[0] != 0:
            buf.zero_()
            raise RuntimeError(f"flashmla_b200: a kernel on {buf.device} gave up a bounded wait (code {vals[0]}, {vals[1]} threads)")


def set_impl(impl: int) -> None:
    """Force a kernel family (0 auto, 1 portable mma.sync kernel, 2 tcgen05 kernel)."""
    global _impl_override
    assert impl in (0, 1, 2)
    _impl_override = impl


@dataclasses.dataclass
class FlashMLASchedMeta:
    """
    A class that stores the tile scheduler metadata of FlashMLA
    """

    @dataclasses.dataclass
    class Config:
        b: int
        s_q: int
        h_q: int
        page_block_size: int
        h_k: int

        causal: bool
        is_fp8_kvcache: bool
        topk: Optional[int]

        extra_page_block_size: Optional[int]
        extra_topk: Optional[int]

    have_initialized: bool = False

    config: Optional[Config] = None

    tile_scheduler_metadata: Optional[torch.Tensor] = None   # (num_sm_parts, 8), dtype torch.int32.
    num_splits: Optional[torch.Tensor] = None                # (batch_size + 1), dtype torch.int32.

    # Not in the reference: how the stored schedule was made.  Sparse decode without per-request lengths uses one
    # partition per request where that fits (and then needs no combine step); with lengths it uses the general partition
    # count.  The reference's partition count never depends on the lengths, so it accepts a call that switches between
    # the two on one sched_meta: here the schedule is made again for such a call.
    uniform_costs: Optional[bool] = None


# the fields of a schedule's configuration and what the caller knows them as
_CONFIG_NAMES = (("b", "batch_size"), ("s_q", "seq_len_q"), ("h_q", "num_heads_q"), ("page_block_size", "page_block_size"),
                 ("h_k", "num_heads_k"), ("causal", "causal"), ("is_fp8_kvcache", "is_fp8_kvcache"),
                 ("topk", "the last dim of indices_in_kvcache"), ("extra_page_block_size", "the page_block_size of extra_k_cache"),
                 ("extra_topk", "the last dim of extra_indices_in_kvcache"))


def get_mla_metadata(*args, **kwargs) -> Tuple[FlashMLASchedMeta, None]:
    """
    Returns an empty FlashMLASchedMeta; the scheduling metadata is generated by the first
    flash_mla_with_kvcache call that uses it.  Arguments are accepted and ignored for
    compatibility with the old interface.  Returns (FlashMLASchedMeta, None).
    """
    return FlashMLASchedMeta(), None


def _make_sched_meta(b, s_q, num_sm_parts, device, seqlens_k=None, topk=-1, extra_topk=0,
                     topk_length=None, extra_topk_length=None):
    """A schedule for callers of the C ABI (the calls below make theirs on the way)."""
    host = _capi.host()
    meta = torch.empty((num_sm_parts, host.META_INTS), dtype=torch.int32, device=device)
    num_splits = torch.empty((b + 1,), dtype=torch.int32, device=device)
    a = _capi.SchedMetaArgs(
        b=b, s_q=s_q, block_size_n=host.BLOCK_SIZE_N, fixed_overhead_num_blocks=host.FIXED_OVERHEAD_NUM_BLOCKS,
        topk=topk, extra_topk=extra_topk,
        topk_length=ptr(topk_length), extra_topk_length=ptr(extra_topk_length), seqlens_k=ptr(seqlens_k),
        meta=ptr(meta), num_splits=ptr(num_splits), num_sm_parts=num_sm_parts, stream=torch.cuda.current_stream(device).cuda_stream)
    _capi.check(_capi.lib().mla_get_sched_meta(a), "mla_get_sched_meta")
    return meta, num_splits


def flash_mla_with_kvcache(
    q: torch.Tensor,
    k_cache: torch.Tensor,
    block_table: Optional[torch.Tensor],
    cache_seqlens: Optional[torch.Tensor],
    head_dim_v: int,
    tile_scheduler_metadata: FlashMLASchedMeta,
    num_splits: None = None,
    softmax_scale: Optional[float] = None,
    causal: bool = False,
    is_fp8_kvcache: bool = False,
    indices: Optional[torch.Tensor] = None,
    attn_sink: Optional[torch.Tensor] = None,
    extra_k_cache: Optional[torch.Tensor] = None,
    extra_indices_in_kvcache: Optional[torch.Tensor] = None,
    topk_length: Optional[torch.Tensor] = None,
    extra_topk_length: Optional[torch.Tensor] = None,
    is_causal: Optional[bool] = None,
) -> Tuple[torch.Tensor, torch.Tensor]:
    """
    MLA decode with a paged KV cache.  Same contract as the reference's flash_mla_with_kvcache
    (flash_mla/flash_mla_interface.py:53-173):

        q: (batch_size, seq_len_q, num_heads_q, 576) bf16 (sparse FP8 also 512, with the 584-byte records)
        k_cache: dense: (num_blocks, 64, num_heads_k, 576) bf16;
                 sparse FP8: (num_blocks, page_block_size, 1, 656) bytes -- per token 512 e4m3 values,
                 4 fp32 scales (one per 128 values), 64 bf16 RoPE values; or, with 512-wide queries,
                 (num_blocks, page_block_size, 1, 584) bytes -- per block page_block_size x (448 e4m3 + 64 bf16 RoPE)
                 followed by page_block_size x (7 e8m0 scales + 1 pad byte)
        block_table: (batch_size, max_num_blocks_per_seq) int32 (dense)
        cache_seqlens: (batch_size) int32 (dense)
        head_dim_v: 512
        tile_scheduler_metadata: the FlashMLASchedMeta returned by get_mla_metadata(); may be reused while
                 shapes and cache_seqlens / topk_length / extra_topk_length stay the same
        num_splits: must be None
        softmax_scale: default 1 / sqrt(576)
        causal: dense attention only (`is_causal` is accepted as an alias)
        indices: (batch_size, seq_len_q, topk) int32, page * page_block_size + offset, -1 = invalid
        attn_sink: (num_heads_q) fp32; scales the output by exp(lse) / (exp(lse) + exp(attn_sink))
        extra_k_cache / extra_indices_in_kvcache / topk_length / extra_topk_length: as in the reference

    Returns (out (batch_size, seq_len_q, num_heads_q, 512), softmax_lse (batch_size, num_heads_q, seq_len_q) fp32).
    """
    if is_causal is not None:
        causal = is_causal
    sched_meta = tile_scheduler_metadata
    indices_in_kvcache = indices
    assert isinstance(sched_meta, FlashMLASchedMeta), "tile_scheduler_metadata must be of type FlashMLASchedMeta"
    assert num_splits is None, "num_splits must be None"

    q_shape, k_shape = q.shape, k_cache.shape
    topk = indices_in_kvcache.shape[-1] if indices_in_kvcache is not None else None
    extra_k_page_block_size = extra_k_cache.shape[1] if extra_k_cache is not None else None
    extra_topk = extra_indices_in_kvcache.shape[-1] if extra_indices_in_kvcache is not None else None
    if softmax_scale is None:
        softmax_scale = q_shape[-1] ** (-0.5)

    if not sched_meta.have_initialized:
        if indices_in_kvcache is not None:
            assert not causal, "causal must be False when indices_in_kvcache is not None (i.e. sparse attention is enabled)"
        sched_meta.have_initialized = True
        sched_meta.config = FlashMLASchedMeta.Config(
            q_shape[0], q_shape[1], q_shape[2], k_shape[1], k_shape[2],
            causal, is_fp8_kvcache, topk, extra_k_page_block_size, extra_topk)
    else:
        cfg = sched_meta.config
        assert cfg is not None
        given = (q_shape[0], q_shape[1], q_shape[2], k_shape[1], k_shape[2], causal, is_fp8_kvcache, topk, extra_k_page_block_size, extra_topk)
        if given != (cfg.b, cfg.s_q, cfg.h_q, cfg.page_block_size, cfg.h_k, cfg.causal, cfg.is_fp8_kvcache, cfg.topk,
                     cfg.extra_page_block_size, cfg.extra_topk):
            for (name, what), value in zip(_CONFIG_NAMES, given):
                assert getattr(cfg, name) == value, (
                    f"sched_meta.config.{name} must be equal to {what}. Your input arguments are inconsistent with sched_meta. "
                    "Please make sure the input arguments are consistent across different invocations of flash_mla_with_kvcache on the same sched_meta.")

    host = _capi.host()
    if topk is not None:
        assert not causal, "causal must be False when sparse attention is enabled"
        assert is_fp8_kvcache, "is_fp8_kvcache must be True when sparse attention is enabled"
        uniform = topk_length is None and extra_topk_length is None
        if sched_meta.tile_scheduler_metadata is not None and sched_meta.uniform_costs != uniform:
            sched_meta.tile_scheduler_metadata = sched_meta.num_splits = None      # made under the other partition rule
        sched_meta.uniform_costs = uniform
        out, lse, sched_meta.tile_scheduler_metadata, sched_meta.num_splits = host.sparse_decode(
            q, k_cache, indices_in_kvcache, topk_length, attn_sink,
            sched_meta.tile_scheduler_metadata, sched_meta.num_splits,
            extra_k_cache, extra_indices_in_kvcache, extra_topk_length, head_dim_v, softmax_scale, _impl_override, _kernel_timer)
    else:
        assert indices_in_kvcache is None and attn_sink is None and extra_k_cache is None and extra_indices_in_kvcache is None and topk_length is None and extra_topk_length is None, "indices_in_kvcache, attn_sink, extra_k_cache, extra_indices_in_kvcache, topk_length and extra_topk_length must be None when dense attention is used."
        assert block_table is not None and cache_seqlens is not None, "block_table and cache_seqlens must be provided when dense attention is used."
        out, lse, sched_meta.tile_scheduler_metadata, sched_meta.num_splits = host.dense_decode(
            q, k_cache, head_dim_v, cache_seqlens, block_table, softmax_scale, causal,
            sched_meta.tile_scheduler_metadata, sched_meta.num_splits, _impl_override, _kernel_timer)
    return out, lse


def flash_mla_sparse_fwd(
    q: torch.Tensor,
    kv: torch.Tensor,
    indices: torch.Tensor,
    sm_scale: float,
    d_v: int = 512,
    attn_sink: Optional[torch.Tensor] = None,
    topk_length: Optional[torch.Tensor] = None,
) -> Tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
    """
    Token-sparse MLA prefill forward; same contract as the reference's flash_mla_sparse_fwd
    (flash_mla/flash_mla_interface.py:176-211, checks of csrc/api/sparse_fwd.h:101-243):

        q [s_q, h_q, 576] bf16; kv [s_kv, 1, 576] bf16; indices [s_q, 1, topk] int32 (invalid: < 0 or >= s_kv);
        attn_sink [h_q] fp32 (optional); topk_length [s_q] int32 (optional)
    Returns (out [s_q, h_q, 512] bf16, max_logits [s_q, h_q] fp32, lse [s_q, h_q] fp32).
    """
    return _capi.host().sparse_prefill(q, kv, indices, sm_scale, d_v, attn_sink, topk_length, _impl_override, _kernel_timer)
