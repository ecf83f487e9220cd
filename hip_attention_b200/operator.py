"""``hip_attention_12``: hierarchical mask estimation + block-sparse attention on B200.

The call signature, argument semantics, returned metadata and cached-mask behaviour of the reference's
``dual_stage_quadratic_hip_attention`` (``src/hip_attn/v1_2/attention_extend.py:1918-3133``).  A call is carried out by
the extension module ``_host`` (``csrc/host.cpp``): argument checks, device memory from torch's caching allocator, and
the launches of ``libhipattn_sm100.so`` on the current stream of q's device.

What differs from the reference by design:

* chunk lists are kept once per (batch, query block) as int32 -- with the head max-reduce every head
  selects the same chunks -- and widened / expanded to the reference's per-head int64 layout only in
  the returned metadata;
* equal scores are ordered by chunk position (lower first), where the reference leaves it open;
* pages of any positive size are accepted;
* K smaller than ``sink + window`` (no chunk to scan) yields an empty selection instead of failing.
"""
from __future__ import annotations

import os
import threading
from typing import Optional

import torch
from torch import Tensor

from . import _lib as L
from .metadata import (HiPAttentionArgs, HiPAttentionCacheAccessStatistics, HiPAttentionOutputMetadata,
                       HiPAttentionStageInputCache, ScanStage)

_DT = {torch.float32: L.F32, torch.float16: L.F16, torch.bfloat16: L.BF16}
# an fp8 KV cache: e5m2 values, handed over as float8_e5m2 or as the uint8 view the serving adapter makes of it
# (paged_hip.py:409-418); every value is read as the 16-bit number it converts to exactly
_FP8 = (torch.float8_e5m2, torch.uint8)
_host_module = None
_host_lock = threading.Lock()


def host():
    """The host extension, loaded once.  There is no fallback: a missing build is an error."""
    global _host_module
    if _host_module is None:
        L.load()
        with _host_lock:
            if _host_module is None:
                try:
                    from . import _host
                except ImportError as e:
                    raise L.HipAttnError(f"the host extension of {L.LIB_PATH} cannot be loaded ({e}): build it with "
                                         "`python -m hip_attention_b200.build`") from e
                _host.bind(ScanStage, HiPAttentionOutputMetadata, HiPAttentionStageInputCache, HiPAttentionCacheAccessStatistics,
                           L.HipAttnError, torch.cuda)
                _host_module = _host
    return _host_module


def _stream(device) -> int:
    return torch.cuda.current_stream(device).cuda_stream


def status_word(device) -> Tensor:
    """Device status word (one int32 per device) the kernels OR their HIPATTN_STATUS_* bits into."""
    dev = torch.device(device)
    return host().status_word(dev.index if dev.index is not None else torch.cuda.current_device())


def read_status(device, reset: bool = True) -> int:
    """Synchronising read of the status word (0 = clean)."""
    w = status_word(device)
    v = int(w.item())
    if reset and v:
        w.zero_()
    return v


def _tokens(dense: Optional[Tensor], cache: Optional[Tensor], table: Optional[Tensor], seq_lens: Optional[Tensor],
            what: str) -> L.Tokens:
    """K or V as the C ABI takes it, for callers of the library's functions through ctypes."""
    t = L.Tokens()
    if cache is not None:
        if cache.ndim != 4 or cache.stride(-1) != 1:
            raise ValueError(f"{what}_cache must be [n_pages, page_size, kv_heads, head_dim] with a contiguous last dim")
        if table is None or table.ndim != 2 or seq_lens is None or seq_lens.ndim != 1:
            raise ValueError("paged KV needs block_table [B, pages] and cache_seq_lens [B]")
        if table.dtype not in (torch.int32, torch.int64) or seq_lens.dtype not in (torch.int32, torch.int64):
            raise ValueError("block_table and cache_seq_lens must be int32 or int64")
        if table.stride(1) != 1:
            raise ValueError("block_table rows must be contiguous")
        if not seq_lens.is_contiguous():
            raise ValueError("cache_seq_lens must be contiguous")
        t.cache = cache.data_ptr()
        t.fp8_e5m2 = int(cache.dtype in _FP8)
        t.stride_page, t.stride_off, t.stride_ch = cache.stride(0), cache.stride(1), cache.stride(2)
        t.block_table = table.data_ptr()
        t.table_stride_b = table.stride(0)
        t.cache_seq_lens = seq_lens.data_ptr()
        t.n_pages = cache.shape[0]
        t.table_width = table.shape[1]
        t.table_is_i64 = int(table.dtype == torch.int64)
        t.seq_lens_is_i64 = int(seq_lens.dtype == torch.int64)
        t.page_size = cache.shape[1]
    else:
        if dense is None:
            raise ValueError(f"{what} is None and no {what}_cache was given")
        if dense.ndim != 4 or dense.stride(-1) != 1:
            raise ValueError(f"{what} must be [B, T, kv_heads, head_dim] with a contiguous last dim")
        t.dense = dense.data_ptr()
        t.fp8_e5m2 = int(dense.dtype in _FP8)
        t.stride_b, t.stride_t, t.stride_h = dense.stride(0), dense.stride(1), dense.stride(2)
    return t


class PhaseTimer:
    """Optional per-phase CUDA-event timing of one call (events are recorded on the current stream;
    read them with ``milliseconds()`` after a synchronise)."""

    def __init__(self):
        self.marks = []

    def mark(self, name: str) -> None:
        ev = torch.cuda.Event(enable_timing=True)
        ev.record()
        self.marks.append((name, ev))

    def milliseconds(self) -> dict:
        out = {}
        for (_, e0), (name, e1) in zip(self.marks[:-1], self.marks[1:]):
            out[name] = out.get(name, 0.0) + e0.elapsed_time(e1)
        return out


def hip_attention_impl(q: Tensor, k: Optional[Tensor], v: Optional[Tensor], args: HiPAttentionArgs,
                       cached_metadata: Optional[HiPAttentionOutputMetadata] = None, *, return_lse: bool = False,
                       debug: Optional[dict] = None, score_reduce=None, timer: Optional[PhaseTimer] = None,
                       v_ready: Optional[torch.cuda.Event] = None, shared: Optional[dict] = None, out: Optional[Tensor] = None,
                       lse: Optional[Tensor] = None, fork=None, beside: bool = False):
    """Implementation behind ``hip_attention_12``.

    ``return_lse`` adds the base-2 log-sum-exp [B, TQ, H]; ``score_reduce(score_int32)`` is called after every scan
    stage, before the selection: a KV-head-parallel caller all-reduces (MAX) the head-reduced scores there; ``timer``
    collects per-phase CUDA-event times; ``debug`` collects the per-head outputs of every scan stage.  ``v_ready``: the
    mask estimator reads only q and k, so a caller that streams its inputs to the device may issue the call as soon as q
    and k have arrived and pass the event that marks the arrival of v (dense ``v`` or the value cache); the attention
    launch waits for it.  ``shared``: a dict that calls on the same keys hand on, so that key copies and rope tables are
    prepared once; its entries ``positions`` [B, n] and ``windows`` name the query positions and the sliding windows of
    all of them.  ``out`` [B, TQ, H, D] and
    ``lse`` [B, TQ, H] receive the context and its log-sum-exp.  ``fork``: a fork of the current stream (``host().fork``)
    with calls that do not depend on one another; with ``beside`` a decode call runs beside that stream.  The results may
    be used after ``host().join``."""
    return (_host_module or host()).forward(q, k, v, args, cached_metadata, return_lse, debug, score_reduce, timer, v_ready, shared, out,
                                            lse, fork, beside)


def hip_attention_12(q: Tensor, k: Optional[Tensor], v: Optional[Tensor], args: Optional[HiPAttentionArgs] = None,
                     cached_metadata: Optional[HiPAttentionOutputMetadata] = None):
    """HiP attention: ``(context, metadata) = hip_attention_12(q, k, v, args, cached_metadata)``.

    q [B, TQ, H, D] must already carry the softmax scale; k, v [B, TK, HKV, D], or ``None`` with
    ``args.k_cache / v_cache / block_table / cache_seq_lens`` describing a paged cache.  Passing the
    returned metadata back skips the mask estimator; metadata with ``indices=None`` and a prefix of
    ``stage_caches`` restarts the estimator at the last cached stage.
    """
    return hip_attention_impl(q, k, v, args if args is not None else HiPAttentionArgs(), cached_metadata)
