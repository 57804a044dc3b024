"""Grouped Cross-Attention: host-side mirror of the reference's ``ltriton/gca.py`` boundary.

``attention`` and ``gca_kv_cache`` keep the reference's positional signatures
(``ltriton/gca.py:844`` / ``:846``, called from ``model/DRT.py:380,382``) so a model can
rebind ``model.DRT.gca_attn`` / ``model.DRT.gca_kv_cache`` to them.  ``gca_indexed`` is the
extended entry: it takes the chunk cache and the retrieved indices and never materialises
the gathered copy (``model/DRT.py:193-199`` + ``:321-332`` in the reference); gradients
flow to the cache.

All arithmetic happens in the CUDA library behind the C ABI (``_lib``); shapes, strides, output
allocation and autograd bookkeeping happen in the compiled host path (``_lib.host()``); this file
gives the entry points their names, defaults and meaning.
"""
from __future__ import annotations

from typing import Tuple

import torch

from . import _lib
from ._lib import ALGO_AUTO, ALGO_SIMT, ALGO_TC, ALGO_TC_UNPAIRED  # noqa: F401  (re-exported)


def _status(device: torch.device) -> torch.Tensor:
    return _lib.host().status_word(device.index if device.index is not None else torch.cuda.current_device())


def read_status(device=None, clear: bool = True) -> int:
    """Device-side soft status bits accumulated by the kernels (synchronises)."""
    device = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    word = _status(device)
    val = int(word.item())
    if clear:
        word.zero_()
    return val


def set_status_checks(enabled: bool) -> None:
    """When enabled, every GCA call of this module reads the device status word after its launch
    (one synchronisation per call) and raises ``GcaError`` if a kernel reported that a bounded
    wait expired (outputs invalid).  Off by default; ``HostGcaPipeline`` always checks, at the
    point where it synchronises anyway."""
    _lib.set_check(enabled)


def check_status(device=None, clear: bool = True) -> int:
    """Reads the status word (synchronises).  ``STATUS_TIMEOUT`` -- a kernel gave up a bounded
    on-chip wait, its outputs are not valid -- raises ``GcaError``; other bits (a retrieved index
    outside the cache: that slot was skipped) are returned to the caller."""
    bits = read_status(device, clear)
    if bits & _lib.STATUS_TIMEOUT:
        raise _lib.GcaError("a GCA kernel gave up a bounded wait (GCA_STATUS_TIMEOUT): its outputs are not valid")
    return bits


def _stream() -> int:
    return torch.cuda.current_stream().cuda_stream


def _off_by_one(sm_n: float, softmax_off_by_one: bool) -> float:
    return (float(sm_n) if sm_n else 1.0) if softmax_off_by_one else 0.0


BWD_STAGE_INDEX, BWD_STAGE_KV, BWD_STAGE_Q, BWD_STAGE_ALL = 1, 2, 4, 7
BWD_INDEX_BY_SORT = 8          # flag beside BWD_STAGE_INDEX: build the inverse index by radix sort (same bits)


def gca_backward_stages(q, k_cache, v_cache, indices, weights, dout, lse, sm_scale, *, stages=BWD_STAGE_ALL,
                        bufs=None, softmax_off_by_one=False, algo: int = ALGO_AUTO):
    """The backward of `gca_indexed` without autograd, optionally one stage at a time:
    BWD_STAGE_INDEX, then BWD_STAGE_Q, then BWD_STAGE_KV (the dK/dV kernel reads per-row terms
    that the dQ kernel leaves in the workspace).  `stages | BWD_INDEX_BY_SORT` builds the index
    by radix sort.

    q (N, J, Hq, S, D); caches (N, C, L, Hkv*D); dout like q; lse as returned by
    `gca_forward_with_lse`.  A partial call returns (dq, dk, dv, dw, workspace): pass that tuple
    back as `bufs` for the remaining stages.  A full call returns (dq, dk, dv, dw).
    """
    out = _lib.host().gca_backward(q, k_cache, v_cache, indices, weights, dout, lse, sm_scale, 1.0 if softmax_off_by_one else 0.0,
                                   algo, stages, bufs)
    return out if bufs is None and (stages & BWD_STAGE_ALL) != BWD_STAGE_ALL else out[:4]


def gca_indexed(q: torch.Tensor, k_cache: torch.Tensor, v_cache: torch.Tensor, indices: torch.Tensor,
                weights: torch.Tensor, sm_scale: float, sm_n: float = 0.0, *,
                softmax_off_by_one: bool = False, algo: int = ALGO_AUTO,
                token_major_out: bool = False) -> torch.Tensor:
    """GCA straight from the chunk cache.

    q (N, J, Hq, S, D); caches (N, C, L, Hkv*D) token-major (the layout of
    ``ChunkKVManager``, ``model/DRT.py:88``) or (N, C, L, Hkv, D); indices (N, J, K) integer,
    negative = padding slot; weights (N, J, K).  Returns (N, J, Hq, S, D) in q's dtype.

    ``sm_n`` is accepted for signature compatibility and, exactly like the reference
    kernels, has no effect unless ``softmax_off_by_one=True``, which adds a virtual zero
    logit of weight ``sm_n`` (default 1 when sm_n == 0) to every per-chunk softmax.
    ``token_major_out`` lays the result out as (n, j, s, h, d) in memory (returned as a
    permuted view of the same logical shape), which is what the output projection wants.
    """
    return _lib.host().gca_indexed(q, k_cache, v_cache, indices, weights, sm_scale, _off_by_one(sm_n, softmax_off_by_one), algo,
                                   token_major_out)


def attention(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, weights: torch.Tensor,
              sm_scale: float, sm_n: float = 0.0) -> torch.Tensor:
    """Drop-in for ``ltriton.gca.attention`` (``_attention.apply``, ``ltriton/gca.py:681-844``).

    q (Z, Hq, S, D); k, v (Z, Hkv, K, L, D) pre-gathered chunks; weights (Z, K).
    Differentiable in q, k, v and weights; ``sm_n`` is inert as in the reference kernel
    (its ``l_i = sm_n`` start value is multiplied by zero in the first softmax step,
    ``ltriton/gca.py:48-49,187``).
    """
    return _lib.host().attention(q, k, v, weights, sm_scale)


def gca_kv_cache(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, weights: torch.Tensor,
                 sm_scale: float, sm_n: float = 0.0) -> torch.Tensor:
    """Drop-in for ``ltriton.gca.gca_kv_cache`` (``ltriton/gca.py:846-888``): no autograd;
    q (Z, Hq, Sq, D) with Sq = 1 or 2 while decoding and Sq = 64 for eval prefill
    (``model/DRT.py:379-382``)."""
    return _lib.host().gca_kv_cache(q, k, v, weights, sm_scale)


def gca_indexed_nograd(q, k_cache, v_cache, indices, weights, sm_scale, sm_n: float = 0.0, *,
                       softmax_off_by_one: bool = False, algo: int = ALGO_AUTO, token_major_out: bool = False) -> torch.Tensor:
    """Inference form of ``gca_indexed`` for any Sq in [1, 64] (decode uses 1 or 2 rows); never recorded for autograd."""
    return _lib.host().gca_nograd(q, k_cache, v_cache, indices, weights, sm_scale, _off_by_one(sm_n, softmax_off_by_one), algo,
                                  token_major_out)


def gca_forward_with_lse(q, k_cache, v_cache, indices, weights, sm_scale, *, off_by_one: float = 0.0,
                         algo: int = ALGO_AUTO) -> Tuple[torch.Tensor, torch.Tensor]:
    """Forward returning (out, lse) with lse (N*J, Hq, K, S) in base 2 -- for tests and tools."""
    return _lib.host().gca_forward_lse(q, k_cache, v_cache, indices, weights, sm_scale, off_by_one, algo)
