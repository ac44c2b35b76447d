"""Attention entry point: the reference's ``fst_attention`` on the sm_100a kernels.

Same positional signature as fstattention.py:153 of the reference::

    o = fst_attention(q, k, v, ancestor_idx, ancestor_mask, leaf_idx, sm_scale,
                      BLOCK_M=128, MAX_ANCESTORS=64)

``q`` is ``[Z, H, N, D]``, ``k``/``v`` are ``[Z, H, P + N, D]`` where the first ``P`` rows are a
prefix every query attends to.  The launch is asynchronous on torch's current stream.
"""
from __future__ import annotations

import math
from typing import Optional

import torch

from . import _lib
from .utils import TreeMetadata, metadata_of

_KERNELS = _lib.KERNELS

_DTYPES = {torch.float16: _lib.DTYPE_F16, torch.bfloat16: _lib.DTYPE_BF16,
           torch.float32: _lib.DTYPE_F32}


def _resolve(device) -> torch.device:
    device = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    if device.index is None:
        device = torch.device("cuda", torch.cuda.current_device())
    return device


def last_status(device=None, clear: bool = False) -> int:
    """Device-side status code recorded by attention launches on ``device`` (synchronises).

    The record keeps the first problem it saw until it is cleared: pass ``clear=True`` (or call
    ``clear_status``) once the code has been dealt with, so that later launches report afresh."""
    rec = _lib.host().status_record(_resolve(device).index)
    if rec is None:
        return 0
    code = int(rec[0].item())
    if clear and code != 0:
        rec.zero_()
    return code


def clear_status(device=None) -> None:
    """Zero the status record of ``device`` (asynchronous, on the current stream)."""
    rec = _lib.host().status_record(_resolve(device).index)
    if rec is not None:
        rec.zero_()


def _strides(t):
    st = t.stride()
    if st[3] != 1:
        raise ValueError("the head dimension must be contiguous")
    return [st[0], st[1], st[2]]


def launch_plan(q, prefix, block_m, kernel: str = "auto", kv_splits: Optional[int] = None,
                max_ancestors: int = 64, sm_scale: float = 1.0, kv_heads: Optional[int] = None) -> dict:
    """Which kernels one ``fst_attention`` call on packed metadata launches for ``q`` (shape and
    dtype only), a shared prefix of ``prefix`` rows and the given block size, mirroring the
    dispatch inside the library (for rows on 16-byte boundaries): ``{"kernels":
    [...], "prefix_runs": r}``.  ``max_ancestors`` is the metadata's ancestor bound; of ``sm_scale`` the sign counts,
    and ``kv_heads`` are the heads of K and V where they are fewer than those of ``q``."""
    kv_splits = None if kv_splits is None else int(kv_splits)
    splits, need_ws, umma = _lib.host().splits(q, prefix, block_m, _lib.KERNELS[kernel], kv_splits, sm_scale,
                                               q.shape[1] if kv_heads is None else kv_heads)
    tensor_core = q.dtype in (torch.float16, torch.bfloat16) and q.shape[-1] in (64, 128) \
        and block_m in (16, 32, 64, 128)
    tree = "attn_simt_kernel" if kernel == "simt" or not tensor_core else \
        "attn_mma_kernel" if kernel == "mma" or block_m == 16 else "attn_tma_kernel"
    if tree == "attn_tma_kernel" and prefix == 0 and (kernel == "tree_umma" or (kernel == "auto" and sm_scale > 0 and _lib.lib().fst_attention_tree_kernel(
            q.shape[0], q.shape[1], q.shape[2], q.shape[3], block_m, max_ancestors) == _KERNELS["tree_umma"])):
        tree = "tree_umma_kernel"
    if kernel == "persist" and tree == "attn_tma_kernel" and prefix == 0 and block_m in (64, 128):
        tree = "attn_persist_kernel"                      # by hand only: it measured slower than attn_tma_kernel
    if umma:
        # prefix and tree in one; its runs merge inside unless they are spread over the GPU
        return {"kernels": ["prefix_umma_kernel"] + ["combine_splits_kernel"] * need_ws, "prefix_runs": splits}
    if need_ws:
        return {"kernels": [tree, "combine_splits_kernel"], "prefix_runs": splits}
    return {"kernels": [tree], "prefix_runs": 1}


def fst_attention(q, k, v, ancestor_idx, ancestor_mask=None, leaf_idx=None, sm_scale=None,
                  BLOCK_M=128, MAX_ANCESTORS=64, *, out: Optional[torch.Tensor] = None,
                  return_lse: bool = False, kernel: str = "auto", kv_splits: Optional[int] = None,
                  scatter=None):
    """Fused sparse tree attention forward.

    ``ancestor_idx, ancestor_mask, leaf_idx`` are the tensors returned by
    ``create_fst_attention_kernel_inputs`` (from this package, or the reference's moved to the
    GPU) built with ``block_m=BLOCK_M`` and ``max_ancestors=MAX_ANCESTORS``; index tensors hold
    absolute K/V rows, i.e. the caller adds the prefix length as fstattention.py:211-212 does.
    Alternatively pass a ``TreeMetadata`` as ``ancestor_idx`` and leave the other two ``None``;
    its block size and ancestor bound are used.  Metadata with a leading tree dimension of size
    ``Z`` gives every batch element its own tree.  ``k`` and ``v`` may have fewer heads than ``q``
    (grouped-query attention, ``H`` a multiple of ``H_kv``).

    ``kv_splits`` cuts a call behind a shared prefix into that many runs handled by separate CTAs and
    merged afterwards; ``None`` picks a split that fills the GPU when the tree alone does not.

    ``scatter`` (see ``sharding.GatheredOutput.target``) makes the kernel deliver this call's
    rows into every rank's copy of a full output tensor instead of a local ``out``; the return
    value is then this rank's copy, complete only after the ranks have met.

    Asserts like the reference (fstattention.py:155-157): equal head dims, in {16, 32, 64, 128}.
    """
    if sm_scale is None:
        raise TypeError("sm_scale is required")
    kern = _KERNELS[kernel]
    meta = ancestor_idx if isinstance(ancestor_idx, TreeMetadata) else metadata_of(ancestor_idx, ancestor_mask, leaf_idx)
    if meta is not None and meta is not ancestor_idx and (meta.block_m != BLOCK_M or meta.max_ancestors != MAX_ANCESTORS):
        raise ValueError("BLOCK_M / MAX_ANCESTORS differ from the ones the metadata was built with")
    if scatter is not None:
        tensors = (ancestor_idx, ancestor_mask, leaf_idx, BLOCK_M, MAX_ANCESTORS)
        return _scattered(q, k, v, meta, tensors, sm_scale, kern, scatter, out, return_lse)
    if kv_splits is not None:
        kv_splits = int(kv_splits)
    host = _lib._host or _lib.host()
    if meta is None:
        # the reference's three tensors (fstattention.py:153), which the call packs first
        return host.attention_ref(q, k, v, out, ancestor_idx, ancestor_mask, leaf_idx, BLOCK_M, MAX_ANCESTORS,
                                  sm_scale, kern, kv_splits, bool(return_lse))
    # From the second launch after the precompute on, the launch ahead of this one in the stream
    # cannot be the metadata's writer: the kernel may then fetch its index lists while that launch
    # drains (FST_KERNEL_FLAG_META_STABLE).
    if meta.reads_since_build > 0:
        kern |= _lib.KERNEL_FLAG_META_STABLE
    result = host.attention(q, k, v, out, meta.packed, meta.tree_stride, meta.n_trees, meta.n_blocks, meta.block_m,
                            meta.max_ancestors, sm_scale, kern, kv_splits, bool(return_lse))
    meta.reads_since_build += 1
    return result


def _scattered(q, k, v, meta, tensors, sm_scale, kern, scatter, out, return_lse):
    """``fst_attention(..., scatter=)``: this call's rows into every rank's copy of the full output."""
    assert q.shape[-1] == k.shape[-1] == v.shape[-1] and k.shape[-1] in {16, 32, 64, 128}
    if not (q.is_cuda and k.is_cuda and v.is_cuda):
        raise RuntimeError("fst_attention runs on CUDA tensors only; there is no CPU path")
    if q.dtype not in _DTYPES or k.dtype != q.dtype or v.dtype != q.dtype:
        raise TypeError("q, k, v must share one dtype out of float16, bfloat16, float32")
    Z, H, n_q, D = q.shape
    n_kv, H_kv = k.shape[2], k.shape[1]
    if k.shape != (Z, H_kv, n_kv, D) or v.shape != k.shape or n_kv < n_q or H_kv < 1 or H % H_kv:
        raise ValueError("k and v must be [Z, H_kv, P + N, D] with P >= 0 and H a multiple of H_kv")
    if H_kv != H or n_kv != n_q:
        raise ValueError("scatter= takes neither grouped-query heads nor a shared prefix")
    if out is not None:
        raise ValueError("out= and scatter= exclude each other")
    o = scatter.local
    if o.dtype != q.dtype or o.shape[2:] != q.shape[2:] or not o.is_cuda:
        raise ValueError("the gathered output must have q's dtype, rows and head dimension")
    if not math.isfinite(sm_scale):
        raise ValueError("sm_scale must be finite")
    dev = q.device
    if meta is None:
        ai, am, li, block_m, max_ancestors = tensors
        packed, stride, n_trees = _lib.host().pack(ai, am, li, Z, n_q, 0, block_m, max_ancestors)
    else:
        packed, stride, n_trees = meta.packed, meta.tree_stride, meta.n_trees
        block_m, max_ancestors = meta.block_m, meta.max_ancestors
        if n_trees not in (1, Z):
            raise ValueError("metadata must describe one tree or one tree per batch element")
        if meta.n_blocks != -(-n_q // block_m):
            raise ValueError("metadata block count does not match q")
    if any(t.device != dev for t in (k, v, o, packed)):
        raise RuntimeError("all tensors of a call must be on one device")
    lse = torch.empty((Z * H, n_q), device=dev, dtype=torch.float32) if return_lse else None
    with torch.cuda.device(dev):
        if meta is not None:
            if meta.reads_since_build > 0:
                kern |= _lib.KERNEL_FLAG_META_STABLE
            meta.reads_since_build += 1
        rc = _lib.lib().fst_attention_fwd_scatter(
            q.data_ptr(), k.data_ptr(), v.data_ptr(), scatter.pointer_array, scatter.n_ranks, scatter.rank,
            scatter.z0, scatter.h0, o.shape[0], o.shape[1], lse.data_ptr() if lse is not None else None,
            packed.data_ptr(), stride if n_trees > 1 else 0, Z, H, n_q, n_kv, D,
            *_strides(q), *_strides(k), *_strides(v), *_strides(o), block_m, max_ancestors,
            float(sm_scale), _DTYPES[q.dtype], kern, _lib.host().attention_status(dev.index).data_ptr(),
            torch.cuda.current_stream(dev).cuda_stream)
    _lib.check(rc, "fst_attention_fwd")
    return (o, lse) if return_lse else o


def fst_attention_paged(q, k_tree, v_tree, meta: TreeMetadata, k_pool, v_pool, block_table, prefix_lens,
                        sm_scale, *, max_prefix: Optional[int] = None, pool_layout: str = "NHD",
                        kv_splits: Optional[int] = None, out: Optional[torch.Tensor] = None,
                        return_lse: bool = False):
    """Tree attention behind a prefix held in a paged KV cache (head_dim 64 or 128, fp16 / bf16).

    ``q`` is ``[Z, H, N, D]``; ``k_tree``, ``v_tree`` are the tree nodes' own K/V rows,
    ``[Z, H_kv, N, D]``.  The prefix of batch element ``z`` is rows ``[0, prefix_lens[z])`` of
    the sequence whose pages ``block_table[z]`` lists (int32, on the GPU, as is ``prefix_lens``):
    row ``r`` lives in page ``block_table[z, r // page_size]``.  The pools are
    ``[n_pages, page_size, H_kv, D]`` (``pool_layout="NHD"``) or ``[n_pages, H_kv, page_size, D]``
    (``"HND"``), page_size 16, 32, 64 or 128.  ``max_prefix`` (default: the largest entry of
    ``prefix_lens``, which costs a device synchronisation) sizes the grid.  ``meta`` is the
    ``TreeMetadata`` of the tree (``build_tree_metadata``)."""
    if not isinstance(meta, TreeMetadata):
        raise TypeError("meta must be a TreeMetadata (build_tree_metadata)")
    if pool_layout not in ("NHD", "HND"):
        raise ValueError("pool_layout must be 'NHD' or 'HND'")
    if max_prefix is None:
        max_prefix = int(prefix_lens.max().item())
    host = _lib._host or _lib.host()
    return host.attention_paged(q, k_tree, v_tree, out, meta.packed, meta.tree_stride, meta.n_trees, meta.n_blocks,
                                meta.block_m, meta.max_ancestors, k_pool, v_pool, pool_layout == "NHD", block_table,
                                prefix_lens, int(max_prefix), sm_scale, kv_splits, bool(return_lse))
