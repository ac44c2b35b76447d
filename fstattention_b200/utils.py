"""Tree precompute: the reference's ``utils.py`` surface on top of the CUDA precompute kernel.

``create_fst_attention_kernel_inputs`` keeps the reference's name, arguments, return order,
dtypes and shapes (utils.py:104-129 of the reference) and raises ``RuntimeError`` where the
reference does (more unique ancestors in a block than ``max_ancestors``, utils.py:120), but the
work is done by one kernel launch on the GPU and the tensors it returns live there.
``build_tree_metadata`` is the front door for callers that hold a parent array, which is what a
decoder that rebuilds its tree every step has.
"""
from __future__ import annotations

import weakref
from typing import Optional, Sequence, Union

import torch

from . import _lib

TreeLike = Union[torch.Tensor, Sequence[int], Sequence[Sequence[int]]]

# Same tables as the reference's utils.py:4-24: tree depth that fills a context of 2^k - 4 nodes,
# and the ancestor bound its benchmark uses for it.
DEPTH_MAPPING = {2 ** (10 + i): 7 + i for i in range(8)}
MAX_ANCESTOR_MAPPING = {2 ** (10 + i): 64 for i in range(8)}


class TreeMetadata:
    """Block metadata of one tree or a batch of trees, resident on one GPU.

    Unpacks like the reference's return value: ``ancestor_idx, ancestor_mask, leaf_idx = meta``
    (int64 / bool / int64; a leading tree dimension is present only for a batch of trees).
    ``packed`` is the bit-packed form the attention kernels read; ``fst_attention`` accepts the
    object itself in place of the three tensors.
    """

    def __init__(self, n_trees, n_nodes, block_m, max_ancestors, packed, tree_stride, status,
                 ancestor_idx=None, ancestor_mask=None, leaf_idx=None, batched=False):
        self.n_trees, self.n_nodes = n_trees, n_nodes
        self.block_m, self.max_ancestors = block_m, max_ancestors
        self.n_blocks = -(-n_nodes // block_m)
        self.packed, self.tree_stride, self.status = packed, tree_stride, status
        self.ancestor_idx, self.ancestor_mask, self.leaf_idx = ancestor_idx, ancestor_mask, leaf_idx
        self.batched = batched
        # attention launches that have read the packed form since it was last written: from the
        # second one on, the launch ahead of the call in the stream cannot be the writer
        self.reads_since_build = 0
        self._captured_status = []                        # records that graphs write at their replays
        self._twin = None if ancestor_idx is None else _PackedTwin.of(self)

    def _rebuilt(self) -> None:
        """The buffers have just been written (again)."""
        self.reads_since_build = 0
        if self._twin is not None:
            self._twin.reads_since_build = 0
            self._twin.versions = _versions((self.ancestor_idx, self.ancestor_mask, self.leaf_idx))

    def tensors_untouched(self) -> bool:
        """True while nobody has modified the three reference-format tensors in place."""
        return self._twin is None or _unchanged(self._twin, (self.ancestor_idx, self.ancestor_mask, self.leaf_idx))

    # Saved or deep-copied metadata has tensors of its own, and a twin that belongs to them.
    def __getstate__(self):
        return dict(self.__dict__, _twin=self.tensors_untouched())

    def __setstate__(self, state):
        self.__dict__.update(state)
        self._twin = None if self.ancestor_idx is None else _PackedTwin.of(self)
        if not state["_twin"]:
            self._twin.versions = None
        elif self._twin is not None:
            setattr(self.ancestor_idx, _ORIGIN_ATTR, self._twin)

    def __copy__(self):                                   # the same tensors, hence the same twin
        other = object.__new__(type(self))
        other.__dict__.update(self.__dict__)
        return other

    def __iter__(self):
        if self.ancestor_idx is None:
            raise RuntimeError("metadata was built with reference_format=False")
        return iter((self.ancestor_idx, self.ancestor_mask, self.leaf_idx))

    def _keep_captured(self, status) -> None:
        """A graph clears and writes this record at every replay: it lives as long as the buffers, whatever record a
        later eager build takes, and ``check`` reads it too."""
        if not any(t is status for t in self._captured_status):
            self._captured_status.append(status)

    def check(self) -> "TreeMetadata":
        """Read the device status record (synchronises) and raise on a recorded problem - of the last build, eager
        or replayed from a graph."""
        code, where, detail, _ = _lib.host().read_status(self.status)
        for record in self._captured_status:
            if code == 0 and record is not self.status:
                code, where, detail, _ = _lib.host().read_status(record)
        if code == _lib.DEV_ANCESTOR_OVERFLOW:
            raise RuntimeError(
                f"block {where % 65536} of tree {where // 65536} has {detail} unique ancestors, "
                f"more than max_ancestors={self.max_ancestors}")
        if code == _lib.DEV_MALFORMED_TREE:
            raise ValueError(f"malformed tree: parent[{where}]={detail} must be -1 or an earlier node")
        if code != 0:
            raise RuntimeError(_lib.status_string(code))
        return self

    @property
    def device(self):
        return self.packed.device


def _versions(three):
    """None where nobody counts: tensors loaded or copied under ``torch.inference_mode()``."""
    a, b, c = three
    try:
        return a._version, b._version, c._version
    except RuntimeError:
        return None


def _unchanged(twin, three) -> bool:
    return twin.versions is not None and twin.versions == _versions(three)


# The three tensors handed out by the precompute remember the packed form they came with, so that
# fst_attention(q, k, v, ancestor_idx, ancestor_mask, leaf_idx, ...) can skip re-packing them.
_ORIGIN_ATTR = "_fst_tree_metadata"


class _PackedTwin:
    """What ``ancestor_idx`` carries: the packed form, and weak references to the three tensors it
    belongs to.  (A strong reference back would be a cycle, and buffers as large as a tree's mask
    would then wait for the garbage collector instead of going back to the allocator: building a
    131068-node tree over and over spent more on fresh allocations than on the kernel.)"""
    __slots__ = ("n_trees", "n_blocks", "block_m", "max_ancestors", "packed", "tree_stride", "reads_since_build",
                 "versions", "tensors")

    def __init__(self, n_trees, n_blocks, block_m, max_ancestors, packed, tree_stride, three):
        self.n_trees, self.n_blocks = n_trees, n_blocks
        self.block_m, self.max_ancestors = block_m, max_ancestors
        self.packed, self.tree_stride = packed, tree_stride
        self.reads_since_build = 0
        a, b, c = three
        self.versions = _versions(three)
        self.tensors = weakref.ref(a), weakref.ref(b), weakref.ref(c)

    @classmethod
    def of(cls, meta: TreeMetadata):
        return cls(meta.n_trees, meta.n_blocks, meta.block_m, meta.max_ancestors, meta.packed, meta.tree_stride,
                   (meta.ancestor_idx, meta.ancestor_mask, meta.leaf_idx))

    def __reduce__(self):                                 # a tensor saved or copied on its own is a plain one
        return type(None), ()


def metadata_of(ancestor_idx, ancestor_mask, leaf_idx) -> Optional[_PackedTwin]:
    """The packed form of three tensors handed out together, while nobody has changed them."""
    twin = getattr(ancestor_idx, _ORIGIN_ATTR, None)
    if twin is None:
        return None
    a, b, c = twin.tensors
    if a() is ancestor_idx and b() is ancestor_mask and c() is leaf_idx \
            and _unchanged(twin, (ancestor_idx, ancestor_mask, leaf_idx)):
        return twin
    return None


def _as_parent_tensor(parent: TreeLike, device) -> torch.Tensor:
    if not torch.is_tensor(parent):
        parent = torch.tensor(parent, dtype=torch.int32)
    if parent.dim() not in (1, 2) or parent.numel() == 0:
        raise ValueError("parent must be a non-empty [N] or [T, N] array")
    if parent.is_cuda and parent.dtype == torch.int32 and parent.is_contiguous() and device is None:
        return parent
    if device is None:
        device = parent.device if parent.is_cuda else "cuda"
    if parent.dtype == torch.long and not parent.is_cuda:
        parent = _in_32_bits(parent)
    return parent.to(device=device, dtype=torch.int32, non_blocking=True).contiguous()


def _in_32_bits(parent: torch.Tensor) -> torch.Tensor:
    """What does not fit into 32 bits stays what it is, no node's number."""
    return parent.clamp(-2, 2 ** 31 - 1)


def packed_meta_bytes(n_blocks: int, block_m: int, max_ancestors: int) -> int:
    return int(_lib.lib().fst_packed_meta_bytes(n_blocks, block_m, max_ancestors))


def build_tree_metadata(parent: TreeLike, block_m: int = 64, max_ancestors: int = 32, *,
                        reference_format: bool = True, check: bool = True,
                        device: Union[str, torch.device, None] = None,
                        out: Optional[TreeMetadata] = None) -> TreeMetadata:
    """Parent array(s) -> block metadata, with one kernel launch on the current stream.

    ``parent`` is ``[N]`` (one tree) or ``[T, N]`` (T independent trees of N nodes); entries are
    -1 for roots and otherwise the index of an earlier node.  ``reference_format=False`` skips
    the int64/bool tensors and writes only the packed form.  ``check=False`` skips reading the
    status record, which avoids a device synchronisation; call ``.check()`` later.  ``out``
    reuses the buffers of an earlier result of the same shape (nothing is allocated then).
    """
    par = _as_parent_tensor(parent, device)
    host = _lib._host or _lib.host()
    if out is None:
        n_trees, n_nodes, packed, stride, status, ai, am, li, captured = host.new_metadata(par, block_m, max_ancestors,
                                                                                           bool(reference_format))
        meta = TreeMetadata(n_trees, n_nodes, block_m, max_ancestors, packed, stride, status, ai, am, li, par.dim() == 2)
        if captured:
            meta._keep_captured(status)
        if ai is not None:
            setattr(ai, _ORIGIN_ATTR, meta._twin)
    else:
        meta = out
        n_trees, n_nodes = par.shape if par.dim() == 2 else (1, par.shape[0])
        if (meta.n_trees, meta.n_nodes, meta.block_m, meta.max_ancestors) != (n_trees, n_nodes, block_m, max_ancestors):
            raise ValueError("out= metadata has a different shape")
        for record in meta._captured_status:              # what a replay has left there is about an older build
            if record is not meta.status:
                record.zero_()
        status = host.precompute(par, block_m, max_ancestors, meta.packed, meta.tree_stride, meta.status,
                                 meta.ancestor_idx, meta.ancestor_mask, meta.leaf_idx)
        if status is meta.status:                         # captured into a graph
            meta._keep_captured(status)
        meta.status = status
        meta._rebuilt()
    if check:
        meta.check()
    return meta


def tree_topk_nodes(depth: int = 7, topk: int = 4, left_weight_factor: float = 0.5) -> int:
    """Node count of the forest ``build_tree_topk`` / the reference's ``create_tree`` makes."""
    n = int(_lib.lib().fst_tree_topk_nodes(depth, topk, float(left_weight_factor)))
    if n < 0:
        raise ValueError("forest shape beyond the kernel's limits (a level above 4096 nodes, or more than 32 levels)")
    return n


def build_tree_topk(scores: torch.Tensor, depth: Optional[int] = None, topk: Optional[int] = None,
                    left_weight_factor: float = 0.5, max_nodes: Optional[int] = None, *,
                    return_choice: bool = False, return_scores: bool = False):
    """Grow the speculation tree on the GPU from the heads' top-k candidate scores.

    ``scores`` is a CUDA float32 tensor ``[depth + 1, topk]`` (one tree) or ``[T, depth + 1, topk]``:
    row ``l`` holds the scores (log-probabilities) of head ``l``'s ``topk`` candidates.  The
    forest has the shape of the reference's ``create_tree(depth, topk, left_weight_factor)``
    (utils.py:27-77) - ``topk`` roots, of every level the ``int(size * left_weight_factor)``
    best-scoring nodes (score = sum along the path) expanded into the next head's candidates -
    and with equal scores is exactly that forest.  Returns the parent array, int32 ``[N]`` /
    ``[T, N]`` on the GPU (``N = max_nodes`` or the forest's node count), ready for
    ``dfs_order_device`` / ``build_tree_metadata(parent, check=False)``; with ``return_choice``
    also ``choice`` (``l * topk + k``: which candidate each node stands for) and with
    ``return_scores`` the nodes' path scores.  One launch on the current stream, no host
    synchronisation.
    """
    if not scores.is_cuda or scores.dtype != torch.float32 or scores.dim() not in (2, 3):
        raise TypeError("scores must be a CUDA float32 tensor [depth + 1, topk] or [T, depth + 1, topk]")
    levels, k = scores.shape[-2:]
    depth = levels - 1 if depth is None else depth
    topk = k if topk is None else topk
    if (depth + 1, topk) != (levels, k):
        raise ValueError("scores must have depth + 1 rows of topk entries")
    parent, choice, nscore = (_lib._host or _lib.host()).build_tree_topk(
        scores, depth, topk, float(left_weight_factor), None if max_nodes is None else int(max_nodes), bool(return_choice),
        bool(return_scores))
    extra = tuple(t for t in (choice, nscore) if t is not None)
    return (parent,) + extra if extra else parent


def parent_from_lineage(lineage: torch.Tensor, level_lookup: torch.Tensor) -> torch.Tensor:
    """parent[k] = lineage[k, level_lookup[k] - 1], -1 for level-0 nodes (utils.py:42-44)."""
    lvl = level_lookup.to(lineage.device).long()
    col = (lvl - 1).clamp_min(0).unsqueeze(1)
    par = lineage.gather(1, col).squeeze(1)
    return torch.where(lvl > 0, par, torch.full_like(par, -1))


def _on_host(t, dim: int) -> bool:
    return t.device.type == "cpu" and t.dtype == torch.long and t.dim() == dim


def create_fst_attention_kernel_inputs(lineage: torch.Tensor, level_lookup: torch.Tensor,
                                       block_m: int = 64, max_ancestors: int = 32,
                                       mutate_lineage: bool = True):
    """Drop-in for the reference function of the same name (utils.py:104-129).

    Returns ``ancestor_idx [nb, max_ancestors]`` (int64), ``ancestor_mask [nb, block_m,
    max_ancestors]`` (bool) and ``leaf_idx [nb, block_m]`` (int64) with the reference's values,
    as CUDA tensors.  Raises RuntimeError when a block has more than ``max_ancestors`` unique
    ancestors.  Like the reference (utils.py:124-125) it writes every node into its own lineage
    row as a side effect; pass ``mutate_lineage=False`` to leave ``lineage`` alone.
    """
    native = _on_host(lineage, 2) and _on_host(level_lookup, 1) and lineage.shape[0] == level_lookup.shape[0]
    host = _lib._host or _lib.host()
    built = host.metadata_of_lineage(lineage, level_lookup, block_m, max_ancestors) if native else None
    if built is not None:                                 # the whole of it in one call, for trees of ordinary size
        packed, stride, idx, mask, leaf = built
        setattr(idx, _ORIGIN_ATTR, _PackedTwin(1, idx.shape[0], block_m, max_ancestors, packed, stride, (idx, mask, leaf)))
        if mutate_lineage:
            host.write_self(lineage, level_lookup)
        return idx, mask, leaf
    parent = host.parents_of_lineage(lineage, level_lookup) if native else parent_from_lineage(lineage, level_lookup)
    if parent.dtype == torch.long and parent.is_cuda:
        parent = _in_32_bits(parent)
    meta = build_tree_metadata(parent, block_m, max_ancestors, reference_format=True, check=not native)
    if native:
        # the parents are on the host: so is the check, and nobody waits for the device
        host.check_tree(parent, block_m, max_ancestors)
    if mutate_lineage and native:
        _lib.host().write_self(lineage, level_lookup)
    elif mutate_lineage:
        n = lineage.shape[0]
        rows = torch.arange(n, device=lineage.device)
        lineage[rows, level_lookup.to(lineage.device).long()] = rows
    return meta.ancestor_idx, meta.ancestor_mask, meta.leaf_idx


def lineage_from_parent(parent: Sequence[int]):
    """Parent array -> (lineage, level_lookup) as the reference describes trees (utils.py:42-44).

    Host-side adapter for callers that still want the reference's inputs; CPU tensors.
    """
    n = len(parent)
    level = [0] * n
    for i, p in enumerate(parent):
        if p >= i or p < -1:
            raise ValueError(f"parent[{i}]={p} must be -1 or an earlier node")
        level[i] = 0 if p < 0 else level[p] + 1
    width = max(level) + 1
    lin = torch.full((n, width), -1, dtype=torch.long)
    for i, p in enumerate(parent):
        if p >= 0:
            lin[i, : level[p]] = lin[p, : level[p]]
            lin[i, level[p]] = p
    return lin, torch.tensor(level, dtype=torch.long)


def create_tree(depth: int = 7, topk: int = 4, left_weight_factor: float = 0.5):
    """The reference's synthetic left-weighted forest (utils.py:27-77), built without loops over
    nodes.

    ``topk`` roots; level sizes follow ``size[l] = topk * int(size[l-1] * left_weight_factor)``
    and node ``r`` of a level hangs under node ``r // topk`` of the level above.  With the
    defaults the forest has 2^(depth+3) - 4 nodes.  Returns ``lineage [N, depth + 1]`` (ancestor
    of each node per level, -1 padded, the node itself not included) and ``level_lookup [N]``,
    both int64 on the CPU, equal to what the reference returns.
    """
    sizes = [topk]
    for _ in range(depth):
        sizes.append(topk * int(sizes[-1] * left_weight_factor))
    starts = [0]
    for sz in sizes:
        starts.append(starts[-1] + sz)
    n = starts[-1]
    level = torch.repeat_interleave(torch.arange(len(sizes)), torch.tensor(sizes))
    start_of = torch.tensor(starts[:-1])[level]
    rel = torch.arange(n) - start_of
    parent = torch.where(level > 0, torch.tensor([0] + starts[:-2])[level] + rel // topk,
                         torch.full((n,), -1, dtype=torch.long))
    lineage = torch.full((n, depth + 1), -1, dtype=torch.long)
    anc = parent.clone()
    for step in range(1, depth + 1):                     # ancestor `step` levels up, all nodes at once
        has = anc >= 0
        rows = torch.nonzero(has).squeeze(1)
        lineage[rows, level[rows] - step] = anc[rows]
        anc = torch.where(has, parent[anc.clamp_min(0)], anc)
    return lineage, level.long()


def create_full_attention_mask(lineage: torch.Tensor) -> torch.Tensor:
    """Dense mask "node attends to itself and its ancestors", as the reference builds it
    (utils.py:79-102), on the device ``lineage`` lives on.

    float32 ``[N + 4, N + 4]``: the reference always appends four zero rows and columns (its
    trees have 2^k - 4 nodes), clears the last column while removing the -1 pads and restores
    only the last node's self entry.  For other sizes pad ``mask[:N, :N]`` yourself.
    """
    n = lineage.shape[0]
    dev = lineage.device
    mask = torch.zeros((n, n), dtype=torch.bool, device=dev)
    rows = torch.arange(n, device=dev).unsqueeze(1).expand_as(lineage)
    mask[rows.reshape(-1), lineage.reshape(-1)] = True    # -1 lands in the last column
    mask[torch.arange(n, device=dev), torch.arange(n, device=dev)] = True
    mask[:, -1] = False
    mask[-1, -1] = True
    out = torch.zeros((n + 4, n + 4), dtype=torch.float32, device=dev)
    out[:n, :n] = mask
    return out


def dfs_order(parent: Sequence[int]):
    """Depth-first renumbering of a tree, so that a query block's ancestors are few and local.

    The reference leaves this as a TODO (README.md:19-20): with nodes numbered breadth first a
    block of 64 rows of a deep tree has ancestors all over the tree (a 2579-node chain tree needs
    up to 1613 per block and gathers 8x the bytes); numbered depth first, a block is a few
    root-to-leaf paths.  Returns ``(order, new_parent)``: ``order[i]`` is the old index of the
    node that becomes node ``i`` (pre-order, children in their old relative order) and
    ``new_parent`` is the parent array in the new numbering, still with ``new_parent[i] < i``.
    Permute the tree rows of q/k/v with ``order`` (``x[..., order, :]``) before attention and
    scatter the output back (``out[..., order, :] = o``).  Host code (numpy); trees are small.
    """
    import numpy as np
    par = np.asarray(parent, dtype=np.int64)
    n = par.shape[0]
    if n == 0:
        return [], []
    if np.any(par >= np.arange(n)) or np.any(par < -1):
        raise ValueError("parent[i] must be -1 or an earlier node")
    size = np.ones(n, dtype=np.int64)
    for i in range(n - 1, -1, -1):                       # children come after parents
        if par[i] >= 0:
            size[par[i]] += size[i]
    # position = position of parent + 1 + sizes of earlier siblings; roots are siblings of each other
    pos = np.empty(n, dtype=np.int64)
    next_free = {}                                       # parent (or -1) -> next free position
    for i in range(n):
        p = int(par[i])
        start = next_free.get(p, 0 if p < 0 else pos[p] + 1)
        pos[i] = start
        next_free[p] = start + size[i]
    order = np.empty(n, dtype=np.int64)
    order[pos] = np.arange(n)
    new_parent = np.where(par[order] >= 0, pos[np.clip(par[order], 0, None)], -1)
    return order.tolist(), new_parent.tolist()


def dfs_order_device(parent: TreeLike, *, check: bool = True,
                     device: Union[str, torch.device, None] = None):
    """``dfs_order`` computed on the GPU with one kernel launch on the current stream, for parent
    arrays that already live there (a decoder that builds its tree on the device).

    ``parent`` is ``[N]`` or ``[T, N]`` as for ``build_tree_metadata`` (N <= 8192).  Returns
    ``(order, new_parent)`` as int32 CUDA tensors of the same shape, with the meaning
    ``dfs_order`` gives them; ``new_parent`` goes straight into ``build_tree_metadata``.
    ``check=False`` skips reading the status record (no device synchronisation); a malformed
    tree then leaves both outputs uninitialised."""
    par = _as_parent_tensor(parent, device)
    order, new_parent, status = (_lib._host or _lib.host()).dfs_order(par)
    if check:
        code, where, detail, _ = _lib.host().read_status(status)
        if code == _lib.DEV_MALFORMED_TREE:
            raise ValueError(f"parent[{where}] = {detail} is neither -1 nor an earlier node")
        if code != 0:
            raise RuntimeError(f"fst_dfs_order: device status {code}")
    return order, new_parent
