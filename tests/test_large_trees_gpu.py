"""Metadata of trees beyond the size where the parent array is staged in shared memory, trees with crowded and deep
levels in the device renumbering, and levels large enough to be sorted in the device-built forest."""
import numpy as np
import pytest
import torch

from oracle import tree_oracle as orc
from test_precompute_gpu import _topk_forest_cpu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fst(built_lib):
    import fstattention_b200
    return fstattention_b200


def sets_of(par, lo, hi):
    rows = []
    for k in range(lo, hi):
        x, anc = int(par[k]), []
        while x >= 0:
            anc.append(x)
            x = int(par[x])
        rows.append(anc)
    return rows


@pytest.mark.parametrize("n,bm,ma,kind", [(8193, 64, 64, "near"), (8200, 128, 128, "near"), (9000, 32, 100, "near"),
                                          (20000, 128, 256, "near"), (12001, 64, 128, "inside"), (9000, 24, 40, "near")])
def test_wide_precompute(fst, n, bm, ma, kind):
    """Sampled blocks, bit for bit: ancestors outside and inside the block, partial last blocks, bounds of a slot
    mask's inheritance (128 slots) and past it, odd sizes."""
    i = np.arange(n)
    if kind == "near":                                    # a shallow heap of fan-out 7
        par = np.where(i > 0, (i - 1) // 7, -1)
    else:                                                 # chains of eight inside every block, under one root
        par = np.where(i % 8 > 0, i - 1, np.where(i > 0, 0, -1))
    meta = fst.build_tree_metadata(torch.tensor(par, dtype=torch.int32), bm, ma)
    ai, am, li = (t.cpu().numpy() for t in meta)
    packed_only = fst.build_tree_metadata(torch.tensor(par, dtype=torch.int32), bm, ma, reference_format=False)
    from helpers import decode_packed
    nb = meta.n_blocks
    count, p_ai, p_am, p_li = decode_packed(packed_only.packed[0].cpu().numpy(), nb, bm, ma)
    for b in (0, 1, nb // 3, nb - 2, nb - 1):
        lo, hi = b * bm, min(n, b * bm + bm)
        rows = sets_of(par, lo, hi)
        anc = sorted(set(x for r in rows for x in r))
        assert len(anc) <= ma
        want = np.full(ma, -1)
        want[:len(anc)] = anc
        mask = np.zeros((bm, ma), bool)
        for j, r in enumerate(rows):
            for x in r + ([lo + j] if lo + j in anc else []):
                mask[j, anc.index(x)] = True
        leaf = np.array([-1 if k in anc else k for k in range(lo, lo + bm)])
        for got_i, got_m, got_l in ((ai[b], am[b], li[b]), (p_ai[b], p_am[b], p_li[b])):
            assert np.array_equal(got_i, want) and np.array_equal(got_m[:hi - lo], mask[:hi - lo]), b
            assert np.array_equal(got_l, leaf), b
        assert count[b] == sum(1 for x in anc if x < lo)


@pytest.mark.parametrize("bm,ma", [(128, 128), (128, 127), (64, 128), (100, 31), (32, 33), (16, 16), (1, 5)])
@pytest.mark.parametrize("apart", [1, 37, 1024])
@pytest.mark.parametrize("staged", [False, True])
def test_ancestor_set_and_bitmap_agree(fst, bm, ma, apart, staged):
    """Bounds of up to 128 keep a block's ancestors in a hash set, larger ones in a bitmap: the same metadata, up to a
    block whose list is full, and an error for one ancestor more.  Hubs 1024 apart crowd the hash table's places;
    staged: a tree whose parents fit shared memory."""
    n = (8192 if apart == 37 else 2500) if staged else 131072 if apart == 1024 and bm >= 32 else 9001
    apart = min(apart, (n - 1) // ma)
    for hubs in (1, ma):
        hub = np.arange(hubs) * apart
        i = np.arange(n)
        earlier = np.maximum(np.searchsorted(hub, i), 1)  # hubs below node i, at least one
        par = np.where(i > 0, hub[(i * 7919) % earlier], -1)
        if bm * (hubs > 1) >= ma:
            par[hub] = np.where(np.arange(hubs) > 0, hub[(np.arange(hubs) - 1) // 3], -1)
        else:                                             # fewer rows than ancestors: the hubs are a chain
            par[hub[1:]] = hub[:-1]
            par[0] = -1
        par = torch.tensor(par, dtype=torch.int32, device="cuda")
        got = fst.build_tree_metadata(par, bm, ma)
        want = fst.build_tree_metadata(par, bm, 160)
        assert torch.equal(got.ancestor_idx, want.ancestor_idx[:, :ma])
        assert torch.equal(got.ancestor_mask, want.ancestor_mask[..., :ma])
        assert torch.equal(got.leaf_idx, want.leaf_idx)
        from helpers import decode_packed_raw
        a, b = (decode_packed_raw(m.packed[0].cpu().numpy(), m.n_blocks, bm, w) for m, w in ((got, ma), (want, 160)))
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1][:, :ma]) and np.array_equal(a[2], b[2][..., :ma])
        assert np.array_equal(a[3], b[3])
    if int((got.ancestor_idx >= 0).sum(1).max()) == ma:
        with pytest.raises(RuntimeError, match=f"{ma} unique ancestors"):
            fst.build_tree_metadata(par, bm, ma - 1)


def test_wide_precompute_reports(fst):
    n = 10000
    star = torch.tensor([-1] * 200 + [i % 200 for i in range(200, n)], dtype=torch.int32)
    with pytest.raises(RuntimeError, match="unique ancestors"):
        fst.build_tree_metadata(star, 128, 64)
    bad = star.clone()
    bad[9000] = 9500
    with pytest.raises(ValueError, match="malformed"):
        fst.build_tree_metadata(bad, 64, 128)
    torch.cuda.synchronize()


@pytest.mark.parametrize("n", [1024, 1025, 2049, 4097, 8192])
def test_dfs_order_sizes(fst, n):
    rng = np.random.default_rng(n)
    for par in ([-1] + [int(rng.integers(max(0, i - 50), i)) for i in range(1, n)],
                [-1] + [0 if i < 60 else int(rng.integers(0, 60)) for i in range(1, n)],      # crowded parents
                [-1] + [i - 1 if i < 300 else int(rng.integers(0, 300)) for i in range(1, n)]):
        order, new_parent = fst.dfs_order(par)
        d_order, d_parent = fst.dfs_order_device(par)
        assert d_order.cpu().tolist() == order and d_parent.cpu().tolist() == new_parent


@pytest.mark.parametrize("depth,topk,lwf", [(9, 4, 0.5), (8, 10, 0.2), (3, 600, 0.002), (2, 1024, 0.001)])
def test_sorted_levels_with_random_scores_and_ties(fst, depth, topk, lwf):
    rng = np.random.default_rng(depth)
    scores = np.round(rng.standard_normal((depth + 1, topk)), 1).astype(np.float32)       # many ties, both zeros
    parent, choice, score = _topk_forest_cpu(scores, topk, lwf)
    p, c, s = fst.build_tree_topk(torch.tensor(scores, device="cuda"), left_weight_factor=lwf, return_choice=True,
                                  return_scores=True)
    assert p.cpu().tolist() == parent and c.cpu().tolist() == choice
    assert np.array_equal(s.cpu().numpy(), np.array(score, dtype=np.float32))


def test_a_captured_build_keeps_its_status_record(fst):
    """A graph writes the record it was captured with, which lives on when an eager build takes one of its own (what a
    replay reports there is the next test's)."""
    par = torch.tensor([-1] + [i // 2 for i in range(255)], dtype=torch.int32, device="cuda")
    meta = fst.build_tree_metadata(par, 64, 128, reference_format=False)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        fst.build_tree_metadata(par, 64, 128, out=meta, check=False)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        fst.build_tree_metadata(par, 64, 128, out=meta, check=False)
    record = meta.status.data_ptr()
    fst.build_tree_metadata(par, 64, 128, out=meta, check=False)
    assert meta.status.data_ptr() != record and any(t.data_ptr() == record for t in meta._captured_status)
    want = meta.packed.clone()
    graph.replay()
    assert torch.equal(meta.packed, want) and meta.check() is meta


@pytest.mark.parametrize("made_in_graph", [False, True])
def test_check_sees_what_a_replay_reports(fst, made_in_graph):
    """A problem that only a replay meets is reported by ``check``, also after an eager build in between; the next
    build, eager or replayed, starts afresh."""
    good = torch.tensor([-1] + [i // 2 for i in range(255)], dtype=torch.int32, device="cuda")
    par = good.clone()
    build = lambda **kw: fst.build_tree_metadata(par, 64, 128, reference_format=False, check=False, **kw)
    meta = build()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        meta = build() if made_in_graph else build(out=meta)
        build(out=meta)
    build(out=meta)
    assert len(meta._captured_status) == 1
    par[100] = 200
    graph.replay()
    with pytest.raises(ValueError, match="malformed"):
        meta.check()
    par.copy_(good)
    graph.replay()
    meta.check()
    par[0] = 7
    graph.replay()
    par.copy_(good)
    build(out=meta)
    meta.check()
    par[:] = torch.arange(-1, 255, device="cuda")         # a chain: 255 ancestors
    graph.replay()
    with pytest.raises(RuntimeError, match="unique ancestors"):
        meta.check()


def test_captured_builds_are_kernels_only(fst):
    """A memset node between two kernels costs a captured build some 2.5 us."""
    runtime = pytest.importorskip("cuda.bindings.runtime")
    par = torch.tensor([-1] + [i // 2 for i in range(255)], dtype=torch.int32, device="cuda")
    meta = fst.build_tree_metadata(par, 64, 128, reference_format=False)
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        fst.build_tree_metadata(par, 64, 128, out=meta, check=False)
        fst.dfs_order_device(par, check=False)
    raw = runtime.cudaGraph_t(init_value=graph.raw_cuda_graph())
    err, _, count = runtime.cudaGraphGetNodes(raw, 0)
    err, nodes, count = runtime.cudaGraphGetNodes(raw, count)
    kinds = [runtime.cudaGraphNodeGetType(n)[1] for n in nodes]
    assert len(kinds) == 4 and set(kinds) == {runtime.cudaGraphNodeType.cudaGraphNodeTypeKernel}, kinds


@pytest.mark.parametrize("n,bm,ma", [(8193, 64, 192), (9000, 64, 1000), (9001, 24, 136), (16384, 128, 320), (18945, 128, 320)])
def test_one_tree_and_many_are_built_alike(fst, n, bm, ma):
    """A deep tree alone may take one kernel and a batch of it another: the same metadata, bit for bit."""
    rng = np.random.default_rng(n)
    i = np.arange(n)
    par = np.where(i < 60, i - 1, np.where(i % 8 == 0, rng.integers(30, 60, n), i - 1))      # chains of eight behind a trunk
    par = torch.tensor(par, dtype=torch.int32, device="cuda")
    one = fst.build_tree_metadata(par, bm, ma)
    many = fst.build_tree_metadata(par.expand(6, n).contiguous(), bm, ma)
    for a, b in zip(one, many):
        assert all(torch.equal(a, b[t]) for t in range(6))
    from helpers import decode_packed_raw                 # (the bytes between its parts are nobody's)
    parts = [decode_packed_raw(x.cpu().numpy(), one.n_blocks, bm, ma) for x in (one.packed[0], *many.packed)]
    assert all(np.array_equal(a, b) for other in parts[1:] for a, b in zip(parts[0], other))
