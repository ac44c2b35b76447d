"""The tcgen05 tree kernel at the sizes where it can go wrong: rows that do not fill an item or a 16-row step,
one CTA with several items, ancestor lists that end in either half of a tile or run over many tiles, grouped
K/V heads, strided tensors, scores that outgrow the first reference point."""
import pytest
import torch

from helpers import oracle_attention

pytestmark = pytest.mark.gpu
TOL = {torch.float16: 2e-3, torch.bfloat16: 1.6e-2}


@pytest.fixture(scope="module")
def fst(built_lib):
    import fstattention_b200
    return fstattention_b200


def comb(n, teeth):
    """A chain of ``teeth`` nodes; every later node hangs under one of them in turn: a block's list is as long
    as the chain, whatever block it is."""
    return [i - 1 if i < teeth else (i * 7) % teeth for i in range(n)]


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("bm", [32, 64, 128])
@pytest.mark.parametrize("n,teeth", [(1, 1), (17, 3), (127, 20), (128, 33), (129, 64), (200, 65), (385, 130), (640, 300)])
def test_tree_umma_edges(fst, D, bm, n, teeth):
    par = comb(n, teeth)
    meta = fst.build_tree_metadata(par, bm, 512, reference_format=False)
    dtype = torch.float16 if n % 2 else torch.bfloat16
    g = torch.Generator().manual_seed(n + bm)
    q = torch.randn((2, 4, n, D), generator=g).to(dtype)
    k, v = (torch.randn((2, 2, n, D), generator=g).to(dtype) for _ in range(2))
    o, lse = fst.fst_attention(q.cuda(), k.cuda(), v.cuda(), meta, sm_scale=D ** -0.5, kernel="tree_umma", return_lse=True)
    want = oracle_attention(q, k.repeat_interleave(2, 1), v.repeat_interleave(2, 1), par, D ** -0.5,
                            compute_dtype=torch.float32)
    assert (o.cpu().float() - want.float()).abs().max().item() <= TOL[dtype]
    _, ref = fst.fst_attention(q.cuda().float(), k.cuda().float(), v.cuda().float(), meta, sm_scale=D ** -0.5,
                               kernel="simt", return_lse=True)
    assert (lse - ref).abs().max().item() <= 1e-3
    assert fst.last_status() == 0


@pytest.mark.parametrize("D,bm", [(64, 32), (64, 128), (128, 64)])
def test_tree_umma_many_items_strided(fst, D, bm):
    """Several items per CTA, a tree of its own for every batch element, [Z, N, H, D] storage."""
    from fstattention_b200 import configs
    Z, H, n = 6, 40, 300
    trees = [configs.random_window_tree(s, n, 40) for s in range(Z)]
    meta = fst.build_tree_metadata(trees, bm, 256, reference_format=False)
    g = torch.Generator(device="cuda").manual_seed(1)
    q, k, v = (torch.randn((Z, n, H, D), generator=g, device="cuda").half().permute(0, 2, 1, 3) for _ in range(3))
    out = torch.empty((Z, n, H, D), dtype=torch.float16, device="cuda").permute(0, 2, 1, 3)
    for _ in range(3):
        fst.fst_attention(q, k, v, meta, sm_scale=D ** -0.5, kernel="tree_umma", out=out)
        want = fst.fst_attention(q.float(), k.float(), v.float(), meta, sm_scale=D ** -0.5, kernel="simt")
        assert (out.float() - want).abs().max().item() <= 2e-3
    assert fst.last_status() == 0


@pytest.mark.parametrize("D,bm", [(64, 128), (128, 64)])
@pytest.mark.parametrize("own", ["alone", "chained", "across"])
@pytest.mark.parametrize("n,teeth", [(77, 1), (129, 20), (300, 16), (640, 17), (300, 32), (300, 33), (640, 64), (640, 65), (640, 97), (650, 128)])
def test_tree_umma_merged_round(fst, D, bm, own, n, teeth):
    """The scores of both tiles of an item at once (D 64, block_m 128, bounds of up to 64; longer bounds, and D 128 with block_m 64,
    take the same trees tile by tile): lists that end in any 16-column step or fill the tile; rows that attend to nobody in their block but
    themselves, to their neighbours, and to a column in another 32-column word that nobody else uses.  A value that
    is not finite stays with the rows that attend to it or to one of its fifteen neighbours."""
    par = comb(n, teeth)
    for i in range(teeth, n):
        if own == "chained" and i % 3 and i > teeth or own == "across" and i % 32 == 0 and i > teeth:
            par[i] = i - 1
    for bound in (64, 128, 128 + bm):
        try:
            meta = fst.build_tree_metadata(par, bm, bound, reference_format=False)
            break
        except RuntimeError:                              # with those inside the block there are more
            assert bound < 128 + bm
    longest = int(meta.packed[0, : meta.n_blocks * 4].view(torch.int32).max())
    assert longest <= teeth + 2 and (longest >= teeth or own == "chained" or n < 2 * bm)
    g = torch.Generator().manual_seed(n + teeth)
    q, k, v = (torch.randn((3, 60, n, D), generator=g).half().cuda() for _ in range(3))     # several items a CTA
    o, lse = fst.fst_attention(q, k, v, meta, sm_scale=D ** -0.5, kernel="tree_umma", return_lse=True)
    want, ref = fst.fst_attention(q.float(), k.float(), v.float(), meta, sm_scale=D ** -0.5, kernel="simt", return_lse=True)
    assert (o.float() - want).abs().max().item() <= TOL[torch.float16] and (lse - ref).abs().max().item() <= 1e-3
    x = n - 5
    bad = v.clone()
    bad[:, :, x] = float("nan")
    got = fst.fst_attention(q, k, bad, meta, sm_scale=D ** -0.5, kernel="tree_umma")
    near = reaches(par, x // 16 * 16, x // 16 * 16 + 16).cuda()
    assert torch.isnan(got[:, :, reaches(par, x, x + 1).cuda()]).all() and torch.equal(got[:, :, ~near], o[:, :, ~near])
    assert fst.last_status() == 0


def test_tree_umma_moving_maximum(fst):
    """A late ancestor whose score dwarfs the row's own tile: the accumulator is rescaled."""
    n, D = 400, 128
    par = comb(n, 200)
    meta = fst.build_tree_metadata(par, 64, 256, reference_format=False)
    g = torch.Generator().manual_seed(4)
    q, k, v = (torch.randn((1, 2, n, D), generator=g) for _ in range(3))
    k[:, :, 150:160] *= 12.0
    q, k, v = q.half(), k.half(), v.half()
    o = fst.fst_attention(q.cuda(), k.cuda(), v.cuda(), meta, sm_scale=0.5, kernel="tree_umma").cpu()
    want = oracle_attention(q, k, v, par, 0.5, compute_dtype=torch.float32)
    assert (o.float() - want).abs().max().item() <= 4e-3


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D,bm", [(64, 128), (64, 32), (128, 64)])
def test_tree_umma_rounds_like_the_other_kernel(fst, D, bm, dtype):
    """Both tree kernels round a probability to 16 bits once, against the largest score of its row so far: a weight that
    dominates its row is exactly 1 and costs nothing.  So their errors against 64 bits are alike: 0.99
    to 1.01 of one another over six kinds of trees, the sampling of these 260,000 outputs and more included.  Against
    a reference point that lags the maximum they were 1.09 to 1.20."""
    par = [-1] * 4 + [(i - 4) // 2 for i in range(4, 1020)]
    meta = fst.build_tree_metadata(par, bm, 256, reference_format=False)
    g = torch.Generator().manual_seed(D + bm)
    q, k, v = (torch.randn((1, 4, len(par), D), generator=g).to(dtype) for _ in range(3))
    want = oracle_attention(q, k, v, par, D ** -0.5, compute_dtype=torch.float64).double()
    err = {}
    for kernel in ("tree_umma", "tma"):
        o = fst.fst_attention(q.cuda(), k.cuda(), v.cuda(), meta, sm_scale=D ** -0.5, kernel=kernel).cpu().double()
        err[kernel] = (o - want).norm().item() / want.norm().item()
    assert err["tree_umma"] <= 1.01 * err["tma"], err      # 0.998 to 1.008 here


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D,bm", [(128, 64), (64, 128)])
def test_tree_umma_bound_changes_no_bit(fst, D, bm, dtype):
    """The bound says how long lists may be, not how they are rounded: the own tile's weights are against its own
    largest score, an ancestor tile's against the largest so far, with short bounds as with long ones.  (All
    weights of an item against one reference point were 1.2 to 2.8 % further from 64 bits.)"""
    trees = [fst.parent_from_lineage(*fst.create_tree(7)).tolist(), comb(300, 20), comb(129, 1), comb(640, 60), comb(77, 33)]
    trees.append([-1] + [(i - 1) // 3 if i % 5 else i - 1 for i in range(1, 500)])
    compared = 0
    for par in trees:
        g = torch.Generator(device="cuda").manual_seed(len(par))
        q, k, v = (torch.randn((2, 24, len(par), D), generator=g, device="cuda").to(dtype) for _ in range(3))
        want = None
        for bound in (256, 128, 64):
            try:
                meta = fst.build_tree_metadata(par, bm, bound, reference_format=False)
            except RuntimeError:                          # the tree needs more
                continue
            got = fst.fst_attention(q, k, v, meta, sm_scale=D ** -0.5, kernel="tree_umma", return_lse=True)
            if want is not None:
                assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1]), (len(par), bound)
                compared += bound == 64
            want = want or got
    assert compared >= 4 and fst.last_status() == 0


def test_forest_is_rounded_as_by_the_mma_kernel(fst):
    """D 128, block_m 64, one short list to a block: both kernels wait for the same bytes, so the choice falls on the one that
    is nearer to 64 bits (by 0.3 %), however large the forest."""
    from fstattention_b200 import configs
    trees = configs.jittered_forest(0, 24, 256)
    trees = [t + [0] * (256 - len(t)) for t in trees]
    meta = fst.build_tree_metadata(trees, 64, 64, reference_format=False)
    g = torch.Generator(device="cuda").manual_seed(3)
    q, k, v = (torch.randn((24, 32, 256, 128), generator=g, device="cuda").half() for _ in range(3))
    got, want = (fst.fst_attention(q, k, v, meta, sm_scale=128 ** -0.5, kernel=kernel) for kernel in ("auto", "tma"))
    assert torch.equal(got, want)


def reaches(par, lo, hi):
    """Which nodes attend to one of the nodes lo .. hi - 1."""
    hit = torch.zeros(len(par), dtype=torch.bool)
    for i, p in enumerate(par):
        hit[i] = lo <= i < hi or (p >= 0 and bool(hit[p]))
    return hit


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("bm", [32, 64, 128])
@pytest.mark.parametrize("fill", [float("nan"), float("inf")])
def test_tree_umma_values_that_are_not_finite(fst, D, bm, fill):
    """A row of V that is not finite reaches the rows that attend to it, and else only rows that attend to another of
    the sixteen columns of one step of the product - not the rest of the item, whose weights for it are zero."""
    n = 300
    par = [-1] + [(i - 1) // 3 for i in range(1, n)]
    meta = fst.build_tree_metadata(par, bm, 256, reference_format=False)
    g = torch.Generator(device="cuda").manual_seed(bm)
    q, k, v = (torch.randn((2, 3, n, D), generator=g, device="cuda").half() for _ in range(3))
    clean = fst.fst_attention(q, k, v, meta, sm_scale=D ** -0.5, kernel="tree_umma")
    for x in (299, 200, 137, 40, 5):
        bad = v.clone()
        bad[:, :, x] = fill
        o = fst.fst_attention(q, k, bad, meta, sm_scale=D ** -0.5, kernel="tree_umma")
        hit, near = reaches(par, x, x + 1).cuda(), reaches(par, x // 16 * 16, x // 16 * 16 + 16).cuda()
        assert not torch.isfinite(o[:, :, hit]).any(), x
        if not any(p == x for p in par):                  # nobody's ancestor: in its own item's tile only
            assert torch.equal(o[:, :, ~near], clean[:, :, ~near]), x
        block = x // 128 * 128                            # rows of earlier items do not attend to it at all
        assert torch.equal(o[:, :, :block], clean[:, :, :block]), x
    assert fst.last_status() == 0


def test_tree_umma_behind_a_long_launch(fst):
    """A launch that becomes resident while the one ahead runs for longer than the bound of its waits: no role's
    bound starts before the launch ahead has ended.  (The launch ahead is one CTA that walks a long prefix.)"""
    n, D, prefix = 64, 64, 8_000_000
    meta = fst.build_tree_metadata([-1] + [0] * (n - 1), 64, 64, reference_format=False)
    g = torch.Generator(device="cuda").manual_seed(0)
    long_kv = torch.randn((1, 1, prefix + n, D), generator=g, device="cuda").half()
    q, k, v = (torch.randn((1, 4, n, D), generator=g, device="cuda").half() for _ in range(3))
    small = lambda: fst.fst_attention(q, k, v, meta, sm_scale=0.1, kernel="tree_umma")
    ahead = lambda: fst.fst_attention(q[:, :1], long_kv, long_kv, meta, sm_scale=0.1, kernel="tma", kv_splits=1)
    small()
    want = small()
    start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    start.record()
    ahead()
    end.record()
    torch.cuda.synchronize()
    assert start.elapsed_time(end) > 75.0                 # half as long again as the bound
    ahead()
    got = small()
    torch.cuda.synchronize()
    assert fst.last_status() == 0 and torch.equal(got, want)


@pytest.mark.parametrize("n,H,H_kv", [(16, 16, 2), (17, 16, 2), (32, 8, 2), (33, 8, 2), (64, 8, 4), (65, 8, 4), (9, 12, 2)])
@pytest.mark.parametrize("D", [64, 128])
def test_prefix_heads_share_a_query_tile(fst, n, H, H_kv, D):
    """Grouped-query heads packed into one query tile of the prefix kernel, contiguous and paged."""
    from fstattention_b200 import configs
    par = configs.random_window_tree(n, n, 8)
    meta = fst.build_tree_metadata(par, 32, 128, reference_format=False)
    P, ps = 700, 16
    g = torch.Generator(device="cuda").manual_seed(n)
    q = torch.randn((2, H, n, D), generator=g, device="cuda").half()
    k, v = (torch.randn((2, H_kv, P + n, D), generator=g, device="cuda").half() for _ in range(2))
    want, lse_w = fst.fst_attention(q, k, v, meta, sm_scale=D ** -0.5, kernel="tma_t32", kv_splits=1, return_lse=True)
    got, lse = fst.fst_attention(q, k, v, meta, sm_scale=D ** -0.5, kernel="tma_umma", return_lse=True)
    assert (got.float() - want.float()).abs().max().item() <= 2e-3 and (lse - lse_w).abs().max().item() <= 2e-2
    pages = -(-P // ps)
    pool = torch.zeros((2, 2 * pages, ps, H_kv, D), dtype=torch.float16, device="cuda")
    for kv, src in enumerate((k, v)):
        for z in range(2):
            rows = torch.zeros((pages * ps, H_kv, D), dtype=torch.float16, device="cuda")
            rows[:P] = src[z, :, :P].transpose(0, 1)
            pool[kv, z * pages:(z + 1) * pages] = rows.view(pages, ps, H_kv, D)
    table = torch.arange(2 * pages, dtype=torch.int32, device="cuda").view(2, pages)
    lens = torch.tensor([P, P], dtype=torch.int32, device="cuda")
    o = fst.fst_attention_paged(q, k[:, :, P:].contiguous(), v[:, :, P:].contiguous(), meta, pool[0], pool[1], table, lens,
                                D ** -0.5, max_prefix=P)
    assert (o.float() - want.float()).abs().max().item() <= 2e-3
    assert fst.last_status() == 0
