"""The tcgen05 kernel behind a shared prefix, which walks prefix and tree: prefixes that end inside a tile, query
tiles of one to four blocks, ancestor lists that end inside a tile or run over several, and cuts that leave runs
without a tile or with the tree's tiles only."""
import pytest
import torch

pytestmark = pytest.mark.gpu
TOL = {torch.float16: 2e-3, torch.bfloat16: 1.6e-2}


@pytest.fixture(scope="module")
def fst(built_lib):
    import fstattention_b200
    return fstattention_b200


def comb(n, teeth):
    return [i - 1 if i < teeth else (i * 7) % teeth for i in range(n)]


@pytest.mark.parametrize("bm", [32, 64, 128])
@pytest.mark.parametrize("n,teeth,prefix,splits,D", [
    (1, 1, 1, 1, 128), (17, 3, 127, 1, 64), (33, 8, 128, 2, 128), (64, 20, 129, 3, 128), (65, 40, 300, 2, 64),
    (128, 33, 256, 8, 128), (129, 64, 700, 2, 128), (200, 65, 513, 3, 64), (257, 30, 384, 1, 128),
    (64, 20, 2500, 16, 128), (129, 64, 3000, 12, 64), (385, 130, 1000, 5, 128), (640, 300, 640, 2, 64), (640, 300, 130, 6, 128)])
def test_prefix_and_tree_in_one(fst, n, teeth, prefix, splits, D, bm):
    par = comb(n, teeth)
    meta = fst.build_tree_metadata(par, bm, 512, reference_format=False)
    dtype = torch.float16 if n % 2 else torch.bfloat16
    g = torch.Generator().manual_seed(n + bm)
    q = torch.randn((2, 4, n, D), generator=g).to(dtype)
    k, v = (torch.randn((2, 2, prefix + n, D), generator=g).to(dtype) for _ in range(2))
    qc, kc, vc = q.cuda(), k.cuda(), v.cuda()
    o, lse = fst.fst_attention(qc, kc, vc, meta, sm_scale=D ** -0.5, kernel="tma_umma", kv_splits=splits, return_lse=True)
    want, ref = fst.fst_attention(qc.float(), kc.float(), vc.float(), meta, sm_scale=D ** -0.5, kernel="simt", return_lse=True)
    assert (o.float() - want).abs().max().item() <= TOL[dtype]
    assert (lse - ref).abs().max().item() <= 1e-3
    assert fst.last_status() == 0


@pytest.mark.parametrize("splits", [2, 3, 4, 8])
@pytest.mark.parametrize("prefix,n,teeth", [(128, 60, 1), (257, 60, 20), (640, 100, 70), (1100, 128, 128), (1500, 90, 200), (2304, 128, 300)])
def test_one_query_tile_in_clustered_runs(fst, prefix, n, teeth, splits):
    """One query tile to a K/V head at D 128, in a cluster: K is loaded a tile ahead of V.  Runs of no, one and more tiles,
    of the tree's tiles only, with up to three gathered ones, that go round the ring of six stages and do not."""
    n = max(n, teeth + 20)
    par = comb(n, teeth)
    meta = fst.build_tree_metadata(par, 128, 512, reference_format=False)
    g = torch.Generator(device="cuda").manual_seed(prefix + splits)
    q = torch.randn((3, 25, n, 128), generator=g, device="cuda").half()       # more query tiles than idle SMs: nothing is spread
    k, v = (torch.randn((3, 25, prefix + n, 128), generator=g, device="cuda").half() for _ in range(2))
    o, lse = fst.fst_attention(q, k, v, meta, sm_scale=128 ** -0.5, kernel="tma_umma", kv_splits=splits, return_lse=True)
    want, ref = fst.fst_attention(q.float(), k.float(), v.float(), meta, sm_scale=128 ** -0.5, kernel="simt", return_lse=True)
    assert (o.float() - want).abs().max().item() <= 2e-3 and (lse - ref).abs().max().item() <= 1e-3
    assert fst.last_status() == 0


@pytest.mark.parametrize("rows", [slice(40, 50), slice(700, 710), slice(1100, 1110)])     # prefix, prefix, tree
def test_prefix_moving_maximum(fst, rows):
    """Rows whose scores dwarf the first reference point: the accumulators are rescaled."""
    n, D, prefix = 300, 128, 1000
    par = comb(n, 200)
    meta = fst.build_tree_metadata(par, 64, 256, reference_format=False)
    g = torch.Generator().manual_seed(4)
    q = torch.randn((1, 2, n, D), generator=g).half()
    k, v = (torch.randn((1, 2, prefix + n, D), generator=g) for _ in range(2))
    k[:, :, rows] *= 12.0
    q, k, v = q.cuda(), k.half().cuda(), v.half().cuda()
    for splits in (1, 3):
        o = fst.fst_attention(q, k, v, meta, sm_scale=0.5, kernel="tma_umma", kv_splits=splits)
        want = fst.fst_attention(q.float(), k.float(), v.float(), meta, sm_scale=0.5, kernel="simt")
        assert (o.float() - want).abs().max().item() <= 4e-3


def test_paged_lengths_of_their_own(fst):
    """Sequences without a prefix, with part of a page, and with the longest allowed, next to one another."""
    Z, H, n, D, ps = 4, 4, 70, 128, 16
    lens, longest = [0, 5, 130, 640], 640
    par = comb(n, 20)
    meta = fst.build_tree_metadata(par, 64, 64, reference_format=False)
    g = torch.Generator(device="cuda").manual_seed(0)
    q, kt, vt = (torch.randn((Z, H, n, D), generator=g, device="cuda").half() for _ in range(3))
    pages = longest // ps
    pool = torch.randn((2, Z * pages, ps, H, D), generator=g, device="cuda").half()
    table = torch.randperm(Z * pages, generator=g, device="cuda", dtype=torch.int32).view(Z, pages)
    for splits in (1, 3):
        o = fst.fst_attention_paged(q, kt, vt, meta, pool[0], pool[1], table,
                                    torch.tensor(lens, dtype=torch.int32, device="cuda"), D ** -0.5, max_prefix=longest,
                                    kv_splits=splits)
        for z in range(Z):
            kv = [torch.cat([p[table[z].long()].reshape(-1, H, D)[:lens[z]].transpose(0, 1), t[z]], 1)[None]
                  for p, t in ((pool[0], kt), (pool[1], vt))]
            want = fst.fst_attention(q[z:z + 1].float(), kv[0].float(), kv[1].float(), meta, sm_scale=D ** -0.5, kernel="simt")
            assert (o[z:z + 1].float() - want).abs().max().item() <= 2e-3
    assert fst.last_status() == 0


@pytest.mark.parametrize("ps", [16, 64, 128])
@pytest.mark.parametrize("n,H,H_kv,D", [(70, 4, 4, 128), (200, 4, 2, 64), (30, 8, 2, 128), (60, 16, 2, 64)])
def test_paged_rows_past_the_end(fst, ps, n, H, H_kv, D):
    """What the pool holds past a sequence's end - NaN, infinities - reaches nobody: the outputs are bit for bit
    those of a pool of zeros there.  Ends before, in and behind a 16-row step, in the first, a middle and the last tile."""
    lens = [1, 15, 16, 17, 100, 127, 128, 129, 255, 300, 383, 400]
    Z, longest = len(lens), 400
    meta = fst.build_tree_metadata(comb(n, 20), 32, 64, reference_format=False)
    g = torch.Generator(device="cuda").manual_seed(n)
    q = torch.randn((Z, H, n, D), generator=g, device="cuda").bfloat16()
    kt, vt = (torch.randn((Z, H_kv, n, D), generator=g, device="cuda").bfloat16() for _ in range(2))
    per_seq = -(-longest // ps)
    pool = torch.randn((2, Z * per_seq, ps, H_kv, D), generator=g, device="cuda").bfloat16()
    table = torch.randperm(Z * per_seq, generator=g, device="cuda", dtype=torch.int32).view(Z, per_seq)
    past = torch.zeros((Z * per_seq, ps), dtype=torch.bool, device="cuda")
    for z, end in enumerate(lens):
        for i in range(per_seq):
            past[table[z, i].long(), max(0, min(ps, end - i * ps)):] = True
    lens = torch.tensor(lens, dtype=torch.int32, device="cuda")
    for splits in (None, 1, 2, 3):
        outs = []
        for fill in (0.0, float("nan"), float("inf")):
            pool[:, past] = fill
            outs.append(fst.fst_attention_paged(q, kt, vt, meta, pool[0], pool[1], table, lens, D ** -0.5, max_prefix=longest,
                                                kv_splits=splits, return_lse=True))
        for o, lse in outs:
            assert torch.isfinite(o).all() and torch.equal(o, outs[0][0]) and torch.equal(lse, outs[0][1]), splits
    assert fst.last_status() == 0


def test_lineage_on_the_host_is_checked_there(fst):
    """The bound at which a lineage on the host is refused is the device's, and so is the message."""
    par = comb(300, 90)
    lineage, level = fst.lineage_from_parent(par)
    for bm in (16, 64):
        bound = 60
        while True:                                       # the smallest bound that the device accepts
            try:
                want = fst.build_tree_metadata(par, bm, bound)
                break
            except RuntimeError:
                bound += 1
        got = fst.create_fst_attention_kernel_inputs(lineage.clone(), level, bm, bound)
        assert bound > 60 and all(torch.equal(a, b) for a, b in zip(got, want))
        with pytest.raises(RuntimeError, match="max_ancestors"):
            fst.create_fst_attention_kernel_inputs(lineage.clone(), level, bm, bound - 1)
    bad = lineage.clone()
    bad[5, level[5] - 1] = 7
    with pytest.raises(ValueError, match="malformed"):
        fst.create_fst_attention_kernel_inputs(bad, level, 64, 128)


@pytest.mark.parametrize("D,H,H_kv", [(128, 2, 2), (64, 4, 2)])
@pytest.mark.parametrize("prefix", [1, 129, 300, 2000])
def test_nan_keys_reach_their_rows(fst, prefix, D, H, H_kv):
    """A NaN key is seen by every row that attends to it and by no other: as the only key of a tile or of a run, in
    the prefix and in the tree, with runs in a cluster and spread."""
    n = 70
    par = comb(n, 30)
    attends = torch.zeros((n, prefix + n), dtype=torch.bool)
    attends[:, :prefix] = True
    for i in range(n):
        x = i
        while x >= 0:
            attends[i, prefix + x] = True
            x = par[x]
    meta = fst.build_tree_metadata(par, 32, 64, reference_format=False)
    g = torch.Generator(device="cuda").manual_seed(prefix)
    q = torch.randn((1, H, n, D), generator=g, device="cuda").half()
    k, v = (torch.randn((1, H_kv, prefix + n, D), generator=g, device="cuda").half() for _ in range(2))
    for x in (0, prefix - 1, prefix, prefix + 29, prefix + 50):
        bad = k.clone()
        bad[:, :, x, 3] = float("nan")
        for splits in (None, 1, 2, 3, 12):
            o, lse = fst.fst_attention(q, bad, v, meta, sm_scale=0.1, kernel="tma_umma", kv_splits=splits, return_lse=True)
            for h in range(H):
                assert torch.equal(o[0, h].isnan().all(-1).cpu(), attends[:, x]), (x, splits)
                assert torch.equal(o[0, h].isnan().any(-1).cpu(), attends[:, x]), (x, splits)
                assert torch.equal(lse[h].isnan().cpu(), attends[:, x]), (x, splits)


@pytest.mark.parametrize("n,H,H_kv,D,bm", [(300, 2, 2, 128, 64), (300, 2, 2, 64, 128), (60, 8, 2, 128, 32), (30, 8, 2, 64, 32)])
@pytest.mark.parametrize("fill", [float("nan"), float("inf")])
def test_tree_values_that_are_not_finite(fst, n, H, H_kv, D, bm, fill):
    """A row of V in the tree that is not finite reaches the rows that attend to it, and else only rows that attend to
    another of the sixteen columns of one step of the product; behind a contiguous prefix and a paged one."""
    prefix, ps = 400, 16
    par = [-1] + [(i - 1) // 3 for i in range(1, n)]

    def reaches(lo, hi):
        hit = torch.zeros(n, dtype=torch.bool)
        for i, p in enumerate(par):
            hit[i] = lo <= i < hi or (p >= 0 and bool(hit[p]))
        return hit.cuda()

    meta = fst.build_tree_metadata(par, bm, 128, reference_format=False)
    g = torch.Generator(device="cuda").manual_seed(n)
    q = torch.randn((1, H, n, D), generator=g, device="cuda").half()
    k, v = (torch.randn((1, H_kv, prefix + n, D), generator=g, device="cuda").half() for _ in range(2))
    pools = [t[:, :, :prefix].transpose(1, 2).reshape(prefix // ps, ps, H_kv, D).contiguous() for t in (k, v)]
    table = torch.arange(prefix // ps, dtype=torch.int32, device="cuda")[None]
    lens = torch.tensor([prefix], dtype=torch.int32, device="cuda")
    for splits in (1, 2, 12):
        def call(v, paged):
            if paged:
                return fst.fst_attention_paged(q, k[:, :, prefix:], v[:, :, prefix:], meta, *pools, table, lens, 0.1,
                                               max_prefix=prefix, kv_splits=splits)
            return fst.fst_attention(q, k, v, meta, sm_scale=0.1, kernel="tma_umma", kv_splits=splits)
        for paged in (False, True):
            clean = call(v, paged)
            for x in (n - 1, n * 2 // 3, n // 2 - 3, 20, 5):
                bad = v.clone()
                bad[:, :, prefix + x] = fill
                o = call(bad, paged)
                assert not torch.isfinite(o[:, :, reaches(x, x + 1)]).any(), (x, splits, paged)
                if x not in par:
                    near = reaches(x // 16 * 16, x // 16 * 16 + 16)
                    assert torch.equal(o[:, :, ~near], clean[:, :, ~near]), (x, splits, paged)
    assert fst.last_status() == 0
