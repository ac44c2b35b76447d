"""The fp32-arithmetic kernel at the sizes where it can go wrong: rows that do not fill a CTA, more keys
than a warp lists at once, a prefix that is no multiple of a batch, rows that start off a vector boundary."""
import pytest
import torch

from helpers import oracle_attention
from oracle import tree_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [16, 32, 64, 128])
@pytest.mark.parametrize("n,tree,bm,prefix,shift", [
    (1, "chain", 16, 0, 0), (9, "binary", 16, 0, 1), (31, "binary", 24, 5, 0), (300, "chain", 32, 0, 0),
    (130, "star", 64, 33, 2), (257, "chain", 128, 70, 4)])
def test_simt_edges(built_lib, D, n, tree, bm, prefix, shift):
    import fstattention_b200 as fst
    par = {"chain": lambda i: i - 1, "binary": lambda i: (i - 1) // 2, "star": lambda i: 0}[tree]
    par = [-1] + [par(i) for i in range(1, n)]
    meta = fst.build_tree_metadata(par, bm, 320, reference_format=False)
    g = torch.Generator().manual_seed(n + D)
    rows = prefix + n
    q = torch.randn((2, 3, n, D + shift), generator=g)[..., shift:]
    k, v = (torch.randn((2, 1, rows, D + shift), generator=g)[..., shift:] for _ in range(2))
    dev = [torch.empty((*t.shape[:3], D + shift), device="cuda")[..., shift:].copy_(t) for t in (q, k, v)]
    o, lse = fst.fst_attention(*dev, meta, sm_scale=D ** -0.5, return_lse=True)
    want = oracle_attention(q, k.expand(2, 3, rows, D), v.expand(2, 3, rows, D), par, D ** -0.5, prefix,
                            compute_dtype=torch.float64)
    assert (o.cpu().double() - want.double()).abs().max().item() <= 2e-5
    assert torch.isfinite(lse).all() and fst.last_status() == 0


@pytest.mark.parametrize("D", [16, 32, 64, 128])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_simt_nan_and_infinite_scores(built_lib, D, dtype):
    """A NaN in a key reaches every row that attends to it, also where it is the only key that a group of lanes has,
    and no other row; a score of minus infinity is a weight of zero."""
    import fstattention_b200 as fst
    n, prefix = 70, 5
    par = [-1] + [(i - 1) // 3 for i in range(1, n)]
    meta = fst.build_tree_metadata(par, 32, 64, reference_format=False)
    lineage, _ = orc.lineage_from_parent(par)
    attends = torch.cat([torch.ones(n, prefix), orc.full_attention_mask(lineage, pad_rows=0)], 1).bool()
    g = torch.Generator().manual_seed(D)
    q, k, v = (torch.randn((1, 1, r, D), generator=g).to(dtype) for r in (n, prefix + n, prefix + n))
    call = lambda key: fst.fst_attention(q.cuda(), key.cuda(), v.cuda(), meta, sm_scale=0.3, kernel="simt", return_lse=True)
    for x in (0, 3, prefix, prefix + 1, prefix + 7, prefix + 40):
        bad = k.clone()
        bad[0, 0, x, D // 2] = float("nan")
        o, lse = (t.cpu() for t in call(bad))
        assert torch.equal(o[0, 0].isnan().all(-1), attends[:, x]) and torch.equal(lse[0].isnan(), attends[:, x]), x
        assert torch.isfinite(o[0, 0][~attends[:, x]]).all()
    q[0, 0, :, 0] = q[0, 0, :, 0].abs() + 0.1
    for x in (0, prefix, prefix + 2):                     # every row has other keys as well
        away = k.clone()
        away[0, 0, x, 0] = float("-inf")
        o, _ = (t.cpu() for t in call(away))
        mask = attends.clone()
        mask[:, x] = False
        s = (q[0, 0].double() @ k[0, 0].double().T) * 0.3
        want = torch.softmax(s.masked_fill(~mask, float("-inf")), 1) @ v[0, 0].double()
        assert (o[0, 0].double() - want).abs().max().item() <= (2e-5 if dtype == torch.float32 else 2e-3), x
