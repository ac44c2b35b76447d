"""The fp32-arithmetic kernel at the sizes where it can go wrong: rows that do not fill a CTA, more keys
than a warp lists at once, a prefix that is no multiple of a batch, rows that start off a vector boundary."""
import pytest
import torch

from helpers import oracle_attention

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
