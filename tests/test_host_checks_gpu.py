"""Calls whose tensors do not fit together are refused on the host, before anything is launched, and calls
with unusual but valid tensors are answered."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fst(built_lib):
    import fstattention_b200
    return fstattention_b200


def qkv(Z, H, n, D, n_kv=None, dtype=torch.float16, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn((Z, H, r, D), generator=g, device="cuda").to(dtype) for r in (n, n_kv or n, n_kv or n)]


def test_reference_tensors_describe_the_same_trees(fst):
    Z, n, bm, ma = 3, 100, 32, 64
    idx, mask, leaf = (t.clone() for t in fst.build_tree_metadata([[-1] + [i // 2 for i in range(n - 1)]] * Z, bm, ma))
    q, k, v = qkv(Z, 2, n, 64)
    args = dict(sm_scale=0.125, BLOCK_M=bm, MAX_ANCESTORS=ma)
    want = fst.fst_attention(q, k, v, idx, mask, leaf, **args)
    for a, b, c in ((idx, mask[0], leaf), (idx, mask, leaf[0]), (idx, mask[:2], leaf), (idx, mask, leaf[1:])):
        with pytest.raises(ValueError, match="as many trees"):
            fst.fst_attention(q, k, v, a, b, c, **args)
    # one list of ancestors: the first tree of the others, as ever
    assert torch.equal(fst.fst_attention(q, k, v, idx[0], mask, leaf, **args), want)
    assert torch.equal(fst.fst_attention(q, k, v, idx[:1], mask[:1], leaf[0], **args), want)
