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


def test_paged_prefix_lengths_of_any_stride(fst):
    """Lengths out of a column of a table, and one length for all."""
    Z, H, n, D, ps = 3, 2, 20, 128, 16
    meta = fst.build_tree_metadata([-1] + [0] * (n - 1), 32, 32, reference_format=False)
    q, k, v = qkv(Z, H, n, D)
    pool = torch.randn((2, Z * 8, ps, H, D), generator=torch.Generator(device="cuda").manual_seed(1), device="cuda").half()
    table = torch.arange(Z * 8, dtype=torch.int32, device="cuda").view(Z, 8)
    wide = torch.tensor([[100, 0], [7, 128], [128, 3]], dtype=torch.int32, device="cuda")
    for lens in (wide[:, 0], wide[:1, 0].expand(Z)):
        assert not lens.is_contiguous()
        got, want = (fst.fst_attention_paged(q, k, v, meta, pool[0], pool[1], table, x, 0.1, max_prefix=128)
                     for x in (lens, lens.clone(memory_format=torch.contiguous_format)))
        assert torch.equal(got, want)


def test_tensors_of_one_device(fst):
    """Metadata buffers that were moved to the host (or, with two GPUs, tensors of the other one) are refused."""
    n = 40
    par = torch.tensor([-1] + [0] * (n - 1), dtype=torch.int32, device="cuda")
    meta = fst.build_tree_metadata(par, 32, 32, reference_format=False)
    q, k, v = qkv(1, 2, n, 128)
    pool = torch.zeros((4, 16, 2, 128), dtype=torch.float16, device="cuda")
    table, lens = torch.zeros((1, 4), dtype=torch.int32, device="cuda"), torch.tensor([40], dtype=torch.int32, device="cuda")
    elsewhere = ["cpu"] + ["cuda:1"] * (torch.cuda.device_count() > 1)
    for other in elsewhere:
        meta.packed = meta.packed.to(other)
        for call in (lambda: fst.fst_attention(q, k, v, meta, sm_scale=0.1),
                     lambda: fst.fst_attention(q.float(), k.float(), v.float(), meta, sm_scale=0.1),
                     lambda: fst.fst_attention_paged(q, k, v, meta, pool, pool, table, lens, 0.1, max_prefix=40),
                     lambda: fst.build_tree_metadata(par, 32, 32, out=meta)):
            with pytest.raises(RuntimeError, match="one device"):
                call()
        meta.packed = meta.packed.to("cuda:0")
        for i in (1, 2):
            args = [q, k, v]
            args[i] = args[i].to(other)
            with pytest.raises(RuntimeError, match="one device|CUDA tensors"):
                fst.fst_attention(*args, meta, sm_scale=0.1)
        with pytest.raises((RuntimeError, ValueError), match="one device|out must match"):
            fst.fst_attention(q, k, v, meta, sm_scale=0.1, out=q.to(other))
    fst.fst_attention(q, k, v, meta, sm_scale=0.1)


def test_block_size_of_the_metadata_tensors(fst):
    """Tensors of one block size with another BLOCK_M or MAX_ANCESTORS beside them, with and without ``scatter``."""
    class Copy:
        n_ranks, rank, z0, h0 = 1, 0, 0, 0

    import ctypes
    n = 64
    three = tuple(fst.build_tree_metadata([-1] + [0] * (n - 1), 32, 64))
    q, k, v = qkv(1, 2, n, 64)
    to = Copy()
    to.local = torch.empty_like(q)
    to.pointer_array = (ctypes.c_void_p * 1)(to.local.data_ptr())
    for scatter in (None, to):
        for bm, ma in ((64, 64), (32, 32), (64, 32)):
            with pytest.raises(ValueError, match="BLOCK_M / MAX_ANCESTORS"):
                fst.fst_attention(q, k, v, *three, sm_scale=0.1, BLOCK_M=bm, MAX_ANCESTORS=ma, scatter=scatter)
    want = fst.fst_attention(q, k, v, *three, sm_scale=0.1, BLOCK_M=32, MAX_ANCESTORS=64)
    assert torch.equal(fst.fst_attention(q, k, v, *three, sm_scale=0.1, BLOCK_M=32, MAX_ANCESTORS=64, scatter=to), want)


def test_paged_without_a_prefix(fst):
    """Plain tree attention, and the same checks as with a prefix."""
    Z, H, n, D, ps = 2, 4, 20, 128, 16
    meta = fst.build_tree_metadata([-1] + [0] * (n - 1), 32, 32, reference_format=False)
    q, k, v = qkv(Z, H, n, D)
    pool = torch.zeros((4, ps, H, D), dtype=torch.float16, device="cuda")
    table, lens = torch.zeros((Z, 2), dtype=torch.int32, device="cuda"), torch.zeros(Z, dtype=torch.int32, device="cuda")
    want, want_lse = fst.fst_attention(q, k, v, meta, sm_scale=-0.1, return_lse=True)
    for max_prefix in (None, 0, -1):
        got, lse = fst.fst_attention_paged(q, k, v, meta, pool, pool, table, lens, -0.1, max_prefix=max_prefix, return_lse=True)
        assert torch.equal(got, want) and torch.equal(lse, want_lse)
        for bad, error in (((pool.cpu(), pool, table, lens), RuntimeError), ((pool, pool.float(), table, lens), TypeError),
                           ((pool[:, :, :2], pool[:, :, :2], table, lens), ValueError), ((pool, pool, table.long(), lens), ValueError),
                           ((pool, pool, table, lens[:1]), ValueError), ((pool, pool, table[:1], lens), ValueError)):
            with pytest.raises(error):
                fst.fst_attention_paged(q, k, v, meta, *bad, 0.1, max_prefix=max_prefix)


def test_a_number_of_splits_of_any_type(fst):
    n, prefix = 20, 600
    meta = fst.build_tree_metadata([-1] + [0] * (n - 1), 32, 32)
    q, k, v = qkv(1, 2, n, 64, prefix + n)
    want = fst.fst_attention(q, k, v, meta, sm_scale=0.1, kv_splits=2)
    for splits in (2.0, torch.tensor(2)):
        assert torch.equal(fst.fst_attention(q, k, v, meta, sm_scale=0.1, kv_splits=splits), want)
        idx, mask, leaf = (t.clone() for t in meta)
        idx += prefix
        leaf += prefix
        assert torch.equal(fst.fst_attention(q, k, v, idx, mask, leaf, 0.1, BLOCK_M=32, MAX_ANCESTORS=32, kv_splits=splits), want)


def test_a_plan_for_a_host_tensor_leaves_no_error_behind(fst):
    """launch_plan looks at shape and type; the next launch in the process must not be blamed for the host's device index."""
    q = torch.empty((1, 8, 127, 128), dtype=torch.float16)
    want = fst.launch_plan(q.cuda(), 4096, 64)
    assert fst.launch_plan(q, 4096, 64) == want
    assert torch.equal(torch.ones(8, device="cuda").clone(), torch.ones(8, device="cuda"))
