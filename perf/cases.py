"""What a user of this framework has it do, as a list of measurable cases.

A decoder that speculates with token trees uses the package in a few ways, and each has its
family here:

  layer     one attention call on metadata that is already there (every transformer layer)
  step      one decode step: the tree's metadata rebuilt from its parent array, then one attention
            call per layer
  prefix    one attention call whose tree hangs behind a prompt held in contiguous K/V tensors
  paged     the same with the prompt in a paged KV cache, sequences of different lengths
  reference the call sequence of the original package: lineage tensors on the host, index tensors
            shifted by the prefix length, plain tensors into the attention call
  grow      the tree itself grown on the GPU from top-k scores, renumbered, metadata built
  metadata  metadata of large trees in the reference's tensor format

``listed()`` names twelve cases over these families, ``draw(rng)`` gives others of the same ranges.
Trees come from ``fstattention_b200.configs``, from ``create_tree`` or, for trees that depend on
scores, from the same recurrence with a random choice of the expanded nodes.
"""
import math
import random

import numpy as np
import torch

import fstattention_b200 as fst
from fstattention_b200 import configs

DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16, "fp32": torch.float32}


# ---------------------------------------------------------------------------------------------
# trees
# ---------------------------------------------------------------------------------------------
def scored_tree(nodes, seed):
    """Parent array of a score-driven top-4 forest: of every level a random half (the nodes that
    happened to score best) is expanded into four children each, level by level, cut at ``nodes``."""
    rng = np.random.default_rng(seed)
    parent = [np.full(4, -1, dtype=np.int64)]
    start, size, total = 0, 4, 4
    while total < nodes:
        kept = np.sort(rng.choice(size, max(1, size // 2), replace=False)) + start
        parent.append(np.repeat(kept, 4))
        start, size = total, 4 * kept.size
        total += size
    return np.concatenate(parent)[:nodes].tolist()


def one_tree(kind, nodes, seed):
    if kind == "binary":                       # complete binary tree, breadth first
        return configs.binary_tree(nodes)
    if kind == "medusa":                       # left-weighted static tree, fan-out jittered by the seed
        fan = [c + random.Random(seed + d).choice((-1, 0, 1)) for d, c in enumerate(configs.MEDUSA_FANOUT)]
        tree = configs.left_weighted_tree(fan, nodes)
        return tree + [0] * (nodes - len(tree))
    if kind == "window":                       # dynamic tree, parents drawn from the 64 nodes before
        return configs.random_window_tree(seed, nodes)
    if kind == "deep":                         # chains behind a shared trunk
        return configs.deep_chain_tree(seed, nodes)
    if kind == "scored":                       # the best half of every level expanded
        return scored_tree(nodes, seed)
    if kind == "create":                       # the original package's benchmark forest
        depth = int(math.log2(nodes + 4)) - 3
        return fst.parent_from_lineage(*fst.create_tree(depth)).tolist()
    raise KeyError(kind)


def tree_tensor(case, seed):
    """int32 parent arrays on the GPU: [N], or [T, N] when every batch element has its own tree."""
    if case.get("trees", 1) == 1:
        tree = one_tree(case["tree"], case["nodes"], seed)
    else:
        tree = [one_tree(case["tree"], case["nodes"], seed * 1009 + 31 * i) for i in range(case["trees"])]
    return torch.tensor(tree, dtype=torch.int32, device="cuda")


# Nodes a row attends to besides the prefix (itself and its ancestors), on average.
MEAN_LINEAGE = {"binary": lambda n: math.log2(n + 1) - 1, "medusa": lambda n: 4.5, "window": lambda n: 2 + n / 45,
                "deep": lambda n: 48.0, "scored": lambda n: math.log2(n + 4) - 3, "create": lambda n: math.log2(n + 4) - 3}


# Ancestor bound a user sets for a kind of tree and a block size.
def ancestor_bound(tree, block_m):
    return {"binary": 128, "medusa": 64 if block_m <= 64 else 128, "window": 320 if block_m <= 64 else 384,
            "deep": 128 if block_m <= 64 else 256, "scored": 128, "create": 64}[tree]


# ---------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------
def listed():
    return [
        # The smallest call: 31-node tree in fp32 with four heads, as one checks a model with.
        dict(name="layer_fp32_31", op="layer", tree="binary", nodes=31, trees=1, batch=1, heads=4, kv_heads=4,
             head_dim=64, dtype="fp32", block_m=16, max_ancestors=16, lse=False),
        # A small grouped-query model with an odd tree size, log-sum-exps wanted.
        dict(name="layer_bf16_gqa_77", op="layer", tree="medusa", nodes=77, trees=1, batch=2, heads=16, kv_heads=4,
             head_dim=64, dtype="bf16", block_m=32, max_ancestors=64, lse=True),
        # The everyday decode step: 256-node Medusa tree, sixteen layers of a 32-head model.
        dict(name="step_medusa_256", op="step", tree="medusa", nodes=256, trees=1, heads=32, kv_heads=32,
             head_dim=128, dtype="fp16", block_m=64, max_ancestors=64, layers=16),
        # A dynamic 1024-node tree, regenerated every step.
        dict(name="step_window_1024", op="step", tree="window", nodes=1024, trees=1, heads=32, kv_heads=32,
             head_dim=128, dtype="fp16", block_m=64, max_ancestors=320, layers=4),
        # Batched decoding: 64 sequences, each with a tree of its own.
        dict(name="layer_forest_64x256", op="layer", tree="medusa", nodes=256, trees=64, batch=64, heads=32,
             kv_heads=32, head_dim=128, dtype="fp16", block_m=64, max_ancestors=64, lse=False),
        # A large deep tree.
        dict(name="layer_deep_4096", op="layer", tree="deep", nodes=4096, trees=1, batch=1, heads=64, kv_heads=64,
             head_dim=128, dtype="fp16", block_m=64, max_ancestors=128, lse=False),
        # The top of the original package's benchmark sweep (batch 4, 48 heads, 128-row blocks).
        dict(name="layer_create_65536", op="layer", tree="create", nodes=65532, trees=1, batch=4, heads=48,
             kv_heads=48, head_dim=64, dtype="fp16", block_m=128, max_ancestors=64, lse=False),
        # A tree behind a 4096-token prompt.
        dict(name="prefix_4096", op="prefix", tree="medusa", nodes=256, batch=1, heads=32, kv_heads=32, head_dim=128,
             dtype="fp16", block_m=64, max_ancestors=64, prefix=4096),
        # Serving: eight sequences of different lengths in a paged cache, grouped-query bf16 model.
        dict(name="paged_8x64", op="paged", tree="medusa", nodes=64, batch=8, heads=32, kv_heads=8, head_dim=128,
             dtype="bf16", block_m=64, max_ancestors=64, prefix=3001, page_size=16, layout="NHD"),
        # The original package's own test sequence, host tensors in, 1024-token prefix.
        dict(name="reference_1024", op="reference", depth=7, batch=2, heads=8, head_dim=64, dtype="fp16", block_m=64,
             max_ancestors=64, prefix=1024),
        # A tree of 1020 nodes grown from the scores of eight heads, for four sequences.
        dict(name="grow_4x1020", op="grow", depth=7, topk=4, weight=0.5, trees=4, block_m=64, max_ancestors=128),
        # Metadata of the largest tree in the original package's tables.
        dict(name="metadata_131068", op="metadata", tree="scored", nodes=131068, trees=1, block_m=128,
             max_ancestors=128),
    ]


def log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def fit(rng, room, lo, hi):
    """A count between lo and hi, no larger than ``room`` allows."""
    return log_int(rng, lo, max(lo, min(hi, int(room))))


def heads_of(rng, room):
    """(query heads, K/V heads): multi-head half of the time, else grouped-query."""
    group = rng.choice((1, 1, 1, 2, 4, 8))
    kv = fit(rng, room / group, 1, 64 // group)
    return kv * group, kv


def draw(rng):
    op = rng.choice(("fp32", "layer", "layer", "sweep", "step", "step", "prefix", "prefix", "paged", "paged",
                     "reference", "grow", "metadata"))
    dtype = rng.choice(("fp16", "bf16"))
    head_dim = rng.choice((64, 128))
    if op == "fp32":
        tree, bm = rng.choice(("binary", "medusa")), rng.choice((16, 32, 64))
        heads, kv = heads_of(rng, 16)
        return dict(op="layer", tree=tree, nodes=log_int(rng, 15, 511), trees=1, batch=rng.randint(1, 2), heads=heads,
                    kv_heads=kv, head_dim=rng.choice((16, 32, 64, 128)), dtype="fp32", block_m=bm,
                    max_ancestors=ancestor_bound(tree, bm), lse=rng.random() < 0.3)
    if op == "layer":
        tree = rng.choice(("medusa", "window", "deep", "scored"))
        nodes = log_int(rng, 16, {"medusa": 300, "window": 1024, "deep": 8192, "scored": 8192}[tree])
        bm = rng.choice((32, 64, 64, 128))
        rows = 2 ** 20                                    # rows over all heads and batch elements
        heads, kv = heads_of(rng, rows / nodes)
        batch = fit(rng, rows / nodes / heads, 1, 64)
        return dict(op="layer", tree=tree, nodes=nodes, trees=batch if rng.random() < 0.5 else 1, batch=batch,
                    heads=heads, kv_heads=kv, head_dim=head_dim, dtype=dtype, block_m=bm,
                    max_ancestors=ancestor_bound(tree, bm), lse=rng.random() < 0.3)
    if op == "sweep":
        head_dim = rng.choice((64, 64, 64, 128))
        return dict(op="layer", tree="create", nodes=2 ** rng.randint(10, 16) - 4, trees=1, batch=rng.randint(1, 4),
                    heads=rng.randint(8, 3072 // head_dim), kv_heads=None, head_dim=head_dim,
                    dtype=dtype, block_m=128, max_ancestors=64, lse=False)
    if op == "step":
        tree = rng.choice(("medusa", "window", "scored"))
        nodes = log_int(rng, 16, {"medusa": 300, "window": 1024, "scored": 2048}[tree])
        heads, kv = heads_of(rng, 2 ** 16 / nodes)
        bm = rng.choice((32, 64, 64, 128))
        return dict(op="step", tree=tree, nodes=nodes, trees=1, heads=heads, kv_heads=kv, head_dim=head_dim,
                    dtype=dtype, block_m=bm, max_ancestors=ancestor_bound(tree, bm), layers=log_int(rng, 2, 32))
    if op in ("prefix", "paged"):
        tree = rng.choice(("medusa", "scored"))
        nodes = log_int(rng, 16, 300)
        prefix = log_int(rng, 64, 16384)
        heads, kv = heads_of(rng, 64)
        # at most the work of 64 heads x 8 batch elements x 64 nodes x 8192 rows
        batch = fit(rng, 2 ** 28 / (nodes * heads * prefix), 1, 16)
        bm = rng.choice((32, 64, 64, 128))
        c = dict(op=op, tree=tree, nodes=nodes, batch=batch, heads=heads, kv_heads=kv, head_dim=head_dim, dtype=dtype,
                 block_m=bm, max_ancestors=ancestor_bound(tree, bm), prefix=prefix)
        if op == "paged":
            c.update(page_size=rng.choice((16, 32, 64, 128)), layout=rng.choice(("NHD", "HND")))
        return c
    if op == "reference":
        return dict(op="reference", depth=rng.randint(3, 9), batch=rng.randint(1, 4), heads=rng.randint(1, 16),
                    head_dim=head_dim, dtype="fp16", block_m=rng.choice((64, 128)), max_ancestors=64,
                    prefix=rng.choice((0, log_int(rng, 64, 2048))))
    if op == "grow":
        topk = rng.randint(2, 10)
        return dict(op="grow", depth=rng.randint(3, 8), topk=topk, weight=round(rng.uniform(1.05, 2.0) / topk, 3),
                    trees=log_int(rng, 1, 64), block_m=rng.choice((32, 64, 128)), max_ancestors=512)
    nodes = log_int(rng, 512, 131068)
    return dict(op="metadata", tree="scored", nodes=nodes, trees=fit(rng, 131068 / nodes, 1, 64),
                block_m=rng.choice((32, 64, 128)), max_ancestors=128)


# ---------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------
def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype = DTYPES.get(case.get("dtype"))
    op = case["op"]
    s = {"op": op, "bm": case["block_m"], "ma": case["max_ancestors"]}

    def normal(*shape):
        return torch.randn(shape, generator=gen, device="cuda", dtype=dtype)

    if op == "grow":
        s["args"] = (case["depth"], case["topk"], case["weight"])
        logits = torch.randn((case["trees"], case["depth"] + 1, case["topk"]), generator=gen, device="cuda")
        s["scores"] = torch.log_softmax(logits, dim=-1)
        return s
    if op == "reference":
        D, prefix = case["head_dim"], case["prefix"]
        s["lineage"], s["level"] = fst.create_tree(case["depth"])
        rows = 2 ** (case["depth"] + 3)                   # the forest's node count and four more
        s["q"] = normal(case["batch"], case["heads"], rows, D)
        s["k"], s["v"] = (normal(case["batch"], case["heads"], prefix + rows, D) for _ in range(2))
        s["prefix"], s["scale"] = prefix, D ** -0.5
        return s

    s["parent"] = tree_tensor(case, seed)
    if op == "metadata":
        return s
    # the metadata a decoder holds when a layer is called (and, in a step, the buffers it rebuilds)
    s["meta"] = fst.build_tree_metadata(s["parent"], s["bm"], s["ma"], reference_format=False)
    N, D = case["nodes"], case["head_dim"]
    n_rows = N + 4 if case["tree"] == "create" else N     # the original benchmark pads its forests to 2^k rows
    H, H_kv, Z = case["heads"], case["kv_heads"] or case["heads"], case.get("batch", 1)
    s["scale"] = D ** -0.5
    if op == "paged":
        ps = case["page_size"]
        lens = torch.tensor([random.Random(seed + 7 * z).randint(case["prefix"] // 4, case["prefix"]) for z in range(Z)])
        lens[seed % Z] = case["prefix"]
        per_seq = -(-case["prefix"] // ps)
        n_pages = Z * per_seq + 8
        order = torch.randperm(n_pages, generator=gen, device="cuda")[: Z * per_seq]
        s["table"] = order.to(torch.int32).reshape(Z, per_seq).contiguous()
        s["lens"], s["max_prefix"] = lens.to(torch.int32).cuda(), case["prefix"]
        s["layout"] = case["layout"]
        shape = (n_pages, ps, H_kv, D) if case["layout"] == "NHD" else (n_pages, H_kv, ps, D)
        s["k_pool"], s["v_pool"] = normal(*shape), normal(*shape)
    rows_kv = n_rows + (case["prefix"] if op == "prefix" else 0)
    s["qkv"] = [(normal(Z, H, n_rows, D), normal(Z, H_kv, rows_kv, D), normal(Z, H_kv, rows_kv, D))
                for _ in range(case.get("layers", 1))]
    s["lse"] = bool(case.get("lse", False))
    return s


# ---------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------
def run(s):
    op = s["op"]
    if op in ("layer", "prefix"):
        q, k, v = s["qkv"][0]
        return fst.fst_attention(q, k, v, s["meta"], sm_scale=s["scale"], return_lse=s["lse"])
    if op == "step":
        meta = fst.build_tree_metadata(s["parent"], s["bm"], s["ma"], reference_format=False, check=False, out=s["meta"])
        return [fst.fst_attention(q, k, v, meta, sm_scale=s["scale"]) for q, k, v in s["qkv"]]
    if op == "paged":
        q, k, v = s["qkv"][0]
        return fst.fst_attention_paged(q, k, v, s["meta"], s["k_pool"], s["v_pool"], s["table"], s["lens"], s["scale"],
                                       max_prefix=s["max_prefix"], pool_layout=s["layout"])
    if op == "reference":
        idx, mask, leaf = fst.create_fst_attention_kernel_inputs(s["lineage"], s["level"], block_m=s["bm"],
                                                                 max_ancestors=s["ma"])
        idx += s["prefix"]
        leaf += s["prefix"]
        o = fst.fst_attention(s["q"], s["k"], s["v"], idx, mask, leaf, s["scale"], BLOCK_M=s["bm"], MAX_ANCESTORS=s["ma"])
        return {"o": o, "idx": idx, "mask": mask, "leaf": leaf}
    if op == "grow":
        parent, choice = fst.build_tree_topk(s["scores"], *s["args"], return_choice=True)
        order, parent = fst.dfs_order_device(parent, check=False)
        meta = fst.build_tree_metadata(parent, s["bm"], s["ma"], check=False)
        return (order, parent, choice) + tuple(meta)
    return tuple(fst.build_tree_metadata(s["parent"], s["bm"], s["ma"], check=False))


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------
def metadata_bytes(case, nodes, trees):
    """Parent array in; ancestor indices, mask and leaf indices of every block out."""
    blocks = -(-nodes // case["block_m"])
    per_block = 8 * case["max_ancestors"] + case["block_m"] * case["max_ancestors"] + 8 * case["block_m"]
    return trees * (4 * nodes + blocks * per_block)


def work(case):
    op = case["op"]
    if op == "metadata":
        return {"bytes": metadata_bytes(case, case["nodes"], case["trees"]), "flops": 0}
    if op == "grow":
        n = fst.tree_topk_nodes(case["depth"], case["topk"], case["weight"])
        scores = 4 * (case["depth"] + 1) * case["topk"]
        return {"bytes": case["trees"] * (scores + 12 * n) + metadata_bytes(case, n, case["trees"]), "flops": 0}
    es = 4 if case["dtype"] == "fp32" else 2
    D, H = case["head_dim"], case["heads"]
    if op == "reference":
        n, rows, prefix = 2 ** (case["depth"] + 3) - 4, 2 ** (case["depth"] + 3), case["prefix"]
        z = case["batch"]
        lineage = MEAN_LINEAGE["create"](n)
        return {"bytes": metadata_bytes(case, n, 1) + z * H * (4 * rows + 2 * prefix) * D * es,
                "flops": 4 * D * z * H * rows * (prefix + lineage)}
    n = case["nodes"] + (4 if case["tree"] == "create" else 0)
    H_kv, z, layers = case["kv_heads"] or H, case.get("batch", 1), case.get("layers", 1)
    prefix = case.get("prefix", 0)
    if op == "paged":
        prefix = 0.7 * prefix                             # the sequences' mean length
    kv = 2 * z * H_kv * (n + prefix) * D * es
    qo = 2 * z * H * n * D * es
    flops = 4 * D * z * H * n * (prefix + MEAN_LINEAGE[case["tree"]](n))
    return {"bytes": layers * (kv + qo), "flops": layers * flops}


def tolerance(case):
    """Integers are exact; probabilities and outputs are rounded to the tensors' own type."""
    if case["op"] in ("metadata", "grow"):
        return "exact"
    return {"rel": {"fp32": 1e-5, "fp16": 2e-3, "bf16": 1e-2}[case["dtype"]]}
