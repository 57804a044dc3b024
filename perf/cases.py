"""What this framework is used for, as cases that can be timed and compared.

A training step runs GCA forward and backward over chunks read from the cache, and the retrieval that
chose them with its gradients.  A prefill projects the encoded chunks into the cache and runs the GCA
sub-layer over whole chunks.  A decode step runs the GCA sub-layer and the windowed attention for one new
position per sequence, and a retrieval over every cached landmark when a chunk is complete.  Shapes are
those of the model configuration (12 heads x 64, chunk 64, top-k 8, window 512), of `bench.py` and of the
tests; `draw` spreads the sizes around them.
"""
from __future__ import annotations

import math

import torch

import long_context_modeling_b200 as lcm
from long_context_modeling_b200 import fused_ops

CHUNK = HEAD_DIM = 64
SCALE = 1.0 / math.sqrt(HEAD_DIM)
ESIZE = {"bf16": 2, "fp32": 4}
DTYPE = {"bf16": torch.bfloat16, "fp32": torch.float32}
SLOT_FLOPS = 4 * CHUNK * CHUNK * HEAD_DIM        # QK^T and PV of one (query chunk, head, retrieved chunk)
LARGEST_TRAIN = 8 * 256 * 12 * 8                 # (sequence, chunk, head, slot) of the largest training case


# ---------------------------------------------------------------------------------------------- cases
def listed():
    return [
        # One decode step of one GCA sub-layer for a single sequence: norm, q projection, attention over the
        # retrieved chunks, output projection, residual.  The smallest call a server makes; latency counts.
        dict(name="layer_decode_1", op="layer", n=1, chunks=64, rows=1, heads=12, topk=8),
        # The attention alone for a batch of 32 sequences (`bench.py --workload decode`).
        dict(name="decode_32", op="decode", n=32, chunks=1024, rows=1, heads=12, kv_heads=12, topk=8),
        # The sliding-window attention of the same step, the new position stored into the window by the same
        # call (`bench.py --workload window-decode`).
        dict(name="window_decode_32", op="window", n=32, heads=12, window=512),
        # Retrieval at a chunk boundary over a 16M-token context (`bench.py --workload retrieval`).
        dict(name="retrieve_16m", op="scan", n=1, rows=1, entries=262144, dim=768, topk=8, per_head=False),
        # The same with one choice per head, for two sequences whose caches have an odd length.
        dict(name="retrieve_per_head", op="scan", n=2, rows=1, entries=16411, dim=768, topk=8, per_head=True),
        # Retrieval of a training step, noise and gradients into the landmarks included.
        dict(name="retrieve_train_16k", op="retrieve", n=8, chunks=260, dim=768, topk=8, train=True),
        # Chunk K/V projection of a prefill, written into the cache (`bench.py --workload projection`).
        dict(name="append_16k", op="append", n=8, chunks=260, dim=768),
        # The GCA sub-layer over a ragged prefill: 3 prompts of 37 chunks.
        dict(name="layer_prefill_ragged", op="layer", n=3, chunks=37, rows=64, heads=12, topk=8),
        # Drop-in call on chunks gathered beforehand, grouped-query heads, an odd number of query chunks,
        # forward and backward.
        dict(name="attention_gathered", op="gathered", z=109, heads=8, kv_heads=4, topk=5),
        # The float32 configuration (4096 tokens), forward and backward, with the extra softmax logit.
        dict(name="train_fp32", op="train", n=2, chunks=64, heads=12, kv_heads=12, topk=8, dtype="fp32", off_by_one=True,
             token_major=False),
        # GCA of a training step at 16K tokens, called as the sub-layer calls it: q a view of its projection.
        dict(name="train_16k", op="train", n=8, chunks=256, heads=12, kv_heads=12, topk=8, dtype="bf16", off_by_one=False,
             token_major=True),
        # One long sequence (64K tokens) with more retrieved chunks.
        dict(name="train_64k", op="train", n=1, chunks=1024, heads=12, kv_heads=12, topk=16, dtype="bf16", off_by_one=False,
             token_major=False),
    ]


def _log_int(rng, lo, hi):
    """An integer from lo to hi, even over the logarithm."""
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.5))))))


def draw(rng):
    """A case of the same kinds with other sizes: from one sequence to a full batch, from a handful of chunks
    to the longest of the listed contexts, other head counts, grouped-query heads and other top-k."""
    op = rng.choice(["layer_decode", "decode", "window", "scan", "scan", "retrieve", "append", "layer_prefill", "gathered",
                     "train_fp32", "train", "train"])
    heads = rng.choice([4, 6, 8, 12, 16])
    kv_heads = heads // rng.choice([1, 1, 1, 2])
    dim = rng.choice([512, 768, 768, 1024])
    topk = rng.randint(2, 16)
    if op == "layer_decode":                     # two rows: the step that also carries the landmark position
        return dict(op="layer", n=_log_int(rng, 1, 64), chunks=_log_int(rng, 16, 512), rows=rng.choice([1, 1, 2]),
                    heads=rng.choice([8, 12, 16]), topk=topk)
    if op == "decode":
        return dict(op="decode", n=_log_int(rng, 1, 48), chunks=_log_int(rng, 16, 1024), rows=rng.choice([1, 1, 2]), heads=heads,
                    kv_heads=kv_heads, topk=topk)
    if op == "window":
        return dict(op="window", n=_log_int(rng, 1, 48), heads=heads, window=rng.randint(64, 640))
    if op == "scan":
        n = _log_int(rng, 1, 32)
        return dict(op="scan", n=n, rows=1, entries=_log_int(rng, 256, 262144 // n), dim=768, topk=topk,
                    per_head=rng.random() < 0.3)
    if op == "retrieve":
        n = _log_int(rng, 1, 8)
        return dict(op="retrieve", n=n, chunks=_log_int(rng, 16, 2080 // n), dim=dim, topk=topk, train=rng.random() < 0.5)
    if op == "append":                           # one chunk per sequence while decoding, the whole prompt in a prefill
        n = _log_int(rng, 1, 32)
        return dict(op="append", n=n, chunks=_log_int(rng, 1, 2080 // n * 3 // 4), dim=dim)
    if op == "layer_prefill":
        n = _log_int(rng, 1, 8)
        return dict(op="layer", n=n, chunks=_log_int(rng, 6, 1024 // n), rows=64, heads=rng.choice([8, 12]), topk=topk)
    if op == "gathered":
        return dict(op="gathered", z=_log_int(rng, 3, 1000), heads=heads, kv_heads=kv_heads, topk=rng.randint(2, 8))
    if op == "train_fp32":
        n = _log_int(rng, 1, 4)
        heads = rng.choice([4, 6, 8, 12])
        return dict(op="train", n=n, chunks=_log_int(rng, 6, 128 // n), heads=heads, kv_heads=heads // rng.choice([1, 1, 1, 2]),
                    topk=rng.randint(2, 8), dtype="fp32", off_by_one=rng.random() < 0.5, token_major=False)
    n = _log_int(rng, 1, 8)
    most = max(8, min(1024, LARGEST_TRAIN // (n * heads * topk)))
    return dict(op="train", n=n, chunks=_log_int(rng, 8, most), heads=heads, kv_heads=kv_heads, topk=topk, dtype="bf16",
                off_by_one=rng.random() < 0.2, token_major=rng.random() < 0.5)


# ------------------------------------------------------------------------------------------- inputs
def _normal(g, *shape, dtype=torch.bfloat16, std=1.0):
    return torch.empty(*shape, dtype=dtype, device="cuda").normal_(0.0, std, generator=g)


def _with_zero_landmarks(t):
    """The model clears the landmark row of every cached chunk."""
    t[..., -1, :] = 0
    return t


def _causal_ids(g, n, chunks, topk):
    """Query chunk j (1 .. chunks - 1) retrieves up to topk distinct chunks out of 0 .. j - 2, uniformly; the
    slots beyond hold -1 and weight 0.  Returns int32 ids and float32 weights, (n, chunks - 1, topk)."""
    scores = torch.rand(n, chunks - 1, max(topk, chunks), generator=g, device="cuda")
    j = torch.arange(chunks - 1, device="cuda").view(1, -1, 1)
    scores = scores.masked_fill(torch.arange(scores.shape[2], device="cuda").view(1, 1, -1) >= j, -1.0)
    best, ids = scores.topk(topk, dim=2)
    ids = ids.masked_fill(best < 0, -1)
    w = torch.randn(n, chunks - 1, topk, generator=g, device="cuda").masked_fill(ids < 0, float("-inf"))
    return ids.int().contiguous(), torch.nan_to_num(torch.softmax(w, -1), nan=0.0).contiguous()


def _any_ids(g, n, chunks, topk):
    """topk distinct chunks of the whole cache per sequence (what a decode step has retrieved)."""
    topk = min(topk, chunks)
    ids = torch.rand(n, 1, chunks, generator=g, device="cuda").topk(topk, dim=2).indices
    return ids.int().contiguous(), torch.softmax(torch.randn(n, 1, topk, generator=g, device="cuda"), -1)


def _caches(g, n, chunks, width, dtype=torch.bfloat16):
    return [_with_zero_landmarks(_normal(g, n, chunks, CHUNK, width, dtype=dtype)) for _ in range(2)]


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    op, s = case["op"], {"op": case["op"]}
    if op == "layer":
        n, c, rows, dim = case["n"], case["chunks"], case["rows"], case["heads"] * HEAD_DIM
        layer = lcm.TritonGroupCrossAttention(dim, case["heads"], chunk_topk=case["topk"]).to("cuda", torch.bfloat16).eval()
        with torch.no_grad():
            for p in layer.parameters():
                p.copy_(_normal(g, *p.shape, std=dim ** -0.5) if p.dim() == 2 else 1 + _normal(g, *p.shape, std=0.1))
        prefill = rows == CHUNK
        s["layer"] = layer
        s["hidden"] = _normal(g, n, c if prefill else 1, rows, dim)
        s["k"], s["v"] = _caches(g, n, c, dim)
        s["ids"], s["w"] = (_causal_ids if prefill else _any_ids)(g, n, c, case["topk"])
        s["residual"] = s["hidden"].view(n, -1, dim)
    elif op == "decode":
        n, c = case["n"], case["chunks"]
        s["q"] = _normal(g, n, 1, case["heads"], case["rows"], HEAD_DIM)
        s["k"], s["v"] = _caches(g, n, c, case["kv_heads"] * HEAD_DIM)
        s["ids"], s["w"] = _any_ids(g, n, c, case["topk"])
    elif op == "window":
        n, h, t = case["n"], case["heads"], case["window"] + 1
        qkv = _normal(g, n, 3 * h * HEAD_DIM)            # one stacked projection, as the decode step has it
        s["q"], k_new, v_new = (x.view(n, 1, h, HEAD_DIM).transpose(1, 2) for x in qkv.chunk(3, dim=1))
        s["new"] = (k_new, v_new)
        s["k"], s["v"] = _normal(g, n, h, t, HEAD_DIM), _normal(g, n, h, t, HEAD_DIM)
        s["count"] = torch.full((1,), 1000 + seed % 1000, dtype=torch.int64, device="cuda")
        s["slopes"] = torch.tensor([2.0 ** (-8.0 * (i + 1) / h) for i in range(h)], device="cuda")
        s["window"] = case["window"]
    elif op == "scan":
        n, e, d = case["n"], case["entries"], case["dim"]
        s["q"], s["lmk"] = _normal(g, n, case["rows"], d, std=0.125), _normal(g, n, e, d, std=0.125)
        s["topk"], s["head_dim"] = case["topk"], HEAD_DIM if case["per_head"] else 0
    elif op == "retrieve":
        n, c, d, train = case["n"], case["chunks"], case["dim"], case["train"]
        s["q"], s["lmk"] = (_normal(g, n, c, d, std=0.5).requires_grad_(train) for _ in range(2))
        s["chunks"] = lcm.ChunkKVManager(zero_landmark=True)
        kv = torch.zeros(n, c, CHUNK, HEAD_DIM, dtype=torch.bfloat16, device="cuda")     # retrieval reads landmarks only
        s["chunks"].append(kv, kv, s["lmk"])
        s["topk"], s["train"], s["noise"] = min(case["topk"], c), train, None
        if train:
            s["noise"] = -torch.empty(n, c, c, device="cuda").exponential_(generator=g).log()
            s["dw"] = _normal(g, n, c - 1, s["topk"], dtype=torch.float32)
    elif op == "append":
        n, c, d = case["n"], case["chunks"], case["dim"]
        s["hidden"] = _normal(g, n, c, CHUNK, d)
        s["wk"], s["wv"] = _normal(g, d, d, std=d ** -0.5), _normal(g, d, d, std=d ** -0.5)
        s["capacity"] = c
    elif op == "gathered":
        z, h, hkv, k = case["z"], case["heads"], case["kv_heads"], case["topk"]
        s["q"] = _normal(g, z, h, CHUNK, HEAD_DIM).requires_grad_()
        s["k"], s["v"] = (_with_zero_landmarks(_normal(g, z, hkv, k, CHUNK, HEAD_DIM)).requires_grad_() for _ in range(2))
        s["w"] = torch.softmax(_normal(g, z, k, dtype=torch.float32), -1).requires_grad_()
        s["dout"] = _normal(g, z, h, CHUNK, HEAD_DIM)
    elif op == "train":
        n, c, h, dtype = case["n"], case["chunks"], case["heads"], DTYPE[case["dtype"]]
        s["token_major"], s["off_by_one"] = case["token_major"], case["off_by_one"]
        if s["token_major"]:                             # views of the projection's output and of its gradient
            q, dout = (_normal(g, n, c, CHUNK, h, HEAD_DIM, dtype=dtype).permute(0, 1, 3, 2, 4)[:, 1:] for _ in range(2))
        else:
            q, dout = (_normal(g, n, c - 1, h, CHUNK, HEAD_DIM, dtype=dtype) for _ in range(2))
        s["q"], s["dout"] = q.requires_grad_(), dout
        s["k"], s["v"] = (t.requires_grad_() for t in _caches(g, n, c, case["kv_heads"] * HEAD_DIM, dtype))
        s["ids"], w = _causal_ids(g, n, c, case["topk"])
        s["w"] = w.requires_grad_()
    return s


# --------------------------------------------------------------------------------------------- a pass
def run(s):
    op = s["op"]
    if op == "train":
        o = lcm.gca_indexed(s["q"], s["k"], s["v"], s["ids"], s["w"], SCALE, softmax_off_by_one=s["off_by_one"],
                            token_major_out=s["token_major"])
        return (o, *torch.autograd.grad(o, (s["q"], s["k"], s["v"], s["w"]), s["dout"]))
    if op == "gathered":
        o = lcm.attention(s["q"], s["k"], s["v"], s["w"], SCALE)
        return (o, *torch.autograd.grad(o, (s["q"], s["k"], s["v"], s["w"]), s["dout"]))
    if op == "retrieve":
        ids, w, full = lcm.retrieve(s["q"], s["chunks"], s["topk"], training=s["train"], noise=s["noise"])
        if not s["train"]:
            return ids, w, full.scores, full.n_valid
        return (ids, w, *torch.autograd.grad(w, (s["q"], s["lmk"]), s["dw"]))
    with torch.no_grad():
        if op == "layer":
            return s["layer"].forward_fused(s["hidden"], s["k"], s["v"], s["ids"], s["w"], residual=s["residual"])
        if op == "decode":
            return lcm.gca_indexed_nograd(s["q"], s["k"], s["v"], s["ids"], s["w"], SCALE)
        if op == "window":
            out = fused_ops.window_ring_decode(s["q"], s["k"], s["v"], *s["new"], s["count"], s["window"], s["slopes"], SCALE)
            s["count"] += 1
            return out, s["k"], s["v"]
        if op == "scan":
            return tuple(lcm.lmk_score_topk(s["q"], s["lmk"], s["topk"], q_pos0=s["lmk"].shape[1], head_dim=s["head_dim"]))
        if op == "append":
            cache = lcm.ChunkKVManager(zero_landmark=True, capacity=s["capacity"])
            cache.append_projected(s["hidden"], s["wk"], s["wv"])
            return cache.chunk_k, cache.chunk_v, cache.past_lmk_embeds
    raise ValueError(op)


# ------------------------------------------------------------------------------- what a pass has to do
def _slots(chunks, topk):
    """Retrieved chunks of one sequence and head: query chunk j has j - 1 to choose from."""
    return sum(min(topk, j - 1) for j in range(1, chunks))


def work(case):
    op = case["op"]
    tile = CHUNK * HEAD_DIM * ESIZE[case.get("dtype", "bf16")]       # one chunk of one head
    if op == "layer":
        n, rows, h, k, dim = case["n"], case["rows"], case["heads"], case["topk"], case["heads"] * HEAD_DIM
        if rows == CHUNK:
            c = case["chunks"]
            tokens, slots = n * c * rows, n * h * _slots(c, k)
            return {"bytes": 3 * tokens * dim * 2 + 2 * dim * dim * 2 + 2 * n * c * h * tile,
                    "flops": slots * SLOT_FLOPS + 2 * 2 * n * (c - 1) * rows * dim * dim}
        k = min(k, case["chunks"])
        return {"bytes": 3 * n * rows * dim * 2 + 2 * dim * dim * 2 + 2 * n * k * h * tile,
                "flops": n * rows * (h * k * 4 * CHUNK * HEAD_DIM + 2 * 2 * dim * dim)}
    if op == "decode":
        n, k, rows = case["n"], min(case["topk"], case["chunks"]), case["rows"]
        return {"bytes": 2 * n * k * case["kv_heads"] * tile + 2 * n * case["heads"] * rows * HEAD_DIM * 2,
                "flops": n * rows * case["heads"] * k * 4 * CHUNK * HEAD_DIM}
    if op == "window":
        n, h, t = case["n"], case["heads"], case["window"] + 1
        return {"bytes": 2 * n * h * (t + 1) * HEAD_DIM * 2 + 2 * n * h * HEAD_DIM * 2, "flops": n * h * t * 4 * HEAD_DIM}
    if op == "scan":
        n, e, d = case["n"], case["entries"], case["dim"]
        return {"bytes": n * e * d * 2, "flops": 2 * n * case["rows"] * e * d}
    if op == "retrieve":
        n, c, d = case["n"], case["chunks"], case["dim"]
        pairs = n * c * (c - 1) // 2
        landmarks = 2 * n * c * d * 2
        return {"bytes": landmarks * (2 if case["train"] else 1) + (4 * pairs if case["train"] else 0),
                "flops": 2 * pairs * d + (3 * 2 * n * c * min(case["topk"], c) * d if case["train"] else 0)}
    if op == "append":
        rows, d = case["n"] * case["chunks"] * CHUNK, case["dim"]
        return {"bytes": 3 * rows * d * 2 + 2 * d * d * 2, "flops": 2 * 2 * rows * d * d}
    if op == "gathered":
        z, h, hkv, k = case["z"], case["heads"], case["kv_heads"], case["topk"]
        return {"bytes": 4 * z * h * tile + 4 * z * hkv * k * tile, "flops": 3.5 * z * h * k * SLOT_FLOPS}
    n, c, h, hkv = case["n"], case["chunks"], case["heads"], case["kv_heads"]
    return {"bytes": 4 * n * (c - 1) * h * tile + 4 * n * c * hkv * tile, "flops": 3.5 * n * h * _slots(c, case["topk"]) * SLOT_FLOPS}


def tolerance(case):
    """float32 sums for the scan (ids and packed keys are whole numbers and have to be the same) and for the
    float32 GCA; bf16 results, or weights and gradients computed from bf16 scores, elsewhere."""
    if case["op"] == "scan" or (case["op"] == "retrieve" and not case["train"]):
        return {"rel": 1e-5}
    if case.get("dtype") == "fp32":
        return {"rel": 2e-5}
    return {"rel": 1e-2}
