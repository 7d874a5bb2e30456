"""Cases by which the speed of the hot path is judged.

A case is one pass of block-sparse attention as a program runs it through the public API of
flash_topk_attn_v2.  Its "path" is one of

  train    flash_topk_score -> build_qblock_topk_indices -> flash_topk_attn -> backward
  prefill  the same forward, without gradients
  lists    flash_topk_score -> build_qblock_topk_indices only
  attend   flash_topk_attn -> backward over block lists that the program made by its own rule
           (a first block that everybody reads, a local window and some far blocks)

The other keys: B, N, H, Hkv (kv heads, other than H only where the lists are given), D, dtype,
block (score block = kv block), g (q block), topk, threshold, width (qblock_topk; 0: the default
g * topk; in "attend": length of the lists), pad_head / q_pad_head (virtual rows before token 0
of the key and query grids; the tail completes the last block) and hot (score blocks per head
with a shared direction added to their keys, which skews the scores).
"""

import os
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "flash-topk-attention_b200"))

from flash_topk_attn_v2 import (  # noqa: E402
    build_qblock_topk_indices, flash_topk_attn, flash_topk_score)

_DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16, "fp32": torch.float32}


def _case(**kw):
    c = dict(path="train", B=1, N=1024, H=8, Hkv=0, D=128, dtype="bf16", block=64, g=64, topk=16,
             threshold=1.0, width=0, pad_head=0, q_pad_head=0, hot=0, scale=1.0)
    c.update(kw)
    c["Hkv"] = c["Hkv"] or c["H"]
    return c


def listed():
    return [
        # the smallest call of the test suite: a unit test or a toy model, all latency
        _case(name="train tiny", N=256, H=2, D=64, dtype="fp16", g=32, topk=3, threshold=0.9),
        # the small correctness shape that the project quotes: a short-context model
        _case(name="train small", B=2, N=1024, H=8, D=64, dtype="fp16", g=32),
        # one user's prompt of odd length, forward only
        _case(name="prefill ragged", path="prefill", N=2000, H=16, topk=8, pad_head=20,
              q_pad_head=24),
        # float32 activations with a head dim that is padded (computed in bf16)
        _case(name="train fp32 d96", N=3000, H=12, D=96, dtype="fp32", pad_head=8),
        # grouped kv heads, short lists by a fixed rule: a fine-tuning step of a long-context model
        _case(name="attend grouped", path="attend", B=2, N=4096, H=32, Hkv=8, width=16),
        # ordinary training shapes, at each of the kernels' three head dims
        _case(name="train d64", N=8192, H=16, D=64, topk=32, threshold=0.9, scale=0.5),
        _case(name="train d128 batch", B=4, N=8192, H=16, width=256),
        _case(name="train d256", N=8192, H=16, D=256, topk=32, threshold=0.9, scale=0.5),
        # 128-row blocks, virtual padding, skewed scores: forward of a long odd-length document,
        # and the selection alone at the size the project quotes
        _case(name="prefill 128-row blocks", path="prefill", N=15000, H=16, dtype="fp16",
              block=128, g=128, topk=24, threshold=0.8, pad_head=40, q_pad_head=40, hot=8),
        _case(name="lists 128-row blocks", path="lists", B=2, N=30000, H=32, dtype="fp16",
              block=128, g=128, topk=24, threshold=0.8, pad_head=40, q_pad_head=40, hot=8,
              scale=1.0),
        # long context with the lists capped, so that attention is sparse in earnest
        _case(name="train long capped", N=65536, H=4, topk=64, width=128, hot=32),
        # the headline workload
        _case(name="train headline", N=32768, H=32, topk=32, threshold=0.9, scale=0.5),
    ]


def draw(rng):
    """One more case: lengths log-uniform from 256 to 65536 and mostly not multiples of a block."""
    while True:
        path = rng.choice(["train", "train", "train", "prefill", "prefill", "lists", "attend"])
        block = rng.choice([32, 64, 64, 64, 64, 128])
        g = rng.choice([32, 64, 64, 64, 128])
        n = int(round(256 * 256 ** rng.random()))
        if rng.random() < 0.3:
            n = -(-n // 128) * 128
        heads = rng.choice([1, 2, 4, 8, 12, 16, 32])
        c = _case(path=path, B=rng.choice([1, 1, 1, 2, 4]), N=n, H=heads,
                  D=rng.choice([64, 64, 128, 128, 128, 128, 96, 256]),
                  dtype=rng.choice(["bf16", "bf16", "bf16", "fp16", "fp16", "fp32"]),
                  block=block, g=g, threshold=rng.choice([1.0, 0.9, 0.8]),
                  scale=rng.choice([0.5, 1.0]))
        aligned = n % 128 == 0
        c["pad_head"] = 0 if aligned or rng.random() < 0.5 else rng.randrange(block)
        c["q_pad_head"] = 0 if aligned or rng.random() < 0.5 else rng.randrange(g)
        m = _grid(c["N"], c["block"], c["pad_head"])[0]
        c["topk"] = min(rng.choice([8, 16, 24, 32, 64]), m)
        c["width"] = rng.choice([0, 0, max(1, min(m, c["topk"] * rng.choice([2, 4])))])
        c["hot"] = rng.choice([0, 8]) if m >= 32 else 0
        if path == "attend":
            c["width"] = max(1, min(m, rng.choice([8, 16, 32, 64])))
            c["Hkv"] = heads // rng.choice([1, 2, 4]) if heads % 4 == 0 else heads
            c["hot"] = 0
        if g * c["topk"] > 4096:
            continue
        # small blocks and the largest head dim run further from the tensor peak
        dear = (4 if c["D"] == 256 else 1) * (2 if min(block, g) < 64 else 1)
        if work(c)["flops"] * dear <= 0.5 * work(_HEADLINE)["flops"]:
            return c


def _grid(n, block, head):
    """(blocks, tail) of a grid whose first `head` rows and last `tail` rows are virtual."""
    blocks = -(-(head + n) // block)
    return blocks, blocks * block - head - n


def _rand(shape, gen, dtype, scale=1.0):
    return (torch.randn(shape, generator=gen, device="cuda") * scale).to(dtype)


def prepare(case, seed):
    """Activations as the projections of a layer leave them, [B, N, heads * D], and what a program
    keeps beside them: its settings, the gradient that comes back from the next layer and, where
    it makes its own, the block lists."""
    c = case
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dt = _DTYPES[c["dtype"]]
    B, N, H, Hkv, D = c["B"], c["N"], c["H"], c["Hkv"], c["D"]
    M, kv_tail = _grid(N, c["block"], c["pad_head"])
    QM, q_tail = _grid(N, c["g"], c["q_pad_head"])
    q = _rand((B, N, H * D), gen, dt, c["scale"])
    k = _rand((B, N, Hkv * D), gen, dt, c["scale"])
    if c["hot"]:
        # keys of some blocks of every head lean towards one direction
        u = torch.randn(D, generator=gen, device="cuda")
        rank = torch.rand(B, M, Hkv, generator=gen, device="cuda").argsort(1).argsort(1)
        block_of = (torch.arange(N, device="cuda") + c["pad_head"]) // c["block"]
        lean = (rank < c["hot"]).index_select(1, block_of).to(dt).unsqueeze(-1)
        k = (k.view(B, N, Hkv, D) + lean * (2.0 * u).to(dt)).view(B, N, Hkv * D)
    s = dict(case=c, q=q, k=k, pad=(c["pad_head"], kv_tail), q_pad=(c["q_pad_head"], q_tail))
    if c["path"] != "lists":
        s["v"] = _rand((B, N, Hkv * D), gen, dt)
    if c["path"] in ("train", "attend"):
        s["do"] = _rand((B, N, H * D), gen, dt)
        for name in "qkv":
            s[name].requires_grad_(True)
    if c["path"] == "attend":
        W = c["width"]
        key = torch.rand(B, H, QM, M, generator=gen, device="cuda")
        kv = torch.arange(M, device="cuda")
        own = (torch.arange(QM, device="cuda") * M // QM).unsqueeze(1)
        key += 2.0 * ((kv == 0) | ((kv - own).abs() <= W // 4))
        s["merged"] = key.topk(W, dim=-1).indices.to(torch.int32)
        s["counts"] = torch.full((B, H, QM), W, dtype=torch.int32, device="cuda")
    return s


def run(state):
    s, c = state, state["case"]
    q, k = s["q"], s["k"]
    if c["path"] == "attend":
        merged, counts = s["merged"], s["counts"]
        out = []
    else:
        idx, raw, avg = flash_topk_score(
            q.detach(), k.detach(), c["H"], c["block"], c["topk"], s["pad"], c["threshold"])
        merged, counts, _ = build_qblock_topk_indices(
            idx, c["g"], s["q_pad"], avg, c["width"] or None)
        out = [idx, raw, avg, merged, counts]
    if c["path"] == "lists":
        return out
    o, lse = flash_topk_attn(q, k, s["v"], merged, counts, c["H"], c["g"], c["block"],
                             num_kv_heads=c["Hkv"], kv_padding=s["pad"], q_padding=s["q_pad"])
    out += [o, lse]
    if c["path"] != "prefill":
        out += torch.autograd.grad(o, (q, k, s["v"]), s["do"])
    return out


def work(case):
    c = case
    B, N, H, D = c["B"], c["N"], c["H"], c["D"]
    size = 4 if c["dtype"] == "fp32" else 2
    M, QM = _grid(N, c["block"], c["pad_head"])[0], _grid(N, c["g"], c["q_pad_head"])[0]
    K = min(c["topk"], M)
    q_bytes, kv_bytes = B * N * H * D * size, B * N * c["Hkv"] * D * size
    W = c["width"] or c["g"] * c["topk"]
    nbytes, flops = q_bytes + kv_bytes, 0.0
    if c["path"] == "attend":
        per_block = W
        nbytes += 4 * B * H * QM * W
    else:
        flops += 2.0 * B * H * N * N * D
        nbytes += 12 * B * H * N * K + 4 * B * H * QM * (W + 1)
        # distinct blocks among the picks of a q-block's rows when these pick independently
        per_block = min(W, M, M * (1.0 - (1.0 - K / M) ** c["g"]) if K < M else M)
    if c["path"] != "lists":
        # a product over all listed (query, key) pairs: two forward, five more backward
        product = 2.0 * D * B * H * N * min(N, per_block * c["block"])
        nbytes += kv_bytes + q_bytes + 4 * B * H * N
        flops += 2 * product
        if c["path"] != "prefill":
            nbytes += 2 * q_bytes + 2 * kv_bytes
            flops += 5 * product
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """Relative error of the probabilities and their gradients, which are rounded to 16 bits
    between the products (float32 inputs are computed in bfloat16), and of outputs in that type.
    Block scores are sums in float32: two blocks whose scores tie to the last bits may change
    places, and where the two stand at a cut (the topk, the threshold, the width) another block is
    listed.  That is rare, so it shows in no norm, but it moves single values by their own size."""
    rel = 2e-3 if case["dtype"] == "fp16" else 1e-2
    if case["path"] == "attend":
        return {"rel": rel, "max": 50 * rel}
    return {"rel": rel, "max": 0.9, "differ": 2e-3}


_HEADLINE = listed()[-1]
