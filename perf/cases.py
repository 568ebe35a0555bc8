"""Performance cases of the Video Sparse Attention operator.

A case is one call that a program makes through the public entry points of ``simple_vsa_b200``:

* ``vsa``: ``video_sparse_attn`` on tile-order ``[batch, heads, tokens, head_dim]`` tensors;
* ``routes``: ``b200_sparse_attention``, the fine branch alone on a routing table the caller brings;
* ``raster``: ``video_sparse_attn_raster`` on raster-order ``[batch, tokens, heads, head_dim]`` activations.

``train`` cases run forward and backward and return the output with every gradient, the others are forward passes
without autograd (sampling).  Inputs are N(0,1) as in the operator's benchmarks, gates are sigmoid(N(0,1)), ragged
blocks have their padded rows zeroed, routing tables are drawn without replacement.
"""

from __future__ import annotations

import math

import torch

import simple_vsa_b200 as vsa

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
ELEMENT = {"bf16": 2, "fp16": 2, "fp32": 4}
BLOCKS = {64: (4, 4, 4), 128: (4, 4, 8), 256: (4, 8, 8)}
LARGEST_USEFUL_FLOPS = 14.0 * 80 * 92160 * 180 * 64 * 128      # the largest listed case


def _case(name, op, dtype, batch, heads, tokens, dim, block, topk, **more):
    c = dict(name=name, op=op, dtype=dtype, batch=batch, heads=heads, tokens=tokens, dim=dim, block=block, topk=topk,
             gate=False, ragged=0.0, train=True)
    c.update(more)
    return c


def listed():
    return [
        # the smallest configuration of the benchmark: fp32 numerics check, every launch counts
        _case("train_1k_fp32_d64", "vsa", "fp32", 1, 2, 1024, 64, 64, 4),
        # one denoising step's layer on a thumbnail-sized latent: latency of a sampling call
        _case("infer_4k", "vsa", "bf16", 1, 12, 4096, 128, 64, 8, gate=True, train=False),
        # a short training clip with few heads (a head-sharded rank)
        _case("train_8k", "vsa", "bf16", 1, 8, 8192, 128, 64, 16),
        # the 16k-token training configuration with the learned gate
        _case("train_16k_gate", "vsa", "bf16", 1, 12, 16384, 128, 64, 32, gate=True),
        # the same at head dim 64
        _case("train_16k_d64_gate", "vsa", "bf16", 1, 12, 16384, 64, 64, 32, gate=True),
        # sampling at the middle token count of the benchmarks, 87.5 % sparsity
        _case("infer_40k", "vsa", "bf16", 1, 12, 39936, 128, 64, 78, train=False),
        # large blocks of which a tenth are clipped at the latent's border
        _case("train_40k_block256_ragged", "vsa", "bf16", 1, 40, 40960, 128, 256, 20, ragged=0.1),
        # one eight-head shard of the 92k-token shape, fp16 training
        _case("train_92k_h8_fp16_gate", "vsa", "fp16", 1, 8, 92160, 128, 64, 180, gate=True),
        # the same token count with blocks of 128 tokens
        _case("train_92k_h8_block128_gate", "vsa", "bf16", 1, 8, 92160, 128, 128, 90, gate=True),
        # a transformer layer that keeps raster-order activations; tiles clipped on two axes, 1380 of them
        _case("train_raster_81k", "raster", "bf16", 1, 8, 81000, 128, 64, 172, gate=True, grid_t=20, grid_h=45,
              grid_w=90),
        # the executor alone on skewed routes of the caller
        _case("train_92k_routes_zipf", "routes", "bf16", 1, 40, 92160, 128, 64, 180, zipf=1.1),
        # the headline shape: two samples, forty heads, 92k tokens
        _case("train_92k", "vsa", "bf16", 2, 40, 92160, 128, 64, 180),
    ]


def _log_uniform(rng, low, high):
    return math.exp(rng.uniform(math.log(low), math.log(high)))


def draw(rng):
    """One more case: token counts, heads, sparsity, block volume, head dim, type, direction and entry point vary."""
    while True:
        op = rng.choice(("vsa", "vsa", "vsa", "vsa", "raster", "routes"))
        dtype = rng.choice(("bf16", "bf16", "bf16", "fp16", "fp16", "fp32")) if op == "vsa" else rng.choice(("bf16", "fp16"))
        block = rng.choice((64, 64, 64, 128, 256))
        dim = 128 if op == "raster" else rng.choice((128, 128, 128, 64))
        if dtype == "fp32":
            # the numerics mode: small problems only
            tokens, heads, batch, block, dim = _log_uniform(rng, 512, 4096), rng.randint(1, 8), 1, 64, rng.choice((64, 128))
        else:
            tokens, heads, batch = _log_uniform(rng, 2048, 100000), round(_log_uniform(rng, 1, 40)), rng.choice((1, 1, 1, 2))
        more = {}
        if op == "raster":
            tile = BLOCKS[block]
            t, h = rng.randint(4, 24), rng.randint(12, 60)
            w = min(160, max(8, round(tokens / (t * h))))
            tokens, more = t * h * w, dict(grid_t=t, grid_h=h, grid_w=w)
            blocks = math.prod(-(-n // s) for n, s in zip((t, h, w), tile))
        else:
            blocks = max(8, round(tokens / block))
            tokens = blocks * block
        topk = max(1, round(blocks * rng.choice((0.0625, 0.1, 0.125, 0.125, 0.2))))
        if op == "routes":
            more["zipf"] = rng.choice((0.0, 1.1))
        c = _case("", op, dtype, batch, heads, tokens, dim, block, topk, gate=op != "routes" and rng.random() < 0.5,
                  ragged=rng.choice((0.0, 0.0, 0.1, 0.3)) if op != "raster" else 0.0, train=rng.random() < 0.65, **more)
        del c["name"]
        # head dim 64 and 128 are priced alike: the narrow heads are no cheaper per token pair in softmax work
        if 14.0 * batch * heads * blocks * block * topk * block * 128 <= 0.5 * LARGEST_USEFUL_FLOPS:
            return c


def _normal(shape, dtype, gen):
    return torch.empty(shape, device="cuda", dtype=dtype).normal_(generator=gen)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    B, H, L, D, be = case["batch"], case["heads"], case["tokens"], case["dim"], case["block"]
    dtype = DTYPES[case["dtype"]]
    state = {"case": case}
    shape = (B, L, H, D) if case["op"] == "raster" else (B, H, L, D)
    names = ["q", "k", "v"] + (["gate"] if case["gate"] else [])
    tensors = {n: _normal(shape, dtype, gen) for n in names}
    if case["gate"]:
        tensors["gate"].sigmoid_()
    if case["op"] == "raster":
        state["meta"] = vsa.build_vsa_metadata((case["grid_t"], case["grid_h"], case["grid_w"]), BLOCKS[be], "cuda")
    else:
        blocks = L // be
        sizes = torch.full((blocks,), be, device="cuda", dtype=torch.int32)
        if case["ragged"] > 0:
            clipped = torch.rand(blocks, device="cuda", generator=gen) < case["ragged"]
            smaller = torch.randint(1, be, (blocks,), device="cuda", generator=gen, dtype=torch.int32)
            sizes = torch.where(clipped, smaller, sizes)
            padded = (torch.arange(be, device="cuda")[None, :] >= sizes[:, None]).view(1, 1, L, 1)
            for n in ("q", "k", "v"):
                tensors[n].masked_fill_(padded, 0)
        state["sizes"] = sizes
    if case["op"] == "routes":
        # without replacement from a Zipf(s) distribution over the key blocks (s = 0: uniform): Gumbel Top-K
        blocks = L // be
        weight = -case["zipf"] * torch.log(torch.arange(1, blocks + 1, device="cuda", dtype=torch.float32))
        state["routes"] = torch.empty((B, H, blocks, case["topk"]), device="cuda", dtype=torch.int32)
        for b in range(B):
            for h in range(H):
                u = torch.rand((blocks, blocks), device="cuda", generator=gen).clamp_(1e-12, 1 - 1e-7)
                gumbel = -torch.log(-torch.log(u))
                state["routes"][b, h] = torch.topk(gumbel + weight, case["topk"], dim=-1).indices.to(torch.int32)
    if case["train"]:
        state["dout"] = _normal(shape, dtype, gen)
        for t in tensors.values():
            t.requires_grad_()
    state["tensors"] = tensors
    return state


def _forward(state):
    case, t = state["case"], state["tensors"]
    if case["op"] == "raster":
        return vsa.video_sparse_attn_raster(t["q"], t["k"], t["v"], state["meta"], case["topk"], t.get("gate"))
    if case["op"] == "routes":
        return vsa.b200_sparse_attention(t["q"], t["k"], t["v"], state["routes"], state["sizes"],
                                         block_size=BLOCKS[case["block"]])
    return vsa.video_sparse_attn(t["q"], t["k"], t["v"], state["sizes"], state["sizes"], case["topk"],
                                 BLOCKS[case["block"]], t.get("gate"))


def run(state):
    if not state["case"]["train"]:
        with torch.no_grad():
            return {"out": _forward(state)}
    out = _forward(state)
    leaves = state["tensors"]
    grads = torch.autograd.grad(out, list(leaves.values()), state["dout"])
    return {"out": out.detach(), **{"d" + n: g for n, g in zip(leaves, grads)}}


def work(case):
    """Each operand read once, each result written once; 4 products' worth of flops per query-key pair forward (two
    matrix products), 10 backward (five), over the tokens that are not padding, plus the pooled branch."""
    B, H, L, D, be = case["batch"], case["heads"], case["tokens"], case["dim"], case["block"]
    passes = 14.0 if case["train"] else 4.0
    tensor = float(B * H * L * D * ELEMENT[case["dtype"]])
    full = 1.0 - 0.5 * case["ragged"]
    if case["op"] == "raster":
        blocks = math.prod(-(-case[n] // s) for n, s in zip(("grid_t", "grid_h", "grid_w"), BLOCKS[be]))
        full = L / (blocks * be)
        pairs = B * H * L * case["topk"] * be * full
    else:
        blocks = L // be
        pairs = B * H * L * full * case["topk"] * be * full
    flops = passes * pairs * D
    if case["op"] != "routes":
        flops += (12.0 if case["train"] else 4.0) * B * H * blocks * blocks * D
    # q, k, v, out (and gate); backward: dout, dq, dk, dv (and dgate)
    moved = 4 + case["gate"] + ((4 + case["gate"]) if case["train"] else 0)
    extra = 4.0 * B * H * blocks * case["topk"] if case["op"] == "routes" else 0.0
    return {"bytes": moved * tensor + extra, "flops": flops}


def tolerance(case):
    """Largest relative error of another correct implementation at the same precision.

    16-bit types: results are rounded to 16 bits, and so are the probabilities and score gradients between the two
    products of each pass.  Measured against float64 on the same routes: 2.2e-3 to 3.4e-3 in bf16 (largest difference
    2.6e-2 of the root mean square), 3.5e-4 to 4.3e-4 in fp16, below 4e-7 in fp32; about four times that, and in fp32
    room for sums in another order."""
    return {"bf16": {"rel": 1e-2, "max": 0.1}, "fp16": {"rel": 2e-3, "max": 2e-2},
            "fp32": {"rel": 5e-6, "max": 1e-4}}[case["dtype"]]


def _tiles(case):
    """Raster index of every tile-order token of the (T, H, W) grid, -1 for padding, and the tiles' sizes: tiles in
    raster order, the tokens of a clipped tile packed to its front."""
    (T, H, W), (a, b, c) = [case[n] for n in ("grid_t", "grid_h", "grid_w")], BLOCKS[case["block"]]
    ids = torch.arange(T * H * W, device="cuda").view(T, H, W)
    rows, sizes = [], []
    for t in range(0, T, a):
        for h in range(0, H, b):
            for w in range(0, W, c):
                live = ids[t:t + a, h:h + b, w:w + c].reshape(-1)
                rows.append(torch.nn.functional.pad(live, (0, case["block"] - live.numel()), value=-1))
                sizes.append(live.numel())
    return torch.stack(rows).view(-1), torch.tensor(sizes, device="cuda")


def _exact_slice(case, x, sizes, routes):
    """One (batch, head) slice in float64.  ``x``: q, k, v (and gate, dout) ``[tokens, dim]`` in tile order."""
    be, D, dtype = case["block"], case["dim"], DTYPES[case["dtype"]]
    x = {n: t.double() for n, t in x.items()}
    blocks, scale = sizes.numel(), 1.0 / math.sqrt(D)
    live = torch.arange(be, device="cuda")[None, :] < sizes[:, None]
    blocked = {n: t.reshape(blocks, be, D) for n, t in x.items()}
    grads, pooled, share = {}, case["op"] != "routes", None
    if pooled:
        share = live.double() / sizes.clamp(min=1)[:, None]
        qc, kc, vc = ((blocked[n] * share[..., None]).sum(1) for n in "qkv")
        # the routes are those of scores in the operator's own type (rounded after the product and after the scale),
        # equal scores to the lower block
        rounded = ((qc.to(dtype).double() @ kc.to(dtype).double().T).to(dtype).double() * scale).to(dtype)
        routes = rounded.float().sort(dim=-1, descending=True, stable=True).indices[:, :case["topk"]]
        probs = (qc @ kc.T * scale).softmax(-1)
        out_c = probs @ vc
    out, dq, dk, dv = (torch.zeros_like(blocked["q"]) for _ in range(4))
    step = max(1, int(3e8 / (case["topk"] * be * D * 8)))
    for at in range(0, blocks, step):
        sel = routes[at:at + step].long()
        q, n = blocked["q"][at:at + step], sel.shape[0]
        k, v = (blocked[m][sel].reshape(n, -1, D) for m in "kv")
        s = (q @ k.transpose(1, 2) * scale).masked_fill_(~live[sel].reshape(n, 1, -1), -math.inf)
        p = s.softmax(-1)
        out[at:at + step] = o = p @ v
        if case["train"]:
            do = blocked["dout"][at:at + step]
            ds = p * (do @ v.transpose(1, 2) - (do * o).sum(-1, keepdim=True)) * scale
            dq[at:at + step] = ds @ k
            dk.index_add_(0, sel.reshape(-1), (ds.transpose(1, 2) @ q).reshape(-1, be, D))
            dv.index_add_(0, sel.reshape(-1), (p.transpose(1, 2) @ do).reshape(-1, be, D))
    if pooled:
        gate = blocked.get("gate", torch.ones((), device="cuda", dtype=torch.float64))
        out = out + out_c[:, None] * gate
        if case["train"]:
            do_c = (blocked["dout"] * gate).sum(1)
            ds = probs * (do_c @ vc.T - (do_c * out_c).sum(-1, keepdim=True)) * scale
            dq += (ds @ kc)[:, None] * share[..., None]
            dk += (ds.T @ qc)[:, None] * share[..., None]
            dv += (probs.T @ do_c)[:, None] * share[..., None]
            if case["gate"]:
                grads["dgate"] = blocked["dout"] * out_c[:, None]
    if case["train"]:
        grads.update(dq=dq, dk=dk, dv=dv)
    return {"out": out.reshape(-1, D), **{n: g.reshape(-1, D) for n, g in grads.items()}}


def exact(case, seed):
    """``run``'s outputs in float64, slice by slice; the two largest shapes would take too long."""
    if work(case)["flops"] > 2.5e13:
        return None
    state = prepare(case, seed)
    tensors = {n: t.detach() for n, t in state["tensors"].items()}
    if case["train"]:
        tensors["dout"] = state["dout"]
    raster = case["op"] == "raster"
    if raster:
        rows, sizes = _tiles(case)
    else:
        sizes = state["sizes"]
    names = ["out"] + (["dq", "dk", "dv"] + ["dgate"] * case["gate"] if case["train"] else [])
    result = {n: torch.zeros(tensors["q"].shape, device="cuda", dtype=torch.float64) for n in names}
    for b in range(case["batch"]):
        for h in range(case["heads"]):
            if raster:
                x = {n: t[b, :, h][rows.clamp(min=0)].masked_fill_((rows < 0)[:, None], 0) for n, t in tensors.items()}
            else:
                x = {n: t[b, h] for n, t in tensors.items()}
            got = _exact_slice(case, x, sizes, state["routes"][b, h] if case["op"] == "routes" else None)
            for n, t in got.items():
                if raster:
                    result[n][b, rows[rows >= 0], h] = t[rows >= 0]
                else:
                    result[n][b, h] = t
    return result
