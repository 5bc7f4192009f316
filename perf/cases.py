"""The workloads whose speed is kept track of: what a serving engine has this library do, through its public calls.

Four kinds of case, all at the benchmark's layer shapes (hidden 2048, 256 NVFP4 experts of intermediate 512, top-8, one
bf16 shared expert of 512):

* "blocks": one engine step through `layers` MoE blocks of `tokens` rows each.  An engine calls one block per layer with
  attention in between, so every layer has rows, weights and banks of its own, and a layer's weights have left L2 by the
  time they are read again.  `norm` = the call that also does the residual add and the norm in front of the block;
  `graph` = the step is captured in a CUDA graph once and replayed, as decode loops do; `zipf` > 0 = popularity of the
  experts skewed by a Zipf bias in the router; `out` = the dtype of the block's result.
* "staged": the port for engines that keep their own router: `CachedExperts.execute_device` on the router's ids and
  weights, `x` / `ids` / `out` = the dtypes it hands over.
* "lm_head": the dense NVFP4 matrix-vector product of the vocabulary projection, `m` sequences at a time.
* "host": `run_experts`, the hand-off of host arrays (plan in the slot cache, upload, experts, download).

Every input is drawn from the case's seed, on the GPU where it is large.
"""
import importlib

import numpy as np
import torch

ft = importlib.import_module("ferrum-torrens_b200")

HIDDEN, INTER, EXPERTS, TOP_K, SHARED = 2048, 512, 256, 8, 512
EXPERT_BYTES = 2 * INTER * HIDDEN // 2 + 2 * INTER * HIDDEN // 16 + 4 * INTER + HIDDEN * INTER // 2 + HIDDEN * INTER // 16 + 2 * HIDDEN
DENSE_BYTES = 2 * (EXPERTS * HIDDEN + 2 * SHARED * HIDDEN + HIDDEN * SHARED + HIDDEN)   # router and shared expert
EPS = 1e-6
# f16 bits of the row globals (2^-6, 2^-10): block outputs of O(0.1 .. 1), as checkpoints have
GLOBALS = (0x2400, 0x1400)
VOCAB = 248320
DTYPES = {"bf16": torch.bfloat16, "f32": torch.float32, "i32": torch.int32, "i64": torch.int64}


def _blocks(name, tokens, layers, zipf=0.0, norm=True, graph=False, out="bf16"):
    return {"name": name, "kind": "blocks", "tokens": tokens, "layers": layers, "zipf": zipf, "norm": norm, "graph": graph, "out": out}


def listed():
    return [
        # one sequence being decoded, launched call by call: latency and launches
        _blocks("decode-1", 1, 12),
        # a few sequences, the decode step captured in a graph
        _blocks("decode-8-graph", 8, 8, graph=True),
        # the ordinary decode batch: bound by the stream of nearly all experts
        _blocks("decode-64", 64, 4),
        # a ragged batch between decode and prefill (several decodes and a short prompt), skewed experts
        _blocks("mixed-173-zipf", 173, 2, zipf=1.1),
        # one short prompt
        _blocks("prefill-512-zipf", 512, 2, zipf=1.1),
        # a chunk of a long prompt
        _blocks("prefill-2048-zipf", 2048, 1, zipf=1.1, norm=False),
        # the largest batch: many prompts at once
        _blocks("prefill-8192", 8192, 1, norm=False),
        # engines with a router of their own: a decode batch in f32 with 64-bit ids, and a ragged prompt in bf16
        {"name": "staged-37-f32", "kind": "staged", "tokens": 37, "layers": 4, "x": "f32", "ids": "i64", "out": "f32"},
        {"name": "staged-1000", "kind": "staged", "tokens": 1000, "layers": 1, "x": "bf16", "ids": "i32", "out": "bf16"},
        # the vocabulary projection behind a decode step of one and of 64 sequences
        {"name": "lm-head-1", "kind": "lm_head", "m": 1, "n": VOCAB, "k": HIDDEN},
        {"name": "lm-head-64", "kind": "lm_head", "m": 64, "n": VOCAB, "k": HIDDEN},
        # an engine whose tensors live on the host
        {"name": "host-16", "kind": "host", "tokens": 16},
    ]


def _log_int(rng, lo, hi):
    """An integer of [lo, hi], uniform in its logarithm."""
    return min(hi, max(lo, int(lo * (hi / lo) ** rng.random() + 0.5)))


def draw(rng):
    kind = rng.choice(["blocks"] * 7 + ["staged"] * 2 + ["lm_head"] * 2 + ["host"])
    if kind == "blocks":
        tokens = _log_int(rng, 1, 8192)
        layers = rng.randint(6, 12) if tokens <= 16 else rng.randint(2, 4) if tokens <= 256 else 1
        return {"kind": kind, "tokens": tokens, "layers": layers, "zipf": rng.choice([0.0, 0.0, 0.8, 1.1, 1.2]),
                "norm": rng.random() < 0.6, "graph": tokens <= 256 and rng.random() < 0.4, "out": rng.choice(["bf16", "bf16", "f32"])}
    if kind == "staged":
        tokens = _log_int(rng, 1, 4096)
        return {"kind": kind, "tokens": tokens, "layers": 4 if tokens <= 64 else 1, "x": rng.choice(["bf16", "f32"]),
                "ids": rng.choice(["i32", "i64"]), "out": rng.choice(["bf16", "f32"])}
    if kind == "lm_head":
        # vocabularies are padded to a multiple of 64 in most checkpoints, and to less in some
        n = _log_int(rng, 32768, VOCAB)
        n -= n % rng.choice([64, 64, 4])
        return {"kind": kind, "m": _log_int(rng, 1, 64), "n": n, "k": HIDDEN}
    return {"kind": kind, "tokens": _log_int(rng, 1, 64)}


def _adapter(tokens, layers, seed):
    """An adapter with every expert of `layers` layers resident."""
    moe = ft.B200MoE(0, ft.ExpertShapes(HIDDEN, INTER), layers * EXPERTS, experts=EXPERTS, layers=layers, top_k=TOP_K,
                     shared_inter=SHARED, max_tokens=tokens)
    for l in range(layers):
        ft.synth.fill_banks_on_device(moe, l, 1000 * seed + l, slot0=l * EXPERTS, chunk=256, global_bits=GLOBALS)
    return moe


def _routes(gen, tokens):
    """What a router hands over: distinct experts of every token and their renormalised weights."""
    p = torch.softmax(torch.randn((tokens, EXPERTS), generator=gen, device="cuda") * 0.9, -1)
    w, ids = torch.topk(p, TOP_K, -1)
    return ids, (w / w.sum(-1, keepdim=True)).contiguous()


def prepare(case, seed):
    torch.cuda.set_device(0)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    randn = lambda *shape: torch.randn(shape, generator=gen, device="cuda")
    s = {"case": case}
    if case["kind"] == "lm_head":
        m, n, k = case["m"], case["n"], case["k"]
        s["moe"] = ft.B200MoE(0, ft.ExpertShapes(HIDDEN, INTER), 1, experts=EXPERTS, layers=1, top_k=TOP_K, shared_inter=0, max_tokens=64)
        s["a"] = randn(m, k).to(torch.bfloat16)
        s["packed"] = torch.randint(-2 ** 31, 2 ** 31, (k // 8, n), generator=gen, device="cuda", dtype=torch.int32)
        scale = torch.exp2(torch.rand((k // 16, n), generator=gen, device="cuda") * -6.0)
        s["scale"] = scale.to(torch.float8_e4m3fn).view(torch.uint8)
        s["glob"] = (2.0 ** -6 * (1.0 + torch.rand(n, generator=gen, device="cuda"))).to(torch.float16).view(torch.int16)
        s["c"] = torch.empty((m, n), dtype=torch.float32, device="cuda")
        return s
    tokens, layers = case["tokens"], case.get("layers", 1)
    s["moe"] = moe = _adapter(tokens, layers, seed)
    if case["kind"] == "host":
        s["cache"] = ft.ExpertCache(moe)
        _, slots, _ = s["cache"].ensure_experts(0, np.arange(EXPERTS))
        if slots != list(range(EXPERTS)):
            raise RuntimeError("the slot cache does not start in slot order")
        ids, w = _routes(gen, tokens)
        s["x"], s["ids"], s["w"] = randn(tokens, HIDDEN).cpu().numpy(), ids.cpu().numpy().astype(np.uint32), w.cpu().numpy()
        s["out"] = np.empty(tokens * HIDDEN, np.float32)
        return s
    s["out"] = torch.empty((layers, tokens, HIDDEN), dtype=DTYPES[case["out"]], device="cuda")
    if case["kind"] == "staged":
        s["executor"] = ft.CachedExperts(moe)
        s["reqs"] = []
        for l in range(layers):
            ids, w = _routes(gen, tokens)
            s["reqs"].append(ft.MoEDeviceRequest(l, HIDDEN, INTER, TOP_K, randn(tokens, HIDDEN).to(DTYPES[case["x"]]),
                                                 ids.to(DTYPES[case["ids"]]), w))
        return s
    zipf = case["zipf"] or None
    s["dense"] = [ft.synth.device_dense_weights(1000 * seed + l, "cuda", zipf_alpha=zipf) for l in range(layers)]
    x = randn(layers, tokens, HIDDEN)
    if case["norm"]:
        # attention output, residual stream and norm weight; the skew sits in column 0, which is 1 after the norm
        r, w = randn(layers, tokens, HIDDEN) * 3.0, 1.0 + 0.1 * randn(layers, HIDDEN)
        if zipf:
            x[..., 0], r[..., 0], w[..., 0] = 0.0, 10.0 ** 0.5, 1.0
        s["r"], s["w"] = r.to(torch.bfloat16), w.to(torch.bfloat16)
        s["sum"] = torch.empty((layers, tokens, HIDDEN), dtype=torch.bfloat16, device="cuda")
    elif zipf:
        x[..., 0] = 1.0
    s["x"] = x.to(torch.bfloat16)
    if case["graph"]:
        _step(s)                    # once as it is: a capture does not load modules
        torch.cuda.synchronize()
        s["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s["graph"]):
            _step(s)
    return s


def _step(s):
    """One engine step: every layer's block, in order, on the current stream."""
    moe, out, x = s["moe"], s["out"], s["x"]
    for l, (gate, gate_up, down, shared_gate) in enumerate(s["dense"]):
        if "r" in s:
            moe.moe_block_prenorm(l, x[l], s["r"][l], s["w"][l], EPS, gate, gate_up, down, shared_gate, s["sum"][l], out[l])
        else:
            moe.moe_block(l, x[l], gate, gate_up, down, shared_gate, out[l])


def run(s):
    kind = s["case"]["kind"]
    if kind == "blocks":
        if "graph" in s:
            s["graph"].replay()
        else:
            _step(s)
        return {"out": s["out"], "sum": s["sum"]} if "sum" in s else {"out": s["out"]}
    if kind == "staged":
        for req, out in zip(s["reqs"], s["out"]):
            s["executor"].execute_device(req, out)
        return s["out"]
    if kind == "lm_head":
        return s["moe"].dense_gemv(s["a"], s["packed"], s["scale"], s["glob"], c=s["c"])
    ft.run_experts(s["cache"], s["moe"], s["moe"], 0, HIDDEN, INTER, TOP_K, s["x"], s["ids"], s["w"], s["out"])
    return s["out"]


def _distinct(tokens, zipf):
    """Experts that a batch reaches: the router's logits are N(0, 0.02^2 * hidden) plus the bias."""
    rng = np.random.default_rng(7)
    bias = -zipf * np.log(np.arange(EXPERTS) + 1.0)
    logits = rng.normal(0.0, 0.02 * HIDDEN ** 0.5, (min(tokens, 8192), EXPERTS)) + bias
    return len(np.unique(np.argpartition(logits, -TOP_K, -1)[:, -TOP_K:]))


def work(case):
    if case["kind"] == "lm_head":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": n * k // 2 + n * k // 16 + 2 * n + m * (2 * k + 4 * n), "flops": 2 * m * n * k}
    tokens, layers = case["tokens"], case.get("layers", 1)
    size = {"bf16": 2, "f32": 4}
    routed = _distinct(tokens, case.get("zipf", 0.0)) * EXPERT_BYTES
    flops = 2 * tokens * TOP_K * 3 * HIDDEN * INTER
    if case["kind"] == "blocks":
        rows = 2 + size[case["out"]] + (4 if case["norm"] else 0)      # in, out; residual in and out
        return {"bytes": layers * (routed + DENSE_BYTES + tokens * HIDDEN * rows),
                "flops": layers * (flops + 2 * tokens * (EXPERTS * HIDDEN + 3 * SHARED * HIDDEN))}
    rows = 8 if case["kind"] == "host" else size[case["x"]] + size[case["out"]]
    return {"bytes": layers * (routed + tokens * HIDDEN * rows), "flops": layers * flops}


def tolerance(case):
    # lm_head: exact products of the bf16 rows and the 4-bit weights, f32 sums in any order.  The experts: bf16
    # activations, and 16-bit floats between the two projections and (prefill) per route.
    return {"rel": 1e-5} if case["kind"] == "lm_head" else {"rel": 5e-3, "max": 0.1}
