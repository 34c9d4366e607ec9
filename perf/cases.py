"""Timed cases of the BF16N hot path: what a serving process calls, through the operators of orin_qwen_lossless_b200.ops.

A case is a dict of plain values; prepare() makes what the process holds before the call (encoded weights on the GPU,
activations, the captured graph of a decode step), run() is one pass, work() the bytes and operations a pass cannot do
without, tolerance() how far two correct implementations of the same precision may be apart.

Weights are N(0, 0.02) rounded to BF16 and activations and router logits N(0, 1), as in the benchmark; formats, unit
sizes and layouts are the shape policy's (ops.choose) for the engine that the case names. Expert shapes are the
benchmark's: hidden 2048, intermediate 512, top-8.
"""
from __future__ import annotations

import torch

from orin_qwen_lossless_b200 import ops

HIDDEN, INTER, TOP_K = 2048, 512, 8
PAIR_BYTES, NIBBLE_BYTES = 1.333, 1.52      # stored bytes per weight of the two formats on these weights


def listed():
    return [
        # one decoded token through the vocabulary projection: the headline product
        {"name": "lm_head", "kind": "project", "engine": "llama", "fo": False, "rows": 248320, "K": 2048, "tokens": 1, "x": "bf16"},
        # the verify batch of speculative decoding on a quarter of the vocabulary (the shard of one of four GPUs)
        {"name": "lm_head_verify", "kind": "project", "engine": "llama", "fo": False, "rows": 62080, "K": 2048, "tokens": 4, "x": "bf16"},
        # eight concurrent sequences on half of the vocabulary, stored in fragment order (the layout for batches)
        {"name": "lm_head_fragments", "kind": "project", "engine": "vllm", "fo": True, "rows": 124160, "K": 2048, "tokens": 8, "x": "bf16"},
        # one token through a layer's input projection, launched eagerly: the smallest single call
        {"name": "linear_token", "kind": "linear", "rows": 8192, "K": 2048, "tokens": 1, "bias": False},
        # the same projection on a prompt of a ragged length
        {"name": "linear_prompt", "kind": "linear", "rows": 8192, "K": 2048, "tokens": 1000, "bias": False},
        # the small matrices of all layers for one token (projections, router, shared expert), one captured graph
        {"name": "small_layers", "kind": "layers", "layers": 48, "tokens": 1},
        # routed experts, one token a step, eight steps of a generation in one captured graph, llama.cpp layout
        {"name": "moe_token", "kind": "moe_decode", "engine": "llama", "experts": 256, "tokens": 1, "steps": 8},
        # routed experts, a batch of four tokens a step, vLLM layout
        {"name": "moe_batch", "kind": "moe_decode", "engine": "vllm", "experts": 128, "tokens": 4, "steps": 4},
        # routed experts of a prompt, llama.cpp layout with the workspace that such an engine registers at load
        {"name": "moe_prompt", "kind": "moe_prompt", "engine": "llama", "experts": 256, "tokens": 2048},
        # routed experts of a full prefill batch, vLLM layout
        {"name": "moe_prompt_large", "kind": "moe_prompt", "engine": "vllm", "experts": 256, "tokens": 8192},
        # one drafted token: 2-bit scores, candidates, exact scores of the candidates
        {"name": "draft_token", "kind": "draft", "rows": 62080, "tokens": 1, "bits": 2},
        # loading one tensor: host encode, upload, bit-exact check of the GPU's decode
        {"name": "load_tensor", "kind": "load", "engine": "llama", "rows": 8192, "K": 2048},
    ]


def _log(rng, lo, hi, step=1):
    """An integer from lo to hi, spread over its logarithm, in multiples of step."""
    v = lo * (hi / lo) ** rng.random()
    return min(hi, max(lo, int(v / step) * step))


def draw(rng):
    kind = rng.choice(["project", "project", "linear", "linear", "layers", "moe_decode", "moe_decode", "moe_prompt", "moe_prompt", "draft", "load"])
    if kind == "project":
        fo = rng.random() < 0.3
        return {"kind": kind, "engine": "vllm" if fo else "llama", "fo": fo, "rows": _log(rng, 4096, 131072, 16), "K": rng.choice([512, 1024, 2048, 2048, 4096]),
                "tokens": rng.randint(1, 8), "x": "f32" if not fo and rng.random() < 0.2 else "bf16"}
    if kind == "linear":
        return {"kind": kind, "rows": _log(rng, 1024, 16384, 16), "K": rng.choice([512, 1024, 2048, 2048, 4096]),
                "tokens": rng.randint(1, 8) if rng.random() < 0.4 else _log(rng, 9, 4096), "bias": rng.random() < 0.3}
    if kind == "layers":
        return {"kind": kind, "layers": _log(rng, 4, 48), "tokens": rng.randint(1, 4)}
    if kind == "moe_decode":
        return {"kind": kind, "engine": rng.choice(["llama", "vllm"]), "experts": _log(rng, 16, 128, 8), "tokens": rng.randint(1, 8), "steps": rng.randint(2, 4)}
    if kind == "moe_prompt":
        return {"kind": kind, "engine": rng.choice(["llama", "vllm"]), "experts": _log(rng, 16, 160, 8), "tokens": _log(rng, 9, 8000)}
    if kind == "draft":
        return {"kind": kind, "rows": _log(rng, 16384, 65536, 16), "tokens": rng.randint(1, 4), "bits": rng.choice([2, 4])}
    return {"kind": kind, "engine": rng.choice(["llama", "vllm"]), "rows": _log(rng, 1024, 8192, 16), "K": rng.choice([1024, 2048])}


# ------------------------------------------------------------------ what a process holds before the call

def _dev():
    return torch.device("cuda", torch.cuda.current_device())


def _randn(gen, *shape, dtype=torch.float32):
    return torch.randn(*shape, device=_dev(), generator=gen).to(dtype)


def _weights(gen, rows, K):
    """BF16 weights in host memory, as a loader has them."""
    return (_randn(gen, rows, K) * 0.02).to(torch.bfloat16).cpu()


def _upload(gen, rows, K, choice):
    return ops.upload(*ops.encode(_weights(gen, rows, K), *choice), _dev())


def _experts(gen, experts, engine):
    gate_up = ops.choose(INTER, HIDDEN, experts, engine=engine, expert=True)
    down = ops.choose(HIDDEN, INTER, experts, engine=engine, expert=True)
    return (_upload(gen, experts * INTER, HIDDEN, gate_up), _upload(gen, experts * INTER, HIDDEN, gate_up),
            _upload(gen, experts * HIDDEN, INTER, down))


def _capture(fn):
    """The CUDA graph of fn(), as a decode loop keeps one for each batch size; fn writes to buffers of its own."""
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        fn()
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        fn()
    return g


def prepare(case, seed):
    ops.init()
    gen = torch.Generator(device=_dev()).manual_seed(seed)
    kind, T = case["kind"], case.get("tokens", 0)
    s = {"case": case}
    if kind == "project":
        choice = ops.choose(case["rows"], case["K"], engine=case["engine"], dense_frag_order=case["fo"])
        s["w"] = _upload(gen, case["rows"], case["K"], choice)
        s["x"] = _randn(gen, T, case["K"], dtype=torch.bfloat16 if case["x"] == "bf16" else torch.float32)
    elif kind == "linear":
        s["w"] = _upload(gen, case["rows"], case["K"], ops.choose(case["rows"], case["K"], engine="vllm"))
        s["x"] = _randn(gen, T, case["K"], dtype=torch.bfloat16)
        s["bias"] = _randn(gen, case["rows"], dtype=torch.bfloat16) if case["bias"] else None
    elif kind == "layers":
        nib = (ops.FMT_NIBBLE, 0, False)
        layers = [[_upload(gen, r, k, nib) for r, k in ((2048, 512), (512, 2048), (256, 2048), (2 * INTER, HIDDEN), (HIDDEN, INTER))]
                  for _ in range(case["layers"])]
        wide, narrow = _randn(gen, T, HIDDEN, dtype=torch.bfloat16), _randn(gen, T, INTER, dtype=torch.bfloat16)
        s["out"] = [torch.empty(len(layers), T, rows, device=_dev()) for rows in (2048, 512, 256, HIDDEN)]

        def step():
            for ws, *ys in zip(layers, *s["out"]):
                ops.mmv_group([narrow, wide, wide], ws[:3], ys[:3])       # independent projections and the router
                ops.mmv(ops.mmv_glu(wide, ws[3]), ws[4], out=ys[3])       # shared expert
        s["graph"], s["held"] = _capture(step), (layers, wide, narrow)
    elif kind == "moe_decode":
        E, steps = case["experts"], case["steps"]
        gate, up, down = _experts(gen, E, case["engine"])
        xs = [_randn(gen, T, HIDDEN, dtype=torch.bfloat16) for _ in range(steps)]
        logits = [_randn(gen, T, E) for _ in range(steps)]
        scratch = ops.moe_decode_scratch(T, TOP_K, gate, down, E, _dev())
        outs = [None] * steps

        def step():
            for i in range(steps):
                outs[i] = ops.moe_decode(xs[i], gate, up, down, E, TOP_K, router_logits=logits[i], scratch=scratch)
        s["graph"], s["held"], s["out"] = _capture(step), (gate, up, down, xs, logits, scratch), [v for o in outs for v in o]
    elif kind == "moe_prompt":
        s["experts"] = _experts(gen, case["experts"], case["engine"])
        s["x"] = _randn(gen, T, HIDDEN, dtype=torch.bfloat16)
        s["logits"] = _randn(gen, T, case["experts"])
        if case["engine"] == "llama":
            ops.ensure_workspace((s["experts"][0], s["experts"][1]), (s["experts"][2], None))
    elif kind == "draft":
        w = _weights(gen, case["rows"], HIDDEN)
        quantize = ops.int2_quantize if case["bits"] == 2 else ops.int4_quantize
        s["head"] = ops.DraftHead(case["bits"], *quantize(w.to(_dev())), ops.DEFAULT_CANDIDATES[case["bits"]])
        s["w"] = ops.upload(*ops.encode(w, *ops.choose(case["rows"], HIDDEN, engine="vllm")), _dev())
        s["x"] = _randn(gen, T, HIDDEN, dtype=torch.bfloat16)
    else:
        s["src"] = _weights(gen, case["rows"], case["K"])
        s["choice"] = ops.choose(case["rows"], case["K"], engine=case["engine"])
        n = case["rows"] * case["K"]
        s["plane"] = torch.empty(case["rows"], case["K"], dtype=torch.uint8, device=_dev())       # the loader's storage for
        s["aux"] = torch.zeros(n // 2 + (1 << 17), dtype=torch.uint8, device=_dev())  # the tensor; the rest of aux stays zero
    return s


# ------------------------------------------------------------------ one pass

def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "project":
        return ops.mmv(s["x"], s["w"])
    if kind == "linear":
        return ops.linear(s["x"], s["w"], s["bias"])
    if kind in ("layers", "moe_decode"):
        s["graph"].replay()
        return s["out"]
    if kind == "moe_prompt":
        gate, up, down = s["experts"]
        weights, ids = ops.moe_topk(s["logits"], TOP_K)
        return ops.moe_experts(s["x"], gate, up, down, weights, ids, case["experts"])
    if kind == "draft":
        return ops.draft_logits(s["x"], s["w"], s["head"], case["rows"])
    plane, aux, meta = ops.encode(s["src"], *s["choice"])
    s["plane"].copy_(plane)
    s["aux"][:aux.numel()].copy_(aux)
    w = ops.Weight(s["plane"], s["aux"][:aux.numel()], meta)
    return {"plane": s["plane"], "aux": s["aux"], "equal": ops.roundtrip_equal(w, s["src"])}


# ------------------------------------------------------------------ what a pass cannot do without, and how exact it is

def work(case):
    kind, T = case["kind"], case.get("tokens", 0)
    if kind in ("project", "linear"):
        n, bf16_out = case["rows"] * case["K"], kind == "linear"
        fmt = ops.choose(case["rows"], case["K"], engine="llama" if kind == "project" else "vllm")[0]
        per = NIBBLE_BYTES if fmt == ops.FMT_NIBBLE and not case.get("fo") else PAIR_BYTES
        x_bytes = 4 if case.get("x") == "f32" else 2
        return {"bytes": n * per + T * case["K"] * x_bytes + T * case["rows"] * (2 if bf16_out else 4), "flops": 2.0 * n * T}
    if kind == "layers":
        n = case["layers"] * (2048 * 512 * 2 + 256 * 2048 + 3 * INTER * HIDDEN)
        return {"bytes": n * NIBBLE_BYTES + case["layers"] * T * 4 * (2048 + 512 + 256 + HIDDEN), "flops": 2.0 * n * T}
    if kind == "moe_decode":
        E = case["experts"]
        used = E * (1.0 - (1.0 - TOP_K / E) ** T)
        n = 3 * INTER * HIDDEN
        return {"bytes": case["steps"] * (used * n * PAIR_BYTES + T * (E * 4 + HIDDEN * 6)), "flops": 2.0 * case["steps"] * T * TOP_K * n}
    if kind == "moe_prompt":
        E = case["experts"]
        used = E * (1.0 - (1.0 - TOP_K / E) ** T)
        n = 3 * INTER * HIDDEN
        return {"bytes": used * n * PAIR_BYTES + T * (E * 4 + HIDDEN * 4), "flops": 2.0 * T * TOP_K * n}
    if kind == "draft":
        n = case["rows"] * HIDDEN
        return {"bytes": n * case["bits"] / 8 + n / 128 * 4 + T * case["rows"] * 4, "flops": 2.0 * n * T}
    n = case["rows"] * case["K"]
    return {"bytes": n * 2.0 + n * PAIR_BYTES, "flops": 0.0}


def tolerance(case):
    kind = case["kind"]
    if kind == "load":
        return "exact"                        # stored bytes are the format's
    if kind == "linear":
        return {"rel": 7e-3, "max": 2e-2}     # one BF16 rounding of an FP32 sum: 1.66e-3 from the sum in 64 bits
    if kind == "moe_prompt":
        return {"rel": 1e-2, "max": 5e-2}     # BF16 between the two products and at the end: 2.33e-3 from the layer in 64 bits
    if kind == "moe_decode":
        return {"rel": 1e-5, "max": 1e-4, "differ": 0.0}   # FP32 sums; the chosen experts are whole numbers
    return {"rel": 1e-5, "max": 1e-4}         # FP32 sums of 512 to 4096 exact products: up to 2.1e-6 from the sums in 64 bits
