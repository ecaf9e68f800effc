"""The work a user of this library has it do, as measurable cases: one MoE expert path (router, top-k,
Q2_0 gate/up with SwiGLU, down, weighted combine) in its decode, verify, prefill and draft-head forms,
from device and from host buffers, and the conversion of weights at load time.

`listed()` names the standing cases and `draw(rng)` gives more of the same ranges; `prepare` makes what
a program holds before the call (weights resident in device memory, activations, workspaces, a captured
graph where a program would keep one), `run` is one pass through the public entry points.

Shapes are the repository's own: hidden 2048 / expert width 512 (the benchmark's layer), 2560 / 640
(the reference's model), 512 / 256 and 384 / 640 (the tests'). Values: 2-bit codes uniform, block
scales |N(0, 0.02)| in fp16, activations N(0, 1), router logits N(0, 1) or a Zipf(1.1) law.
"""
from __future__ import annotations

import math

import torch

from flashrt_b200 import moe

Q2_0 = moe.Q2_0_TYPE
SHAPES = ((2048, 512), (2560, 640), (512, 256), (384, 640))   # (hidden, expert width)


def listed() -> list[dict]:
    return [
        # one user, plain decoding: a token through eight layers, one call per layer; latency and launches count
        {"name": "decode_1", "kind": "decode", "T": 1, "n": 2048, "ff": 512, "E": 512, "K": 10, "layers": 8, "router": False},
        # speculative verification: a window of three tokens through a chained stack, replayed from a CUDA graph
        {"name": "verify_3", "kind": "verify", "T": 3, "n": 2048, "ff": 512, "E": 512, "K": 10, "layers": 8},
        # an engine that keeps its activations in host memory: sixteen tokens, eight layers in one call, pinned buffers
        {"name": "host_16", "kind": "host", "T": 16, "n": 2048, "ff": 512, "E": 512, "K": 10, "layers": 8},
        # a ragged batch of users at the reference model's shape, with the router projection in front
        {"name": "decode_37", "kind": "decode", "T": 37, "n": 2560, "ff": 640, "E": 512, "K": 10, "layers": 2, "router": True},
        # the largest decode batch the layer is meant for
        {"name": "decode_64", "kind": "decode", "T": 64, "n": 2048, "ff": 512, "E": 512, "K": 10, "layers": 2, "router": False},
        # a program that names its experts by pointer (moe_hits) over a window of two tokens, and the combine after it
        {"name": "hits_2", "kind": "hits", "T": 2, "n": 2560, "ff": 640, "E": 512, "K": 10, "layers": 4},
        # a short prompt of odd length at the reference model's shape: projection, routing, expert product, combine
        {"name": "prefill_293", "kind": "prefill", "T": 293, "n": 2560, "ff": 640, "E": 512, "K": 10, "zipf": False, "router": True, "bf16": False},
        # a prompt chunk with skewed routing: few experts take most of the tokens, many take a handful
        {"name": "prefill_4096", "kind": "prefill", "T": 4096, "n": 2048, "ff": 512, "E": 512, "K": 10, "zipf": True, "router": False, "bf16": False},
        # a long prompt, uniform routing, bf16 expert rows for the caller's own combine: the largest case
        {"name": "prefill_16384", "kind": "prefill", "T": 16384, "n": 2048, "ff": 512, "E": 512, "K": 10, "zipf": False, "router": False, "bf16": True},
        # the draft head's MoE on ggml-layout weights, one drafted token: the smallest call
        {"name": "draft_1", "kind": "draft", "T": 1, "n": 2560, "ff": 640, "E": 128, "K": 8},
        # the draft head over a prompt: grouped products on ggml-layout weights
        {"name": "draft_prompt_1000", "kind": "draft_prompt", "T": 1000, "n": 2560, "ff": 640, "E": 128, "K": 8},
        # loading: Q8_0 draft-head weights requantized to Q2_0, planar experts laid out for the kernels
        {"name": "load_48", "kind": "load", "E": 48, "n": 2560, "ff": 640},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.999)))))))


def draw(rng) -> dict:
    kind = rng.choice(("decode", "decode", "verify", "host", "hits", "prefill", "prefill", "prefill", "draft", "draft_prompt", "load"))
    n, ff = rng.choice(SHAPES)
    E, K = rng.choice((128, 256, 512)), rng.choice((4, 6, 8, 10))
    c = {"kind": kind, "n": n, "ff": ff, "E": E, "K": K}
    if kind == "decode":
        c.update(T=_log_int(rng, 1, 64), layers=rng.choice((2, 3, 4)), router=n % 256 == 0 and rng.random() < 0.5)
    elif kind == "verify":
        c.update(T=rng.randint(2, 8), layers=rng.choice((2, 4, 6)))
    elif kind == "host":
        c.update(T=_log_int(rng, 1, 64), layers=rng.randint(2, 6))
    elif kind == "hits":
        c.update(T=rng.randint(1, 8), layers=rng.choice((1, 2, 4)))
    elif kind == "prefill":
        T = _log_int(rng, 65, 16384)
        while T * K * n * ff > 16384 * 10 * 2048 * 512:
            T //= 2
        c.update(T=T, zipf=rng.random() < 0.5, router=n % 256 == 0 and T <= 1024 and rng.random() < 0.4, bf16=rng.random() < 0.4)
    elif kind == "draft":
        c.update(T=rng.randint(1, 8), E=128)
    elif kind == "draft_prompt":
        c.update(T=_log_int(rng, 9, 1000), E=128)
    else:
        c = {"kind": "load", "n": n, "ff": ff, "E": rng.randint(3, 48)}
    return c


# ---- inputs -------------------------------------------------------------------------------------

def _gen(seed: int) -> torch.Generator:
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _scales(g, *shape) -> torch.Tensor:
    d = torch.randn(*shape, generator=g, device="cuda").mul_(0.02).abs_().half()
    return d.clamp_(min=6.103515625e-05)


def _planar(g, count: int, n: int, ff: int) -> torch.Tensor:
    """count planar expert blobs (gate, up, down: codes, then scales), uint8 [count][blob]."""
    blob = torch.randint(0, 256, (count, moe.expert_bytes(n, ff)), dtype=torch.uint8, generator=g, device="cuda")
    off = 0
    for rows, cols in ((ff, n), (ff, n), (n, ff)):
        nblk = rows * cols // 64
        blob[:, off + nblk * 16:off + nblk * 18] = _scales(g, count, nblk).view(torch.uint8)
        off += nblk * 18
    return blob


def _tiled(g, count: int, n: int, ff: int) -> torch.Tensor:
    return moe.tile_experts(_planar(g, count, n, ff).view(-1), n, ff, count)


def _ggml(g, count: int, rows: int, cols: int) -> torch.Tensor:
    """count matrices of ggml Q2_0 blocks {fp16 d; 16 code bytes}, back to back."""
    nblk = count * rows * cols // 64
    b = torch.randint(0, 256, (nblk, 18), dtype=torch.uint8, generator=g, device="cuda")
    b[:, :2] = _scales(g, nblk).view(torch.uint8).view(nblk, 2)
    return b.view(-1)


def _logits(g, T: int, E: int, zipf: bool = False) -> torch.Tensor:
    if not zipf:
        return torch.randn(T, E, generator=g, device="cuda")
    rank = torch.randperm(E, generator=g, device="cuda").float() + 1.0
    u = torch.rand(T, E, generator=g, device="cuda").clamp_(1e-7, 1 - 1e-7)
    return (-1.1 * rank.log()[None, :] - (-(u.log())).log()).contiguous()


def _router(g, E: int, n: int):
    w = torch.randn(E + 1, n, generator=g, device="cuda").mul_(n ** -0.5).bfloat16()
    return w[:E].contiguous(), w[E].contiguous()


def prepare(case: dict, seed: int) -> dict:
    g = _gen(seed)
    kind, n, ff, E = case["kind"], case["n"], case["ff"], case["E"]
    K, T, layers = case.get("K", 0), case.get("T", 0), case.get("layers", 1)
    s = dict(case, stride=moe.expert_stride(n, ff))
    if kind in ("decode", "verify", "host"):
        s["weights"] = [_tiled(g, E + 1, n, ff) for _ in range(layers)]
        s["experts"] = [w.data_ptr() for w in s["weights"]]
        s["shared"] = [w.data_ptr() + E * s["stride"] for w in s["weights"]]
        s["x"] = [torch.randn(T, n, generator=g, device="cuda") for _ in range(layers)]
        s["logits"] = [_logits(g, T, E) for _ in range(layers)]
        s["gate"] = [torch.randn(T, generator=g, device="cuda") for _ in range(layers)]
        s["out"] = [torch.empty(T, n, device="cuda") for _ in range(layers)]
        if kind == "host":
            for name in ("x", "logits", "gate", "out"):
                s[name] = [t.cpu().pin_memory() for t in s[name]]
            s["ws"] = moe.workspace(moe.moe_layers_host_workspace_bytes(T, K, n, ff, E))
        else:
            s["ws"] = moe.workspace(moe.moe_layer_workspace_bytes(T, K, n, ff))
        if case.get("router"):
            s["w"] = [_router(g, E, n) for _ in range(layers)]
        if kind == "verify":   # the step is captured once and replayed, as a serving loop does
            s["xs"] = [s["x"][0]] + [torch.empty(T, n, device="cuda") for _ in range(layers)]
            _stack(s)
            torch.cuda.synchronize()
            s["graph"] = torch.cuda.CUDAGraph()
            with torch.cuda.graph(s["graph"]):
                _stack(s)
    elif kind == "hits":
        s["weights"] = [_tiled(g, E + 1, n, ff) for _ in range(layers)]
        s["x"] = [torch.randn(T, n, generator=g, device="cuda") for _ in range(layers)]
        s["ptr"], s["w"] = [], []
        for w in s["weights"]:
            ids, wts = moe.moe_route_topk(_logits(g, T, E), K)
            s["ptr"].append((w.data_ptr() + ids.long() * s["stride"]).contiguous())
            s["w"].append(wts)
        # most of a token's experts are hits; the rest would be served elsewhere
        s["hit_n"] = [torch.randint(max(1, K - 2), K + 1, (T,), dtype=torch.int32, generator=g, device="cuda") for _ in range(layers)]
        s["shexp"] = [torch.randn(T, n, generator=g, device="cuda") for _ in range(layers)]
        s["gate"] = [torch.randn(T, generator=g, device="cuda") for _ in range(layers)]
        s["yh"] = [torch.zeros(T, K, n, device="cuda") for _ in range(layers)]
        s["out"] = [torch.empty(T, n, device="cuda") for _ in range(layers)]
        s["ws"] = moe.workspace(moe.moe_hits_scratch_bytes(K, n, ff, T))
    elif kind == "prefill":
        s["weights"] = _tiled(g, E, n, ff)
        s["x"] = torch.randn(T, n, generator=g, device="cuda").bfloat16().float()   # a bf16 residual stream
        s["logits"] = _logits(g, T, E, case["zipf"])
        s["shexp"] = torch.randn(T, n, generator=g, device="cuda")
        s["gate"] = torch.randn(T, generator=g, device="cuda")
        s["ws"] = moe.workspace(moe.moe_q2.workspace_bytes(T, K, n, ff, E))
        if case["router"]:
            s["w"] = _router(g, E, n)
    elif kind in ("draft", "draft_prompt"):
        s["gate_w"], s["up_w"], s["down_w"] = _ggml(g, E, ff, n), _ggml(g, E, ff, n), _ggml(g, E, n, ff)
        s["gu_stride"], s["d_stride"] = moe.gemv.row_bytes(Q2_0, n) * ff, moe.gemv.row_bytes(Q2_0, ff) * n
        s["x"] = torch.randn(T, n, generator=g, device="cuda")
        s["logits"] = _logits(g, T, E)
        s["shexp"] = torch.randn(T, n, generator=g, device="cuda")
        s["gate"] = torch.randn(T, generator=g, device="cuda")
        if kind == "draft_prompt":
            s["ws"] = moe.workspace(moe.gemm.workspace_bytes(n, T * K))
            s["ws_h"] = moe.workspace(moe.gemm.workspace_bytes(ff, T * K))
    else:
        nblk = 3 * E * n * ff // 64
        src = torch.randint(-127, 128, (nblk * 2, 34), dtype=torch.int8, generator=g, device="cuda").view(torch.uint8)
        src[:, :2] = _scales(g, nblk * 2).view(torch.uint8).view(nblk * 2, 2)
        s["q8_0"] = src.view(-1)
        s["planar"] = _planar(g, E, n, ff).view(-1)
        s["tiled"] = torch.zeros(E * s["stride"], dtype=torch.uint8, device="cuda")
    return s


# ---- the pass -----------------------------------------------------------------------------------

def _stack(s: dict) -> None:
    """The chained stack: every layer's input is the norm of the one before plus its output."""
    for l in range(s["layers"]):
        moe.moe_layer(s["experts"][l], s["stride"], s["E"], s["shared"][l], s["n"], s["ff"], s["xs"][l], s["logits"][l], s["gate"][l], s["K"],
                      out=s["out"][l], ws=s["ws"])
        moe.chain_rmsnorm_unit(s["xs"][l], s["out"][l], out=s["xs"][l + 1])


def _run_decode(s: dict):
    for l in range(s["layers"]):
        lg, gate = s["logits"][l], s["gate"][l]
        if s["router"]:
            lg, gate = moe.router_logits(*s["w"][l], s["x"][l])
        moe.moe_layer(s["experts"][l], s["stride"], s["E"], s["shared"][l], s["n"], s["ff"], s["x"][l], lg, gate, s["K"], out=s["out"][l],
                      ws=s["ws"])
    return s["out"]


def _run_verify(s: dict):
    s["graph"].replay()
    return {"x": s["xs"][1:], "y": s["out"]}


def _run_host(s: dict):
    return moe.moe_layers_host(s["experts"], s["stride"], s["E"], s["shared"], s["n"], s["ff"], s["x"], s["logits"], s["gate"], s["K"], s["out"],
                               s["ws"])


def _run_hits(s: dict):
    for l in range(s["layers"]):
        moe.moe_hits(s["ptr"][l], s["hit_n"][l], s["K"], s["x"][l], s["n"], s["ff"], s["yh"][l], scratch=s["ws"], T=s["T"])
        moe.moe_combine(s["yh"][l], s["w"][l], s["hit_n"][l], s["shexp"][l], s["gate"][l], out=s["out"][l])
    return {"out": s["out"], "yh": s["yh"]}


def _run_prefill(s: dict):
    lg, gate = s["logits"], s["gate"]
    if s["router"]:
        lg, gate = moe.router_logits(*s["w"], s["x"])
    ids, wts = moe.moe_route_topk(lg, s["K"])
    base = s["weights"].data_ptr()
    if s["bf16"]:
        return {"wts": wts, "y": moe.moe_q2.run_ex(base, s["stride"], s["E"], s["n"], s["ff"], s["x"], ids, yd_bf16=True, ws=s["ws"])}
    yd = moe.moe_q2.run(base, s["stride"], s["E"], s["n"], s["ff"], s["x"], ids, ws=s["ws"])
    out = moe.moe_combine(yd.view(s["T"], s["K"], s["n"]), wts, None, s["shexp"], gate)
    return {"wts": wts, "y": yd, "out": out}


def _run_draft(s: dict):
    T, K, n, ff = s["T"], s["K"], s["n"], s["ff"]
    ids, wts = moe.moe_route_topk(s["logits"], K)
    xq = moe.gemv.quantize_q8_1(s["x"])
    hid = moe.gemv.moe_q(Q2_0, s["up_w"], s["gate_w"], xq, ids, n, ff, s["gu_stride"], False)
    hq = moe.gemv.quantize_q8_1(hid.view(T * K, ff))
    y = moe.gemv.moe_q(Q2_0, s["down_w"], None, hq, ids, ff, n, s["d_stride"], True)
    return {"hid": hid, "out": moe.moe_combine(y, wts, None, s["shexp"], s["gate"])}


def _run_draft_prompt(s: dict):
    T, K, n, ff, E = s["T"], s["K"], s["n"], s["ff"], s["E"]
    ids, wts = moe.moe_route_topk(s["logits"], K)
    plan = moe.gemm.moe_prepare(Q2_0, E, s["x"], False, ids, n, s["ws"])
    gate = moe.gemm.moe_run(plan, s["gate_w"], s["gu_stride"], ff)
    up = moe.gemm.moe_run(plan, s["up_w"], s["gu_stride"], ff)
    hid = torch.nn.functional.silu(gate).mul_(up)
    plan_h = moe.gemm.moe_prepare(Q2_0, E, hid, True, ids, ff, s["ws_h"])
    y = moe.gemm.moe_run(plan_h, s["down_w"], s["d_stride"], n)
    return {"hid": hid, "out": moe.moe_combine(y, wts, None, s["shexp"], s["gate"])}


def _run_load(s: dict):
    q2 = moe.convert_q8_0_to_q2_0(s["q8_0"])
    moe.tile_experts(s["planar"], s["n"], s["ff"], s["E"], out=s["tiled"])
    return {"q2": q2, "tiled": s["tiled"]}


_RUN = {"decode": _run_decode, "verify": _run_verify, "host": _run_host, "hits": _run_hits, "prefill": _run_prefill, "draft": _run_draft,
        "draft_prompt": _run_draft_prompt, "load": _run_load}


def run(state: dict):
    return _RUN[state["kind"]](state)


# ---- what a pass cannot do without --------------------------------------------------------------

def _distinct(T: int, E: int, K: int, zipf: bool = False) -> float:
    """Expected number of distinct experts of T tokens with K each."""
    if not zipf:
        return E * (1.0 - (1.0 - K / E) ** T)
    p = [r ** -1.1 for r in range(1, E + 1)]
    lo, hi = 0.0, 1e9   # inclusion of an expert in a token's K: 1 - exp(-c p), c such that they add up to K
    for _ in range(100):
        c = (lo + hi) / 2
        lo, hi = (c, hi) if sum(1 - math.exp(-c * q) for q in p) < K else (lo, c)
    return sum(1 - math.exp(-c * q * T) for q in p)


def work(case: dict) -> dict:
    kind, n, ff, E = case["kind"], case["n"], case["ff"], case["E"]
    K, T, layers = case.get("K", 0), case.get("T", 0), case.get("layers", 1)
    blob = 3 * n * ff // 64 * 18
    if kind == "load":   # Q8_0 in, Q2_0 out; planar in, tiled out
        return {"bytes": 3 * E * n * ff // 64 * (68 + 18) + 2 * E * blob, "flops": 0}
    shared = 1 if kind in ("decode", "verify", "host") else 0
    D = _distinct(T, E, K, case.get("zipf", False))
    row = T * n * 4
    b = (D + shared) * blob + 2 * row + T * E * 4   # each expert once, activations in, rows out, logits
    f = 6.0 * T * (K + shared) * n * ff
    if kind == "prefill":
        b += T * K * n * (2 if case["bf16"] else 4) + (0 if case["bf16"] else row) - (row if case["bf16"] else 0)   # the per-slot rows; the shared rows
    elif kind == "hits":
        b += T * K * n * 4 + row - T * E * 4
    elif kind in ("draft", "draft_prompt"):
        b += T * K * ff * 4 + row
    if case.get("router"):
        b += (E + 1) * n * 2
        f += 2.0 * T * (E + 1) * n
    return {"bytes": b * layers, "flops": f * layers}


def tolerance(case: dict):
    """Sums are fp32, but activations pass through int8 codes twice (x and the hidden row): another
    order of additions moves a hidden value by about 1e-7 of itself and tips a code at one in some
    ten thousand values; a tipped code (1/127 of its block's largest value) moves an expert row of
    width ff by about 1.5e-3 of its RMS, a few thousandths at its worst element. Weights at load time are
    whole bytes. bf16 rows carry a rounding of 2^-9 each."""
    if case["kind"] == "load":
        return "exact"
    if case.get("bf16"):
        return {"rel": 4e-3, "max": 2e-2}
    return {"rel": 3e-4, "max": 1e-2}
