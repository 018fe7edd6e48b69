"""The work that users of this library have it do, as measurable cases: MoE layer calls from one decode token to an
8192-token prefill over the five block formats, directly or replayed as a CUDA graph, and the call sequence of an engine
that drives the path matrix by matrix (the WeightFormat adapter's protocol).

A case is a dict of plain values:
  kind      "layer": MoeLayer.forward for each of `layers` stacked layers; "engine": router, routing, per-matrix products
  tokens    tokens of the pass (1..128: decode / speculative verification, above: prefill)
  hidden, experts, topk, ff, gating, norm, shared, bias      the layer's shape (gating 1: softmax, 2: sigmoid)
  gate, down                                                 block formats of the gate and up banks / the down bank
  layout    bank layout of IQ3_S experts ("codes": the default; "gguf": the GGUF-sized one)
  dtype, out   activation and output types; residual: the layer call adds the skip connection
  graph     the pass is captured once and replayed, as a decode loop does; otherwise it is launched call by call
  skew      Zipf-like expert popularity (the hottest expert holds about ten times the mean)
"""
from __future__ import annotations

import ctypes
import functools
import math

import torch

from tqllm_b200 import capi, moe, synth

TORCH = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
TYPE = {"q4_k": synth.Q4_K, "iq3_s": synth.IQ3_S, "iq4_xs": synth.IQ4_XS, "iq4_nl": synth.IQ4_NL, "nvfp4g": synth.NVFP4G}
NAME_OF = {v: k for k, v in TYPE.items()}
DISTINCT = 24          # experts quantised one by one; a bank of more experts repeats them in a seeded order


def _of_config(config: str, tokens: int, **more) -> dict:
    """a case on one of the package's layer shapes"""
    s = synth.CONFIGS[config]
    case = dict(kind="layer", tokens=tokens, layers=1, hidden=s.hidden, experts=s.experts, topk=s.topk, ff=s.ff, gating=s.gating, norm=s.norm,
                shared=s.shared, bias=s.sel_bias, gate=NAME_OF[s.types[0]], down=NAME_OF[s.types[2]], layout="codes", dtype=s.act_dtype,
                out="f32" if s.act_dtype == "f32" else "bf16", residual=False, graph=False, skew=False)
    case.update(more)
    return case


def listed() -> list[dict]:
    return [
        # one chat user on the 512-expert IQ3_S model, launched call by call: latency of the launches and the host path
        _of_config("c2", 1, name="c2 decode 1"),
        # the decode step of 64 concurrent users through four stacked layers, replayed as a graph: weight streaming
        _of_config("c2", 64, name="c2 decode 64 x4", layers=4, graph=True),
        # a handful of users on the NVFP4 checkpoint, with the skip connection
        _of_config("c3", 8, name="c3 decode 8", residual=True, graph=True),
        # 16 users on the wide Q4_K sigmoid-routed model
        _of_config("c4", 16, name="c4 decode 16", graph=True),
        # a verification step of a few speculative drafts on the IQ4_XS / IQ4_NL model
        _of_config("c5", 24, name="c5 decode 24", graph=True),
        # a small fp32 model, an odd token count
        _of_config("c1", 7, name="c1 f32 7"),
        # shapes that belong to no configuration: ragged tokens, odd expert count, 16-bit floats
        _of_config("c1", 77, name="own q4_k 77", hidden=2560, experts=60, topk=6, ff=768, dtype="f16", out="f16"),
        # a chunk of a chunked prefill, between decode and prefill densities
        _of_config("c2", 509, name="c2 chunk 509"),
        # the prefill of a prompt on each large shape
        _of_config("c3", 4096, name="c3 prefill 4096", residual=True),
        _of_config("c4", 2047, name="c4 prefill 2047"),
        _of_config("c5", 8192, name="c5 prefill 8192 skew", skew=True),
        # an engine that calls the products matrix by matrix with its own groups (the adapter's protocol): prompt of 600
        _of_config("c4", 600, name="engine c4 600", kind="engine", dtype="f16"),
    ]


def _log_uniform(rng, lo: int, hi: int) -> int:
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.5)))))))


def draw(rng) -> dict:
    kind = rng.choice(["decode", "decode", "decode", "prefill", "prefill", "engine"])
    tokens = {"decode": lambda: _log_uniform(rng, 1, 128), "prefill": lambda: _log_uniform(rng, 129, 8192),
              "engine": lambda: _log_uniform(rng, 1, 1024)}[kind]()
    case = _of_config(rng.choice(["c1", "c2", "c2", "c3", "c4", "c5"]), tokens)
    if rng.random() < 0.35:                                     # a shape of no configuration
        fmt = rng.choice(["q4_k", "iq3_s", "iq4_xs", "nvfp4g"])
        unit = 128 if fmt == "nvfp4g" else 256
        case.update(hidden=256 * rng.randint(4, 20), ff=unit * rng.randint(512 // unit, 2048 // unit), gate=fmt,
                    down="iq4_nl" if fmt == "iq4_xs" and rng.random() < 0.5 else fmt, gating=rng.choice([1, 1, 2]), shared=rng.random() < 0.4)
        expert = 3 * case["hidden"] * case["ff"] * 0.56
        case["experts"] = _log_uniform(rng, 8, min(512, int(3e9 / expert)))
        case["topk"] = rng.randint(1, min(10, case["experts"] // 2))
        case["bias"] = case["gating"] == 2
    if case["dtype"] != "f32":
        case["dtype"] = rng.choice(["bf16", "bf16", "f16"])
    case["out"] = rng.choice([case["dtype"], case["dtype"], "f32"])
    case["layout"] = "gguf" if case["gate"] == "iq3_s" and rng.random() < 0.25 else "codes"
    if kind == "engine":
        case.update(kind="engine", dtype="f16", out="bf16", shared=False)
    else:
        case["residual"] = rng.random() < 0.3
        case["graph"] = kind == "decode" and rng.random() < 0.5
        case["skew"] = tokens >= 64 and case["gating"] == 1 and rng.random() < 0.3
    most = [work(c) for c in listed() if c["name"] == "c5 prefill 8192 skew"][0]
    while work(case)["flops"] > most["flops"] or work(case)["bytes"] > most["bytes"]:
        case["tokens"] = max(1, case["tokens"] * 3 // 4)
    return case


def _popularity(case) -> list[float]:
    """probability that a token selects the expert, expert by expert (skew: a power law whose first expert has ten times the mean)"""
    e, k = case["experts"], case["topk"]
    if not case["skew"]:
        return [k / e] * e
    lo, hi = 0.0, 4.0
    for _ in range(40):
        a = 0.5 * (lo + hi)
        total = sum(r ** -a for r in range(1, e + 1))
        lo, hi = (a, hi) if e / total < 10.0 else (lo, a)
    return [min(1.0, k * r ** -a / total) for r in range(1, e + 1)]


def work(case) -> dict:
    """the GGUF blocks of the experts that are touched, router weights, activations in and out; two operations per weight and assignment"""
    n, h, f, e = case["tokens"], case["hidden"], case["ff"], case["experts"]
    touched = sum(1.0 - (1.0 - p) ** n for p in _popularity(case)) + (1 if case["shared"] else 0)
    expert = 2 * synth.raw_bytes(TYPE[case["gate"]], f, h) + synth.raw_bytes(TYPE[case["down"]], h, f)
    size = {"f32": 4, "f16": 2, "bf16": 2}
    rows = n * h * (size[case["dtype"]] + size[case["out"]] * (2 if case["residual"] else 1))
    per_layer = touched * expert + 4 * e * h + rows
    flops = 6.0 * h * f * n * (case["topk"] + (1 if case["shared"] else 0)) + 2.0 * n * h * e
    return {"bytes": case["layers"] * per_layer, "flops": case["layers"] * flops}


def tolerance(case) -> dict:
    """Products of 16-bit operands (weights or activations rounded to 11 bits, two products and SwiGLU in a row) summed in fp32:
    about 1e-3; a bf16 result adds its own 2^-9 per value."""
    return {"rel": 5e-3 if case["out"] == "bf16" else 2e-3}


@functools.lru_cache(maxsize=None)
def _router_scale(hidden: int, experts: int, topk: int) -> float:
    return synth.solve_router_scale(synth.LayerShape("own", hidden, experts, topk, 256))


def _shape(case) -> synth.LayerShape:
    t = TYPE[case["gate"]]
    return synth.LayerShape("own", case["hidden"], case["experts"], case["topk"], case["ff"], case["gating"], case["norm"], 0.0, case["shared"],
                            (t, t, TYPE[case["down"]]), case["bias"], case["dtype"])


def _gen(seed: int) -> torch.Generator:
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _layer(case, g: torch.Generator) -> moe.MoeLayer:
    """a resident layer: N(0, 0.02) weights in the case's block formats; softmax routers whose top-k mass is about 0.6, sigmoid
    routers with a small balancing bias (a trained bias evens out the expert loads)"""
    s, dev = _shape(case), "cuda"
    scale = _router_scale(s.hidden, s.experts, s.topk) if s.gating == synth.SOFTMAX else 1.0
    router = torch.randn(s.experts, s.hidden, generator=g, device=dev) * (0.02 * scale)
    bias = torch.randn(s.experts, generator=g, device=dev) * 0.01 if s.sel_bias else None

    def bank(type_id, rows, cols, experts):
        m = min(experts, DISTINCT)
        raw = [synth.quantize(type_id, torch.randn(rows, cols, generator=g, device=dev) * 0.02) for _ in range(m)]
        order = torch.randint(0, m, (experts,), generator=g, device=dev) if experts > m else torch.arange(m, device=dev)
        return torch.stack(raw)[order].reshape(-1)

    dims = ((s.ff, s.hidden), (s.ff, s.hidden), (s.hidden, s.ff))
    raw = tuple(bank(t, r, c, s.experts) for t, (r, c) in zip(s.types, dims))
    shared = tuple(bank(t, r, c, 1) for t, (r, c) in zip(s.types, dims)) if s.shared else None
    return moe.MoeLayer(s, router, raw, shared, bias, iq3s_layout=case["layout"])


def _skew(case, layer: moe.MoeLayer, x: torch.Tensor) -> torch.Tensor:
    """a direction that every token shares, along which the router rows fall with the expert's rank: expert popularity with the
    hottest expert at about ten times the mean; returns the shifted tokens"""
    d = torch.zeros(case["hidden"], device="cuda")
    d[::5] = 1.0
    d /= d.norm()
    x = (x.float() + 3.0 * d).to(x.dtype)
    fall = torch.log(torch.arange(1, case["experts"] + 1, device="cuda", dtype=torch.float32))[:, None] * d[None, :] / 3.0
    probe, base, lo, hi = x[:1024].float(), layer.router_w.clone(), 0.0, 12.0
    for _ in range(14):
        c = 0.5 * (lo + hi)
        ids = (probe @ (base - c * fall).T).topk(case["topk"], -1).indices
        hot = torch.bincount(ids.flatten(), minlength=case["experts"]).float()
        lo, hi = (c, hi) if float(hot.max() / hot.mean()) < 10.0 else (lo, c)
    layer.router_w.copy_(base - c * fall)
    return x


class _Engine:
    """buffers of an engine that runs the layer matrix by matrix: fp16 rows in, bf16 rows between the products and out"""

    def __init__(self, case, layer: moe.MoeLayer, x: torch.Tensor):
        n, k, e = case["tokens"], case["topk"], case["experts"]
        lib, dev = capi.lib, "cuda"
        self.layer, self.x, self.n, self.k = layer, x, n, k
        self.rows = n > 8                                       # more tokens than this: grouped products; else id lists
        new = lambda *shape, dtype: torch.empty(*shape, dtype=dtype, device=dev)
        self.logits = new(n, e + 1, dtype=torch.float32)
        self.ids, self.weights = new(n, k, dtype=torch.int32), new(n, k, dtype=torch.float32)
        self.counts, self.groups = new(e, dtype=torch.int32), new(e, n, dtype=torch.int32)
        self.plan = new(lib.b2moe_plan_ints(e, n * k, 0), dtype=torch.int32)
        self.dws = new(max(16, lib.b2moe_dispatch_workspace_bytes(e, n * k)), dtype=torch.uint8)
        self.g, self.u = new(n * k, case["ff"], dtype=torch.bfloat16), new(n * k, case["ff"], dtype=torch.bfloat16)
        self.act = new(n * k, case["ff"], dtype=torch.float16)
        self.y = new(n * k, case["hidden"], dtype=torch.bfloat16)
        self.out = new(n, case["hidden"], dtype=torch.bfloat16)
        self.gate, self.up, self.down = (ctypes.byref(b.c) for b in (layer.gate, layer.up, layer.down))
        need = max(lib.b2moe_expert_matvec_workspace_bytes(self.gate, n, k), lib.b2moe_expert_matvec_workspace_bytes(self.down, n, k),
                   lib.b2moe_expert_gemm_gateup_workspace_bytes(self.gate, n, k, capi.F16))
        self.ws = new(need, dtype=torch.uint8)

    def step(self):
        lib, s, n, k, check = capi.lib, torch.cuda.current_stream().cuda_stream, self.n, self.k, capi.check
        sh, e, h = self.layer.shape, self.layer.experts, self.layer.shape.hidden
        p = lambda t: t.data_ptr()
        ws = (p(self.ws), self.ws.numel(), s)
        check(lib.b2moe_router(p(self.layer.router_w), None, p(self.x), capi.F16, p(self.logits), e + 1, h, e, n, s), "router")
        if sh.gating == synth.SOFTMAX:
            check(lib.b2moe_topk_softmax(p(self.logits), e + 1, p(self.ids), p(self.weights), None, e, k, n, 0.0, s), "top-k")
        else:
            check(lib.b2moe_route_sigmoid(p(self.logits), e + 1, p(self.layer.sel_bias), p(self.ids), p(self.weights), e, k, int(sh.norm), 0.0, n, s),
                  "route")
        if self.rows:
            check(lib.b2moe_dispatch(p(self.ids), n, k, e, 0, p(self.plan), p(self.dws), self.dws.numel(), s), "group")
            check(lib.b2moe_plan_to_groups(p(self.plan), n, k, e, p(self.counts), p(self.groups), s), "group")
            lists = (p(self.counts), p(self.groups), n, k)
            check(lib.b2moe_expert_gemm_gateup(self.gate, self.up, p(self.x), capi.F16, p(self.act), capi.F16, *lists, *ws), "gate/up")
            check(lib.b2moe_expert_gemm(self.down, p(self.act), capi.F16, p(self.y), capi.BF16, *lists, 1, *ws), "down")
        else:
            for m, y in ((self.gate, self.g), (self.up, self.u)):
                check(lib.b2moe_expert_matvec(m, p(self.x), capi.F16, p(y), capi.BF16, p(self.ids), n, k, 0, *ws), "gate, up")
            check(lib.b2moe_swiglu(p(self.g), p(self.u), capi.BF16, p(self.act), capi.F16, self.act.numel(), s), "swiglu")
            check(lib.b2moe_expert_matvec(self.down, p(self.act), capi.F16, p(self.y), capi.BF16, p(self.ids), n, k, 1, *ws), "down")
        check(lib.b2moe_sum_rows(p(self.y), None, capi.BF16, p(self.weights), None, p(self.out), capi.BF16, h, k, n, s), "sum")
        return self.out


class _Layers:
    """stacked resident layers that read the same tokens, with their output buffers, and the captured pass where the case has one"""

    def __init__(self, case, layers, x, residual):
        self.layers, self.x, self.residual = layers, x, residual
        self.outs = [torch.empty(case["tokens"], case["hidden"], dtype=TORCH[case["out"]], device="cuda") for _ in layers]
        for layer in layers:
            layer.reserve(case["tokens"])
        self.graph = None
        if case["graph"]:
            stream = torch.cuda.Stream()
            stream.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(stream):
                self.launch()
            stream.synchronize()
            self.graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(self.graph, stream=stream):
                self.launch()

    def launch(self):
        for layer, out in zip(self.layers, self.outs):
            layer.forward(self.x, out=out, residual=self.residual)

    def step(self):
        if self.graph is not None:
            self.graph.replay()
        else:
            self.launch()
        return self.outs


def prepare(case, seed):
    g = _gen(seed)
    layers = [_layer(case, g) for _ in range(case["layers"])]
    x = torch.randn(case["tokens"], case["hidden"], generator=g, device="cuda").to(TORCH[case["dtype"]])
    if case["skew"]:
        x = _skew(case, layers[0], x)
    if case["kind"] == "engine":
        return _Engine(case, layers[0], x)
    residual = torch.randn(case["tokens"], case["hidden"], generator=g, device="cuda").to(TORCH[case["out"]]) if case["residual"] else None
    return _Layers(case, layers, x, residual)


def run(state):
    return state.step()
