"""The work that a user of this package has it do, as cases that can be timed.

Four kinds, each through the package's public entry points:

  "layer"      one MoE sublayer as a forward runs it: router-logits projection, router, pack, experts (with or without the
               shared expert), combine, residual.  One token (a single conversation's decode step) to 16384 (a long
               prefill chunk).  Below 128 tokens the router projection is the streaming form, from there on the
               tensor-core one; the layer itself picks its expert kernels by the token count.
  "launchers"  the same block as a host that calls launcher by launcher issues it in prefill: BF16 activations handed
               over as they are, the served matrix-unit numerics (BF16 per-slot dots), the caller's own work buffers.
  "mix"        the hyper-connection mix in front of the block: the per-token forms for decode, the tensor-core forms
               for multi-token forwards.
  "dense"      a quantized dense projection: the streaming form for decode, the tensor-core form for prefill.

Decode steps can be replayed as CUDA graphs ("graph": True), as a serving loop does, or issued call by call.
Activations are N(0, 1) in BF16, weights N(0, 0.02) quantized with the package's own quantizer, router weights
N(0, 0.02) in FP32; expert popularity is level, N(0, 0.5) or Zipf(1.1) by a bias on the logits.
"""
import math

import torch

from strixite_b200 import kernels as K
from strixite_b200.kernels import Act, MoeMath, QDeviceView
from strixite_b200.layer import MoeBuffers, MoeLayer, MoeWeights

ROUTER_WMMA_MIN = 128  # tokens from which a forward takes the tensor-core router projection
MIX_WMMA_MIN = 64      # ... the tensor-core hyper-connection mix
DENSE_WMMA_MIN = 64    # ... the tensor-core dense projections
MIX_STREAMS = 4


def _layer(name, T, shared=True, gu=4, dn=4, bias="none", graph=False, d=4096, E=512, k=10, I=1024):
    return dict(name=name, kind="layer", T=T, d=d, E=E, k=k, I=I, gu_bits=gu, dn_bits=dn, shared=shared, bias=bias, graph=graph)


def listed():
    return [
        # one conversation, one token a step: every launch and every call shows
        _layer("layer_decode_1", 1),
        # two conversations of eight rows each (one token and seven drafts), replayed as a graph
        _layer("layer_decode_16", 16, graph=True),
        # a ragged continuous batch of eight conversations, uneven expert load, Q8 down weights
        _layer("layer_ragged_37", 37, dn=8, bias="normal"),
        # a wide decode batch or a short prompt: nearly every expert is touched by a few tokens
        _layer("layer_batch_150", 150),
        # a medium prompt of an odd length
        _layer("layer_prefill_777", 777),
        # a prefill chunk
        _layer("layer_prefill_4096", 4096),
        # a long prefill chunk over Zipf-popular experts, no shared expert
        _layer("layer_prefill_16384", 16384, shared=False, dn=8, bias="zipf"),
        # a prefill of a host that keeps its own call sequence and BF16 buffers
        dict(name="launchers_prefill_1200", kind="launchers", T=1200, d=4096, E=512, k=10, I=1024, gu_bits=4, dn_bits=4, bias="none"),
        # the hyper-connection mix in a decode step, replayed as a graph
        dict(name="mix_decode_16", kind="mix", T=16, d=4096, r=320, bits=8, G=64, graph=True),
        # the hyper-connection mix in a prefill chunk
        dict(name="mix_prefill_4096", kind="mix", T=4096, d=4096, r=320, bits=8, G=64, graph=False),
        # a dense projection of a small decode batch, call by call
        dict(name="dense_decode_8", kind="dense", T=8, N=8192, K=4096, bits=8, G=64, graph=False),
        # a dense projection of a prompt of an odd length
        dict(name="dense_prefill_1000", kind="dense", T=1001, N=8192, K=4096, bits=4, G=128, graph=False),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["layer", "layer", "layer", "layer", "launchers", "mix", "dense"])
    if kind == "layer":
        T = _log_int(rng, 1, 12000)
        small = T <= 300 and rng.random() < 0.2  # a small all-Q8 layer beside the full-width one
        c = _layer("", T, shared=rng.random() < 0.6, dn=rng.choice([4, 8]), bias=rng.choice(["none", "normal", "zipf"]),
                   graph=T <= 64 and rng.random() < 0.5)
        if small:
            c.update(d=1024, E=64, k=4, I=256, gu_bits=8, dn_bits=8, shared=False)
    elif kind == "launchers":
        c = dict(kind=kind, T=_log_int(rng, 256, 4096), d=4096, E=512, k=10, I=1024, gu_bits=4, dn_bits=rng.choice([4, 8]),
                 bias=rng.choice(["none", "normal"]))
    elif kind == "mix":
        T = _log_int(rng, 1, 8192)
        c = dict(kind=kind, T=T, d=rng.choice([2560, 4096]), r=320, bits=rng.choice([4, 8]), G=64, graph=T < MIX_WMMA_MIN and rng.random() < 0.5)
    else:
        T = _log_int(rng, 1, 4096)
        N, Kd = rng.choice([(8192, 4096), (4096, 4096), (2048, 4096), (4096, 1024), (2560, 4096), (4104, 2048)])
        bits = rng.choice([4, 8])
        c = dict(kind=kind, T=T, N=N, K=Kd, bits=bits, G=128 if bits == 4 else 64, graph=T < DENSE_WMMA_MIN and rng.random() < 0.5)
    c.pop("name", None)
    return c


def _gen(seed, dev):
    return torch.Generator(device=dev).manual_seed(int(seed) * 7919 + 17)


def _quantized(g, rows, cols, bits, G, std=0.02, unit=2048):
    """A [rows, cols] weight, N(0, std), quantized in slabs (the FP32 form of a whole layer's experts would not fit)."""
    q = torch.empty((rows, cols // 2 if bits == 4 else cols), dtype=torch.uint8, device=g.device)
    s = torch.empty((rows, cols // G), dtype=torch.int16, device=g.device)
    m = torch.empty_like(s)
    err = torch.zeros(4, dtype=torch.int32, device=g.device)
    slab = max(unit, (1 << 27) // cols)
    for lo in range(0, rows, slab):
        hi = min(rows, lo + slab)
        v = K.quantize(torch.randn((hi - lo, cols), generator=g, device=g.device) * std, G, bits, err=err)
        q[lo:hi], s[lo:hi], m[lo:hi] = v.q, v.scale, v.minv
    return QDeviceView(q, s, m, rows, cols, G, bits)


def _bias(c, seed):
    """Per-expert logit bias [E + 1]; the last entry belongs to the shared expert's gate."""
    g = torch.Generator().manual_seed(int(seed) * 31 + 5)
    b = torch.zeros(c["E"] + 1)
    if c["bias"] == "normal":
        b[: c["E"]] = torch.randn(c["E"], generator=g) * 0.5
    elif c["bias"] == "zipf":
        b[: c["E"]] = -1.1 * torch.log(torch.randperm(c["E"], generator=g) + 1.0)
    return b


def _captured(fn):
    """fn as a CUDA graph, after the warm-up that a capture needs."""
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        fn()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        fn()
    return graph


# ---- prepare: what a program holds before the call -----------------------------------------------------------------

def prepare(case, seed):
    state = {"layer": _prepare_block, "launchers": _prepare_block, "mix": _prepare_mix, "dense": _prepare_dense}[case["kind"]](case, seed)
    state["call"] = {"layer": _layer_call, "launchers": _launcher_calls, "mix": _mix_calls, "dense": _dense_call}[case["kind"]]
    state["graph"] = _captured(lambda: state["call"](state)) if case.get("graph") else None
    return state


def _prepare_block(c, seed):
    dev = torch.device("cuda")
    g = _gen(seed, dev)
    T, d, E, k, I = c["T"], c["d"], c["E"], c["k"], c["I"]
    G = {4: 128, 8: 64}
    w = MoeWeights(_quantized(g, E * 2 * I, d, c["gu_bits"], G[c["gu_bits"]]), _quantized(g, E * d, I, c["dn_bits"], G[c["dn_bits"]]))
    shared = c.get("shared", True)
    if shared:
        w.shared_gate_up, w.shared_down = _quantized(g, 2 * I, d, 8, 64), _quantized(g, d, I, 8, 64)
    wr = torch.randn((E + 1, d), generator=g, device=dev) * 0.02
    s = dict(T=T, d=d, E=E, k=k, I=I, w=w, wr=wr, bias=_bias(c, seed).to(dev), shared=shared,
             planes=K.router_prepare(wr, 3) if T >= ROUTER_WMMA_MIN else None,
             x=torch.randn((T, d), generator=g, device=dev).to(torch.bfloat16),
             logits=torch.empty((T, E + 1), dtype=torch.float32, device=dev), x_out=torch.empty((T, d), dtype=torch.bfloat16, device=dev))
    if c["kind"] == "layer":
        s["layer"] = MoeLayer(w, E, k, MoeBuffers(T, d, I, E, k, dev, shared))
        s["y"] = torch.empty((T, d), dtype=torch.float32, device=dev)
        return s
    bf = dict(dtype=torch.bfloat16, device=dev)
    nbytes = K.moe_route_workspace_bytes(T, k, E)
    s.update(ids=torch.empty((T, k), dtype=torch.int32, device=dev), coef=torch.empty((T, k), dtype=torch.float32, device=dev),
             ws=torch.empty(nbytes // 4, dtype=torch.int32, device=dev), ws_bytes=nbytes, h=torch.empty((T * k, I), **bf),
             partial=torch.empty((T * k, d), dtype=torch.float32, device=dev), y=torch.empty((T, d), **bf),
             sh_h=torch.empty((T, I), **bf), sh_y=torch.empty((T, d), **bf),
             router_err=torch.zeros(4, dtype=torch.int32, device=dev), expert_err=torch.zeros(4, dtype=torch.int32, device=dev))
    return s


def _prepare_mix(c, seed):
    dev = torch.device("cuda")
    g = _gen(seed, dev)
    T, d, r, H, bits, G = c["T"], c["d"], c["r"], MIX_STREAMS, c["bits"], c["G"]
    wmma = T >= MIX_WMMA_MIN
    f32 = dict(dtype=torch.float32, device=dev)
    s = dict(T=T, d=d, r=r, wmma=wmma, wd=_quantized(g, r + H, H * d, bits, G, std=0.05),
             wu=K.to_chunk_major(_quantized(g, H * d, r, bits, G, std=0.2)),
             x=torch.randn((T, H * d), generator=g, device=dev).to(torch.bfloat16),
             norm_w=torch.randn(H * d, generator=g, device=dev) * 0.1, h=torch.empty((T, r), **f32), w_in=torch.empty((T, H), **f32),
             inv=torch.empty((T, H), **f32), u=torch.empty((T, d), dtype=torch.bfloat16, device=dev))
    if wmma:
        s["ws_d"] = torch.empty(K.hc_wmma_workspace_bytes(T, H, d, r + H, bits, G), dtype=torch.uint8, device=dev)
        s["ws_u"] = torch.empty(K.hc_mix_up_wmma_workspace_bytes(T, H, d, r, bits, G), dtype=torch.uint8, device=dev)
    return s


def _prepare_dense(c, seed):
    dev = torch.device("cuda")
    g = _gen(seed, dev)
    return dict(T=c["T"], w=_quantized(g, c["N"], c["K"], c["bits"], c["G"]),
                x=torch.randn((c["T"], c["K"]), generator=g, device=dev).to(torch.bfloat16),
                y=torch.empty((c["T"], c["N"]), dtype=torch.bfloat16, device=dev))


# ---- run: one pass ---------------------------------------------------------------------------------------------------

def run(state):
    if state["graph"] is not None:
        state["graph"].replay()
        return state["out"]
    return state["call"](state)


def _logits(s):
    if s["planes"] is not None:
        K.router_logits_wmma(s["x"], s["planes"], s["bias"], s["logits"])
    else:
        K.router_logits(s["x"], s["wr"], s["bias"], s["logits"])


def _layer_call(s):
    _logits(s)
    s["layer"].forward(s["x"], s["logits"], s["y"])
    K.residual_add(s["x"], s["y"], s["x_out"])
    b = s["layer"].buf
    s["out"] = {"x": s["x_out"], "y": s["y"], "logits": s["logits"], "ids": b.ids, "coef": b.coef}
    return s["out"]


def _launcher_calls(s):
    T, E, k, w, m = s["T"], s["E"], s["k"], s["w"], MoeMath.WmmaF16
    _logits(s)
    K.moe_router(s["logits"], E + 1, T, E, k, None, 1, 0, s["ids"], s["coef"], Act.F32, s["router_err"])
    K.linear_qw_wmma_swiglu(s["x"], w.shared_gate_up, s["sh_h"], T, Act.BF16)
    K.linear_qw_wmma(s["sh_h"], w.shared_down, s["sh_y"], T, Act.BF16)
    K.moe_group_routes(s["ids"], T, k, E, s["ws"], s["ws_bytes"], s["expert_err"])
    K.linear_qw_experts_gather_grouped_swiglu(s["x"], w.gate_up, E, s["ws"], s["ws_bytes"], T, k, s["h"], Act.BF16, m)
    add = K.MoeSharedAdd(s["sh_y"], s["logits"].data_ptr() + 4 * E, E + 1, E, s["router_err"])
    K.linear_qw_experts_combine_grouped(s["h"], w.down, E, s["ids"], s["coef"], s["ws"], s["ws_bytes"], s["partial"], T, k, s["y"],
                                        Act.BF16, m, shared=add)
    K.residual_add(s["x"], s["y"], s["x_out"])
    return {"x": s["x_out"], "y": s["y"], "logits": s["logits"], "ids": s["ids"], "coef": s["coef"]}


def _mix_calls(s):
    T, d, r, H = s["T"], s["d"], s["r"], MIX_STREAMS
    if s["wmma"]:
        K.hc_mix_down_wmma(s["x"], s["wd"], T, H, d, r, True, 1e-6, s["h"], s["w_in"], s["inv"], s["ws_d"], Act.BF16)
        K.hc_mix_up_wmma(s["h"], s["wu"], s["x"], s["norm_w"], s["inv"], T, H, d, s["u"], s["ws_u"], Act.BF16)
    else:
        K.hc_mix_down(s["x"], s["wd"], T, H, d, r, True, 1e-6, s["h"], s["w_in"], s["inv"], Act.BF16)
        K.hc_mix_up(s["h"], s["wu"], s["x"], s["norm_w"], s["inv"], T, H, d, s["u"], Act.BF16)
    s["out"] = {"u": s["u"], "h": s["h"], "w_in": s["w_in"], "inv": s["inv"]}
    return s["out"]


def _dense_call(s):
    if s["T"] >= DENSE_WMMA_MIN:
        K.linear_qw_wmma(s["x"], s["w"], s["y"], s["T"], Act.BF16)
    else:
        K.linear_qw(s["x"], s["w"], s["y"], s["T"], Act.BF16)
    s["out"] = s["y"]
    return s["y"]


# ---- work and tolerance ----------------------------------------------------------------------------------------------

def _q_bytes(rows, cols, bits):
    return rows * cols * bits / 8 + 4 * rows * cols / (128 if bits == 4 else 64)


def _distinct_experts(c):
    """Experts that a pass touches: the router's draw on logits of the path's distribution, N(0, 0.02^2 d) plus the bias."""
    g = torch.Generator().manual_seed(1)
    T = min(c["T"], 4096)
    logits = torch.randn((T, c["E"]), generator=g) * (0.02 * math.sqrt(c["d"])) + _bias(c, 1)[: c["E"]]
    return int(torch.unique(logits.topk(c["k"], dim=1).indices).numel())


def work(c):
    T = c["T"]
    if c["kind"] == "dense":
        return {"bytes": c["N"] * c["K"] * c["bits"] / 8 + 4 * c["N"] * c["K"] / c["G"] + 2 * T * (c["N"] + c["K"]), "flops": 2.0 * T * c["N"] * c["K"]}
    if c["kind"] == "mix":
        n, rows = MIX_STREAMS * c["d"], 2 * c["r"] + MIX_STREAMS
        weights = rows * n * (c["bits"] / 8 + 4 / c["G"]) + 4 * n
        return {"bytes": weights + 2 * T * (n + c["d"]) + 4 * T * (c["r"] + 2 * MIX_STREAMS), "flops": 2.0 * T * n * rows}
    d, I, E, k = c["d"], c["I"], c["E"], c["k"]
    experts = _distinct_experts(c)
    b = experts * (_q_bytes(2 * I, d, c["gu_bits"]) + _q_bytes(d, I, c["dn_bits"])) + 4 * (E + 1) * (d + T)
    b += 2 * T * d * 2 + (4 if c["kind"] == "layer" else 2) * T * d + 8 * T * k  # x in and out, y, ids and coefficients
    f = 2.0 * T * (k * 3 * I * d + (E + 1) * d)
    if c.get("shared", True):
        b += _q_bytes(2 * I, d, 8) + _q_bytes(d, I, 8)
        f += 2.0 * T * 3 * I * d
    return {"bytes": b, "flops": f}


def tolerance(c):
    # BF16 (or F16) operands and BF16 intermediates; expert ids may swap where two logits tie to the last bits of an FP32 sum
    return {"rel": 1e-2, "differ": 1e-3}
