"""The work that a program has this framework do, as cases that can be timed and compared.

Hidden size 4096 with 256 filter groups, 7- and 128-tap inner filters and 16 poles is the 7B-shaped stack of
``bench.py``; 768 channels in fp32 is its configuration for the short filter.  A stack repeats (short, medium, long)
Hyena layers, so the cases that stand for a whole model run one such triple.
"""
import math

import torch
import torch.nn.functional as F

from vortex_b200 import HyenaInferenceEngine, hyena_ops
from vortex_b200.cache import HyenaCascadeFIRInferenceParams, HyenaCascadeIIRInferenceParams

BF16, F32 = "bf16", "f32"
TAPS = {"se": 7, "mr": 128}
POLES = 16
GROUP = 16                      # channels that share a filter
MOST = 131072 * 4096            # tokens x channels of the largest call
HIDDEN = (512, 768, 1024, 2048, 4096)


def listed():
    return [
        # one token of one sequence through a triple: the interactive decode step, launch and host time
        dict(name="decode_b1", path="decode", layers="se,mr,li", B=1, D=4096),
        # one token of 64 sequences: the serving decode step, every cache read and written
        dict(name="decode_b64", path="decode", layers="se,mr,li", B=64, D=4096),
        # a short prompt of ragged length prefilled through a triple, caches written
        dict(name="prompt_1003", path="fused", layers="se,mr,li", B=1, L=1003, D=4096, grouped=False),
        # batch prefill of the medium filter (the default workload of bench.py)
        dict(name="prefill_mr", path="fused", layers="mr", B=4, L=8192, D=4096, grouped=False),
        # batch prefill of the short filter, odd batch and odd length
        dict(name="prefill_se_odd", path="fused", layers="se", B=7, L=2047, D=4096, grouped=False),
        # batch prefill of the long filter with a modal system of real poles per channel
        dict(name="prefill_li", path="fused", layers="li", B=4, L=8192, D=4096, grouped=False),
        # long-context prefill of the same layer: one long sequence
        dict(name="prefill_li_long", path="fused", layers="li", B=1, L=131072, D=4096, grouped=False),
        # long-context prefill, complex poles shared by groups of 16 channels
        dict(name="prefill_li_grouped", path="fused", layers="li", B=1, L=131072, D=4096, grouped=True),
        # the engine methods that a model calls when only its engine was exchanged (featurizer, then the gated filter)
        dict(name="engine_mr", path="engine", layers="mr", B=4, L=8192, D=4096),
        # the same for a prompt of odd length through a triple, parallel_iir among it
        dict(name="engine_4001", path="engine", layers="se,mr,li", B=1, L=4001, D=4096),
        # a training step of the gate-conv-gate operator: forward, then all four gradients
        dict(name="train_gcg", path="train", B=2, L=8192, D=4096, K=128),
        # the short filter in fp32, small: fits L2, latency and one pass over memory
        dict(name="prefill_se_f32", path="f32", B=1, L=2048, D=768),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["decode", "fused", "fused", "fused", "engine", "train", "f32"])
    D = rng.choice(HIDDEN)
    layers = rng.choice(["se", "mr", "li", "se,mr,li"])
    if path == "decode":
        return dict(path=path, layers=layers, B=_log(rng, 1, 128), D=D)
    if path == "f32":
        L = _log(rng, 64, 16384)
        return dict(path=path, B=_log(rng, 1, max(1, 16384 // L)), L=L, D=768)
    top = {"fused": MOST // 3 if layers == "se,mr,li" else MOST, "engine": MOST // 16, "train": MOST // 8}[path]
    L = _log(rng, 130, min(131072, top // D))
    B = _log(rng, 1, max(1, min(32, top // D // L)))
    if path == "train":
        return dict(path=path, B=B, L=L, D=D, K=rng.choice([4, 7, 32, 128]))
    case = dict(path=path, layers=layers, B=B, L=L, D=D)
    if path == "fused":
        case["grouped"] = layers == "li" and rng.random() < 0.4
    return case


def _layer(kind, i, D, grouped, randn, rand, dt):
    """Weights of one Hyena layer as a checkpoint holds them: 3-tap featurizer, inner filter or modal system, skip."""
    c = {"kind": kind, "engine": HyenaInferenceEngine(layer_idx=i), "w3": (randn(3 * D, 1, 3) / 3 ** 0.5).to(dt)}
    if kind == "li":
        rows = D // GROUP if grouped else D
        c["kw"] = dict(log_poles=torch.log(0.9 + 0.099 * rand(rows, POLES))[..., None], residues=randn(rows, POLES),
                       D=randn(D).to(dt))
        if grouped:
            c["theta"], c["res_im"] = math.pi * rand(rows, POLES), randn(rows, POLES)
    else:
        K = TAPS[kind]
        h = randn(D // GROUP, 1, K) / K ** 0.5
        if kind == "mr":
            h = h * torch.exp(-(0.01 + 0.09 * rand(D // GROUP, 1, 1)) * torch.arange(K, device="cuda"))
        c["kw"] = dict(h=h.to(dt), D=0.5 * randn(D).to(dt) if kind == "mr" else None)
    return c


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    dt = torch.float32 if case["path"] == "f32" else torch.bfloat16
    B, D = case["B"], case["D"]

    def randn(*shape, dtype=torch.float32):
        return torch.randn(*shape, device="cuda", generator=g, dtype=dtype)

    def rand(*shape):
        return torch.rand(*shape, device="cuda", generator=g)

    s = {"case": case, "dims": (D, 1, D, POLES, D // GROUP)}
    if case["path"] == "train":
        G = D // GROUP
        s["x"], s["B"], s["C"] = (randn(B, case["L"], G, GROUP, dtype=dt).requires_grad_() for _ in range(3))
        s["dy"] = randn(B, case["L"], G, GROUP, dtype=dt)
        s["h"] = (randn(G, 1, case["K"]) / case["K"] ** 0.5).to(dt).requires_grad_()
        return s
    if case["path"] == "f32":
        s["u"] = randn(B, case["L"], 3 * D)
        s["w3"] = randn(3 * D, 1, 3) / 3 ** 0.5
        s["h"] = randn(D // GROUP, 1, 7) / 7 ** 0.5
        return s
    kinds = case["layers"].split(",")
    s["layers"] = [_layer(k, i, D, case.get("grouped", False), randn, rand, dt) for i, k in enumerate(kinds)]
    s["fir"], s["iir"] = HyenaCascadeFIRInferenceParams(), HyenaCascadeIIRInferenceParams()
    if case["path"] == "decode":
        # one projection output per layer, and the caches as earlier decode steps leave them (fp32)
        s["u"] = [randn(B, 3 * D, dtype=dt) for _ in kinds]
        for i, k in enumerate(kinds):
            (s["iir"] if k == "li" else s["fir"]).fir_state_dict[i] = randn(B, 3 * D, 2)
            if k == "li":
                s["iir"].state_dict[i] = randn(B, D, POLES)
            else:
                s["fir"].fir_inner_state_dict[i] = randn(B, D, TAPS[k] - 1)
        return s
    s["u"] = randn(B, case["L"], 3 * D, dtype=dt)
    if case["path"] == "engine":
        for c in s["layers"]:
            if c["kind"] != "li":       # the model hands the filter over with one row per channel
                c["rows"] = c["kw"]["h"].repeat_interleave(GROUP, 0)
    return s


def _decode(s):
    out = []
    for i, (c, u) in enumerate(zip(s["layers"], s["u"])):
        ip = s["iir"] if c["kind"] == "li" else s["fir"]
        out.append(c["engine"].fused_decode(u, c["w3"], None, s["dims"], ip, **c["kw"]))
        out += [ip.fir_state_dict[i], ip.state_dict[i] if c["kind"] == "li" else ip.fir_inner_state_dict[i]]
    return out


def _fused(s):
    out = []
    for i, c in enumerate(s["layers"]):
        if "theta" in c:                # complex poles: the operator's own entry point
            kw = c["kw"]
            out += hyena_ops.hyena_li_fwd(s["u"], c["w3"], None, kw["log_poles"], kw["residues"], kw["D"], theta=c["theta"],
                                          res_im=c["res_im"], want_state=True)
            continue
        ip = s["iir"] if c["kind"] == "li" else s["fir"]
        out.append(c["engine"].fused_prefill(s["u"], c["w3"], None, s["dims"], inference_params=ip, **c["kw"]))
        out += [ip.fir_state_dict[i], ip.state_dict[i] if c["kind"] == "li" else ip.fir_inner_state_dict[i]]
    return out


def _engine(s):
    out, L, G = [], s["u"].shape[1], s["case"]["D"] // GROUP
    for i, c in enumerate(s["layers"]):
        e, kw = c["engine"], c["kw"]
        z, fs = e.parallel_fir(F.conv1d, s["u"], c["w3"], None, L, dims=s["dims"], gate=False, inference_params=s["fir"])
        out += [z, fs]
        if c["kind"] == "li":
            out.append(e.parallel_iir(z, None, kw["D"], L, kw["log_poles"], kw["residues"], None, s["dims"], i,
                                      inference_params=s["iir"]))
            out.append(s["iir"].state_dict[i])
        else:
            out += e.parallel_fir(F.conv1d, z, c["rows"], kw["D"], L, dims=s["dims"], groups=G, gated_bias=c["kind"] == "mr",
                                  dim_last=False, fir_length=TAPS[c["kind"]], gate=True, inference_params=s["fir"])
    return out


def run(state):
    s = state
    path = s["case"]["path"]
    if path == "decode":
        return _decode(s)
    if path == "fused":
        return _fused(s)
    if path == "engine":
        return _engine(s)
    if path == "f32":
        return hyena_ops.hyena_se_fwd(s["u"], s["w3"], None, s["h"], layout="split", want_state=True)
    y = hyena_ops.two_pass_chunked_gate_conv_gate(s["x"], s["B"], s["C"], s["h"])
    return [y.detach(), *torch.autograd.grad(y, (s["x"], s["B"], s["C"], s["h"]), s["dy"])]


def _weights(kind, D, grouped, e):
    """Bytes of a layer's weights."""
    n = 9 * D * e
    if kind == "li":
        return n + D * e + (D // GROUP if grouped else D) * POLES * 4 * (4 if grouped else 2)
    return n + D // GROUP * TAPS[kind] * e + (D * e if kind == "mr" else 0)


def _ops(kind, grouped):
    """Operations for one sample of one channel: featurizer, two gates and the filter (a modal one as its recurrence)."""
    return 18 + 2 + (2 * TAPS[kind] + 2 if kind != "li" else (12 if grouped else 4) * POLES + 2)


def work(case):
    B, D = case["B"], case["D"]
    if case["path"] == "train":
        n = B * case["L"] * D
        # forward: x, B, C in, y out; backward: dy, x, B, C in, three gradients out
        return {"bytes": 22 * n + 4 * D // GROUP * case["K"], "flops": n * (6 * case["K"] + 8)}
    if case["path"] == "f32":
        n = B * case["L"] * D
        return {"bytes": 16 * n + 4 * B * D * 12 + _weights("se", D, False, 4), "flops": n * _ops("se", False)}
    nbytes = flops = 0
    for kind in case["layers"].split(","):
        g = case.get("grouped", False)
        inner = POLES * (2 if g else 1) if kind == "li" else TAPS[kind] - 1
        n = B * D * case.get("L", 1)
        nbytes += _weights(kind, D, g, 2)
        flops += n * _ops(kind, g)
        if case["path"] == "decode":
            nbytes += 8 * n + 2 * 4 * B * D * (6 + inner)
        else:
            # the engine's two calls hand the featurizer's output over in memory
            nbytes += (20 if case["path"] == "engine" else 8) * n + B * D * (6 * 2 + inner * (4 if kind == "li" else 2))
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # four times the distance to the same path in 64 bits.  One rounding of a bf16 result: 1.7e-3 (fused, decode); the
    # filter output rounded too (train): 2.9e-3; featurizer output, k*v and filter output rounded (engine): 4.0e-3
    return {"rel": {"f32": 1e-6, "engine": 1.6e-2, "train": 1.2e-2}.get(case["path"], 7e-3)}
