"""The work whose speed is measured: what a program that uses this library has it do.

Six kinds of work, each through the public entry points:

  decode          a slice of the layers of one decode step: fb_moe_layer_decode for every layer (router, top-10, expert
                  gate/up, SwiGLU, down, combine), device tensors in and out
  decode_host     the same step with pinned host activations in and host results out, waited for in every call
  branch_decode   the whole decode branch of a layer: 513-row router, selection, shared FP8 expert, routed experts,
                  combine with the residual write
  prefill         one layer over a prompt chunk from given router logits: route, grouped gate/up, grouped down, combine
  branch_prefill  the whole prefill branch of a layer: router projection, route, shared expert, grouped GEMMs, combine
                  with the residual write
  linear          the FP8-row projection at any number of tokens (up to 16: the decode-width entry point), the same
                  projection of several layers one after another as a step has them

Every expert layer holds 512 experts of hidden size 2560, top-10; weights, routers and activations follow the
distributions of the repository's benchmark. States rotate and every layer has its own weights, so that weights
come from memory and not from the cache, as in a model that is larger than the cache.
"""
import math

import torch

from fngine_b200 import lib as L
from fngine_b200 import linear, moe, prefill, synth

H, EXPERTS, TOPK = L.HIDDEN, L.EXPERTS, L.TOPK

FORMATS = {"iq3_s": L.FMT_IQ3_S, "iq4_nl": L.FMT_IQ4_NL, "iq3_xxs": L.FMT_IQ3_XXS, "iq2_s": L.FMT_IQ2_S,
           "iq4_xs": L.FMT_IQ4_XS, "q2_0": L.FMT_Q2_0}

# gate/up format, down format, intermediate size: the two of the benchmark definition, the engine's native shape,
# and the other pairs a pack can hold (decode only)
TUNED = [("iq3_s", "iq3_s", 512), ("iq4_nl", "iq4_nl", 512), ("iq3_s", "iq4_nl", 640)]
OTHER = [("iq2_s", "iq4_nl", 640), ("iq3_xxs", "iq4_nl", 640), ("iq4_xs", "iq4_nl", 640), ("iq2_s", "q2_0", 640)]

# name: rows, k, epilogue. The projections of the engine's layers, the vocabulary matrix, the benchmark's GEMM.
PROJECTIONS = {
    "gdn_qkvz": (16384, 2560, "store_bf16"),
    "gdn_out": (2560, 6144, "gr_write"),
    "shared_gate_up": (1280, 2560, "swiglu"),
    "shared_down": (2560, 640, "shared_scale"),
    "dense_9216": (9216, 2560, "store_bf16"),
    "lm_head": (248320, 2560, "store_f32"),
}


def listed():
    return [
        # one user's token through the benchmark's layers: the smallest decode step, bound by latency and launches
        dict(name="decode_iq3s_t1", kind="decode", gate_up="iq3_s", down="iq3_s", inter=512, tokens=1, dtype="f32", layers=8),
        # a full decode batch: every layer reads some 140 experts
        dict(name="decode_iq3s_t16", kind="decode", gate_up="iq3_s", down="iq3_s", inter=512, tokens=16, dtype="f32", layers=8),
        # the IQ4_NL experts of the multi-token-prediction layer at its larger batch
        dict(name="decode_iq4nl_t8", kind="decode", gate_up="iq4_nl", down="iq4_nl", inter=512, tokens=8, dtype="f32", layers=8),
        # the pair that the reference's expert pool takes by default, an odd batch, bf16 activations
        dict(name="decode_iq2s_t5", kind="decode", gate_up="iq2_s", down="iq4_nl", inter=640, tokens=5, dtype="bf16", layers=8),
        # host buffers in and out, a wait in every call: a program that keeps its activations on the host
        dict(name="decode_host_t4", kind="decode_host", gate_up="iq3_s", down="iq3_s", inter=512, tokens=4, dtype="f32", layers=8),
        # the engine's own decode layer: native shape, shared expert beside the routed ones, residual streams
        dict(name="branch_decode_t4", kind="branch_decode", gate_up="iq3_s", down="iq4_nl", inter=640, tokens=4, layers=8),
        # the benchmark's prompt chunk with its skewed expert popularity: the largest
        dict(name="prefill_iq3s_8192", kind="prefill", gate_up="iq3_s", down="iq3_s", inter=512, tokens=8192, popularity="zipf"),
        # a short prompt, every expert hit by a token or two
        dict(name="prefill_iq4nl_96", kind="prefill", gate_up="iq4_nl", down="iq4_nl", inter=512, tokens=96, popularity="flat"),
        # an ordinary chunk of ragged length through the engine's own prefill layer
        dict(name="branch_prefill_1003", kind="branch_prefill", gate_up="iq3_s", down="iq4_nl", inter=640, tokens=1003),
        # the vocabulary projection of one token: the largest weight that decode streams
        dict(name="lm_head_t1", kind="linear", weight="lm_head", tokens=1, path="auto", layers=1),
        # the output projections of a few layers at a small batch, with the residual write
        dict(name="gdn_out_t4", kind="linear", weight="gdn_out", tokens=4, path="auto", layers=8),
        # the benchmark's dense GEMM, exact activations
        dict(name="dense_4096", kind="linear", weight="dense_9216", tokens=4096, path="auto", layers=1),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choices(["decode", "decode_host", "branch_decode", "prefill", "branch_prefill", "linear"],
                       weights=[30, 8, 10, 17, 8, 27])[0]
    case = dict(kind=kind)
    if kind == "linear":
        case["tokens"] = _log_int(rng, 1, 16) if rng.random() < 0.5 else _log_int(rng, 17, 4096)
        names = [n for n in PROJECTIONS if n != "lm_head" or case["tokens"] <= 16]
        case["weight"] = rng.choice(names)
        case["path"] = "a8" if case["tokens"] > 16 and rng.random() < 0.25 else "auto"
        case["layers"] = 1 if case["weight"] == "lm_head" or case["tokens"] > 512 else 8
        return case
    pair = rng.choice(TUNED * 2 + OTHER if kind == "decode" else TUNED)
    case["gate_up"], case["down"], case["inter"] = pair
    if kind in ("prefill", "branch_prefill"):
        case["tokens"] = _log_int(rng, 17, 8192 if kind == "prefill" and case["inter"] == 512 else 4096)
        if kind == "prefill":
            case["popularity"] = rng.choice(["zipf", "flat"])
    else:
        case["tokens"] = _log_int(rng, 1, 16)
        case["layers"] = 4 if pair in OTHER else rng.choice([4, 6, 8])
        if kind != "branch_decode":
            case["dtype"] = rng.choice(["f32", "bf16"])
    return case


# ---------------------------------------------------------------- states
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _experts(case, seed):
    return moe.synth_layer(FORMATS[case["gate_up"]], FORMATS[case["down"]], case["inter"], EXPERTS, seed)


def _router(gen, rows):
    return (torch.randn(rows, H, generator=gen, device="cuda") * 0.02).to(torch.bfloat16)


def _fp8_weight(gen, n, k):
    """Values ~ N(0,1) as E4M3 codes, one bf16 scale per row ~ U(0.001, 0.01)."""
    codes = torch.empty(n, k, dtype=torch.uint8, device="cuda")
    step = 1 << 14
    for r in range(0, n, step):
        v = torch.randn(min(step, n - r), k, generator=gen, device="cuda")
        codes[r:r + step] = v.to(torch.float8_e4m3fn).view(torch.uint8)
    scales = 0.001 + 0.009 * torch.rand(n, generator=gen, device="cuda")
    return linear.Fp8RowWeight(codes, scales.to(torch.bfloat16))


def _shared(gen, cls, *args):
    return cls(_fp8_weight(gen, 1280, H), _fp8_weight(gen, H, 640), *args)


def _prepare_decode(case, seed):
    gen = _gen(seed)
    T, n = case["tokens"], case["layers"]
    host, branch = case["kind"] == "decode_host", case["kind"] == "branch_decode"
    dt = torch.bfloat16 if branch or case["dtype"] == "bf16" else torch.float32
    layers = [_experts(case, 1000 * (seed % 1000003) + l) for l in range(n)]
    s = dict(layers=layers, ws=moe.DecodeWorkspace(layers[0]),
             routers=[_router(gen, L.ROUTER_ROWS if branch else EXPERTS) for _ in range(n)],
             x=[torch.randn(T, H, generator=gen, device="cuda").to(dt) for _ in range(n)],
             y=[torch.empty(T, H, dtype=torch.float32, device="cuda") for _ in range(n)])
    if host:
        s["x_dev"], s["y_dev"] = torch.empty_like(s["x"][0]), torch.empty_like(s["y"][0])
        s["x"] = [x.cpu().pin_memory() for x in s["x"]]
        s["y"] = [torch.empty(T, H, dtype=torch.float32).pin_memory() for _ in range(n)]
    if branch:
        s["shared"] = [_shared(gen, moe.SharedExpert) for _ in range(n)]
        s["inj"] = [torch.randn(T, 4, generator=gen, device="cuda") * 1e-6 for _ in range(n)]
        s["X0"] = torch.randn(T, 4, H, generator=gen, device="cuda")
        s["X"] = torch.empty_like(s["X0"])
        s["aux"] = torch.cuda.Stream()
    return s


def _prepare_prefill(case, seed):
    gen = _gen(seed)
    T, branch = case["tokens"], case["kind"] == "branch_prefill"
    s = dict(layer=_experts(case, seed), ws=prefill.PrefillWorkspace(T, case["inter"]),
             x=torch.randn(T, H, generator=gen, device="cuda").to(torch.bfloat16),
             y=torch.empty(T, H, dtype=torch.float32, device="cuda"))
    if branch:
        s["router"] = _router(gen, L.ROUTER_ROWS)
        s["shared"] = _shared(gen, prefill.SharedExpertPrefill, T)
        s["inj"] = torch.randn(T, 4, generator=gen, device="cuda") * 1e-6
        s["X0"] = torch.randn(T, 4, H, generator=gen, device="cuda")
        s["X"] = torch.empty_like(s["X0"])
        s["logits"] = torch.empty(T, L.ROUTER_ROWS, dtype=torch.float32, device="cuda")
    else:
        logits = (s["x"] @ _router(gen, EXPERTS).t()).float()
        if case["popularity"] == "zipf":
            logits += torch.from_numpy(synth.zipf_router_bias(seed)).cuda()
        s["logits"] = logits
    return s


def _prepare_linear(case, seed):
    gen = _gen(seed)
    T, layers = case["tokens"], case["layers"]
    n, k, kind = PROJECTIONS[case["weight"]]
    s = dict(calls=[], out=[])
    for _ in range(layers):
        w = _fp8_weight(gen, n, k)
        x = torch.randn(T, k, generator=gen, device="cuda").to(torch.bfloat16)
        if kind == "store_bf16":
            out = torch.empty(T, n, dtype=torch.bfloat16, device="cuda")
            epi = linear.store_bf16(out)
        elif kind == "store_f32":
            out = torch.empty(T, n, dtype=torch.float32, device="cuda")
            epi = linear.store_f32(out)
        elif kind == "swiglu":
            out = torch.empty(T, n // 2, dtype=torch.bfloat16, device="cuda")
            epi = linear.swiglu(out)
        elif kind == "shared_scale":
            gate = torch.randn(T, L.ROUTER_ROWS, generator=gen, device="cuda")
            out = torch.empty(T, n, dtype=torch.float32, device="cuda")
            epi = linear.shared_scale(out, gate.view(-1)[L.ROUTER_ROWS - 1:], L.ROUTER_ROWS)
        else:  # residual streams; every pass adds to them again
            out = torch.zeros(T, 4, n, dtype=torch.float32, device="cuda")
            epi = linear.gr_write(out, torch.randn(T, 4, generator=gen, device="cuda"))
        work = linear.linear_fp8_decode_workspace(w) if T <= 16 else linear.linear_fp8_workspace(w, T)
        s["calls"].append((x, w, epi, work))
        s["out"].append(out)
    s["decode"] = T <= 16
    s["path"] = L.FP8_PATH_A8 if case["path"] == "a8" else L.FP8_PATH_AUTO
    return s


def prepare(case, seed):
    if case["kind"] == "linear":
        s = _prepare_linear(case, seed)
    elif case["kind"] in ("prefill", "branch_prefill"):
        s = _prepare_prefill(case, seed)
    else:
        s = _prepare_decode(case, seed)
    s["kind"] = case["kind"]
    return s


# ---------------------------------------------------------------- one pass
def run(s):
    kind = s["kind"]
    if kind == "decode":
        for w, layer, x, y in zip(s["routers"], s["layers"], s["x"], s["y"]):
            moe.moe_layer_decode(w, layer, x, s["ws"], y)
        return s["y"]
    if kind == "decode_host":
        for w, layer, x, y in zip(s["routers"], s["layers"], s["x"], s["y"]):
            moe.moe_layer_decode_host(w, layer, x, s["ws"], s["x_dev"], s["y_dev"], y)
        return s["y"]
    if kind == "branch_decode":
        s["X"].copy_(s["X0"])  # a new step's residual streams
        for i, layer in enumerate(s["layers"]):
            moe.forward_moe_decode(s["routers"][i], s["shared"][i], layer, s["x"][i], s["ws"], s["inj"][i], s["X"],
                                   s["y"][i], aux_stream=s["aux"])
        return s["y"], s["X"]
    if kind == "prefill":
        prefill.moe_layer_prefill(s["logits"], s["layer"], s["x"], s["ws"], s["y"])
        return s["y"]
    if kind == "branch_prefill":
        s["X"].copy_(s["X0"])  # a new chunk's residual streams
        prefill.forward_moe_prefill(s["router"], s["shared"], s["layer"], s["x"], s["ws"], s["inj"], s["X"], s["logits"],
                                    s["y"])
        return s["y"], s["X"]
    for x, w, epi, work in s["calls"]:
        if s["decode"]:
            linear.linear_fp8_decode(x, w, epi, work)
        else:
            linear.linear_fp8(x, w, epi, work, path=s["path"])
    return s["out"]


# ---------------------------------------------------------------- what a pass cannot do without
def _distinct_experts(tokens, popularity="flat"):
    """Expected number of distinct experts that `tokens` tokens choose."""
    if popularity == "flat":
        return EXPERTS * (1.0 - (1.0 - TOPK / EXPERTS) ** tokens)
    p = [(r + 1.0) ** -1.1 for r in range(EXPERTS)]
    z = TOPK / sum(p)
    return sum(1.0 - (1.0 - min(1.0, z * v)) ** tokens for v in p)


def work(case):
    T = case["tokens"]
    if case["kind"] == "linear":
        n, k, kind = PROJECTIONS[case["weight"]]
        out = {"store_bf16": 2 * n, "store_f32": 4 * n, "swiglu": n, "shared_scale": 4 * n, "gr_write": 2 * 16 * n}[kind]
        return {"bytes": case["layers"] * (n * k + 2 * n + T * (2 * k + out)), "flops": case["layers"] * 2.0 * T * n * k}
    inter = case["inter"]
    blob = synth.blob_bytes(FORMATS[case["gate_up"]], FORMATS[case["down"]], inter)
    flops = 2.0 * T * TOPK * 3 * H * inter
    x_bytes = 4 if case.get("dtype") == "f32" else 2
    nbytes = _distinct_experts(T, case.get("popularity", "flat")) * blob + T * H * (x_bytes + 4)
    if case["kind"] == "prefill":
        nbytes += T * EXPERTS * 4
    else:
        nbytes += EXPERTS * H * 2
        flops += 2.0 * T * EXPERTS * H
    if case["kind"] in ("branch_decode", "branch_prefill"):
        nbytes += 3 * 640 * H + T * 4 * H * 8
        flops += 2.0 * T * 3 * 640 * H
    return {"bytes": case.get("layers", 1) * nbytes, "flops": case.get("layers", 1) * flops}


def tolerance(case):
    if case["kind"] == "linear":
        if case["path"] == "a8":
            return {"rel": 1e-2}  # a token's E4M3 codes may round the other way at a tie
        kind = PROJECTIONS[case["weight"]][2]
        if kind in ("store_bf16", "swiglu"):
            return {"rel": 1e-2}  # bf16 results
        # fp32 results: the decode-width path keeps the activations whole, the wide one to 2^-17 of a row's maximum
        return {"rel": 1e-5 if case["tokens"] <= 16 else 1e-4}
    if case["kind"] in ("prefill", "branch_prefill"):
        return {"rel": 5e-3}  # bf16 weights, activations and intermediate rows
    return {"rel": 1e-3}  # 8-bit activations: a code of h may round the other way
