"""Performance cases: the calls that programs built on this package make, over the range of sizes they make them at.

Shapes come from the configurations the package carries (the 128M, 370M and 1.3B layers and LMs), the grid of
`opbench.py --sweep`, and generic short and ragged sizes.  A case is a dict of plain values:

  kind    op_forward      O = forward_raw(...): the operator without autograd (inference; `chained`: the decode-loop entry)
          op_train        O = flash_mhf(...), then the five gradients through autograd
          layer_forward   y = mhffn_layer(...) without autograd: projection, fused prologue, operator, projection
          layer_train     the same, then the gradients of x and of all parameters through autograd
          lm_forward      logits of the decoder LM around the layer, without autograd
  B, S    sequences and tokens per sequence (S = 1: one decoding step of B sequences)
  H, Hkuv, E, De, Dh     FFN heads, K/U/V heads, sub-networks per head, their width, head dimension
  bshd    op cases: Q is a [B,H,S,d_h] view of [B,S,H,d_h] memory, as a layer hands it over
  scaled  op cases: the eager layer's three constants are not 1

Everything is bf16 with fp32 routing weights, as the model runs; the float32 check mode is a test aid and not timed.
"""
import math

import torch

import flashmhf_b200 as fm

#: (H, Hkuv, E, De, Dh) of the shipped layers and of the sweep's corners.
LAYER_128M = (8, 8, 8, 256, 96)
LAYER_370M = (8, 8, 11, 256, 128)
LAYER_1P3B = (16, 16, 22, 256, 128)
SWEEP_D64 = (16, 16, 16, 192, 64)
SWEEP_D128 = (16, 16, 16, 320, 128)
SHAPES = (LAYER_128M, LAYER_370M, LAYER_1P3B, SWEEP_D64, SWEEP_D128)
MAX_FLOPS = 1.3e13   # no drawn case does more than the largest listed one


def _case(kind, B, S, shape, name=None, **more):
    H, Hkuv, E, De, Dh = shape
    c = {"kind": kind, "B": B, "S": S, "H": H, "Hkuv": Hkuv, "E": E, "De": De, "Dh": Dh}
    c.update(more)
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # one decoding step of a small batch through the small layer: the shortest call there is, latency and launches
        _case("op_forward", 8, 1, LAYER_370M, "op_decode_370m_8", chained=False, bshd=False, scaled=False),
        # one decoding step of 64 sequences in a decode loop over the 1.3B layers: bound by streaming the weights
        _case("op_forward", 64, 1, LAYER_1P3B, "op_decode_1p3b_64", chained=True, bshd=False, scaled=False),
        # prefill of one long prompt, Q as the layer's projection lays it out
        _case("op_forward", 1, 8192, LAYER_1P3B, "op_prefill_1p3b", chained=False, bshd=True, scaled=False),
        # a short ragged batch with K/U/V heads shared by two query heads and the eager layer's scaling constants
        _case("op_train", 3, 333, (8, 4, 5, 192, 128), "op_train_ragged_gqa", bshd=False, scaled=True),
        # the headline workload: the 370M layer's operator, forward and backward, at a training step's batch
        _case("op_train", 16, 2048, LAYER_370M, "op_train_370m", bshd=False, scaled=False),
        # the narrow heads of the sweep
        _case("op_train", 4, 4096, SWEEP_D64, "op_train_d64", bshd=False, scaled=False),
        # a large point of the sweep
        _case("op_train", 16, 4096, SWEEP_D128, "op_train_large", bshd=False, scaled=False),
        # the whole layer in a decoding step of the 1.3B model
        _case("layer_forward", 64, 1, LAYER_1P3B, "layer_decode_1p3b_64"),
        # the whole layer over a batch of prompts of the 128M model (96-wide heads)
        _case("layer_forward", 8, 2048, LAYER_128M, "layer_forward_128m"),
        # fine-tuning on one short sequence
        _case("layer_train", 1, 200, LAYER_128M, "layer_train_128m_short"),
        # the layer's part of a training step of the 370M model
        _case("layer_train", 4, 2048, LAYER_370M, "layer_train_370m"),
        # one request through the whole 128M model
        _case("lm_forward", 8, 2048, LAYER_128M, "lm_forward_128m"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    while True:
        kind = rng.choice(("op_forward", "op_forward", "op_train", "op_train", "layer_forward", "layer_train", "lm_forward"))
        if kind == "lm_forward":
            c = _case(kind, rng.randint(1, 8), _log_int(rng, 32, 2048), LAYER_128M)
        else:
            decode = kind.endswith("forward") and rng.random() < 0.4
            B = _log_int(rng, 1, 256) if decode else rng.randint(1, 16)
            S = 1 if decode else _log_int(rng, 40, 8192)
            H, Hkuv, E, De, Dh = rng.choice(SHAPES)
            if kind.startswith("op") and rng.random() < 0.4:      # away from the shipped layers
                Dh, De, E = rng.choice((64, 96, 128)), 64 * rng.randint(1, 6), rng.randint(1, 32)
                Hkuv = rng.choice((H, H // 2))
            c = _case(kind, B, S, (H, Hkuv, E, De, Dh))
            if kind.startswith("op"):
                c["bshd"], c["scaled"] = rng.random() < 0.5, rng.random() < 0.25
            if kind == "op_forward":
                c["chained"] = decode and rng.random() < 0.5
        if work(c)["flops"] <= MAX_FLOPS:
            return c


def _normal(g, *shape, std=1.0, dtype=torch.bfloat16):
    return torch.randn(*shape, device="cuda", generator=g).mul_(std).to(dtype)


def _op_inputs(c, g):
    B, H, S, Dh = c["B"], c["H"], c["S"], c["Dh"]
    Q = _normal(g, B, S, H, Dh).transpose(1, 2) if c["bshd"] else _normal(g, B, H, S, Dh)
    K, U, V = (_normal(g, c["Hkuv"], c["E"], c["De"], Dh, std=0.02) for _ in range(3))
    R = torch.randn(B, H, S, c["E"], device="cuda", generator=g).sigmoid_()
    return Q, K, U, V, R.div_(R.sum(-1, keepdim=True))


def _normed(c):
    """Per-head RMSNorm in front of the router and the operator: on in the 370M and 1.3B configurations, off in the 128M one."""
    return c["Dh"] != 96


def _layer_params(c, g):
    H, Hkuv, E, Dh = c["H"], c["Hkuv"], c["E"], c["Dh"]
    hid, I = H * Dh, E * c["De"]
    p = {n: _normal(g, hid, hid, std=0.02) for n in ("w_self", "w_self_2")}
    p.update({n: _normal(g, I, Hkuv * Dh, std=0.02) for n in ("gate_weight", "up_weight", "down_weight")})
    p["router"] = _normal(g, H, Dh, E, std=0.02)
    if _normed(c):
        p["q_norm"] = torch.ones(H, Dh, device="cuda", dtype=torch.bfloat16)
    return p


def prepare(case, seed):
    c, kind = case, case["kind"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    s = {"kind": kind, "case": c}
    if kind.startswith("op"):
        ins = _op_inputs(c, g)
        s["scaling"] = (math.sqrt(c["H"]), math.sqrt(c["H"]), math.sqrt(3 / 8)) if c["scaled"] else (1.0, 1.0, 1.0)
        if kind == "op_train":
            ins = tuple(t.requires_grad_(True) for t in ins)
            s["dO"] = _normal(g, c["B"], c["H"], c["S"], c["Dh"])
        s["ins"] = ins
    elif kind.startswith("layer"):
        hid = c["H"] * c["Dh"]
        s["x"], s["p"] = _normal(g, c["B"], c["S"], hid), _layer_params(c, g)
        s["kw"] = {"H": c["H"], "Hkuv": c["Hkuv"], "E": c["E"], "apply_rmsnorm": _normed(c), "eps": 1e-5}
        if kind == "layer_train":
            s["x"].requires_grad_(True)
            s["leaves"] = [s["x"]] + [t.requires_grad_(True) for t in s["p"].values()]
            s["dy"] = _normal(g, c["B"], c["S"], hid)
    else:
        from flashmhf_b200 import lm
        cfg = lm.LMConfig.lm_128m()
        with torch.device("cuda"):
            s["model"] = lm.DecoderLM(cfg).to(torch.bfloat16).init_weights(seed=seed)
        s["ids"] = torch.randint(0, cfg.vocab_size, (c["B"], c["S"]), device="cuda", generator=g)
    return s


def run(state):
    s, kind = state, state["kind"]
    if kind == "op_forward":
        return fm.forward_raw(*s["ins"], scaling=s["scaling"], chained=s["case"]["chained"])
    if kind == "op_train":
        O = fm.flash_mhf(*s["ins"], *s["scaling"])
        return (O.detach(),) + torch.autograd.grad(O, s["ins"], s["dO"])
    if kind == "layer_forward":
        with torch.no_grad():
            return fm.mhffn_layer(s["x"], s["p"], **s["kw"])
    if kind == "layer_train":
        y = fm.mhffn_layer(s["x"], s["p"], **s["kw"])
        return (y.detach(),) + torch.autograd.grad(y, s["leaves"], s["dy"])
    with torch.no_grad():
        return s["model"](s["ids"])


def work(case):
    """Forward: three products of 2*T*H*I*d_h; backward: six (a recompute of the intermediate is a choice, not counted).
    Bytes: inputs read once, outputs written once; what a layer passes between its parts is not counted."""
    c, train = case, case["kind"].endswith("train")
    H, Hkuv, E, Dh = c["H"], c["Hkuv"], c["E"], c["Dh"]
    T, I, hid = c["B"] * c["S"], c["E"] * c["De"], c["H"] * c["Dh"]
    op_flops = (18 if train else 6) * T * H * I * Dh
    w_bytes = 3 * 2 * Hkuv * I * Dh
    if c["kind"].startswith("op"):
        q, r = 2 * T * hid, 4 * T * H * E
        if train:   # Q, K, U, V, R, dO in; O, dQ, dK, dU, dV, dR out
            return {"bytes": 4 * q + 2 * r + 2 * w_bytes, "flops": op_flops}
        return {"bytes": 2 * q + r + w_bytes, "flops": op_flops}
    proj = 2 * (6 if train else 2) * T * hid * hid + (6 if train else 2) * T * hid * E
    p_bytes = w_bytes + 2 * (2 * hid * hid + H * Dh * E + hid)
    if c["kind"].startswith("layer"):
        x = 2 * T * hid
        return {"bytes": (4 * x + 2 * p_bytes) if train else (2 * x + p_bytes), "flops": op_flops + proj}
    layers, vocab = 10, 50280
    attn = 8 * T * hid * hid + 2 * T * c["S"] * hid        # four projections, causal scores and values
    return {"bytes": layers * (p_bytes + 8 * hid * hid) + 2 * vocab * hid + 2 * T * vocab + 2 * T * hid + 8 * T,
            "flops": layers * (op_flops + proj + attn) + 2 * T * hid * vocab}


def tolerance(case):
    """bf16 results of fp32 sums: 2^-9 of rounding per value, and the bf16 intermediate in front of the second product
    moves with the order of the first sum; ten layers of it for the LM."""
    return {"rel": 2e-2 if case["kind"] == "lm_forward" else 1e-2, "max": 0.25}
