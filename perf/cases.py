"""Performance cases of the W4A8 library: what a serving program has it do, through its public entry points.

Every case is a dict of plain values; "kind" says which calls one pass makes:

  norm_quantize   RMSNorm + activation quantizer of the S rows a decode step holds (launch_rmsnorm_quantize_x_q8)
  quantize        activation quantizer alone, over a prefill's rows (launch_quantize_x_q8)
  linear          quantize + product of S rows with `layers` matrices one after the other (linear): decode for S <= 16,
                  prefill / verify above
  mlp             one MLP block: norm + quantize, gate and up sharing the quantized rows, activation + quantize, down
  layer           the matrices of one transformer layer back to back: QKV, O, gate, up, down
  splitk          quantize + split-K product for a verify step's few dozen rows (launch_gemm_bm16_splitk)
  moe             routed-expert MLP block (moe_block)

The path is inference only: it has no backward.  scale_dtype is 0 for fp32 group scales, 1 for fp16.
"""
import importlib
import math

import torch
import torch.nn.functional as F

w4a8 = importlib.import_module("dgx-serving_b200")

EPS = 1e-6
DEV = "cuda"


def listed():
    return [
        # one decode token entering a layer: the smallest call, launch and latency only
        {"name": "norm_quantize_1", "kind": "norm_quantize", "S": 1, "K": 5120},
        # the quantizer over a long prompt, memory traffic only
        {"name": "quantize_8192", "kind": "quantize", "S": 8192, "K": 5120},
        # single-stream decode of the 27B-class gate/up shape; several layers' matrices so that none stays in L2
        {"name": "linear_1", "kind": "linear", "S": 1, "K": 5120, "N": 17408, "layers": 4, "scale_dtype": 0},
        # the vocabulary projection of one decode token, fp16 scales
        {"name": "lm_head_1", "kind": "linear", "S": 1, "K": 5120, "N": 151936, "layers": 1, "scale_dtype": 1},
        # a whole MLP block of single-stream decode
        {"name": "mlp_decode_1", "kind": "mlp", "S": 1, "K": 5120, "N": 17408, "act": 0, "scale_dtype": 0},
        # batched decode through the matrices of a 12B-class layer
        {"name": "layer_decode_8", "kind": "layer", "S": 8, "K": 3840, "QKV": 4096, "N": 15360, "scale_dtype": 0},
        # the widest batch the decode path takes, fp16 scales
        {"name": "linear_16", "kind": "linear", "S": 16, "K": 5120, "N": 17408, "layers": 3, "scale_dtype": 1},
        # a speculative-decoding verify step: few rows, long K, K split over the SMs
        {"name": "splitk_48", "kind": "splitk", "S": 48, "K": 15360, "N": 3840, "splitk": 0, "layers": 2, "scale_dtype": 0},
        # a short prompt of ragged length, fp16 scales
        {"name": "linear_333", "kind": "linear", "S": 333, "K": 3840, "N": 15360, "layers": 1, "scale_dtype": 1},
        # a prefill chunk of the 27B-class gate/up shape
        {"name": "linear_2048", "kind": "linear", "S": 2048, "K": 5120, "N": 17408, "layers": 1, "scale_dtype": 0},
        # routed experts of a 35B-A3B-class block: batched decode and a prefill chunk
        {"name": "moe_8", "kind": "moe", "S": 8, "K": 2048, "N": 768, "experts": 128, "topk": 8, "act": 0, "scale_dtype": 0},
        {"name": "moe_512", "kind": "moe", "S": 512, "K": 2048, "N": 768, "experts": 128, "topk": 8, "act": 0, "scale_dtype": 0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _k(rng, lo, hi):
    return max(lo, 32 * (_log(rng, lo, hi) // 32))


def draw(rng):
    kind = rng.choice(["norm_quantize", "quantize", "decode", "decode", "prefill", "prefill", "mlp", "layer", "splitk", "moe"])
    sd = rng.choice([0, 1])
    if kind == "norm_quantize":
        return {"kind": kind, "S": _log(rng, 1, 64), "K": _k(rng, 2048, 17408)}
    if kind == "quantize":
        return {"kind": kind, "S": _log(rng, 64, 8192), "K": _k(rng, 2048, 5120)}
    if kind == "decode":
        return {"kind": "linear", "S": _log(rng, 1, 16), "K": _k(rng, 2048, 15360), "N": _log(rng, 2048, 20000), "layers": 3, "scale_dtype": sd}
    if kind == "prefill":
        return {"kind": "linear", "S": _log(rng, 17, 2048), "K": _k(rng, 2048, 5120), "N": _log(rng, 2048, 17408), "layers": 1, "scale_dtype": sd}
    if kind == "mlp":
        return {"kind": kind, "S": _log(rng, 1, 512), "K": _k(rng, 2048, 5120), "N": _k(rng, 4096, 17408), "act": rng.choice([0, 1]), "scale_dtype": sd}
    if kind == "layer":
        return {"kind": kind, "S": _log(rng, 1, 16), "K": _k(rng, 2048, 5120), "QKV": _log(rng, 2048, 8192), "N": _k(rng, 4096, 15360), "scale_dtype": sd}
    if kind == "splitk":
        return {"kind": kind, "S": _log(rng, 17, 96), "K": _k(rng, 3840, 17408), "N": _log(rng, 1024, 5120), "splitk": rng.choice([0, 2, 4]), "layers": 2, "scale_dtype": sd}
    return {"kind": "moe", "S": _log(rng, 1, 512), "K": 2048, "N": 768, "experts": rng.choice([64, 128]), "topk": rng.choice([4, 8]), "act": rng.choice([0, 1]), "scale_dtype": sd}


# ---- inputs ----------------------------------------------------------------------------------------------------------
def _gen(seed, salt=0):
    return torch.Generator(device=DEV).manual_seed((int(seed) * 1000003 + salt) % (1 << 62))


def _weights(g, n, k, sd, gain=1.0):
    """Packed int4 weights, every nibble uniform, and group scales |N(0, 0.02)|/7."""
    wq = torch.empty((n, k // 2), dtype=torch.uint8, device=DEV).random_(0, 256, generator=g)
    sw = torch.empty((n, k // 32), dtype=torch.float32, device=DEV).normal_(0.0, 0.02, generator=g).abs_().mul_(gain / 7.0)
    return wq, (sw.half() if sd else sw)


def _rows(g, s, k, outliers=False):
    x = torch.empty((s, k), dtype=torch.float32, device=DEV).normal_(generator=g)
    if outliers:                       # prefill activations: 1 % of the entries are 20 times larger
        x = torch.where(torch.empty_like(x).uniform_(generator=g) < 0.01, x * 20.0, x)
    return x


class _Quant:
    """Scratch of one quantized activation matrix."""

    def __init__(self, s, k):
        self.xq = torch.empty((s, k), dtype=torch.int8, device=DEV)
        self.xs = torch.empty((s, k // 32), dtype=torch.float32, device=DEV)
        self.xsum = torch.empty((s, k // 32), dtype=torch.int32, device=DEV)


def _f32(*shape):
    return torch.empty(shape, dtype=torch.float32, device=DEV)


def _inputs(c, seed):
    """Everything random of a case, from its seed alone (prepare and exact share it)."""
    kind, s, k = c["kind"], c["S"], c["K"]
    g = _gen(seed)
    st = {"x": _rows(g, s, k, outliers=s > 16)}
    sd = c.get("scale_dtype", 0)
    if kind in ("norm_quantize", "mlp"):
        st["w"] = _f32(k).normal_(1.0, 0.1, generator=g)
    if kind in ("linear", "splitk"):
        st["mats"] = [_weights(g, c["N"], k, sd) for _ in range(c["layers"])]
    elif kind == "mlp":               # scales of the first two products such that gate and up have a spread near 1
        gain = 4.4 * math.sqrt(1.0 / k) * 7.0 / 0.02 / 8.0 * 1.2
        st["mats"] = [_weights(g, c["N"], k, sd, gain), _weights(g, c["N"], k, sd, gain), _weights(g, k, c["N"], sd)]
    elif kind == "layer":
        st["mats"] = [_weights(g, n, kk, sd) for n, kk in _layer_shapes(c)]
        st["xo"], st["xd"] = _rows(g, s, k), _rows(g, s, c["N"])
    elif kind == "moe":
        e, topk, mi = c["experts"], c["topk"], c["N"]
        gain = 4.4 * math.sqrt(1.0 / k) * 7.0 / 0.02 / 8.0 * 1.2
        st["gu"] = _weights(g, e * 2 * mi, k, sd, gain)
        st["dn"] = _weights(g, e * k, mi, sd, gain)
        score = torch.empty((s, e), device=DEV).normal_(generator=g)
        val, idx = score.topk(topk, dim=1)
        st["idx"], st["dw"] = idx.to(torch.int32).reshape(-1).contiguous(), torch.softmax(val, dim=1).reshape(-1).contiguous()
    return st


def _layer_shapes(c):
    """(rows, K) of QKV, O, gate, up, down."""
    return [(c["QKV"], c["K"]), (c["K"], c["K"]), (c["N"], c["K"]), (c["N"], c["K"]), (c["K"], c["N"])]


def prepare(case, seed):
    c = dict(case)
    kind, s, k = c["kind"], c["S"], c["K"]
    st = _inputs(c, seed)
    st["c"] = c
    if kind != "moe":
        st["q"] = _Quant(s, k)
    if kind in ("linear", "splitk"):
        st["y"] = [_f32(s, c["N"]) for _ in st["mats"]]
    if kind == "splitk":
        st["ws"] = torch.empty(max(16, w4a8.gemm_splitk_workspace_bytes(s, c["N"], k, c["splitk"])), dtype=torch.uint8, device=DEV)
    elif kind == "mlp":
        st["qh"] = _Quant(s, c["N"])
        st["g"], st["u"], st["y"] = _f32(s, c["N"]), _f32(s, c["N"]), _f32(s, k)
    elif kind == "layer":
        st["qd"] = _Quant(s, c["N"])
        st["y"] = [_f32(s, n) for n, _ in _layer_shapes(c)]
    elif kind == "moe":
        st["ws"] = torch.empty(w4a8.moe_layout_for(s, c["topk"], k, c["N"], c["experts"]).bytes, dtype=torch.uint8, device=DEV)
        st["y"] = _f32(s, k)
    return st


def run(st):
    c = st["c"]
    kind, s, k, sd = c["kind"], c["S"], c["K"], c.get("scale_dtype", 0)
    if kind == "moe":
        w4a8.moe_block(st["x"], st["gu"][0], st["gu"][1], st["dn"][0], st["dn"][1], st["idx"], st["dw"], st["y"], s, c["topk"], k, c["N"],
                       c["experts"], st["ws"], sd, c["act"])
        return st["y"]
    q = st["q"]
    if kind == "norm_quantize":
        w4a8.launch_rmsnorm_quantize_x_q8(st["x"], st["w"], EPS, 0, None, q.xq, q.xs, q.xsum, k, s)
        return {"xq": q.xq, "xs": q.xs, "xsum": q.xsum}
    if kind == "quantize":
        w4a8.launch_quantize_x_q8(st["x"], q.xq, q.xs, q.xsum, k, s)
        return {"xq": q.xq, "xs": q.xs, "xsum": q.xsum}
    if kind == "linear":
        for (wq, sw), y in zip(st["mats"], st["y"]):
            w4a8.linear(st["x"], q.xq, q.xs, q.xsum, wq, sw, y, s, c["N"], k, sd)
        return st["y"]
    if kind == "splitk":
        w4a8.launch_quantize_x_q8(st["x"], q.xq, q.xs, q.xsum, k, s)
        for (wq, sw), y in zip(st["mats"], st["y"]):
            w4a8.launch_gemm_bm16_splitk(q.xq, q.xs, wq, sw, y, s, c["N"], k, sd, c["splitk"], st["ws"])
        return st["y"]
    if kind == "mlp":
        (wg, sg), (wu, su), (wd, sdn) = st["mats"]
        qh = st["qh"]
        w4a8.launch_rmsnorm_quantize_x_q8(st["x"], st["w"], EPS, 0, None, q.xq, q.xs, q.xsum, k, s)
        if s <= 16:
            w4a8.gemv_multi(q.xq, q.xs, [wg, wu], [sg, su], [st["g"], st["u"]], [c["N"], c["N"]], k, s, sd)
        else:
            w4a8.launch_gemm_mmq_w4a8(q.xq, q.xs, wg, sg, st["g"], s, c["N"], k, sd)
            w4a8.launch_gemm_mmq_w4a8(q.xq, q.xs, wu, su, st["u"], s, c["N"], k, sd)
        w4a8.launch_glu_quantize_x_q8(st["g"], st["u"], c["act"], None, qh.xq, qh.xs, qh.xsum, c["N"], s)
        w4a8.linear(None, qh.xq, qh.xs, qh.xsum, wd, sdn, st["y"], s, k, c["N"], sd, 1)
        return {"gate": st["g"], "up": st["u"], "out": st["y"]}
    # layer: QKV and gate/up share one quantized input each; the attention between the products is not this library's
    qd, y, m, shapes = st["qd"], st["y"], st["mats"], _layer_shapes(c)
    w4a8.linear(st["x"], q.xq, q.xs, q.xsum, m[0][0], m[0][1], y[0], s, shapes[0][0], k, sd)
    w4a8.linear(st["xo"], q.xq, q.xs, q.xsum, m[1][0], m[1][1], y[1], s, k, k, sd)
    w4a8.launch_quantize_x_q8(st["x"], q.xq, q.xs, q.xsum, k, s)
    w4a8.gemv_multi(q.xq, q.xs, [m[2][0], m[3][0]], [m[2][1], m[3][1]], [y[2], y[3]], [c["N"], c["N"]], k, s, sd)
    w4a8.linear(st["xd"], qd.xq, qd.xs, qd.xsum, m[4][0], m[4][1], y[4], s, k, c["N"], sd)
    return y


# ---- what a pass cannot do without -----------------------------------------------------------------------------------
def _matrix(n, k, sd):
    return n * (k // 2) + n * (k // 32) * (2 if sd else 4)


def work(case):
    c = case
    kind, s, k, sd = c["kind"], c["S"], c["K"], c.get("scale_dtype", 0)
    x, q = 4 * s * k, s * k + 8 * s * (k // 32)
    if kind in ("norm_quantize", "quantize"):
        return {"bytes": x + q + (4 * k if kind == "norm_quantize" else 0), "flops": 6.0 * s * k}
    if kind in ("linear", "splitk"):
        return {"bytes": x + c["layers"] * (_matrix(c["N"], k, sd) + 4 * s * c["N"]), "flops": 2.0 * s * c["N"] * k * c["layers"]}
    if kind == "mlp":
        return {"bytes": x + 4 * k + 2 * _matrix(c["N"], k, sd) + _matrix(k, c["N"], sd) + 4 * s * (2 * c["N"] + k), "flops": 6.0 * s * c["N"] * k}
    if kind == "layer":
        sh = _layer_shapes(c)
        return {"bytes": 2 * x + 4 * s * c["N"] + sum(_matrix(n, kk, sd) + 4 * s * n for n, kk in sh), "flops": sum(2.0 * s * n * kk for n, kk in sh)}
    slots = s * c["topk"]
    touched = c["experts"] * (1.0 - (1.0 - c["topk"] / c["experts"]) ** s)          # expected number of experts with a token
    return {"bytes": 2 * x + 8 * slots + touched * (_matrix(2 * c["N"], k, sd) + _matrix(k, c["N"], sd)), "flops": 6.0 * slots * c["N"] * k}


def tolerance(case):
    kind = case["kind"]
    if kind == "quantize":            # one division and one rounding per element: nothing to differ in
        return "exact"
    if kind == "norm_quantize":       # the norm's sum of squares in another order moves a value across a rounding tie
        return {"rel": 1e-6, "max": 1e-5, "differ": 1e-4}
    if kind in ("linear", "layer", "splitk"):       # fp32 sums of K/32 scaled group dots in another order
        return {"rel": 2e-6, "max": 2e-5}
    # two products with a quantizer between them: where the first one's fp32 sums are taken in another order, a value near
    # a rounding tie of the int8 grid moves by a whole step
    return {"rel": 4e-4, "max": 2e-2}


# ---- 64-bit reference --------------------------------------------------------------------------------------------------
def _quantized(x32):
    """The int8 grid of fp32 rows (the quantizer is part of the operation, so in its own precision), back in 64 bits."""
    s, k = x32.shape
    b = x32.reshape(s, k // 32, 32)
    m = b.abs().amax(dim=2, keepdim=True)
    d = m / torch.full_like(m, 127.0)              # a true division: torch multiplies by 1/127 for a plain number
    q = torch.where(d > 0, torch.round(b / torch.where(d > 0, d, torch.ones_like(d))), torch.zeros_like(b)).clamp_(-127, 127)
    return q, d


def _dequantized(x32):
    q, d = _quantized(x32)
    return (q.double() * d.double()).reshape(x32.shape)


def _product(xd, wq, sw):
    """xd[S,K] in 64 bits times the packed matrix, in slices of rows."""
    n, k = wq.shape[0], wq.shape[1] * 2
    out = torch.empty((xd.shape[0], n), dtype=torch.float64, device=DEV)
    for r in range(0, n, 16384):
        w = wq[r:r + 16384]
        v = torch.stack([w & 15, w >> 4], dim=2).reshape(-1, k // 32, 32).to(torch.float64) - 8.0
        v = (v * sw[r:r + 16384].double().unsqueeze(2)).reshape(-1, k)
        out[:, r:r + 16384] = xd @ v.t()
    return out


def _act(g, u, act):
    return (F.gelu(g, approximate="tanh") if act else F.silu(g)) * u


def exact(case, seed):
    c = dict(case)
    kind, s = c["kind"], c["S"]
    st = _inputs(c, seed)
    if kind in ("norm_quantize", "quantize"):
        x = st["x"]
        if kind == "norm_quantize":
            x = x.double()
            x = x * torch.rsqrt(x.square().mean(dim=1, keepdim=True) + EPS) * st["w"].double()
        d = x.double().reshape(s, c["K"] // 32, 32).abs().amax(dim=2) / 127.0
        return {"xq": None, "xs": d, "xsum": None}
    if kind in ("linear", "splitk"):
        xd = _dequantized(st["x"])
        return [_product(xd, *m) for m in st["mats"]]
    if kind == "mlp":
        x = st["x"].double()
        x = (x * torch.rsqrt(x.square().mean(dim=1, keepdim=True) + EPS) * st["w"].double()).float()
        xd = _dequantized(x)
        g, u = _product(xd, *st["mats"][0]), _product(xd, *st["mats"][1])
        return {"gate": g, "up": u, "out": _product(_dequantized(_act(g, u, c["act"]).float()), *st["mats"][2])}
    if kind == "layer":
        xd, xo, xdn = _dequantized(st["x"]), _dequantized(st["xo"]), _dequantized(st["xd"])
        return [_product(r, *m) for r, m in zip((xd, xo, xd, xd, xdn), st["mats"])]
    xd, mi, k, topk = _dequantized(st["x"]), c["N"], c["K"], c["topk"]
    out = torch.zeros((s, k), dtype=torch.float64, device=DEV)
    idx, dw = st["idx"].reshape(s, topk), st["dw"].reshape(s, topk).double()
    for e in range(c["experts"]):
        t, j = torch.nonzero(idx == e, as_tuple=True)
        if t.numel() == 0:
            continue
        gu = _product(xd[t], st["gu"][0][e * 2 * mi:(e + 1) * 2 * mi], st["gu"][1][e * 2 * mi:(e + 1) * 2 * mi])
        h = _dequantized(_act(gu[:, :mi], gu[:, mi:], c["act"]).float())
        out.index_add_(0, t, _product(h, st["dn"][0][e * k:(e + 1) * k], st["dn"][1][e * k:(e + 1) * k]) * dw[t, j].unsqueeze(1))
    return out
