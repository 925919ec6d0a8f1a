"""The work whose speed this repository answers for, as cases that call its public entry points.

A case is a dict of plain values; `kind` names the path it takes:

  gemv     batch-1 y = W x with x, W and y on the device (`wv_matvec_dev`), one matrix after the other as a decode
           loop does it; `formats` is the list of packed formats (or FormatNone element types), `shapes` says
           whether every format also runs at the transposed shape (FFN up and down)
  batch    several activation rows against `mats` matrices of one shape, device pointers: prefill, small batches
  block    single-token decode of a stack of decoder blocks (`decode.BlockDecoder`), embedding row in, optionally the
           LM head (final norm in its prologue) and the token pick
  forward  `dense.Forward` on host arrays: the drop-in call of a host program, bias and activation included
  convert  a weight matrix on the host packed, written to the wire form, read back, made resident and dequantised

Weights are N(0, 0.02^2), activations N(0, 1), as in the repository's benchmark; inside a decoder block the activations
are what the block makes of them (heavy-tailed SwiGLU products in front of the down projection among them).
"""
from __future__ import annotations

import ctypes as C
import itertools
import math

import numpy as np
import torch

import welvet_b200 as wv
from welvet_b200 import _lib, decode, dense, quant, sampling, weights

# name -> (quant.Format value, BlockWeights, FormatNone element type)
FORMATS = {
    "Q8_0": (1, 0, 1), "Q4_0": (2, 0, 1), "Q4_1": (3, 0, 1), "Q5_0": (4, 0, 1), "Q5_1": (5, 0, 1),
    "Q2_K": (6, 0, 1), "Q3_K": (7, 0, 1), "Q4_K": (8, 0, 1), "Q5_K": (9, 0, 1), "Q6_K": (10, 0, 1),
    "IQ1_S": (11, 0, 1), "IQ2_XXS": (12, 0, 1), "IQ2_XS": (13, 0, 1), "IQ3_XXS": (14, 0, 1), "IQ3_S": (15, 0, 1),
    "IQ4_NL": (16, 0, 1), "IQ4_XS": (17, 0, 1), "TernaryPacked": (18, 0, 1), "BinaryPacked_g128": (19, 128, 1),
    "BinaryPacked_g32": (19, 32, 1), "AffinePacked_g64": (20, 64, 1), "none_f32": (0, 0, 1), "none_f16": (0, 0, 2), "none_bf16": (0, 0, 3),
}
CLASSIC = ("Q4_0", "Q4_1", "Q5_0", "Q5_1", "Q8_0", "AffinePacked_g64")
KQUANT = ("Q2_K", "Q3_K", "Q4_K", "Q5_K", "Q6_K")
SMALL = ("IQ1_S", "IQ2_XXS", "IQ2_XS", "IQ3_XXS", "IQ3_S", "IQ4_NL", "IQ4_XS", "TernaryPacked", "BinaryPacked_g128")
PLAIN = ("none_f32", "none_f16", "none_bf16")
ACTS = {"linear": dense.ActivationLinear, "silu": dense.ActivationSilu, "gelu": dense.ActivationGELU, "relu": dense.ActivationReLU}
EPS, THETA = 1e-5, 10000.0


def listed():
    return [
        # one Dense call of a host program: 4096 x 4096 in Q4_0, batch 1 (the reference's smallest configuration)
        {"name": "forward_one", "kind": "forward", "format": "Q4_0", "rows": 4096, "cols": 4096, "batch": 1, "act": "linear", "bias": False},
        # the same call with a few rows, a bias and an activation, on an FFN-wide layer
        {"name": "forward_rows", "kind": "forward", "format": "Q8_0", "rows": 14336, "cols": 4096, "batch": 8, "act": "silu", "bias": True},
        # the format sweep at the FFN shapes of an 8B model, in three families
        {"name": "gemv_classic", "kind": "gemv", "formats": ",".join(CLASSIC), "rows": 4096, "cols": 14336, "transposed": True},
        {"name": "gemv_kquant", "kind": "gemv", "formats": ",".join(KQUANT), "rows": 4096, "cols": 14336, "transposed": True},
        {"name": "gemv_small_codes", "kind": "gemv", "formats": ",".join(SMALL), "rows": 4096, "cols": 14336, "transposed": True},
        # unquantised weights, all three element types, at the attention shape
        {"name": "gemv_plain", "kind": "gemv", "formats": ",".join(PLAIN), "rows": 4096, "cols": 4096, "transposed": False},
        # a layer width that is no multiple of a quant block
        {"name": "gemv_ragged", "kind": "gemv", "formats": "Q8_0,Q4_0,Q4_K,IQ3_S", "rows": 2730, "cols": 1022, "transposed": True},
        # several rows against square matrices: speculative or small-batch decode, a short prompt, a prefill slice
        {"name": "batch_4", "kind": "batch", "format": "Q4_K", "rows": 4096, "cols": 4096, "batch": 4, "mats": 8},
        {"name": "batch_33", "kind": "batch", "format": "Q8_0", "rows": 4096, "cols": 4096, "batch": 33, "mats": 8},
        {"name": "batch_256", "kind": "batch", "format": "Q4_K", "rows": 14336, "cols": 4096, "batch": 256, "mats": 4},
        # a token through four blocks of an 8B-shaped stack at position 2048, the LM head and top-k sampling
        {"name": "decode_token", "kind": "block", "format": "Q4_K", "layers": 4, "d": 4096, "heads": 32, "kv_heads": 8, "head_dim": 128,
         "ffn": 14336, "pos": 2048, "head": "Q4_K", "vocab": 128256, "top_k": 40},
        # a checkpoint matrix (a K or V projection) packed, stored, loaded and dequantised
        {"name": "convert", "kind": "convert", "format": "Q4_K", "rows": 1024, "cols": 4096},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["forward", "gemv", "gemv", "gemv", "gemv_plain", "ragged", "batch", "batch", "block", "convert"])
    if kind == "forward":
        return {"kind": "forward", "format": rng.choice(("Q4_0", "Q8_0", "Q4_K", "Q6_K", "IQ4_XS", "none_bf16")), "rows": _log(rng, 256, 14336),
                "cols": 32 * _log(rng, 8, 256), "batch": _log(rng, 1, 16), "act": rng.choice(sorted(ACTS)), "bias": rng.random() < 0.5}
    if kind == "gemv":
        # whole quant blocks per row; rows and columns are anything else
        cols = 32 * _log(rng, 16, 512)
        names = [n for n in CLASSIC + KQUANT + SMALL if (n != "BinaryPacked_g128" or cols % 128 == 0) and (n != "AffinePacked_g64" or cols % 64 == 0)]
        return {"kind": "gemv", "formats": ",".join(rng.sample(names, rng.randint(2, 6))), "rows": _log(rng, 512, min(32768, 58720256 // cols)),
                "cols": cols, "transposed": False}
    if kind == "gemv_plain":
        return {"kind": "gemv", "formats": ",".join(rng.sample(PLAIN, rng.randint(1, 2))), "rows": _log(rng, 512, 8192), "cols": 8 * _log(rng, 64, 1024),
                "transposed": False}
    if kind == "ragged":
        cols = 2 * _log(rng, 100, 1400)
        cols += 2 if cols % 32 == 0 else 0
        names = [n for n in CLASSIC + KQUANT + SMALL if n not in ("BinaryPacked_g128", "AffinePacked_g64")]
        return {"kind": "gemv", "formats": ",".join(rng.sample(names, rng.randint(2, 4))), "rows": _log(rng, 256, 4096), "cols": cols, "transposed": False}
    if kind == "batch":
        rows, cols, batch = _log(rng, 1024, 14336), 256 * _log(rng, 4, 32), _log(rng, 2, 384)
        while rows * cols * batch > 14336 * 4096 * 256 * 2:
            batch //= 2
        return {"kind": "batch", "format": rng.choice(("Q4_K", "Q8_0", "Q4_0", "Q6_K", "Q5_1", "IQ3_S", "none_bf16") if batch <= 16 else
                                                      ("Q4_K", "Q8_0", "Q4_0", "Q6_K", "Q5_1", "IQ3_S")), "rows": rows, "cols": cols, "batch": batch, "mats": 2}
    if kind == "block":
        hd = rng.choice((64, 128))
        kv = rng.choice((4, 8))
        heads = kv * rng.choice((1, 2, 4, 8))
        return {"kind": "block", "format": rng.choice(("Q4_K", "Q8_0", "Q4_0", "Q6_K")), "layers": rng.randint(1, 3), "d": 256 * _log(rng, 4, 20),
                "heads": heads, "kv_heads": kv, "head_dim": hd, "ffn": 256 * _log(rng, 8, 56), "pos": _log(rng, 1, 12000),
                "head": rng.choice(("", "Q8_0", "Q4_K")), "vocab": _log(rng, 8000, 100000), "top_k": rng.choice((1, 20, 50))}
    return {"kind": "convert", "format": rng.choice(("Q4_K", "Q8_0", "Q4_0", "Q6_K", "IQ4_XS", "TernaryPacked")), "rows": _log(rng, 256, 2048),
            "cols": 32 * _log(rng, 8, 128)}


# ------------------------------------------------------------------ what a program has in hand
_keys = itertools.count(1 << 40)
_stream = None


def _start():
    """The library bound to the device, and the one stream all calls go to."""
    global _stream
    if _stream is None:
        torch.cuda.set_device(0)
        wv.init(0)
        _stream = torch.cuda.Stream()
    return _stream.cuda_stream


class _Resident:
    """A matrix packed on the device and kept resident until the last reference to it goes."""

    def __init__(self, name, rows, cols, gen, scale=0.02):
        fmt, bw, dt = FORMATS[name]
        self.key, self.rows, self.cols, self._evict = next(_keys), rows, cols, _lib.lib().wv_blob_evict
        w = torch.randn(rows * cols, device="cuda", generator=gen) * scale
        torch.cuda.synchronize()
        _lib.check(_lib.lib().wv_pack_upload_dev(self.key, fmt, dt, bw, w.data_ptr(), rows, cols, None))

    def __del__(self):
        self._evict(self.key)


def prepare(case, seed):
    st = _start()
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    s = _PREPARE[case["kind"]](case, gen, np.random.default_rng(seed))
    s["stream"], s["kind"] = st, case["kind"]
    torch.cuda.synchronize()
    return s


def _prepare_gemv(case, gen, rng):
    shapes = [(case["rows"], case["cols"])] + ([(case["cols"], case["rows"])] if case["transposed"] else [])
    jobs = []
    for rows, cols in shapes:
        x = torch.randn(cols, device="cuda", generator=gen)
        for f in case["formats"].split(","):
            jobs.append((_Resident(f, rows, cols, gen), x, torch.zeros(rows, device="cuda")))
    return {"jobs": jobs}


def _prepare_batch(case, gen, rng):
    x = torch.randn(case["batch"], case["cols"], device="cuda", generator=gen)
    return {"batch": case["batch"], "jobs": [(_Resident(case["format"], case["rows"], case["cols"], gen), x,
                                              torch.zeros(case["batch"], case["rows"], device="cuda")) for _ in range(case["mats"])]}


def _prepare_block(case, gen, rng):
    d, kd, f = case["d"], case["kv_heads"] * case["head_dim"], case["format"]
    msl = case["pos"] + 128
    cfg = decode.BlockConfig(d, case["heads"], case["kv_heads"], case["head_dim"], case["ffn"], msl, EPS, THETA)
    shapes = decode.projection_shapes(cfg)
    work = {"q": torch.zeros(shapes["q"][0], device="cuda"), "k": torch.zeros(kd, device="cuda"), "v": torch.zeros(kd, device="cuda"),
            "attn": torch.zeros(shapes["q"][0], device="cuda"), "ffn": torch.zeros(case["ffn"], device="cuda")}
    s = {"d": d, "pos": case["pos"], "work": work, "mats": [], "decs": [], "caches": [], "gammas": []}
    s["emb"] = _Resident("none_f32", 8, d, gen, 1.0)
    for _ in range(case["layers"]):
        mats = {n: _Resident(f, r, c, gen) for n, (r, c) in shapes.items()}
        ck, cv = (torch.randn(msl, kd, device="cuda", generator=gen) for _ in range(2))
        g1, g2 = (1 + 0.1 * torch.randn(d, device="cuda", generator=gen) for _ in range(2))
        bufs = {n: t.data_ptr() for n, t in work.items()}
        bufs.update(attn_norm=g1.data_ptr(), ffn_norm=g2.data_ptr(), cache_k=ck.data_ptr(), cache_v=cv.data_ptr())
        s["decs"].append(decode.BlockDecoder(cfg, {n: m.key for n, m in mats.items()}, bufs))
        s["mats"].append(mats)
        s["caches"] += [ck, cv]
        s["gammas"] += [g1, g2]
    s["h"] = torch.zeros(d, device="cuda")
    if case["head"]:
        s["head"] = _Resident(case["head"], case["vocab"], d, gen)
        s["vocab"], s["top_k"], s["u"] = case["vocab"], case["top_k"], float(rng.random())
        s["logits"] = torch.zeros(case["vocab"], device="cuda")
        s["gamma"] = 1 + 0.1 * torch.randn(d, device="cuda", generator=gen)
        s["head_args"] = ((C.c_uint64 * 1)(s["head"].key), (C.c_void_p * 1)(s["logits"].data_ptr()), (C.c_int * 1)(case["vocab"]))
    return s


def _prepare_forward(case, gen, rng):
    fmt, bw, dt = FORMATS[case["format"]]
    w = rng.standard_normal(case["rows"] * case["cols"], np.float32) * np.float32(0.02)
    layer = dense.NewConfigured(case["cols"], case["rows"], ACTS[case["act"]], dt, quant.Format(fmt), w, bw)
    if case["bias"]:
        layer.Weights.Bias = rng.normal(0, 0.1, case["rows"])
    quant.EnsureResident(layer.Weights.Packed)
    return {"layer": layer, "x": rng.standard_normal((case["batch"], case["cols"]), np.float32)}


def _prepare_convert(case, gen, rng):
    fmt, bw, dt = FORMATS[case["format"]]
    return {"fmt": quant.Format(fmt), "bw": bw, "dt": dt, "rows": case["rows"], "cols": case["cols"],
            "w": rng.standard_normal(case["rows"] * case["cols"], np.float32) * np.float32(0.02)}


_PREPARE = {"gemv": _prepare_gemv, "batch": _prepare_batch, "block": _prepare_block, "forward": _prepare_forward, "convert": _prepare_convert}


# ------------------------------------------------------------------ one pass
def run(s):
    return _RUN[s["kind"]](s, s["stream"])


def _run_gemv(s, st):
    L, check = _lib.lib(), _lib.check
    for m, x, y in s["jobs"]:
        check(L.wv_matvec_dev(m.key, x.data_ptr(), y.data_ptr(), 1, m.cols, m.rows, st))
    return [y for _, _, y in s["jobs"]]


def _run_batch(s, st):
    L, check, batch = _lib.lib(), _lib.check, s["batch"]
    for m, x, y in s["jobs"]:
        check(L.wv_matvec_dev(m.key, x.data_ptr(), y.data_ptr(), batch, m.cols, m.rows, st))
    return [y for _, _, y in s["jobs"]]


def _run_block(s, st):
    h = s["h"].data_ptr()
    _lib.check(_lib.lib().wv_decode_row_dev(s["emb"].key, 3, h, st))     # the token's embedding row
    for dec in s["decs"]:
        dec.step(h, s["pos"], st)
    out = {"h": s["h"], "caches": s["caches"]}
    if "head" in s:
        keys, ptrs, outs = s["head_args"]
        decode.MatVecFusedCUDA(keys, h, ptrs, s["d"], outs, dnorm_gamma=s["gamma"].data_ptr(), norm_eps=EPS, stream=st)
        # the host needs the token to go on: the one synchronisation of a decode loop
        out["token"] = sampling.SampleTopKCUDA(s["logits"].data_ptr(), s["vocab"], s["top_k"], 0.8, u=s["u"], stream=st)
        out["logits"] = s["logits"]
    return out


def _run_forward(s, st):
    pre, post = dense.Forward(s["layer"], s["x"])
    return [pre, post]


def _run_convert(s, st):
    store = weights.New(s["rows"], s["cols"], s["w"], s["dt"], s["fmt"], s["bw"])
    wire = weights.EncodePackedWire(store.Packed)
    back = weights.DecodePackedWire(s["fmt"], s["rows"], s["cols"], wire, s["dt"])
    return [back.Raw, back.Scales, back.Mins, quant.Unpack(back)]


_RUN = {"gemv": _run_gemv, "batch": _run_batch, "block": _run_block, "forward": _run_forward, "convert": _run_convert}


# ------------------------------------------------------------------ what a pass cannot do without
def _packed(name, rows, cols):
    fmt, bw, dt = FORMATS[name]
    n = [C.c_size_t() for _ in range(3)]
    _lib.check(_lib.lib().wv_pack_sizes(fmt, dt, bw, rows, cols, *(C.byref(v) for v in n)))
    return n[0].value + 4 * n[1].value + 4 * n[2].value


def work(case):
    kind = case["kind"]
    if kind == "gemv":
        r, c, names = case["rows"], case["cols"], case["formats"].split(",")
        shapes = [(r, c)] + ([(c, r)] if case["transposed"] else [])
        return {"bytes": sum(_packed(f, a, b) + 4 * (a + b) for a, b in shapes for f in names), "flops": 2 * r * c * len(shapes) * len(names)}
    if kind == "batch":
        r, c, b, m = case["rows"], case["cols"], case["batch"], case["mats"]
        return {"bytes": m * (_packed(case["format"], r, c) + 4 * b * r) + 4 * b * c, "flops": 2 * m * b * r * c}
    if kind == "forward":
        r, c, b = case["rows"], case["cols"], case["batch"]
        return {"bytes": _packed(case["format"], r, c) + 4 * b * (c + 2 * r), "flops": 2 * b * r * c}
    if kind == "convert":
        n = case["rows"] * case["cols"]
        return {"bytes": 8 * n + 2 * _packed(case["format"], case["rows"], case["cols"]), "flops": 0}
    cfg = decode.BlockConfig(case["d"], case["heads"], case["kv_heads"], case["head_dim"], case["ffn"], case["pos"] + 128)
    shapes = decode.projection_shapes(cfg).values()
    kd, qd, t = case["kv_heads"] * case["head_dim"], case["heads"] * case["head_dim"], case["pos"] + 1
    nbytes = case["layers"] * (sum(_packed(case["format"], r, c) for r, c in shapes) + 8 * t * kd)
    flops = case["layers"] * (sum(2 * r * c for r, c in shapes) + 4 * t * qd)
    if case["head"]:
        nbytes += _packed(case["head"], case["vocab"], case["d"]) + 4 * case["vocab"]
        flops += 2 * case["vocab"] * case["d"]
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """Largest relative error of a correct implementation at the precision of the path, about four times what the
    path shows against the same product in float64 over its own dequantised weights."""
    kind = case["kind"]
    if kind == "convert":
        return "exact"           # packed bytes and dequantised floats are defined bit for bit
    if kind == "block":
        return {"rel": 4e-4}     # 2e-5 per projection, through up to four blocks (measured 4e-5 .. 9e-5)
    r, c, batch, names = case["rows"], case["cols"], case.get("batch", 1), (case.get("formats") or case["format"]).split(",")
    if c % 32 or names[0].startswith("none"):
        return {"rel": 2e-6}     # float32 products and sums over the dequantised weights (measured 1e-7 .. 3e-7)
    if batch >= 6 or (batch > 1 and _packed(names[0], r, c) > 64e6):
        return {"rel": 1.2e-3}   # TF32 operands: 11 significant bits each (measured 2.9e-4)
    return {"rel": 1e-4}         # activations as 16-bit block fixed point (measured 2.1e-5)
