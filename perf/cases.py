"""The work whose speed counts: calls a program makes through this package's public entry points.

Every case is one call (or one kind of call) of the emulated FP8 GEMM. The listed cases are this repository's own
configurations -- the 256-cube of the ada profile, decode steps of 16 rows, tall-skinny mixed-format shapes, the
4096-cube, the FP8 projection stack, a slab of the sharded problem with special codes -- and, for what those leave out,
generic shapes: ragged sizes, FP8 output, `accumulate` with a K that is no multiple of 16, operands in host memory.
`draw` gives calls of the same kinds over the whole range of sizes. Results are bit-exact by definition of the
framework: the tolerance is "exact" everywhere.
"""
from __future__ import annotations

import math
import warnings

import torch

import mmaemu_b200 as mm

_FP8 = {"e4m3": torch.float8_e4m3fn, "e5m2": torch.float8_e5m2}
_OUT = {"float32": torch.float32, "bfloat16": torch.bfloat16, "float16": torch.float16,
        "float8_e4m3fn": torch.float8_e4m3fn, "float8_e5m2": torch.float8_e5m2}
_OUT_BYTES = {"float32": 4, "bfloat16": 2, "float16": 2, "float8_e4m3fn": 1, "float8_e5m2": 1}

# the largest listed case, in multiply-accumulates; drawn cases stay below it (kinds that run slower per product lower)
_MOST = 8192 * 24576 * 8192
_DRAW_MOST = {"scaled_mm": _MOST // 8, "quantized": _MOST // 16, "host": _MOST // 16, "accumulate": _MOST // 64}


def _case(entry, profile, M, N, K, fa="e4m3", fb="e4m3", out="bfloat16", fast=False, splits=1, scheme="none",
          sigma=4.0, special=False, name=None):
    """splits: 0 = the profile's split-K table decides ("auto"), 1 = unsplit, else (splits, scheme)."""
    c = {"entry": entry, "profile": profile, "M": M, "N": N, "K": K, "fa": fa, "fb": fb, "out": out, "fast": fast,
         "splits": splits, "scheme": scheme, "sigma": sigma, "special": special}
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # a small layer, or a unit test of a model: launches and host work count
        _case("scaled_mm", "ada", 256, 256, 256, splits=0, sigma=2.0, name="small_256_ada"),
        # one decode step of a served model: 16 sequences, a projection of 4096 columns
        _case("scaled_mm", "hopper", 16, 4096, 8192, fa="e5m2", splits=0, sigma=8.0, name="decode_16x4096x8192"),
        # the same through a wide down projection, where cuBLASLt splits K in two
        _case("scaled_mm", "hopper-te", 16, 8192, 28672, fa="e5m2", splits=0, sigma=8.0, name="decode_16x8192x28672_split"),
        # a short prefill with fast accumulation: one chain over K per output and few output tiles
        _case("scaled_mm", "hopper", 64, 4096, 4096, fast=True, name="prefill_64x4096x4096_fast"),
        # tall-skinny, activations in E5M2, fp32 out (a gradient-like product)
        _case("scaled_mm", "hopper", 128, 4096, 16384, fa="e5m2", out="float32", splits=0, sigma=8.0, name="tall_128x4096x16384_f32"),
        # sizes that fill no tile, E4M3 x E5M2, E4M3 out with a result scale, the ada profile with slow accumulation
        _case("scaled_mm", "ada", 1000, 2064, 1936, fb="e5m2", out="float8_e4m3fn", sigma=2.0, name="ragged_1000x2064x1936_f8"),
        # fp32 accumulators of operands of any size: K is no multiple of 16
        _case("accumulate", "hopper", 517, 1003, 2001, out="float32", sigma=2.0, name="accumulate_517x1003x2001"),
        # the headline workload of the benchmark
        _case("scaled_mm", "hopper", 4096, 4096, 4096, name="cube_4096"),
        # the same from and to host memory
        _case("host", "hopper", 4096, 4096, 4096, name="host_cube_4096"),
        # projection stack: bf16 activations of 8192 tokens quantised inside the call, fused QKV weights
        _case("quantized", "hopper-te", 8192, 5760, 1920, fast=True, splits=0, name="projection_8192x5760x1920"),
        # one GPU's rows of the sharded problem: saturated, subnormal and NaN codes, fp16 out
        _case("scaled_mm", "ada", 2048, 16384, 8192, out="float16", fast=True, sigma=16.0, special=True, name="slab_2048x16384x8192_ada"),
        # the projection stack at the largest width (operands quantised with an amax-derived scale: the full E4M3 range)
        _case("scaled_mm", "hopper-te", 8192, 24576, 8192, fast=True, splits=0, sigma=80.0, name="projection_8192x24576x8192"),
    ]


def _log_int(rng, lo, hi, step=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(step, int(round(v / step)) * step)


def draw(rng):
    entry = rng.choices(("scaled_mm", "quantized", "accumulate", "host"), (12, 2, 2, 2))[0]
    most = _DRAW_MOST[entry]
    while True:
        if entry == "scaled_mm" and rng.random() < 0.35:
            M = rng.randint(1, 16)                                   # decode steps
            N, K = _log_int(rng, 256, 16384, 16), _log_int(rng, 512, 32768, 16)
        else:
            M, N, K = _log_int(rng, 16, 8192), _log_int(rng, 64, 24576, 16), _log_int(rng, 128, 16384, 16)
        if entry == "accumulate":
            N, K = max(1, N - rng.randint(0, 15)), K - rng.randint(0, 31)
        if entry == "quantized":
            M = max(M, 64)
        if M * N * K <= most:
            break
    profile = rng.choice(("hopper", "hopper", "hopper-te", "ada", "ada-te"))
    fa, fb = ("e4m3", "e4m3") if entry == "quantized" or rng.random() < 0.5 else rng.choice((("e5m2", "e4m3"), ("e4m3", "e5m2")))
    out = "float32" if entry == "accumulate" else rng.choice(("bfloat16", "bfloat16", "bfloat16", "float32", "float16", "float8_e4m3fn"))
    splits, scheme = 1, "none"
    if entry == "scaled_mm" and M <= 256 and K >= 2048 and rng.random() < 0.4:
        splits = rng.randint(2, 8)
        scheme = "contiguous" if profile.startswith("hopper") else rng.choice(("serial", "pairwise"))
    sigma = rng.choice((1.0, 2.0, 4.0, 8.0, 16.0))
    return _case(entry, profile, M, N, K, fa, fb, out, rng.random() < 0.5, splits, scheme, sigma,
                 entry == "scaled_mm" and rng.random() < 0.2)


def _codes(rows, K, fmt, sigma, special, g):
    """Gaussian operands in FP8; `special`: 1 % of the codes subnormal or +-largest, a NaN code in 1 % of the rows."""
    x = (torch.randn(rows, K, generator=g, device="cuda") * sigma).clamp(-448.0, 448.0).to(_FP8[fmt])
    if special:
        u = x.view(torch.uint8)
        pick = torch.rand(rows, K, generator=g, device="cuda")
        values = torch.tensor([0x01, 0x83, 0x7E, 0xFE] if fmt == "e4m3" else [0x01, 0x82, 0x7B, 0xFB], dtype=torch.uint8, device="cuda")
        which = torch.randint(0, 4, (rows, K), generator=g, device="cuda")
        u.copy_(torch.where(pick < 0.01, values[which], u))
        n = max(1, rows // 100)
        r = torch.randperm(rows, generator=g, device="cuda")[:n]
        u[r, torch.randint(0, K, (n,), generator=g, device="cuda")] = 0x7F
    return x


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    M, N, K, s = case["M"], case["N"], case["K"], case["sigma"]
    warnings.simplefilter("ignore", mm.UnverifiedSplitWarning)       # the drawn splits need not be recorded ones
    warnings.simplefilter("ignore", mm.UnvalidatedEnvelopeWarning)
    kw = {"use_fast_accum": case["fast"], "profile": case["profile"],
          "splitk": "auto" if case["splits"] == 0 else (1 if case["splits"] == 1 else (case["splits"], case["scheme"]))}
    st = {"entry": case["entry"], "kw": kw}
    scales = torch.exp2(torch.rand(2, generator=g, device="cuda") * 4 - 2)
    if case["entry"] == "quantized":
        x = torch.randn(M, K, generator=g, device="cuda")
        w = torch.randn(N, K, generator=g, device="cuda") * 0.02
        qx, qw = 448.0 / x.abs().max(), 448.0 / w.abs().max()
        st.update(x=x.to(torch.bfloat16), quant_scale=qx.reshape(1), sa=(1.0 / qx).reshape(1), sb=(1.0 / qw).reshape(1),
                  b=(w * qw).clamp(-448, 448).to(torch.float8_e4m3fn).t())
    else:
        st.update(a=_codes(M, K, case["fa"], s, case["special"], g), sa=scales[0].reshape(1), sb=scales[1].reshape(1))
        b = _codes(N, K, case["fb"], s, case["special"], g)
        st["b"] = b if case["entry"] == "accumulate" else b.t()
    if case["entry"] == "accumulate":
        return st
    kw["out_dtype"] = _OUT[case["out"]]
    if case["out"].startswith("float8"):
        kw["scale_result"] = (2.0 ** -5 / scales.prod()).reshape(1)
    if case["entry"] == "host":
        st["a"] = st["a"].cpu().pin_memory()
        st["b"] = b.cpu().pin_memory().t()
        st.update(sa=st["sa"].cpu(), sb=st["sb"].cpu())
        if "scale_result" in kw:
            kw["scale_result"] = kw["scale_result"].cpu()
        kw["out"] = torch.empty(M, N, dtype=kw["out_dtype"], pin_memory=True)
    return st


def run(state):
    entry, kw = state["entry"], state["kw"]
    if entry == "scaled_mm":
        return mm.scaled_mm(state["a"], state["b"], state["sa"], state["sb"], **kw)
    if entry == "quantized":
        return mm.quantized_scaled_mm(state["x"], state["quant_scale"], state["b"], state["sa"], state["sb"], **kw)
    if entry == "accumulate":
        return mm.accumulate(state["a"], state["b"], **kw)
    return mm.scaled_mm_host(state["a"], state["b"], state["sa"], state["sb"], **kw)


def work(case):
    M, N, K = case["M"], case["N"], case["K"]
    a_bytes = 2 if case["entry"] == "quantized" else 1               # bf16 activations or FP8 codes
    return {"bytes": M * K * a_bytes + N * K + M * N * _OUT_BYTES[case["out"]], "flops": 2 * M * N * K}


def tolerance(case):
    return "exact"
