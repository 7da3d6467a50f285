"""The work that users of this framework have it do, as cases that can be timed and compared.

Every case calls public entry points only: the quantised layers (`RPTCLinear`, `FactorizedRPTCLinear`), the decoder model
(`RPTCLlama.step` / `prefill`), the drop-in functions of `rptc_kernels`, the decoders (`ops.decompress`,
`rptc.dequantize`) and the encoder behind layer quantisation (`quantize_hf.round_weights`).  A case is a dict of plain
values whose `kind` names the path.  Layer shapes are those of the Llama-2-7B and 70B shapes that this repository's
benchmark and tests use; drawn cases spread over the ranges around them, odd sizes included.
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.abspath("let-it-slide_b200"))      # the package folder of the tree this runs in

import quantize_hf  # noqa: E402
import rptc  # noqa: E402
import rptc_kernels  # noqa: E402
from rptc_b200 import (CODE_HASH, CODE_LITE, CODE_LUT, LAYOUT_ROWMAJOR, LAYOUT_TILED, LAYOUT_UNITMAJOR,  # noqa: E402
                       Format, ops)
from rptc_b200.linear import RPTCLinear  # noqa: E402
from rptc_b200.llama import LlamaConfig, RPTCLlama  # noqa: E402

CODES = {"hash": CODE_HASH, "lut": CODE_LUT, "lite": CODE_LITE}
LAYOUTS = {"rowmajor": LAYOUT_ROWMAJOR, "unitmajor": LAYOUT_UNITMAJOR, "tiled": LAYOUT_TILED}


def listed():
    seven_b = dict(hidden=4096, layers=32, heads=32, kv_heads=32, ffn=11008, vocab=32000)
    return [
        # one token through one attention projection: the smallest call of the quantised layer, host and launches count
        dict(name="linear_t1", kind="linear", m=4096, n=4096, tokens=1, code="hash", K=2),
        # eight sequences decoded together, the widest layer of a block (gate and up fused)
        dict(name="linear_t8", kind="linear", m=22016, n=4096, tokens=8, code="hash", K=2),
        # a prompt of ordinary length through the down projection: few tiles of work, a long reduction
        dict(name="linear_t512", kind="linear", m=4096, n=11008, tokens=512, code="hash", K=2),
        # the layer that quantize_hf swaps into a Hugging Face model: the gate projection (344 rows per bank, not a
        # multiple of a row block) for one token of generation ...
        dict(name="packed_t1", kind="packed", m=11008, n=4096, tokens=1, L=16, banks=32, dtype="float16"),
        # ... and an attention projection for a short prompt
        dict(name="packed_t256", kind="packed", m=4096, n=4096, tokens=256, L=16, banks=32, dtype="float16"),
        # the drop-in function of the reference extension, as its tests call it
        dict(name="dropin_matvec", kind="dropin", fn="matvec_16_8", m=4096, n=4096),
        # packed weights expanded to dense fp16 (before a library GEMM, or to inspect them): the largest layer
        dict(name="decompress", kind="decompress", m=8192, n=28672, code="lut", K=3, L=16, S=0, layout="tiled"),
        # symbols of a quantised matrix back to weights, the reference's `dequantize`
        dict(name="dequantize", kind="dequantize", rows=4096, length=4096, L=16),
        # the encoder while a layer is quantised: one alphabet per bank of rows, the row batches of the driver's default
        dict(name="encode", kind="encode", m=1024, n=1024, L=16, banks=32, batch=8),
        # generation, batch 1, the headline shape: a continuation of eight tokens behind a 128-token prompt
        dict(name="decode_b1", kind="decode", rows=1, context=128, steps=8, **seven_b),
        # sixteen sequences at once
        dict(name="decode_b16", kind="decode", rows=16, context=128, steps=4, **seven_b),
        # a long prompt through the whole model: the largest pass
        dict(name="prefill_2048", kind="prefill", rows=1, tokens=2048, **seven_b),
    ]


# ---- drawn cases ---------------------------------------------------------------------------------------------------
def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _mult(rng, lo, hi, step):
    """A multiple of `step` between lo and hi, spread over the logarithm."""
    return min(hi // step, max(-(-lo // step), round(_log(rng, lo, hi) / step))) * step


def _shape(rng, most):
    """Heads, MLP width and depth of a model of at most `most` block weights: hidden sizes of the tests and the benchmark."""
    while True:
        hidden = rng.choice([512, 1024, 2048, 4096, 4096, 8192])
        heads = hidden // 128
        kv_heads = rng.choice([h for h in (heads, heads // 4, heads // 8) if h >= 1])
        ffn = _mult(rng, 2 * hidden, 4 * hidden, 256)
        layers = 2 * round(_log(rng, 1, 16))
        vocab = rng.choice([1024, 8000, 32000])
        if layers * hidden * (2 * hidden + 2 * kv_heads * 128 + 3 * ffn) <= most:
            return dict(hidden=hidden, layers=layers, heads=heads, kv_heads=kv_heads, ffn=ffn, vocab=vocab)


def draw(rng):
    kind = rng.choice(["linear", "linear", "linear", "packed", "packed", "dropin", "decompress", "dequantize", "encode",
                       "decode", "decode", "prefill"])
    if kind == "linear":
        tokens = round(_log(rng, 1, 2048)) if rng.random() < 0.7 else rng.randint(1, 16)
        code, K = rng.choice([("hash", 2)] * 4 + [("lut", 2), ("lut", 4), ("lite", 2), ("lite", 4)])
        return dict(kind=kind, m=_mult(rng, 1024, 28672, 256), n=_mult(rng, 1024, 14336, 256), tokens=tokens, code=code, K=K)
    if kind == "packed":
        banks = rng.choice([8, 16, 32])
        per_bank = rng.choice([_mult(rng, 32, 11008 // banks, 8), _mult(rng, 128, max(128, 11008 // banks), 128)])
        return dict(kind=kind, m=banks * per_bank, n=_mult(rng, 512, 11008, 64), tokens=round(_log(rng, 1, 512)),
                    L=rng.choice([12, 14, 16, 16]), banks=banks, dtype=rng.choice(["float16", "float32", "bfloat16"]))
    if kind == "dropin":
        fn = rng.choice(["matvec_16_8", "matvec_16_6", "matvec_t_16", "matvec_t_14", "decompress"])
        return dict(kind=kind, fn=fn, m=_mult(rng, 1024, 16384, 32), n=_mult(rng, 2048, 16384, 64 if "_t_" in fn or fn == "decompress" else 2048))
    if kind == "decompress":
        code, K = rng.choice([("lut", 2), ("lut", 3), ("lut", 4), ("hash", 2), ("lite", 2), ("lite", 4)])
        layout = rng.choice(["tiled", "tiled", "rowmajor", "unitmajor"])
        return dict(kind=kind, m=_mult(rng, 1024, 8192, 32), n=_mult(rng, 1024, 28672, 128), code=code, K=K,
                    L=rng.choice([14, 16, 16]) if code == "lut" else 16, S=0 if code == "lut" else 8, layout=layout)
    if kind == "dequantize":
        return dict(kind=kind, rows=round(_log(rng, 1, 4096)), length=round(_log(rng, 100, 8192)), L=rng.randint(8, 16))
    if kind == "encode":
        banks = rng.choice([8, 16, 32])
        m = banks * 8 * rng.randint(1, 1024 // (banks * 8))
        return dict(kind=kind, m=m, n=round(_log(rng, 64, 1024 * 1024 // m)) if m > 128 else round(_log(rng, 64, 4096)),
                    L=rng.randint(8, 16), banks=banks, batch=8)
    if kind == "decode":
        shape = _shape(rng, 6.4e9)
        rows = rng.choice([1, 1, 1, 2, 4, rng.randint(1, 16), 16])
        return dict(kind=kind, rows=rows, context=round(_log(rng, 16, 1000)), steps=4, **shape)
    tokens = round(_log(rng, 16, 2048))
    return dict(kind=kind, rows=rng.choice([1, 1, min(4, 2048 // tokens)]), tokens=tokens, **_shape(rng, 6.4e9))


# ---- what a user's program has in hand -------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _words(g, shape):
    """Packed codes: every bit stream is a valid trellis path, so uniform words are a quantised weight matrix."""
    return torch.randint(-2**31, 2**31 - 1, shape, dtype=torch.int32, device="cuda", generator=g)


def _alphabet(g, L):
    """2^L Gaussian quantiles in a random order, fp32: the codebook of the table code."""
    M = 1 << L
    q = (2 * torch.arange(M, dtype=torch.float64, device="cuda") + 1) / (2 * M)
    return (math.sqrt(2.0) * torch.erfinv(2 * q - 1))[torch.randperm(M, generator=g, device="cuda")].float()


def _codebook(g, code, L, S):
    return _alphabet(g, L).half() if code == "lut" else torch.randn(2 << S, generator=g, device="cuda").half()


def _config(case, max_pos):
    return LlamaConfig(max_pos=max_pos, **{k: case[k] for k in ("hidden", "layers", "heads", "kv_heads", "ffn", "vocab")})


def prepare(case, seed):
    kind, g = case["kind"], _gen(seed)
    s = {"case": case}
    if kind == "linear":
        code, K = case["code"], case["K"]
        fmt = Format(CODES[code], K, 16, 0 if code == "lut" else 8, LAYOUT_TILED)
        s["layer"] = RPTCLinear.random(case["n"], case["m"], fmt, 0.02, seed)
        s["x"] = torch.randn(case["tokens"], case["n"], generator=g, device="cuda").half()
    elif kind == "packed":
        m, n, banks = case["m"], case["n"], case["banks"]
        symbols = torch.randint(0, 4, (m, n), dtype=torch.int32, device="cuda", generator=g)
        alphabets = torch.stack([_alphabet(g, case["L"]) for _ in range(banks)])
        s["layer"] = quantize_hf.FactorizedRPTCLinear.from_parts(
            symbols, alphabets, 0.001 * torch.randn(m, generator=g, device="cuda"), 0.001 * torch.randn(n, generator=g, device="cuda"),
            0.02 * (0.5 + torch.rand(m, generator=g, device="cuda")), 0.5 + torch.rand(n, generator=g, device="cuda"))
        s["x"] = torch.randn(case["tokens"], n, generator=g, device="cuda").to(getattr(torch, case["dtype"]))
    elif kind == "dropin":
        m, n, fn = case["m"], case["n"], case["fn"]
        s["x"] = torch.randn(n, generator=g, device="cuda").half()
        if fn == "decompress":
            s["fn"], L = rptc_kernels.decompress, 16
            s["codes"], s["out"] = _words(g, (m, n // 16)), torch.empty((m, n), dtype=torch.float16, device="cuda")
        elif "_t_" in fn:
            s["fn"], L = getattr(rptc_kernels, "decompress_" + fn), int(fn[-2:])
            s["codes"], s["out"] = _words(g, (n // 64, m, 4)), torch.zeros(m, dtype=torch.float16, device="cuda")
        else:
            s["fn"], L = getattr(rptc_kernels, "decompress_" + fn + "_1"), None
            s["codes"], s["out"] = _words(g, (n // 2048, m, 128)), torch.empty(m, dtype=torch.float16, device="cuda")
        s["lut"] = _codebook(g, "hash", 16, int(fn[-1])) if L is None else _codebook(g, "lut", L, 0)
    elif kind == "decompress":
        s["fmt"] = Format(CODES[case["code"]], case["K"], case["L"], case["S"], LAYOUTS[case["layout"]])
        s["codes"] = _words(g, (case["m"] * case["n"] * case["K"] // 32,))
        s["lut"] = _codebook(g, case["code"], case["L"], case["S"])
        s["out"] = torch.empty((case["m"], case["n"]), dtype=torch.float16, device="cuda")
    elif kind == "dequantize":
        s["symbols"] = torch.randint(0, 4, (case["rows"], case["length"]), dtype=torch.int32, device="cuda", generator=g)
        s["alphabet"] = _alphabet(g, case["L"])
    elif kind == "encode":
        s["weights"] = torch.randn(case["m"], case["n"], generator=g, device="cuda")
        s["importance"] = 0.5 + torch.rand(case["n"], generator=g, device="cuda")
        order = torch.randperm(1 << case["L"], generator=g, device="cuda")
        s["permute"] = lambda alphabet: alphabet[order]
    else:
        rows = case["rows"]
        length = case["context"] + case["steps"] if kind == "decode" else case["tokens"]
        model = RPTCLlama(_config(case, length), rows=rows, seed=seed % 9973)
        tokens = torch.randint(0, case["vocab"], (rows, length), generator=g, device="cuda", dtype=torch.int32)
        s["model"] = model
        if kind == "prefill":
            s["tokens"] = tokens
        else:                                   # the prompt is in the caches, the step is captured, the continuation is known
            model.prefill(tokens[:, : case["context"]])
            model.capture()
            s["start"] = torch.full((rows,), case["context"], dtype=torch.int32, device="cuda")
            s["next"] = tokens[:, case["context"]:].t().contiguous()
            s["logits"] = torch.empty((case["steps"], rows, case["vocab"]), dtype=torch.float16, device="cuda")
    return s


# ---- one pass --------------------------------------------------------------------------------------------------------
@torch.no_grad()
def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind in ("linear", "packed"):
        return s["layer"](s["x"])
    if kind == "dropin":
        if case["fn"] == "decompress":
            s["fn"](s["codes"], s["lut"], s["out"])
        else:
            if "_t_" in case["fn"]:
                s["out"].zero_()                # this function adds into its output
            s["fn"](s["codes"], s["lut"], s["x"], s["out"])
        return s["out"]
    if kind == "decompress":
        return ops.decompress(s["codes"], s["lut"], case["m"], case["n"], s["fmt"], out=s["out"])
    if kind == "dequantize":
        return rptc.dequantize(s["alphabet"], s["symbols"])
    if kind == "encode":
        return quantize_hf.round_weights(s["permute"], s["weights"], s["importance"], case["L"], case["banks"], case["batch"])
    model = s["model"]
    if kind == "prefill":
        return model.prefill(s["tokens"])
    # Scores a given continuation of the cached prompt: back to the end of the prompt, then token by token, keeping the
    # logits of every position.
    model.reset()
    model.pos.copy_(s["start"])
    for ids, out in zip(s["next"], s["logits"]):
        model.ids.copy_(ids)
        model.step()
        out.copy_(model.logits)
    return s["logits"]


# ---- what a pass cannot do without -----------------------------------------------------------------------------------
def _block_weights(case):
    q, kv = case["heads"] * 128, case["kv_heads"] * 128
    return case["layers"] * (case["hidden"] * (q + 2 * kv) + q * case["hidden"] + 3 * case["hidden"] * case["ffn"])


def work(case):
    kind = case["kind"]
    if kind == "linear":
        m, n, t = case["m"], case["n"], case["tokens"]
        table = 2 << 16 if case["code"] == "lut" else 4 << 8
        return {"bytes": m * n * case["K"] / 8 + table + 2 * (m + n) + 2 * t * (m + n), "flops": 2 * t * m * n}
    if kind == "packed":
        m, n, t = case["m"], case["n"], case["tokens"]
        width = 4 if case["dtype"] == "float32" else 2
        return {"bytes": m * n / 4 + case["banks"] * (2 << case["L"]) + 8 * (m + n) + width * t * (m + n), "flops": 2 * t * m * n}
    if kind == "dropin":
        m, n = case["m"], case["n"]
        if case["fn"] == "decompress":
            return {"bytes": m * n / 4 + 2 * m * n + (2 << 16), "flops": 0}
        table = 2 << int(case["fn"][-2:]) if "_t_" in case["fn"] else 4 << int(case["fn"][-1])
        return {"bytes": m * n / 4 + table + 2 * n + 2 * m, "flops": 2 * m * n}
    if kind == "decompress":
        m, n = case["m"], case["n"]
        return {"bytes": m * n * case["K"] / 8 + 2 * m * n + (2 << case["L"] if case["code"] == "lut" else 4 << case["S"]), "flops": 0}
    if kind == "dequantize":
        return {"bytes": 8 * case["rows"] * case["length"] + (4 << case["L"]), "flops": 0}
    if kind == "encode":
        # per row, position and state: one difference, two products, one sum, and a quarter of three comparisons
        m, n = case["m"], case["n"]
        return {"bytes": 8 * m * n + case["banks"] * (4 << case["L"]), "flops": m * n * (1 << case["L"]) * 4.75}
    w, rows, hidden, vocab = _block_weights(case), case["rows"], case["hidden"], case["vocab"]
    kv_row = 4 * case["layers"] * case["kv_heads"] * 128             # bytes of one position's keys and values
    head = 2 * vocab * hidden
    if kind == "decode":
        mid = case["context"] + case["steps"] / 2
        step = w / 4 + head + rows * (kv_row * (mid + 1) + 2 * hidden + 2 * vocab)
        flops = 2 * rows * (w + vocab * hidden) + 4 * rows * case["layers"] * case["heads"] * 128 * mid
        return {"bytes": case["steps"] * step, "flops": case["steps"] * flops}
    t = case["tokens"]
    return {"bytes": w / 4 + head + rows * t * (kv_row + 2 * hidden) + 2 * rows * vocab,
            "flops": rows * (2 * t * w + 2 * case["layers"] * case["heads"] * 128 * t * t + 2 * vocab * hidden)}


def tolerance(case):
    kind = case["kind"]
    if kind in ("decompress", "dequantize", "encode") or case.get("fn") == "decompress":
        return "exact"                                               # a decode selects table entries; the encoder's fp32 steps are fixed
    if kind in ("decode", "prefill"):
        return {"rel": 2e-2}                                         # every layer stores fp16 activations
    if kind == "packed" and case["dtype"] == "bfloat16":
        return {"rel": 5e-3}
    return {"rel": 2e-3}                                             # fp16 operands and results, fp32 sums
