"""Tensor-level front end of the C ABI: thin argument checking, no arithmetic of its own."""
from __future__ import annotations

import ctypes

import torch

from . import _lib
from ._lib import (CODE_HASH, CODE_LITE, CODE_LUT, LAYOUT_CHUNKED, LAYOUT_ROWMAJOR, LAYOUT_TILED, LAYOUT_UNITMAJOR,
                  XORDER_NATURAL, Format, call, check, lib, ptr, native)


def _cuda_contig(t: torch.Tensor, name: str, dtype: torch.dtype | None = None) -> None:
    if not t.is_cuda:
        raise RuntimeError(f"{name} must be a CUDA tensor")
    if not t.is_contiguous():
        raise RuntimeError(f"{name} must be contiguous")
    if dtype is not None and t.dtype != dtype:
        raise RuntimeError(f"{name} must have dtype {dtype}, got {t.dtype}")


def _ld(t: torch.Tensor, width: int) -> int:
    return t.stride(0) if t.shape[0] > 1 else max(width, t.stride(0))


def units_per_row(n: int, K: int) -> int:
    if (n * K) % 128:
        raise RuntimeError(f"n*K = {n * K} bits per row is not a whole number of 128-bit units")
    return n * K // 128


def codes_shape(m: int, n: int, K: int, layout: int) -> tuple[int, ...]:
    nu = units_per_row(n, K)
    if layout == LAYOUT_ROWMAJOR:
        return (m, nu * 4)
    if layout == LAYOUT_CHUNKED:
        return (nu // 32, m, 128)
    if layout == LAYOUT_UNITMAJOR:
        return (nu, m, 4)
    return (m // 32, nu, 32, 4)


def repack(codes: torch.Tensor, src_layout: int, dst_layout: int, m: int, n_units: int) -> torch.Tensor:
    """Packed codes in `src_layout` -> a new tensor in `dst_layout` (rptc_repack)."""
    _cuda_contig(codes, "codes", torch.int32)
    if codes.numel() != m * n_units * 4:
        raise RuntimeError("codes has the wrong number of elements")
    if dst_layout == LAYOUT_ROWMAJOR:
        shape = (m, n_units * 4)
    elif dst_layout == LAYOUT_CHUNKED:
        shape = (n_units // 32, m, 128)
    elif dst_layout == LAYOUT_UNITMAJOR:
        shape = (n_units, m, 4)
    else:
        shape = (m // 32, n_units, 32, 4)
    out = torch.empty(shape, dtype=torch.int32, device=codes.device)
    call("rptc_repack", codes.device, ptr(codes), src_layout, ptr(out), dst_layout, m, n_units)
    return out


def decompress(codes: torch.Tensor, lut: torch.Tensor, m: int, n: int, fmt: Format, out: torch.Tensor | None = None,
               carry_in: torch.Tensor | None = None) -> torch.Tensor:
    """Packed codes -> dense fp16 [m, n] (rptc_decompress)."""
    if out is not None and carry_in is None:
        status = native().decompress(codes, lut, m, n, fmt, out)      # None: something is not as the kernel reads it
        if status is not None:
            check(status, "rptc_decompress")
            return out
    _cuda_contig(codes, "codes", torch.int32)
    _cuda_contig(lut, "lut", torch.float16)
    if lut.numel() != fmt.lut_numel():
        raise RuntimeError(f"lut must have {fmt.lut_numel()} elements, got {lut.numel()}")
    if codes.numel() * 32 != m * n * fmt.K:
        raise RuntimeError("codes has the wrong number of elements for m, n, K")
    if out is None:
        out = torch.empty((m, n), dtype=torch.float16, device=codes.device)
    else:
        if not out.is_cuda or out.dtype != torch.float16 or out.dim() != 2 or out.shape != (m, n) or out.stride(1) != 1:
            raise RuntimeError("out must be a CUDA fp16 [m, n] tensor with unit column stride")
    if carry_in is not None:
        _cuda_contig(carry_in, "carry_in", torch.int32)
    call("rptc_decompress", codes.device, ptr(codes), ptr(lut), ptr(carry_in), ptr(out), out.stride(0), m, n, ctypes.byref(fmt))
    return out


def check_alphabet(alphabet: torch.Tensor) -> None:
    if alphabet.dim() != 1 or alphabet.shape[0] not in [1 << L for L in range(3, 17)]:
        raise RuntimeError(f"the alphabet must be one row of 2^L entries, L = 3 to 16, got {tuple(alphabet.shape)}")


def dequantize(alphabet: torch.Tensor, symbols: torch.Tensor) -> torch.Tensor:
    """2-bit symbols int32 [rows, length] -> alphabet[state], rounded to fp16, in the alphabet's dtype (fp16 or fp32)
    (rptc_dequantize)."""
    _cuda_contig(alphabet, "alphabet")
    _cuda_contig(symbols, "symbols", torch.int32)
    if alphabet.dtype not in (torch.float16, torch.float32):
        raise RuntimeError("alphabet must be fp16 or fp32")
    check_alphabet(alphabet)
    rows, length = symbols.shape
    out = torch.empty((rows, length), dtype=alphabet.dtype, device=symbols.device)
    if out.numel():
        call("rptc_dequantize", symbols.device, alphabet.data_ptr(), symbols.data_ptr(), out.data_ptr(), int(alphabet.dtype == torch.float32), rows,
             length, alphabet.numel().bit_length() - 1)
    return out


def pack_symbols(symbols: torch.Tensor, bits: int, row_words: int) -> torch.Tensor:
    """Symbols int32 [rows, length] -> ROWMAJOR words int32 [rows, row_words], first symbol on top (rptc_pack_symbols)."""
    _cuda_contig(symbols, "symbols", torch.int32)
    rows, length = symbols.shape
    words = torch.empty((rows, row_words), dtype=torch.int32, device=symbols.device)
    call("rptc_pack_symbols", symbols.device, ptr(symbols), ptr(words), rows, length, row_words, bits)
    return words


def gemv_acc(codes: torch.Tensor, lut: torch.Tensor, x: torch.Tensor, acc: torch.Tensor, m: int, n: int, fmt: Format,
             x_order: int = XORDER_NATURAL, carry_in: torch.Tensor | None = None) -> None:
    """acc[b, :m] += W x[b]  (fp32 accumulator; rptc_gemv).  x: fp16 [b, n] or [n]."""
    _cuda_contig(codes, "codes", torch.int32)
    _cuda_contig(lut, "lut", torch.float16)
    if x.dim() == 1:
        x = x.unsqueeze(0)
    if acc.dim() == 1:
        acc = acc.unsqueeze(0)
    if not x.is_cuda or x.dtype != torch.float16 or x.stride(1) != 1 or x.shape[1] != n:
        raise RuntimeError("x must be a CUDA fp16 [batch, n] tensor with unit column stride")
    if not acc.is_cuda or acc.dtype != torch.float32 or acc.stride(1) != 1 or acc.shape[1] < m or acc.shape[0] != x.shape[0]:
        raise RuntimeError("acc must be a CUDA fp32 [batch, >=m] tensor")
    if codes.numel() * 32 != m * n * fmt.K:
        raise RuntimeError("codes has the wrong number of elements for m, n, K")
    if lut.numel() != fmt.lut_numel():
        raise RuntimeError(f"lut must have {fmt.lut_numel()} elements, got {lut.numel()}")
    call("rptc_gemv", codes.device, ptr(codes), ptr(lut), ptr(carry_in), ptr(x), x.stride(0) if x.shape[0] > 1 else max(n, x.stride(0)),
         ptr(acc), acc.stride(0) if acc.shape[0] > 1 else max(m, acc.stride(0)), m, n, x.shape[0], x_order, ctypes.byref(fmt))


def gemv_norm_input(codes: torch.Tensor, lut: torch.Tensor, acc: torch.Tensor, m: int, n: int, fmt: Format, rows: int,
                    prev_acc: torch.Tensor | None, signs_out: torch.Tensor | None, scale_out: float, h_in: torch.Tensor,
                    h_out: torch.Tensor, w_norm: torch.Tensor, eps: float, signs_in: torch.Tensor | None,
                    clear: torch.Tensor | None = None, carry_in: torch.Tensor | None = None) -> None:
    """acc += W x with x = H(s_in * rmsnorm(h_in + s_out * H(prev_acc) * scale_out) * w_norm), computed inside the
    launch; the updated residual goes to h_out (rptc_gemv_glued).  `clear` is zeroed by the launch."""
    from ._lib import GemvInput
    d = GemvInput(ptr(prev_acc), 0 if prev_acc is None else _ld(prev_acc, n), ptr(signs_out), scale_out, eps,
                  ptr(signs_in), ptr(h_in), ptr(h_out), _ld(h_in, n), ptr(w_norm), ptr(clear), 0 if clear is None else clear.numel())
    call("rptc_gemv_glued", codes.device, ptr(codes), ptr(lut), ptr(carry_in), ctypes.byref(d), ptr(acc), _ld(acc, m), m, n, rows,
         ctypes.byref(fmt))


def gemv_swiglu_input(codes: torch.Tensor, lut: torch.Tensor, acc: torch.Tensor, m: int, n: int, fmt: Format, rows: int,
                      prev_acc: torch.Tensor, signs_out: torch.Tensor | None, scale_out: float, signs_in: torch.Tensor | None,
                      block: int, clear: torch.Tensor | None = None, carry_in: torch.Tensor | None = None) -> None:
    """acc += W x with x = H(s_in * silu(g) * u), (g | u) = s_out * H(prev_acc) * scale_out, made inside the launch
    block by block (rptc_gemv_swiglu).  `clear` is zeroed by the launch."""
    call("rptc_gemv_swiglu", codes.device, ptr(codes), ptr(lut), ptr(carry_in), ptr(prev_acc), _ld(prev_acc, 2 * n), ptr(signs_out),
         scale_out, ptr(signs_in), block, ptr(acc), _ld(acc, m), m, n, rows, ctypes.byref(fmt), ptr(clear),
         0 if clear is None else clear.numel())


def gemv_finish(acc: torch.Tensor, y: torch.Tensor, m: int, scale: float = 1.0, accumulate: bool = False,
                clear: bool = True) -> None:
    """y = fp16(scale * acc) (+ y); optionally zero acc (rptc_gemv_finish)."""
    if acc.dim() == 1:
        acc = acc.unsqueeze(0)
    if y.dim() == 1:
        y = y.unsqueeze(0)
    call("rptc_gemv_finish", acc.device, ptr(acc), acc.stride(0) if acc.shape[0] > 1 else max(m, acc.stride(0)), ptr(y),
         y.stride(0) if y.shape[0] > 1 else max(m, y.stride(0)), m, acc.shape[0], scale, int(accumulate), int(clear))


def gemv(codes: torch.Tensor, lut: torch.Tensor, x: torch.Tensor, m: int, n: int, fmt: Format,
         x_order: int = XORDER_NATURAL, carry_in: torch.Tensor | None = None) -> torch.Tensor:
    """Convenience: allocate a zeroed fp32 accumulator, run the fused matvec, return fp16 [b, m]."""
    xb = x.unsqueeze(0) if x.dim() == 1 else x
    acc = torch.zeros((xb.shape[0], m), dtype=torch.float32, device=x.device)
    gemv_acc(codes, lut, xb, acc, m, n, fmt, x_order, carry_in)
    y = torch.empty((xb.shape[0], m), dtype=torch.float16, device=x.device)
    gemv_finish(acc, y, m, clear=False)
    return y[0] if x.dim() == 1 else y


def gemm(codes: torch.Tensor, lut: torch.Tensor, x: torch.Tensor, m: int, n: int, fmt: Format,
         out: torch.Tensor | None = None, carry_in: torch.Tensor | None = None, invariant: bool = False) -> torch.Tensor:
    """y[t] = W x[t] for a block of tokens on the tensor cores (rptc_gemm).  x: fp16 [tokens, n].  `invariant`: a token's
    result does not depend on the number of tokens (rptc_gemm_invariant)."""
    _cuda_contig(codes, "codes", torch.int32)
    _cuda_contig(lut, "lut", torch.float16)
    if not x.is_cuda or x.dtype != torch.float16 or x.dim() != 2 or x.stride(1) != 1 or x.shape[1] != n:
        raise RuntimeError("x must be a CUDA fp16 [tokens, n] tensor with unit column stride")
    if out is None:
        out = torch.empty((x.shape[0], m), dtype=torch.float16, device=x.device)
    call("rptc_gemm_invariant" if invariant else "rptc_gemm", codes.device, ptr(codes), ptr(lut), ptr(carry_in), ptr(x), x.stride(0), ptr(out),
         out.stride(0), m, n, x.shape[0], ctypes.byref(fmt))
    return out


def hadamard(x: torch.Tensor, signs: torch.Tensor | None, block: int, transpose: bool = False, scale: float = 1.0,
             out: torch.Tensor | None = None, clear_in: bool = False, residual: torch.Tensor | None = None) -> torch.Tensor:
    """Block-diagonal randomized Hadamard transform along the last axis (rptc_hadamard).

    x: fp16 or fp32 [rows, n]; result fp16 [rows, n] (+ residual)."""
    squeeze = x.dim() == 1
    if squeeze:
        x = x.unsqueeze(0)
    if not x.is_cuda or x.dim() != 2 or x.stride(1) != 1 or x.dtype not in (torch.float16, torch.float32):
        raise RuntimeError("x must be a CUDA fp16/fp32 [rows, n] tensor with unit column stride")
    rows, n = x.shape
    if out is None:
        out = torch.empty((rows, n), dtype=torch.float16, device=x.device)
    if signs is not None:
        _cuda_contig(signs, "signs", torch.float16)
    if residual is not None and residual.dim() == 1:
        residual = residual.unsqueeze(0)
    call("rptc_hadamard", x.device, ptr(x), int(x.dtype == torch.float32), _ld(x, n), ptr(out), _ld(out, n), ptr(signs), ptr(residual),
         0 if residual is None else _ld(residual, n), rows, n, block, int(transpose), scale, int(clear_in))
    return out[0] if squeeze else out


def swiglu_hadamard(acc: torch.Tensor, out: torch.Tensor, signs_out: torch.Tensor | None, signs_in: torch.Tensor | None,
                    n: int, block: int, scale_out: float, scale_in: float = 1.0, clear: bool = True) -> torch.Tensor:
    """Fused gated-MLP middle (rptc_swiglu_hadamard): acc fp32 [rows, 2n] -> out fp16 [rows, n]."""
    call("rptc_swiglu_hadamard", acc.device, ptr(acc), _ld(acc, 2 * n), ptr(out), _ld(out, n), ptr(signs_out), ptr(signs_in),
         acc.shape[0], n, block, scale_out, scale_in, int(clear))
    return out


def swiglu_hadamard_f16(gate_up: torch.Tensor, out: torch.Tensor, signs_out: torch.Tensor | None, signs_in: torch.Tensor | None,
                        n: int, block: int, scale_out: float, scale_in: float = 1.0) -> torch.Tensor:
    """Fused gated-MLP middle from the fp16 output of a matrix product (rptc_swiglu_hadamard_f16):
    gate_up fp16 [rows, 2n] -> out fp16 [rows, n]."""
    call("rptc_swiglu_hadamard_f16", gate_up.device, ptr(gate_up), _ld(gate_up, 2 * n), ptr(out), _ld(out, n), ptr(signs_out),
         ptr(signs_in), gate_up.shape[0], n, block, scale_out, scale_in)
    return out


def rmsnorm(x: torch.Tensor, w: torch.Tensor, out: torch.Tensor, eps: float) -> torch.Tensor:
    rows, n = x.shape
    call("rptc_rmsnorm", x.device, ptr(x), _ld(x, n), ptr(w), ptr(out), _ld(out, n), rows, n, eps)
    return out


def rope_cache(qkv: torch.Tensor, pos: torch.Tensor, kcache: torch.Tensor, vcache: torch.Tensor, hq: int, hkv: int, d: int,
               theta: float) -> None:
    rows = qkv.shape[0]
    call("rptc_rope_cache", qkv.device, ptr(qkv), _ld(qkv, qkv.shape[1]), ptr(pos), ptr(kcache), ptr(vcache), rows, hq, hkv, d,
         kcache.shape[1], theta)


def rope_cache_prompt(qkv: torch.Tensor, rows: int, tokens: int, kcache: torch.Tensor, vcache: torch.Tensor, hq: int, hkv: int, d: int,
                      theta: float) -> None:
    """RoPE of q (in place) and k, and the cache writes of k and v, for a whole prompt (rptc_rope_cache_prompt):
    qkv fp16 [rows * tokens, (hq + 2 hkv) d]."""
    call("rptc_rope_cache_prompt", qkv.device, ptr(qkv), _ld(qkv, qkv.shape[1]), rows, tokens, ptr(kcache), ptr(vcache), hq, hkv, d,
         kcache.shape[1], theta)


def rope_angles(tokens: int, theta: float, device) -> torch.Tensor:
    """Cosines and sines of positions 0 .. tokens-1 for 128-wide heads, fp32 [tokens, 64, 2] (rptc_rope_angles)."""
    out = torch.empty((tokens, 64, 2), dtype=torch.float32, device=device)
    call("rptc_rope_angles", out.device, ptr(out), tokens, theta)
    return out


def prompt_norm(y: torch.Tensor | None, signs_out: torch.Tensor | None, scale_out: float, h: torch.Tensor, w_norm: torch.Tensor, eps: float,
                signs_in: torch.Tensor | None, out: torch.Tensor) -> torch.Tensor:
    """h += output transform of the product y; out = input transform of rmsnorm(h), many rows (rptc_prompt_norm)."""
    rows, n = h.shape
    call("rptc_prompt_norm", h.device, ptr(y), 0 if y is None else _ld(y, n), ptr(signs_out), scale_out, ptr(h), _ld(h, n), ptr(w_norm), eps,
         ptr(signs_in), ptr(out), _ld(out, n), rows, n)
    return out


def prompt_qkv(qkv: torch.Tensor, signs_out: torch.Tensor | None, scale: float, rows: int, tokens: int, kcache: torch.Tensor,
               vcache: torch.Tensor, hq: int, hkv: int, angles: torch.Tensor) -> None:
    """Output transform of the fused qkv product + RoPE + cache writes for a whole prompt (rptc_prompt_qkv)."""
    call("rptc_prompt_qkv", qkv.device, ptr(qkv), _ld(qkv, qkv.shape[1]), ptr(signs_out), scale, rows, tokens, ptr(kcache), ptr(vcache), hq, hkv,
         kcache.shape[1], ptr(angles))


def attn_decode(qkv: torch.Tensor, pos: torch.Tensor, kcache: torch.Tensor, vcache: torch.Tensor, out: torch.Tensor, hq: int,
                hkv: int, d: int, signs_in: torch.Tensor | None = None) -> torch.Tensor:
    rows = qkv.shape[0]
    call("rptc_attn_decode", qkv.device, ptr(qkv), _ld(qkv, qkv.shape[1]), ptr(pos), ptr(kcache), ptr(vcache), ptr(out),
         _ld(out, out.shape[1]), rows, hq, hkv, d, kcache.shape[1], d ** -0.5, ptr(signs_in))
    return out


def qkv_attn_decode(acc: torch.Tensor, signs_out: torch.Tensor | None, scale_out: float, pos: torch.Tensor, kcache: torch.Tensor,
                    vcache: torch.Tensor, out: torch.Tensor, heads: int, kv_heads: int, theta: float,
                    signs_in: torch.Tensor | None) -> torch.Tensor:
    """Output transform of the fused qkv layer + RoPE + KV append + attention (+ per-head input transform of the
    output projection) in one launch (rptc_qkv_attn_decode)."""
    rows = acc.shape[0]
    call("rptc_qkv_attn_decode", acc.device, ptr(acc), _ld(acc, acc.shape[1]), ptr(signs_out), scale_out, ptr(pos), ptr(kcache),
         ptr(vcache), ptr(out), _ld(out, out.shape[1]), rows, heads, kv_heads, kcache.shape[1], theta, ptr(signs_in))
    return out


def finish_norm_hadamard(acc: torch.Tensor | None, signs_out: torch.Tensor | None, scale_out: float, h: torch.Tensor,
                         w_norm: torch.Tensor, eps: float, signs_in: torch.Tensor | None, transform_in: bool,
                         out: torch.Tensor) -> torch.Tensor:
    """h += output transform of acc; out = input transform of rmsnorm(h) (rptc_finish_norm_hadamard)."""
    rows, n = h.shape
    call("rptc_finish_norm_hadamard", h.device, ptr(acc), 0 if acc is None else _ld(acc, n), ptr(signs_out), scale_out, ptr(h), _ld(h, n),
         ptr(w_norm), eps, ptr(signs_in), int(transform_in), ptr(out), _ld(out, n), rows, n)
    return out


def qkv_finish(acc: torch.Tensor, signs_out: torch.Tensor | None, scale: float, q_out: torch.Tensor, kcache: torch.Tensor,
               vcache: torch.Tensor, pos: torch.Tensor, hq: int, hkv: int, block: int, theta: float) -> None:
    """Output transform of the fused qkv layer + RoPE + KV-cache append (rptc_qkv_finish)."""
    rows = acc.shape[0]
    call("rptc_qkv_finish", acc.device, ptr(acc), _ld(acc, acc.shape[1]), ptr(signs_out), scale, ptr(q_out), _ld(q_out, q_out.shape[1]),
         ptr(kcache), ptr(vcache), ptr(pos), rows, hq, hkv, kcache.shape[1], block, theta)


def dense_gemv(W: torch.Tensor, x: torch.Tensor, out: torch.Tensor | None = None) -> torch.Tensor:
    """y[b] = W x[b] for a dense fp16 W [m, n] (rptc_dense_gemv)."""
    squeeze = x.dim() == 1
    if squeeze:
        x = x.unsqueeze(0)
    m, n = W.shape
    if out is None:
        out = torch.empty((x.shape[0], m), dtype=torch.float16, device=x.device)
    o2 = out.unsqueeze(0) if out.dim() == 1 else out
    for b0 in range(0, x.shape[0], 16):                 # the kernel takes up to sixteen activation rows per launch
        xb, ob = x[b0:b0 + 16], o2[b0:b0 + 16]
        call("rptc_dense_gemv", W.device, ptr(W), W.stride(0), ptr(xb), _ld(xb, n), ptr(ob), _ld(ob, m), m, n, xb.shape[0])
    return out[0] if squeeze and out.dim() == 2 else out


def embed(table: torch.Tensor, ids: torch.Tensor, out: torch.Tensor) -> torch.Tensor:
    call("rptc_embed", table.device, ptr(table), ptr(ids), ptr(out), _ld(out, table.shape[1]), ids.shape[0], table.shape[1])
    return out


def embed_mailbox(table: torch.Tensor, slots: torch.Tensor, steps_done: torch.Tensor, ids: torch.Tensor, out: torch.Tensor,
                  timeout_ms: int = 2000) -> None:
    """Embedding rows of the ids the host posts in `slots` (pinned int64: sequence << 32 | id); waits for them, bounded
    (rptc_embed_mailbox)."""
    if not slots.is_pinned() or slots.dtype != torch.int64 or steps_done.dtype != torch.int32:
        raise RuntimeError("slots must be a pinned int64 host tensor and steps_done an int32 device tensor")
    call("rptc_embed_mailbox", table.device, ptr(table), ptr(slots), ptr(steps_done), ptr(ids), ptr(out), _ld(out, table.shape[1]),
         ids.shape[0], table.shape[1], table.shape[0], timeout_ms)


def next_token(logits: torch.Tensor, next_ids: torch.Tensor, ids: torch.Tensor | None = None, pos: torch.Tensor | None = None,
               mirror: torch.Tensor | None = None, steps_done: torch.Tensor | None = None) -> None:
    """Greedy choice + feedback + position bump in one launch (rptc_next_token).  `mirror`: pinned host int64."""
    rows, n = logits.shape
    if next_ids.dtype != torch.int64 or (mirror is not None and (mirror.dtype != torch.int64 or not mirror.is_pinned())):
        raise RuntimeError("next_ids must be int64 and mirror a pinned int64 host tensor")
    call("rptc_next_token", logits.device, ptr(logits), _ld(logits, n), rows, n, ptr(next_ids), ptr(ids), ptr(pos), ptr(mirror),
         ptr(steps_done))


def viterbi_encode(alphabet: torch.Tensor, pos_weight: torch.Tensor, samples: torch.Tensor, workspace_limit: int = 12 << 30):
    """Code-A trellis encoder on the GPU (rptc_viterbi_encode): samples fp32 [rows, n] -> (symbols int32 [rows, n],
    loss fp32 [rows])."""
    return viterbi_encode_banked(alphabet[None, :], pos_weight, samples, workspace_limit)


def quantiles(sorted_values: torch.Tensor, L: int) -> torch.Tensor:
    """2^L evenly spaced quantiles of each row of sorted fp32 values [banks, n] -> fp32 [banks, 2^L] (rptc_quantiles)."""
    _cuda_contig(sorted_values, "sorted_values", torch.float32)
    out = torch.empty((sorted_values.shape[0], 1 << L), dtype=torch.float32, device=sorted_values.device)
    call("rptc_quantiles", out.device, ptr(sorted_values), sorted_values.shape[0], sorted_values.shape[1], L, ptr(out))
    return out


def encoder_rows_at_once(L: int, n: int, sms: int, workspace_limit: int) -> int:
    """How many rows of n samples go through the encoder at once.  More than the kernel has in flight (one row per SM at L = 16, two
    at L = 15) only shorten the tail of the last ones, so beyond 4 GiB of survivor memory it is no more than those: 2.4 GB
    at L = 16 and n = 4096.  Whole sets of them, so that no launch ends with idle SMs."""
    fit = workspace_limit // lib().rptc_viterbi_workspace_bytes(1, n, L)
    flight = sms // 2 * 2 if L == 16 else 2 * sms
    most = max(flight, (4 << 30) // lib().rptc_viterbi_workspace_bytes(1, n, L))
    rows = max(1, min(65535, fit, most))
    return rows // flight * flight if rows >= flight else rows


def viterbi_encode_banked(alphabets: torch.Tensor, pos_weight: torch.Tensor, samples: torch.Tensor, workspace_limit: int = 12 << 30,
                          least_rows: int = 1):
    """The same for `alphabets` [banks, 2^L] whose banks own equal groups of consecutive rows of `samples`
    (rptc_viterbi_encode_rows).  Rows go through in batches whose survivor memory stays under `workspace_limit`
    (encoder_rows_at_once), and in smaller ones, down to `least_rows`, where the device has no room for that."""
    banks, M = alphabets.shape
    L = M.bit_length() - 1
    if M != 1 << L:
        raise RuntimeError("the alphabet must have 2^L entries")
    alphabets = alphabets.to(torch.float32).contiguous()
    pos_weight = pos_weight.to(torch.float32).contiguous()
    samples = samples.to(torch.float32).contiguous()
    rows, n = samples.shape
    if rows % banks:
        raise RuntimeError("the banks must hold equally many rows")
    symbols = torch.empty((rows, n), dtype=torch.int32, device=samples.device)
    loss = torch.empty(rows, dtype=torch.float32, device=samples.device)
    if rows == 0:
        return symbols, loss
    per_bank = rows // banks
    step = min(rows, encoder_rows_at_once(L, n, torch.cuda.get_device_properties(samples.device).multi_processor_count, workspace_limit))
    while True:
        need = lib().rptc_viterbi_workspace_bytes(step, n, L)
        try:
            ws = torch.empty(need, dtype=torch.uint8, device=samples.device)
            break
        except torch.OutOfMemoryError:
            if step <= least_rows:
                raise
            step = max(least_rows, step // 2)
    for r0 in range(0, rows, step):
        bank, inside = divmod(r0, per_bank)
        call("rptc_viterbi_encode_rows", samples.device, ptr(alphabets[bank:]), per_bank, inside, ptr(pos_weight), ptr(samples[r0:]), n,
             min(step, rows - r0), n, L, ptr(symbols[r0:]), n, ptr(loss[r0:]), ptr(ws), need)
    return symbols, loss


def device_status() -> None:
    """Raises if a kernel reported a timed-out wait since the last call."""
    check(lib().rptc_device_status(), "rptc_device_status")
