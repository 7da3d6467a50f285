"""GPU parity of the fused dequant-GEMM (tcgen05): against the product of the bit-exact decoded
weights (checked against the CPU oracle) with the same activations.

Two kinds of check.  Exact: with the identity matrix as activations every output is one weight plus zeros, so the
product must equal the decoded matrix bit for bit, for every column of every BASELINE shape (a mis-decoded weight at
a producer-group, k-step or tile boundary cannot hide).  Random inputs: fp16 operands, fp32 accumulation in TMEM, one
rounding to fp16 -> |y - exact| <= 2^-11 |exact| + 2e-5 * ||w_row|| * ||x_t|| (0.08 absolute at n = 4096 with N(0,1)
data, where one wrong weight moves an output by about 1)."""
import numpy as np
import pytest
import torch

import rptc_oracle as o
from gpu_util import GEMV_FP32_TOL, assert_same_bits, lut_for_oracle, rand_lut, rand_words, to_dev

pytestmark = pytest.mark.gpu


def _run(code, K, L, S, m, n, tokens, seed=0, check_oracle=True):
    from rptc_b200 import Format, ops
    rng = np.random.default_rng(seed)
    w = rand_words(rng, m, n, K)
    lut = rand_lut(rng, code, L, S)
    fmt = Format(code, K, L, S, o.LAYOUT_TILED)
    codes = to_dev(o.from_rowmajor(w, o.LAYOUT_TILED))
    lut_d = to_dev(lut)
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn((tokens, n), dtype=torch.float16, device="cuda", generator=g)
    y = ops.gemm(codes, lut_d, x, m, n, fmt)
    torch.cuda.synchronize()
    ops.device_status()
    dense = ops.decompress(codes, lut_d, m, n, fmt)
    if check_oracle:
        ref_w = o.decode(w[:32], lut_for_oracle(lut, code, S), n, code=code, K=K, L=L, S=S)
        assert np.array_equal(dense[:32].cpu().numpy().view(np.uint16), ref_w.view(np.uint16))
    exact = x.double() @ dense.double().t()
    scale = x.double().norm(dim=1)[:, None] * dense.double().norm(dim=1)[None, :]
    err = (y.double() - exact).abs()
    tol = 2.0**-11 * exact.abs() + GEMV_FP32_TOL * scale + 1e-4
    worst = (err / tol).max().item()
    print(f"gemm {m}x{n}x{tokens}: max err {err.max().item():.4g}, max err/tol {worst:.3f}")
    assert worst <= 1.0, f"max err/tol {worst:.3f}"


@pytest.mark.parametrize("m,n,tokens", [(128, 64, 256), (128, 512, 256), (256, 4096, 512), (128, 1024, 100), (384, 2048, 300)])
def test_gemm_hash_small(m, n, tokens):
    _run(o.CODE_B, 2, 16, 8, m, n, tokens, seed=m + n + tokens)


@pytest.mark.parametrize("code,K,L,S", [(o.CODE_A, 2, 16, 0), (o.CODE_A, 4, 16, 0), (o.CODE_A, 2, 14, 0), (o.CODE_B, 2, 16, 6),
                                        (o.CODE_C, 2, 16, 9), (o.CODE_C, 4, 16, 9)])
def test_gemm_all_codes(code, K, L, S):
    _run(code, K, L, S, 256, 2048, 384, seed=code * 7 + K)


@pytest.mark.parametrize("m,n,tokens", [(4096, 4096, 2048), (22016, 4096, 512), (4096, 11008, 512)])
def test_gemm_llama_shapes(m, n, tokens):
    _run(o.CODE_B, 2, 16, 8, m, n, tokens, seed=3, check_oracle=False)


@pytest.mark.parametrize("m,n", [(4096, 4096), (11008, 4096), (4096, 11008), (28672, 8192), (384, 2048)])
def test_gemm_identity_activations_give_the_decoded_matrix_bit_for_bit(m, n):
    from rptc_b200 import Format, ops
    fmt = Format()
    g = torch.Generator(device="cuda").manual_seed(m + n)
    codes = torch.randint(-2**31, 2**31 - 1, ops.codes_shape(m, n, 2, fmt.layout), dtype=torch.int32, device="cuda", generator=g)
    lut = torch.randn(512, dtype=torch.float16, device="cuda", generator=g)
    dense = ops.decompress(codes, lut, m, n, fmt)
    y = ops.gemm(codes, lut, torch.eye(n, dtype=torch.float16, device="cuda"), m, n, fmt)       # [n, m]
    torch.cuda.synchronize()
    ops.device_status()
    assert_same_bits(y, dense.t(), f"gemm {m}x{n}")


@pytest.mark.parametrize("code,K,L,S", [(o.CODE_A, 2, 16, 0), (o.CODE_A, 4, 16, 0), (o.CODE_A, 2, 14, 0), (o.CODE_B, 2, 16, 6),
                                        (o.CODE_C, 2, 16, 9), (o.CODE_C, 4, 16, 9)])
def test_gemm_identity_all_codes_and_a_column_shard(code, K, L, S):
    """Every code, plus a column shard with its 16-bit history (carry_in), against the numpy oracle."""
    from rptc_b200 import Format, ops
    m, n = 256, 2048
    rng = np.random.default_rng(code * 11 + K + L)
    w = rand_words(rng, m, 2 * n, K)                        # a row of 2n columns; the right half is the shard
    lut = rand_lut(rng, code, L, S)
    ref = o.decode(w, lut_for_oracle(lut, code, S), 2 * n, code=code, K=K, L=L, S=S)
    nw = w.shape[1] // 2
    fmt = Format(code, K, L, S, o.LAYOUT_TILED)
    eye = torch.eye(n, dtype=torch.float16, device="cuda")
    left = ops.gemm(to_dev(o.from_rowmajor(w[:, :nw], o.LAYOUT_TILED)), to_dev(lut), eye, m, n, fmt)
    right = ops.gemm(to_dev(o.from_rowmajor(w[:, nw:], o.LAYOUT_TILED)), to_dev(lut), eye, m, n, fmt,
                     carry_in=to_dev(np.ascontiguousarray(w[:, nw - 1])))
    torch.cuda.synchronize()
    assert_same_bits(left, torch.from_numpy(ref[:, :n]).cuda().t(), "left shard")
    assert_same_bits(right, torch.from_numpy(ref[:, n:]).cuda().t(), "right shard")


def test_gemm_carry_in_column_shard():
    from rptc_b200 import Format, ops
    rng = np.random.default_rng(5)
    m, n, tokens = 128, 2048, 256
    w = rand_words(rng, m, n, 2)
    lut = rand_lut(rng, o.CODE_B, S=8)
    fmt = Format(o.CODE_B, 2, 16, 8, o.LAYOUT_TILED)
    x = torch.randn((tokens, n), dtype=torch.float16, device="cuda")
    full = ops.gemm(to_dev(o.from_rowmajor(w, o.LAYOUT_TILED)), to_dev(lut), x, m, n, fmt).float()
    nw = w.shape[1]
    left, right = w[:, : nw // 2], w[:, nw // 2:]
    y1 = ops.gemm(to_dev(o.from_rowmajor(left, o.LAYOUT_TILED)), to_dev(lut), x[:, : n // 2].contiguous(), m, n // 2, fmt).float()
    y2 = ops.gemm(to_dev(o.from_rowmajor(right, o.LAYOUT_TILED)), to_dev(lut), x[:, n // 2:].contiguous(), m, n // 2, fmt,
                  carry_in=to_dev(np.ascontiguousarray(left[:, -1]))).float()
    assert (full - (y1 + y2)).abs().max() <= 3 * 2.0**-11 * full.abs().max()      # three fp16 roundings of exact fp32 sums


def test_linear_prefill_path_matches_effective_weight():
    from rptc_b200.linear import RPTCLinear
    lin = RPTCLinear.random(4096, 1024, seed=9)
    x = torch.randn((300, 4096), dtype=torch.float16, device="cuda")
    y = lin(x).float()
    ref = x.float() @ lin.effective_weight().t()
    assert (y - ref).abs().max() <= 1e-2 * ref.abs().max()


@pytest.mark.parametrize("code,K,L,S", [(o.CODE_B, 2, 16, 8), (o.CODE_A, 2, 16, 0), (o.CODE_C, 4, 16, 8)])
@pytest.mark.parametrize("m,n,tokens", [(128, 448, 9), (256, 1024, 128), (384, 2112, 129), (4096, 1088, 100), (256, 4160, 257), (1152, 4032, 640)])
def test_gemm_tiles_and_splits(code, K, L, S, m, n, tokens):
    """One and two token halves, tiles past the last row, and a reduction shared by one, two and four CTAs (uneven parts)."""
    _run(code, K, L, S, m, n, tokens, seed=m + n + tokens)


def test_gemm_invariant_gives_a_token_the_same_bits_in_any_company():
    from rptc_b200 import Format, ops
    fmt, (m, n) = Format(), (512, 4096)
    g = torch.Generator(device="cuda").manual_seed(5)
    codes = torch.randint(-2**31, 2**31 - 1, ops.codes_shape(m, n, 2, fmt.layout), dtype=torch.int32, device="cuda", generator=g)
    lut = torch.randn(512, dtype=torch.float16, device="cuda", generator=g)
    x = torch.randn((5000, n), generator=g, device="cuda").half()
    full = ops.gemm(codes, lut, x, m, n, fmt, invariant=True)
    for tokens in (9, 128, 200, 1000):
        assert torch.equal(ops.gemm(codes, lut, x[:tokens], m, n, fmt, invariant=True), full[:tokens]), tokens


@pytest.mark.parametrize("code,K,L,S", [(o.CODE_B, 2, 16, 8), (o.CODE_A, 2, 16, 0), (o.CODE_A, 4, 14, 0), (o.CODE_C, 4, 16, 9)])
@pytest.mark.parametrize("m,n", [(128, 64), (1152, 576), (4096, 2048), (7168, 1024)])
def test_gemm_of_few_tokens_in_narrow_tiles(code, K, L, S, m, n):
    """Tiles of 32 and 64 rows against the wide ones, whose order of additions they keep: the same bits."""
    from rptc_b200 import Format, ops
    rng = np.random.default_rng(m + n)
    w, lut, fmt = rand_words(rng, m, n, K), to_dev(rand_lut(rng, code, L, S)), Format(code, K, L, S, o.LAYOUT_TILED)
    codes = to_dev(o.from_rowmajor(w, o.LAYOUT_TILED))
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn((2048, n), dtype=torch.float16, device="cuda", generator=g)
    wide = ops.gemm(codes, lut, x, m, n, fmt, invariant=True)
    for tokens in (1, 8, 31, 100, 127, 128, 129, 300):
        y = torch.full((tokens + 1, m), 7.0, dtype=torch.float16, device="cuda")
        ops.gemm(codes, lut, x[:tokens], m, n, fmt, invariant=True, out=y[:tokens])
        assert torch.equal(y[:tokens], wide[:tokens]) and (y[tokens] == 7.0).all(), tokens
    _run(code, K, L, S, m, n, 30, seed=m)


@pytest.mark.parametrize("code,K,L,S", [(o.CODE_B, 2, 16, 8), (o.CODE_A, 2, 16, 0), (o.CODE_A, 4, 16, 0), (o.CODE_C, 4, 16, 8)])
@pytest.mark.parametrize("m,n,tokens", [(64, 4096, 80), (32, 8192, 97), (160, 11008, 112), (1056, 8256, 193), (288, 4160, 385), (4096, 4096, 160)])
def test_layer_of_some_hundred_tokens(code, K, L, S, m, n, tokens):
    """Products that share an accumulator between the groups of a row block: rows past a tile's end, a last tile of few tokens, ranges
    that start inside a tile."""
    from rptc_b200 import Format, ops
    from rptc_b200.linear import RPTCLinear
    g = torch.Generator(device="cuda").manual_seed(m + n + tokens)
    fmt = Format(code, K, L, S, o.LAYOUT_TILED)
    codes = torch.randint(-2**31, 2**31 - 1, ops.codes_shape(m, n, K, fmt.layout), dtype=torch.int32, device="cuda", generator=g)
    lut = torch.randn(fmt.lut_numel(), dtype=torch.float16, device="cuda", generator=g)
    x = torch.randn((tokens, n), dtype=torch.float16, device="cuda", generator=g)
    y = RPTCLinear(n, m, fmt, codes, lut, 0.5)(x) * 2
    torch.cuda.synchronize()
    ops.device_status()
    dense = ops.decompress(codes, lut, m, n, fmt).double()
    err = (y.double() - x.double() @ dense.t()).abs()
    bound = y.double().abs() * 2.0**-11 + 2e-5 * dense.norm(dim=1)[None, :] * x.double().norm(dim=1)[:, None] + 1e-4
    assert float((err / bound).max()) <= 1.0


@pytest.mark.parametrize("code,K,L,S", [(o.CODE_A, 4, 16, 0), (o.CODE_A, 2, 16, 0), (o.CODE_B, 2, 16, 8)])
@pytest.mark.parametrize("m,n,tokens", [(1280, 4160, 49), (1792, 1088, 64), (2304, 2240, 57), (1280, 4160, 96), (128, 40960, 50), (128, 41024, 96), (96, 38400, 17)])
def test_layer_whose_tiles_have_several_parts(code, K, L, S, m, n, tokens):
    """Few row blocks, so that two or four groups of warps take parts of the same rows' steps, segments that are not a multiple of
    the parts, and tables that leave few stages of activations.  The layer twice on inputs that differ in every step: a step's
    sums taken from another step's activations cannot come out right in both."""
    from rptc_b200 import Format, ops
    from rptc_b200.linear import RPTCLinear
    g = torch.Generator(device="cuda").manual_seed(m + n + tokens)
    fmt = Format(code, K, L, S, o.LAYOUT_TILED)
    codes = torch.randint(-2**31, 2**31 - 1, ops.codes_shape(m, n, K, fmt.layout), dtype=torch.int32, device="cuda", generator=g)
    lut = torch.randn(fmt.lut_numel(), dtype=torch.float16, device="cuda", generator=g)
    layer = RPTCLinear(n, m, fmt, codes, lut, 0.25)
    dense = ops.decompress(codes, lut, m, n, fmt).double()
    for _ in range(2):
        x = torch.randn((tokens, n), dtype=torch.float16, device="cuda", generator=g)
        y = layer(x) * 4
        torch.cuda.synchronize()
        ops.device_status()
        err = (y.double() - x.double() @ dense.t()).abs()
        bound = y.double().abs() * 2.0**-11 + 2e-5 * dense.norm(dim=1)[None, :] * x.double().norm(dim=1)[:, None] + 1e-4
        assert float((err / bound).max()) <= 1.0


@pytest.mark.parametrize("code,K,L,S", [(o.CODE_B, 2, 16, 8), (o.CODE_A, 2, 16, 0), (o.CODE_C, 4, 16, 8)])
@pytest.mark.parametrize("m,n,tokens", [(288, 64, 700), (14368, 1024, 512), (32, 128, 3000), (1056, 192, 65)])
def test_layer_of_many_rows_with_a_partial_last_tile(code, K, L, S, m, n, tokens):
    """Any multiple of 32 weight rows and any number of activation rows, whichever product is estimated to be the faster one."""
    from rptc_b200 import Format, ops
    from rptc_b200.linear import RPTCLinear
    g = torch.Generator(device="cuda").manual_seed(m + n + tokens)
    fmt = Format(code, K, L, S, o.LAYOUT_TILED)
    codes = torch.randint(-2**31, 2**31 - 1, ops.codes_shape(m, n, K, fmt.layout), dtype=torch.int32, device="cuda", generator=g)
    lut = torch.randn(fmt.lut_numel(), dtype=torch.float16, device="cuda", generator=g)
    x = torch.randn((tokens, n), dtype=torch.float16, device="cuda", generator=g)
    y = RPTCLinear(n, m, fmt, codes, lut, 0.5)(x) * 2
    torch.cuda.synchronize()
    ops.device_status()
    dense = ops.decompress(codes, lut, m, n, fmt).double()
    err = (y.double() - x.double() @ dense.t()).abs()
    bound = y.double().abs() * 2.0**-11 + 2e-5 * dense.norm(dim=1)[None, :] * x.double().norm(dim=1)[:, None] + 1e-4
    assert float((err / bound).max()) <= 1.0


@pytest.mark.parametrize("code,K,L,S", [(o.CODE_B, 2, 16, 8), (o.CODE_A, 2, 16, 0)])
@pytest.mark.parametrize("m,n,tokens", [(4096, 11008, 512), (4096, 4096, 9), (1280, 4160, 96), (160, 11008, 112), (1056, 8256, 193), (128, 41024, 50), (8192, 4096, 40),
                                        (1024, 14336, 256)])
def test_layers_of_nine_rows_and_more_repeat_themselves(code, K, L, S, m, n, tokens):
    """Several segments to a tile: their sums are added up in one order, so equal calls give equal bits, transforms or none."""
    from rptc_b200 import Format, ops
    from rptc_b200.linear import RPTCLinear
    g = torch.Generator(device="cuda").manual_seed(m + n + tokens)
    layer = RPTCLinear.random(n, m, Format(code, K, L, S, o.LAYOUT_TILED), 0.02, 1, incoherent=m % 256 == 0 and n % 256 == 0)
    x = torch.randn((tokens, n), dtype=torch.float16, device="cuda", generator=g)
    first = layer(x)
    for _ in range(20):
        assert torch.equal(layer(x), first)
    ref = x.float() @ layer.effective_weight().t()
    assert (first.float() - ref).abs().max() <= 1e-2 * ref.abs().max()
    ops.device_status()


def test_layer_without_transforms_takes_more_rows_than_a_grid_has():
    from rptc_b200 import Format
    from rptc_b200._lib import RPTCError
    from rptc_b200.linear import RPTCLinear
    x = torch.randn((70001, 64), dtype=torch.float16, device="cuda", generator=torch.Generator(device="cuda").manual_seed(2))
    layer = RPTCLinear.random(64, 128, Format(), 0.5, 3, incoherent=False)
    y = layer(x)
    ref = x.float() @ layer.effective_weight().t()
    assert (y.float() - ref).abs().max() <= 2e-3 * ref.abs().max()
    with pytest.raises(RPTCError):
        RPTCLinear.random(256, 256, Format(), 0.5, 3)(torch.zeros((70001, 256), dtype=torch.float16, device="cuda"))
