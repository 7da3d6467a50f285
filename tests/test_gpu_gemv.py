"""GPU parity: the fused dequant-GEMV against the CPU oracle (fp64 product of bit-exact weights).

Tolerance (derived in gpu_util.py from the kernels' arithmetic).  The general kernels multiply in fp16 pairs and add eight
products per fp16 accumulator before widening to fp32: |y - exact| <= 1.5e-4 ||w_row|| ||x|| + 2^-11 |exact|, which is
0.6 absolute at n = 4096 with N(0,1) data -- below the ~1 that ONE mis-decoded weight moves an output by (the
reference's fully fp16-accumulated product, inference.cu:263,270-276, is about 200 times looser).  The TILED
layout's products are summed in fp32 (mma.sync up to two rows, tcgen05 above): 2e-5 ||w_row|| ||x||, checked for even batches.  Wrong weights are hunted exactly, column by column, in
test_gpu_probe.py; this file checks the arithmetic on random inputs.
"""
import numpy as np
import pytest
import torch

import rptc_oracle as o
from gpu_util import GEMV_FP32_TOL, GEMV_HFMA2_TOL, bits, check_product, lut_for_oracle, rand_lut, rand_words, to_dev

pytestmark = pytest.mark.gpu


def _check(y, w16, x16, rel=None, what=""):
    """rel defaults to the bound of the kernel that serves this batch size (odd: the wider one of the general kernels)."""
    if rel is None:
        rel = GEMV_HFMA2_TOL if x16.shape[0] in (1, 3, 5, 7) else GEMV_FP32_TOL      # odd batches end in a batch-1 launch
    exact = o.matvec_exact(w16, x16)
    check_product(y, exact, np.linalg.norm(w16.astype(np.float64), axis=1), np.linalg.norm(x16.astype(np.float64), axis=1), rel, what)


CASES = [(o.CODE_B, 2, 16, 8), (o.CODE_B, 2, 16, 6), (o.CODE_A, 2, 16, 0), (o.CODE_A, 4, 16, 0), (o.CODE_A, 2, 14, 0),
         (o.CODE_C, 2, 16, 9), (o.CODE_C, 4, 16, 9)]


@pytest.mark.parametrize("code,K,L,S", CASES)
@pytest.mark.parametrize("batch", [1, 2, 3, 4, 8])
@pytest.mark.parametrize("m,n", [(64, 2048), (4096, 4096), (352, 11008)])
def test_gemv_native_layout(code, K, L, S, batch, m, n):
    from rptc_b200 import Format, ops
    if code != o.CODE_B and batch not in (1, 4) :
        pytest.skip("batch sweep runs on the headline code only")
    rng = np.random.default_rng(hash((code, K, L, S, batch, m, n)) % 2**32)
    w = rand_words(rng, m, n, K)
    lut = rand_lut(rng, code, L, S)
    x = rng.standard_normal((batch, n)).astype(np.float16)
    w16 = o.decode(w, lut_for_oracle(lut, code, S), n, code=code, K=K, L=L, S=S)
    y = ops.gemv(to_dev(o.from_rowmajor(w, o.LAYOUT_TILED)), to_dev(lut), to_dev(x), m, n,
                 Format(code, K, L, S, o.LAYOUT_TILED))
    torch.cuda.synchronize()
    ops.device_status()
    _check(y.float().cpu().numpy(), w16, x)


@pytest.mark.parametrize("layout", [o.LAYOUT_ROWMAJOR, o.LAYOUT_CHUNKED, o.LAYOUT_UNITMAJOR])
def test_gemv_legacy_layouts(layout):
    from rptc_b200 import Format, ops
    rng = np.random.default_rng(51 + layout)
    m, n = 128, 4096
    w = rand_words(rng, m, n, 2)
    lut = rand_lut(rng, o.CODE_B, S=8)
    x = rng.standard_normal((1, n)).astype(np.float16)
    w16 = o.decode(w, lut, n, code=o.CODE_B, S=8)
    y = ops.gemv(to_dev(o.from_rowmajor(w, layout)), to_dev(lut), to_dev(x), m, n, Format(o.CODE_B, 2, 16, 8, layout))
    _check(y.float().cpu().numpy(), w16, x, GEMV_HFMA2_TOL)      # the general kernel is an HFMA2 kernel


def test_gemv_carry_in_and_column_sharding():
    # a row-parallel (column-sharded) layer: shard s decodes units [s*U/2, (s+1)*U/2) and needs the 16 bits
    # before its first unit; the partial products add up to the unsharded result
    from rptc_b200 import Format, ops
    rng = np.random.default_rng(61)
    m, n = 256, 8192
    w = rand_words(rng, m, n, 2)
    lut = rand_lut(rng, o.CODE_B, S=8)
    x = rng.standard_normal((2, n)).astype(np.float16)
    w16 = o.decode(w, lut, n, code=o.CODE_B, S=8)
    nw = w.shape[1]
    left, right = w[:, : nw // 2], w[:, nw // 2:]           # two column shards of the row-major stream
    acc = torch.zeros((2, m), dtype=torch.float32, device="cuda")
    fmt = Format(o.CODE_B, 2, 16, 8, o.LAYOUT_TILED)
    xd = to_dev(x)
    ops.gemv_acc(to_dev(o.from_rowmajor(left, o.LAYOUT_TILED)), to_dev(lut), xd[:, : n // 2], acc, m, n // 2, fmt)
    carry = np.ascontiguousarray(left[:, -1])               # last word of the left shard = the right shard's history
    ops.gemv_acc(to_dev(o.from_rowmajor(right, o.LAYOUT_TILED)), to_dev(lut), xd[:, n // 2:], acc, m, n // 2, fmt,
                 carry_in=to_dev(carry))
    torch.cuda.synchronize()
    _check(acc.cpu().numpy(), w16, x)


def test_gemv_finish_accumulate_and_clear():
    from rptc_b200 import ops
    acc = torch.arange(64, dtype=torch.float32, device="cuda").reshape(2, 32).contiguous()
    y = torch.ones((2, 32), dtype=torch.float16, device="cuda")
    ops.gemv_finish(acc, y, 32, scale=0.5, accumulate=True, clear=True)
    torch.cuda.synchronize()
    assert torch.equal(y.float().cpu(), 1 + 0.5 * torch.arange(64, dtype=torch.float32).reshape(2, 32))
    assert bool((acc == 0).all())


def test_gemv_all_ones_codebook_known_answer():
    # rptc_kernels/tests/test_decompress.py:11,38 — with an all-ones LUT every output equals sum(x)
    from rptc_b200 import Format, ops
    rng = np.random.default_rng(71)
    m, n = 512, 8192
    w = rand_words(rng, m, n, 2)
    lut = np.ones(1 << 16, dtype=np.float16)
    x = rng.standard_normal((1, n)).astype(np.float16)
    y = ops.gemv(to_dev(o.from_rowmajor(w, o.LAYOUT_TILED)), to_dev(lut), to_dev(x), m, n,
                 Format(o.CODE_A, 2, 16, 0, o.LAYOUT_TILED))
    s = x.astype(np.float64).sum()
    assert np.allclose(y.float().cpu().numpy(), s, atol=2.0**-11 * abs(s) + 1.5e-4 * np.sqrt(n) * np.linalg.norm(x.astype(np.float64)))


@pytest.mark.parametrize("m,n", [(4096, 4096), (11008, 4096), (4096, 11008), (28672, 8192)])
def test_gemv_full_size_linearity(m, n):
    # BASELINE-size layers: checked through properties that need no CPU decode — linearity in x and
    # agreement with decompress-then-matmul on the GPU's own bit-exact decompress output
    from rptc_b200 import Format, ops
    g = torch.Generator(device="cuda").manual_seed(m * 7 + n)
    codes = torch.randint(-2**31, 2**31 - 1, (m // 32, n // 64, 32, 4), dtype=torch.int32, device="cuda", generator=g)
    lut = torch.randn(512, dtype=torch.float16, device="cuda", generator=g)
    x = torch.randn((2, n), dtype=torch.float16, device="cuda", generator=g)
    fmt = Format(o.CODE_B, 2, 16, 8, o.LAYOUT_TILED)
    y = ops.gemv(codes, lut, x, m, n, fmt).float()
    ysum = ops.gemv(codes, lut, (x[0] + x[1]).unsqueeze(0), m, n, fmt).float()      # the fp16 sum is the input of both sides
    dense = ops.decompress(codes, lut, m, n, fmt)
    ref = (x.double() @ dense.double().T)
    scale = dense.double().norm(dim=1)[None, :] * x.double().norm(dim=1)[:, None]
    err = (y.double() - ref).abs()
    tol = GEMV_FP32_TOL * scale + 2.0**-11 * ref.abs() + 1e-4                        # two rows: mma.sync
    assert bool((err <= tol).all()), f"max err/tol {(err / tol).max().item():.3f}"
    # batch 1 (HFMA2 kernel) on the fp16 sum of the two rows, against the same product
    xs = (x[0] + x[1]).unsqueeze(0)
    ref_s = xs.double() @ dense.double().T
    err_s = (ysum.double() - ref_s).abs()
    tol_s = GEMV_HFMA2_TOL * dense.double().norm(dim=1)[None, :] * xs.double().norm() + 2.0**-11 * ref_s.abs() + 1e-4
    assert bool((err_s <= tol_s).all()), f"batch 1 max err/tol {(err_s / tol_s).max().item():.3f}"


@pytest.mark.parametrize("code,K,L,S", [(o.CODE_B, 2, 16, 8), (o.CODE_A, 2, 16, 0), (o.CODE_A, 4, 14, 0), (o.CODE_C, 4, 16, 8)])
@pytest.mark.parametrize("m,n,batch", [(32, 64, 3), (32, 128, 16), (128, 64 * 149, 17), (160, 320, 33), (1056, 2112, 5), (4096, 1088, 64), (384, 4160, 48)])
def test_gemv_few_rows_at_tile_and_range_edges(code, K, L, S, m, n, batch):
    """Rows past a tile's end, ranges that start inside a tile, parts of a segment without a step, one to four groups of 16 tokens."""
    from rptc_b200 import Format, ops
    g = torch.Generator(device="cuda").manual_seed(m + n + batch)
    fmt = Format(code, K, L, S, o.LAYOUT_TILED)
    codes = torch.randint(-2**31, 2**31 - 1, ops.codes_shape(m, n, K, fmt.layout), dtype=torch.int32, device="cuda", generator=g)
    lut = torch.randn(fmt.lut_numel(), dtype=torch.float16, device="cuda", generator=g)
    x = torch.randn((batch, n), dtype=torch.float16, device="cuda", generator=g)
    dense = ops.decompress(codes, lut, m, n, fmt).double()
    exact = x.double() @ dense.t()
    y = ops.gemv(codes, lut, x, m, n, fmt)
    torch.cuda.synchronize()
    ops.device_status()
    check_product(y.float().cpu().numpy(), exact.cpu().numpy(), dense.norm(dim=1).cpu().numpy(), x.double().norm(dim=1).cpu().numpy(), GEMV_FP32_TOL)


@pytest.mark.parametrize("m,n,batch", [(16, 8, 3), (17, 40, 5), (1000, 4096, 16), (40000, 520, 9), (37, 8200, 8), (2500, 8232, 13)])
def test_dense_gemv_of_many_rows(m, n, batch):
    """Rows and columns that are not whole tiles, x in one and in several chunks of columns, one and several rounds of tiles."""
    from rptc_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(m + n)
    W, x = torch.randn((m, n), generator=g, device="cuda").half(), torch.randn((batch, n), generator=g, device="cuda").half()
    exact = x.double() @ W.double().t()
    y = ops.dense_gemv(W, x)
    check_product(y.float().cpu().numpy(), exact.cpu().numpy(), W.double().norm(dim=1).cpu().numpy(), x.double().norm(dim=1).cpu().numpy(), GEMV_FP32_TOL)


@pytest.mark.parametrize("code,K,L,S", [(o.CODE_B, 2, 16, 8), (o.CODE_A, 2, 16, 0), (o.CODE_A, 4, 14, 0), (o.CODE_C, 4, 16, 8)])
@pytest.mark.parametrize("layout", [o.LAYOUT_ROWMAJOR, o.LAYOUT_CHUNKED])
@pytest.mark.parametrize("m,n", [(32, 2048), (64, 64), (96, 6208), (1056, 4096), (4096, 10240)])
def test_gemv_of_layouts_with_a_row_together(code, K, L, S, layout, m, n):
    """Fewer rows than CTAs, chunks of fewer than 32 units, ranges that start inside a chunk.  The fp16 roundings of the n / 64 units add
    in quadrature, so the bound, measured at n = 4096, grows as n falls."""
    from rptc_b200 import Format, ops
    if layout == o.LAYOUT_CHUNKED and (n * K // 128) % 32:
        pytest.skip("whole chunks only")
    g = torch.Generator(device="cuda").manual_seed(m + n)
    fmt = Format(code, K, L, S, layout)
    codes = torch.randint(-2**31, 2**31 - 1, (m * n * K // 32,), dtype=torch.int32, device="cuda", generator=g)
    lut = torch.randn(fmt.lut_numel(), dtype=torch.float16, device="cuda", generator=g)
    x = torch.randn((1, n), dtype=torch.float16, device="cuda", generator=g)
    dense = ops.decompress(codes, lut, m, n, fmt).double()
    y = ops.gemv(codes, lut, x, m, n, fmt)
    torch.cuda.synchronize()
    ops.device_status()
    check_product(y.float().cpu().numpy(), (x.double() @ dense.t()).cpu().numpy(), dense.norm(dim=1).cpu().numpy(), x.double().norm(dim=1).cpu().numpy(),
                  GEMV_HFMA2_TOL * (4096 / min(n, 4096)) ** 0.5)


@pytest.mark.parametrize("code,K,L,S", [(o.CODE_B, 2, 16, 8), (o.CODE_A, 2, 16, 0), (o.CODE_A, 4, 14, 0), (o.CODE_C, 2, 16, 8), (o.CODE_C, 4, 16, 8)])
@pytest.mark.parametrize("m,n", [(256, 256), (512, 1536), (1280, 2304), (4096, 4096), (768, 3072), (22016, 1024), (9984, 2048), (1024, 5120)])
def test_layer_of_one_row(code, K, L, S, m, n):
    """The product makes the input transform (blocks of 256 to 4096, spans that the row ends inside) and puts down sums that the output
    transform adds up: few and many CTAs in a row block; the last size has a kernel in front.  Activations and results are rounded to fp16,
    2^-11 of each value at most."""
    from rptc_b200 import Format, ops
    from rptc_b200.linear import RPTCLinear
    layer = RPTCLinear.random(n, m, Format(code, K, L, S, o.LAYOUT_TILED), 0.02, m + n)
    g = torch.Generator(device="cuda").manual_seed(m * 3 + n)
    x = torch.randn(1, n, generator=g, device="cuda").half()
    y = layer(x)
    want = x.double() @ layer.effective_weight().double().t()
    assert (y.double() - want).norm() <= 2.0**-10 * want.norm()
    for _ in range(5 if n <= 4096 else 0):                     # sums in a fixed order
        assert torch.equal(layer(x), y)
    # history in front of the rows (a shard of a layer whose reduction is cut)
    layer.carry_in = torch.randint(-2**31, 2**31 - 1, (m,), dtype=torch.int32, device="cuda", generator=g)
    want = x.double() @ layer.effective_weight().double().t()
    carried = layer(x)
    assert (carried.double() - want).norm() <= 2.0**-10 * want.norm() and not torch.equal(carried, y)
    ops.device_status()


@pytest.mark.parametrize("code,K,L,S", [(o.CODE_B, 2, 16, 8), (o.CODE_B, 2, 16, 6), (o.CODE_A, 2, 16, 0), (o.CODE_A, 4, 14, 0), (o.CODE_C, 4, 16, 8)])
@pytest.mark.parametrize("layout,x_order,quirk", [(o.LAYOUT_ROWMAJOR, 0, 0), (o.LAYOUT_CHUNKED, 0, 0), (o.LAYOUT_CHUNKED, 1, o.QUIRK_K2_LANE0_CARRY)])
@pytest.mark.parametrize("m,n", [(32, 2048), (32, 16384), (160, 6144), (1056, 8192), (96, 10240), (96, 12288), (4128, 4096), (22016, 2048), (64, 51200), (64, 81920)])
def test_timed_matvec_stores_and_adds(code, K, L, S, layout, x_order, quirk, m, n):
    """rptc_gemv_timed: a warp and several per row, one and many rows a warp, the last sizes beyond the shared memory that the HASH code and all codes
    leave, and both sides of the line in the legacy order (beyond either a kernel and one behind it).
    The same product as rptc_gemv's, a store and an addition in fp16, a positive time."""
    from rptc_b200 import Format, ops
    from rptc_b200._lib import native
    if quirk and K != 2 or layout == o.LAYOUT_CHUNKED and (n * K // 128) % 32:
        pytest.skip("not defined")
    g = torch.Generator(device="cuda").manual_seed(m + n)
    fmt = Format(code, K, L, S, layout, quirk)
    codes = torch.randint(-2**31, 2**31 - 1, (m * n * K // 32,), dtype=torch.int32, device="cuda", generator=g)
    lut = torch.randn(fmt.lut_numel(), dtype=torch.float16, device="cuda", generator=g)
    x = torch.randn(n, dtype=torch.float16, device="cuda", generator=g)
    acc = torch.zeros((1, m), device="cuda")
    ops.gemv_acc(codes, lut, x, acc, m, n, fmt, x_order=x_order)
    want = acc[0].clone()
    acc.zero_()
    y = torch.full((m,), 7.0, dtype=torch.float16, device="cuda")
    assert native().gemv_timed(codes, lut, x, acc, y, m, n, x_order, 0, fmt) > 0
    # the same fp16 products, summed in another order in fp32, then one rounding
    scale = want.abs().max().item()
    assert (y.float() - want).abs().max().item() <= 2e-5 * scale * 16 + 2.0**-11 * scale
    first = y.clone()
    assert native().gemv_timed(codes, lut, x, acc, y, m, n, x_order, 1, fmt) > 0
    assert (y.float() - 2 * first.float()).abs().max().item() <= (2e-5 * 16 + 2.0**-9) * scale
    assert not acc.any()
    ops.device_status()


@pytest.mark.parametrize("layout", [o.LAYOUT_ROWMAJOR, o.LAYOUT_CHUNKED])
@pytest.mark.parametrize("m,n,at", [(2048, 2048, 0), (8192, 8192, 0), (4096, 4096, 1024), (1024, 6144, 5120), (6144, 2048, 2046)])
@pytest.mark.parametrize("accumulate", [0, 1])
def test_timed_matvec_whose_result_replaces_its_activations(layout, m, n, at, accumulate):
    """y lies over x, all of it or a part: the product reads x as it was before the call."""
    from rptc_b200 import Format, ops
    from rptc_b200._lib import native
    g = torch.Generator(device="cuda").manual_seed(m + n)
    fmt = Format(o.CODE_B, 2, 16, 8, layout)
    codes = torch.randint(-2**31, 2**31 - 1, (m * n * 2 // 32,), dtype=torch.int32, device="cuda", generator=g)
    lut = torch.randn(fmt.lut_numel(), dtype=torch.float16, device="cuda", generator=g)
    room = torch.randn(max(n, at + m), dtype=torch.float16, device="cuda", generator=g)
    x, y = room[:n], room[at:at + m]
    before = room.clone()
    acc = torch.zeros((1, m), device="cuda")
    ops.gemv_acc(codes, lut, x, acc, m, n, fmt)
    want = acc[0] + (y.float() if accumulate else 0.0)
    acc.zero_()
    assert native().gemv_timed(codes, lut, x, acc, y, m, n, 0, accumulate, fmt) > 0
    scale = want.abs().max().item()
    # the same fp16 products, summed in another order in fp32, rounded to fp16 (twice where the result is added to y)
    assert (y.float() - want).abs().max().item() <= (2e-5 * 16 + 2.0**-10) * scale
    before[at:at + m] = y
    assert torch.equal(room, before)


@pytest.mark.parametrize("code,K,L,S", [(o.CODE_B, 2, 16, 8), (o.CODE_A, 2, 16, 0), (o.CODE_C, 4, 16, 8)])
@pytest.mark.parametrize("m,n", [(512, 4096), (768, 2048), (1536, 2048), (2048, 2048), (4096, 1024), (3840, 3584), (7936, 1280)])
@pytest.mark.parametrize("rows", [9, 31, 32, 72, 73, 96])
def test_layer_whose_sums_are_added_up_in_front_of_or_in_its_output_transform(code, K, L, S, m, n, rows):
    """Blocks of 256 to 4096, many and few sums a value, both sides of the lines in rows.  Activations and results are rounded to fp16, 2^-11 of
    each value at most."""
    from rptc_b200 import Format, ops
    from rptc_b200.linear import RPTCLinear
    layer = RPTCLinear.random(n, m, Format(code, K, L, S, o.LAYOUT_TILED), 0.02, m + n)
    g = torch.Generator(device="cuda").manual_seed(m + rows)
    x = torch.randn(rows, n, generator=g, device="cuda").half()
    y = layer(x)
    want = x.double() @ layer.effective_weight().double().t()
    assert (y.double() - want).norm() <= 2.0**-10 * want.norm()
    assert torch.equal(layer(x), y)                            # sums in a fixed order
    ops.device_status()
