"""The `rptc` / `rptc_lite` modules (reference function names) against the golden vectors produced by
the reference's own code: the encoder on CPU, the decoder (CUDA kernels) in the GPU-marked tests."""
import numpy as np
import pytest
import torch


def test_rptc_quantize_matches_reference_encoder(golden):
    import rptc
    alphabet = torch.from_numpy(golden["enc8_alphabet"])
    for s, want_q, want_loss in zip(golden["enc8_samples"], golden["enc8_symbols"], golden["enc8_loss"]):
        q, loss = rptc.quantize(alphabet, torch.eye(len(s)), torch.from_numpy(s))
        assert np.array_equal(q.numpy(), want_q)
        assert abs(float(loss) - want_loss) <= 1e-5 * max(1.0, abs(want_loss))


def test_rptc_lite_quantize_and_index_match_reference(golden):
    import rptc_lite
    assert np.array_equal(rptc_lite.index_fn(torch.from_numpy(golden["c_index_states"]), 16, 9).numpy(), golden["c_index"])
    alphabet = torch.from_numpy(golden["encc_alphabet"])
    for s, want_q, want_loss in zip(golden["encc_samples"], golden["encc_symbols"], golden["encc_loss"]):
        q, loss = rptc_lite.quantize(alphabet, 8, 5, 4, torch.ones(s.shape), torch.from_numpy(s))
        assert np.array_equal(q.numpy(), want_q)
        assert abs(float(loss) - want_loss) <= 1e-5 * max(1.0, abs(want_loss))


def test_pack_symbols_matches_oracle():
    import rptc
    import rptc_oracle as o
    rng = np.random.default_rng(0)
    for bits, T in ((2, 100), (4, 37), (8, 16)):
        sym = rng.integers(0, 1 << bits, (3, T))
        got = rptc.pack_symbols(torch.from_numpy(sym), bits).numpy().view(np.uint32)
        assert np.array_equal(got, o.pack_symbols(sym, bits))


def test_dequantize_refuses_cpu_tensors():
    import rptc
    with pytest.raises(RuntimeError):
        rptc.dequantize(torch.zeros(65536), torch.zeros(16, dtype=torch.int32))


@pytest.mark.gpu
def test_rptc_dequantize_on_gpu_matches_reference(golden):
    import rptc
    for L in (16, 14):
        alphabet = torch.from_numpy(golden[f"a{L}_alphabet"]).cuda()
        sym = torch.from_numpy(golden[f"a{L}_symbols"]).cuda()
        got = rptc.dequantize(alphabet, sym)
        want = golden[f"a{L}_decoded"].astype(np.float16).astype(np.float32)       # fp16 codebook on the device
        assert np.array_equal(got.cpu().numpy(), want)
        assert np.array_equal(rptc.dequantize(alphabet, sym[0]).cpu().numpy(), want[0])


@pytest.mark.gpu
def test_rptc_lite_dequantize_on_gpu_matches_reference(golden):
    import rptc_lite
    alphabet = torch.from_numpy(golden["c_alphabet"]).cuda()
    sym = torch.from_numpy(golden["c_symbols"]).cuda()
    got = rptc_lite.dequantize(alphabet, 16, 9, 4, sym)
    want = golden["c_decoded"].astype(np.float16).astype(np.float32)
    assert np.array_equal(got.cpu().numpy(), want)


@pytest.mark.gpu
def test_config0_quantize_pack_decompress_matvec():
    """BASELINE config 0 in small: rows of iid N(0,1) weights, quantised with the reference's trellis
    (L = 16 state bits, K = 2), then decompress + matvec on the GPU."""
    import rptc
    from rptc_b200 import CODE_LUT, LAYOUT_ROWMAJOR, LAYOUT_TILED, Format, ops
    from rptc_b200.linear import gaussian_codebook
    g = torch.Generator(device="cuda").manual_seed(42)
    m, n = 32, 1024
    W = torch.randn((m, n), device="cuda", generator=g)
    fmt = Format(CODE_LUT, 2, 16, 0, LAYOUT_TILED)
    alphabet = gaussian_codebook(fmt, g, "cuda").float()
    q, loss = rptc.quantize_rows(alphabet, torch.ones(n, device="cuda"), W)
    recon = rptc.dequantize(alphabet, q)
    mse = ((recon - W) ** 2).mean().item()
    assert abs(loss.sum().item() / (m * n) - mse) < 5e-3           # the encoder's own loss is the decode error
    assert mse < 0.12                                              # 2-bit TCQ of a unit Gaussian (scalar Lloyd-Max is 0.1175)
    words = rptc.pack_symbols(q, 2)
    codes = ops.repack(words.contiguous(), LAYOUT_ROWMAJOR, LAYOUT_TILED, m, n // 64)
    x = torch.randn((1, n), dtype=torch.float16, device="cuda", generator=g)
    y = ops.gemv(codes, alphabet.half(), x, m, n, fmt).float()
    ref = x.float() @ recon.t()
    assert (y - ref).abs().max() <= 2e-3 * recon.norm(dim=1).max() * x.float().norm() + 1e-2


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.float64])
@pytest.mark.parametrize("rows,length,L", [(1, 1, 4), (3, 7, 8), (2, 256, 16), (5, 1001, 11), (1, 8193, 16), (4096, 700, 16), (2500, 1027, 14)])
def test_dequantize_over_pieces_and_tails(rows, length, L, dtype):
    """Rows that are and are not whole pieces of 256 symbols, aligned or not, through L2 and through the table."""
    import rptc
    g = torch.Generator(device="cuda").manual_seed(rows + length)
    alphabet = torch.randn(1 << L, generator=g, device="cuda", dtype=torch.float64).to(dtype)
    sym = torch.randint(0, 4, (rows, length), generator=g, device="cuda", dtype=torch.int32)
    got = rptc.dequantize(alphabet, sym)
    states = torch.zeros((rows, length), dtype=torch.int64, device="cuda")
    for back in range((L + 1) // 2):                        # the symbols that the state's L bits come from
        states[:, back:] |= sym[:, : length - back].long() << (2 * back)
    assert got.dtype == dtype and torch.equal(got, alphabet.half().to(dtype)[states & ((1 << L) - 1)])
    assert torch.equal(rptc.pack_symbols(sym, 2).cpu(), rptc.pack_symbols(sym.cpu(), 2))


@pytest.mark.parametrize("L,n,limit,want", [(16, 4096, 12 << 30, 148), (16, 1024, 12 << 30, 888), (16, 4096, 1 << 30, 63), (16, 65536, 1 << 20, 1), (15, 4096, 12 << 30, 296),
                                            (8, 4096, 12 << 30, 65416)])
def test_encoder_rows_at_once_needs_no_gpu(L, n, limit, want):
    """Survivor memory is 2^(L-4) bytes per row and position: whole sets of the rows in flight, 4 GiB beyond one set."""
    from rptc_b200 import ops
    assert ops.encoder_rows_at_once(L, n, 148, limit) == want


@pytest.mark.parametrize("shape", [(65535,), (100,), (4,), (1 << 17,), (2, 32768), (0,)])
def test_dequantize_refuses_an_alphabet_that_is_not_a_table(shape):
    """The state indexes 2^L entries: any other length would silently use its first ones."""
    from rptc_b200 import lib, ops
    with pytest.raises(RuntimeError, match="2\\^L entries"):
        ops.check_alphabet(torch.zeros(shape))
    for L in (3, 16):
        ops.check_alphabet(torch.zeros(1 << L))
    for L in (0, 2, 17):
        assert lib().rptc_dequantize(1 << 8, 1 << 8, 1 << 8, 1, 1, 1, L, None) == -1


@pytest.mark.gpu
def test_dequantize_refuses_odd_alphabets_on_the_gpu():
    import rptc
    sym = torch.zeros(8, dtype=torch.int32, device="cuda")
    for n in (100, 65535):
        with pytest.raises(RuntimeError, match="2\\^L entries"):
            rptc.dequantize(torch.zeros(n, device="cuda"), sym)


@pytest.mark.gpu
@pytest.mark.parametrize("rows,length", [(512, 4096), (4096, 4096)])
def test_dequantize_keeps_stream_order_under_dependent_launch(rows, length):
    """With rptc_set_pdl on, the kernel in front lets this one start early; it neither reads nor writes anything before that one is
    done: here the memory that the decoder in front still reads its codes from becomes the result."""
    import ctypes

    from rptc_b200 import CODE_LUT, LAYOUT_TILED, Format, lib, ops
    g = torch.Generator(device="cuda").manual_seed(rows)
    m, n, L = 4096, 8192, 16
    fmt = Format(CODE_LUT, 2, L, 0, LAYOUT_TILED)
    codes = torch.randint(-2**31, 2**31 - 1, ops.codes_shape(m, n, 2, fmt.layout), dtype=torch.int32, device="cuda", generator=g)
    lut = torch.randn(1 << L, generator=g, device="cuda").half()
    symbols = torch.randint(0, 4, (rows, length), generator=g, device="cuda", dtype=torch.int32)
    want_dense, want = ops.decompress(codes, lut, m, n, fmt), ops.dequantize(lut, symbols)
    out, stream = torch.empty_like(want_dense), torch.cuda.current_stream().cuda_stream
    shared = torch.empty(max(codes.numel(), want.numel() // 2), dtype=torch.int32, device="cuda")
    lib().rptc_set_pdl(1)
    try:
        for _ in range(20):
            shared[: codes.numel()].copy_(codes.reshape(-1))
            assert lib().rptc_decompress(shared.data_ptr(), lut.data_ptr(), None, out.data_ptr(), n, m, n, ctypes.byref(fmt), stream) == 0
            assert lib().rptc_dequantize(lut.data_ptr(), symbols.data_ptr(), shared.data_ptr(), 0, rows, length, L, stream) == 0
            assert torch.equal(out, want_dense)
            assert torch.equal(shared.view(torch.float16)[: want.numel()].view(want.shape), want)
    finally:
        lib().rptc_set_pdl(0)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("L", [3, 4, 9])
def test_dequantize_and_decompress_by_either_route(L, dtype):
    """What the native call takes and what it leaves to the converting path: 64-bit and strided symbols, other types, a
    single row; outputs with a stride, and those that are refused."""
    import rptc
    from rptc_b200 import CODE_LUT, LAYOUT_TILED, Format, ops
    g = torch.Generator(device="cuda").manual_seed(L)
    alphabet = torch.randn(1 << L, generator=g, device="cuda").to(dtype)
    wide = torch.randint(0, 4, (6, 300), generator=g, device="cuda")
    want = rptc.dequantize(alphabet, wide)
    assert torch.equal(rptc.dequantize(alphabet, wide.int()), want) and torch.equal(rptc.dequantize(alphabet, wide[2].int()), want[2])
    strided = torch.zeros((6, 600), dtype=torch.int32, device="cuda")[:, ::2]
    strided.copy_(wide)
    assert torch.equal(rptc.dequantize(alphabet, strided), want)
    m, n = 64, 256
    fmt = Format(CODE_LUT, 2, max(L, 8), 0, LAYOUT_TILED)
    codes = torch.randint(-2**31, 2**31 - 1, ops.codes_shape(m, n, 2, fmt.layout), dtype=torch.int32, device="cuda", generator=g)
    lut = torch.randn(fmt.lut_numel(), generator=g, device="cuda").half()
    dense = ops.decompress(codes, lut, m, n, fmt)
    out = torch.empty((m, n + 16), dtype=torch.float16, device="cuda")
    assert torch.equal(ops.decompress(codes, lut, m, n, fmt, out=out[:, :n]), dense)
    for refused in (out, out[:, :n].float(), out[: m // 2, :n], torch.empty((n, m), dtype=torch.float16, device="cuda").t()):
        with pytest.raises(Exception):
            ops.decompress(codes, lut, m, n, fmt, out=refused)
