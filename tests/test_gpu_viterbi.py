"""The CUDA trellis encoder (csrc/viterbi.cu) against the reference's own encoder output (golden vectors), against
the torch restatement on the CPU, and on BASELINE's single-linear case: Gaussian weights encoded at L = 16, packed,
decoded and multiplied on the GPU."""
import numpy as np
import pytest
import torch

import rptc_oracle as o

pytestmark = pytest.mark.gpu


def test_cuda_encoder_reproduces_the_reference_encoder(golden):
    import rptc
    alphabet = torch.from_numpy(golden["enc8_alphabet"]).cuda()
    samples = torch.from_numpy(golden["enc8_samples"]).cuda()
    weights = torch.ones(samples.shape[1], device="cuda")
    sym, loss = rptc.quantize_rows(alphabet, weights, samples)
    assert sym.dtype == torch.int32
    assert np.array_equal(sym.cpu().numpy(), golden["enc8_symbols"])
    np.testing.assert_allclose(loss.cpu().numpy(), golden["enc8_loss"], rtol=1e-5)


@pytest.mark.parametrize("L,n,rows,ties", [(4, 9, 3, False), (6, 40, 5, False), (10, 130, 9, False), (8, 64, 6, True), (12, 50, 130, False)])
def test_cuda_encoder_matches_the_cpu_recurrence(L, n, rows, ties):
    import rptc
    g = torch.Generator().manual_seed(L * 100 + n)
    alphabet = torch.randn(1 << L, generator=g)
    if ties:
        alphabet = (alphabet * 2).round() / 2             # few distinct values: equal costs everywhere, first minimum wins
    samples = torch.randn(rows, n, generator=g)
    if ties:
        samples = (samples * 2).round() / 2
    weights = 0.5 + torch.rand(n, generator=g)
    want_sym, want_loss = rptc.quantize_rows(alphabet, weights, samples)               # torch, on the CPU
    got_sym, got_loss = rptc.quantize_rows(alphabet.cuda(), weights.cuda(), samples.cuda())
    assert torch.equal(got_sym.cpu(), want_sym)
    torch.testing.assert_close(got_loss.cpu(), want_loss, rtol=1e-5, atol=1e-6)
    # the symbols walk the trellis to the cost the encoder reports
    for r in range(min(rows, 3)):
        dec = o.dequantize_symbols(alphabet.numpy(), want_sym[r].numpy())
        cost = float((weights.numpy().astype(np.float64) * (samples[r].numpy().astype(np.float64) - dec) ** 2).sum())
        assert abs(cost - float(got_loss[r])) <= 1e-4 * max(1.0, cost)


def test_single_linear_gaussian_weights_at_L16():
    """BASELINE's single-linear case at 256 x 4096: N(0,1) weights, Gaussian-quantile alphabet in a seeded random order,
    encoded at L = 16 / 2 bits per weight, packed, decoded bit-exactly and multiplied by one fp16 vector."""
    import rptc
    from rptc_b200 import CODE_LUT, LAYOUT_ROWMAJOR, LAYOUT_TILED, Format, ops
    m, n, L = 256, 4096, 16
    g = torch.Generator(device="cuda").manual_seed(42)
    W = torch.randn(m, n, generator=g, device="cuda")
    M = 1 << L
    q = (2 * torch.arange(M, dtype=torch.float64, device="cuda") + 1) / (2 * M)
    alphabet = (2.0 ** 0.5 * torch.erfinv(2 * q - 1)).float()[torch.randperm(M, generator=g, device="cuda")]      # rptc.py:143-146
    sym, loss = rptc.quantize_rows(alphabet, torch.ones(n, device="cuda"), W)
    assert int(sym.min()) >= 0 and int(sym.max()) <= 3
    W_hat = rptc.dequantize(alphabet, sym)                                            # CUDA decompress of the packed symbols
    mse = float(((W - W_hat.float()) ** 2).mean())
    assert 0.06 < mse < 0.09, mse                      # 2 bits per weight: the distortion-rate bound is 0.0625
    torch.testing.assert_close(loss / n, ((W - alphabet[_states(sym, L)]) ** 2).mean(dim=1), rtol=1e-4, atol=1e-5)
    lut16 = alphabet.half()
    for r in (0, 17, m - 1):                           # bit-exact against the oracle's sequential decode
        want = o.dequantize_symbols(lut16.cpu().numpy(), sym[r].cpu().numpy())
        assert np.array_equal(W_hat[r].half().cpu().numpy().view(np.uint16), want.view(np.uint16))
    words = rptc.pack_symbols(sym)
    fmt = Format(CODE_LUT, 2, L, 0, LAYOUT_TILED)
    codes = ops.repack(words.contiguous(), LAYOUT_ROWMAJOR, LAYOUT_TILED, m, n // 64)
    x = torch.randn(n, generator=g, device="cuda").half()
    y = ops.gemv(codes, lut16, x, m, n, fmt).float()
    want = W_hat.half().float() @ x.float()
    assert (y - want).abs().max().item() <= 2e-3 * float(W_hat.float().norm(dim=1).max() * x.float().norm())


def _states(sym: torch.Tensor, L: int) -> torch.Tensor:
    """The state visited at every position of every row (the last L bits of the symbol stream)."""
    state = torch.zeros(sym.shape[0], dtype=torch.int64, device=sym.device)
    out = torch.empty(sym.shape, dtype=torch.int64, device=sym.device)
    for i in range(sym.shape[1]):
        state = ((state << 2) | sym[:, i].long()) & ((1 << L) - 1)
        out[:, i] = state
    return out


@pytest.mark.parametrize("L,n,banks,per_bank", [(5, 7, 2, 3), (9, 33, 1, 2), (10, 12, 3, 1), (13, 21, 2, 5), (14, 9, 1, 3), (15, 1, 1, 2), (15, 12, 2, 2),
                                                (15, 5, 100, 3), (16, 11, 1, 1), (16, 2, 2, 3), (16, 6, 51, 3)])
def test_banked_encoder_at_the_edges_of_its_variants(L, n, banks, per_bank):
    """One and two rows per CTA, one CTA and a pair of CTAs per row, banks with a row left over."""
    import rptc
    from rptc_b200 import ops
    g = torch.Generator().manual_seed(L * 100 + n)
    alphabets = (torch.randn(banks, 1 << L, generator=g) * 64).round() / 64          # equal entries: ties
    samples = torch.randn(banks * per_bank, n, generator=g)
    weights = 0.5 + torch.rand(n, generator=g)
    sym, loss = ops.viterbi_encode_banked(alphabets.cuda(), weights.cuda(), samples.cuda())
    for b in range(banks):
        rows = slice(b * per_bank, (b + 1) * per_bank)
        want_sym, want_loss = rptc.quantize_rows(alphabets[b], weights, samples[rows])
        assert torch.equal(sym[rows].cpu(), want_sym), b
        torch.testing.assert_close(loss[rows].cpu(), want_loss, rtol=1e-6, atol=0)
    # a workspace that holds two rows only: parts of banks
    again, _ = ops.viterbi_encode_banked(alphabets[:2].cuda(), weights.cuda(), samples[: min(banks, 2) * per_bank].cuda(),
                                         workspace_limit=2 * (n << (L - 4)) + 1024)
    assert torch.equal(again, sym[: again.shape[0]])


@pytest.mark.parametrize("L,n,banks,per_bank", [(6, 20, 4, 5), (12, 30, 3, 7), (15, 9, 5, 3), (16, 7, 4, 5), (16, 5, 90, 2), (15, 4, 110, 3)])
@pytest.mark.parametrize("at_once", [1, 2, 3, 8, 296])
def test_encoder_takes_ranges_that_start_and_end_inside_banks(L, n, banks, per_bank, at_once):
    from rptc_b200 import ops
    from rptc_b200._lib import lib
    g = torch.Generator(device="cuda").manual_seed(L * 100 + n)
    alphabets = (torch.randn(banks, 1 << L, generator=g, device="cuda") * 64).round() / 64
    samples = torch.randn(banks * per_bank, n, generator=g, device="cuda")
    weights = 0.5 + torch.rand(n, generator=g, device="cuda")
    want, want_loss = ops.viterbi_encode_banked(alphabets, weights, samples)
    got, loss = ops.viterbi_encode_banked(alphabets, weights, samples, workspace_limit=at_once * lib().rptc_viterbi_workspace_bytes(1, n, L))
    assert torch.equal(got, want) and torch.equal(loss, want_loss)


def test_layer_quantisation_keeps_its_memory_bounded():
    """At L = 16 and 4096 columns a row's survivors are 16 MiB: the rows of a whole layer at once would take 8.6 GB here.  With less memory
    than the rows in flight need, batch_size rows at once are enough."""
    import quantize_hf as q
    g = torch.Generator(device="cuda").manual_seed(5)
    weights, importance = torch.randn(512, 4096, generator=g, device="cuda"), 0.5 + torch.rand(4096, generator=g, device="cuda")
    permute = q.seeded_permute(3)
    torch.cuda.empty_cache()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    symbols, alphabets = q.round_weights(permute, weights, importance, 16, 32, 8)
    assert torch.cuda.max_memory_allocated() - before < 3 << 30
    torch.cuda.empty_cache()
    limit = (torch.cuda.memory_reserved() + (400 << 20)) / torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction(limit)
    try:
        again, _ = q.round_weights(permute, weights, importance, 16, 32, 8)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert torch.equal(again, symbols)


def test_encoder_of_no_rows_returns_nothing():
    import rptc
    sym, loss = rptc.quantize_rows(torch.randn(256, device="cuda"), torch.ones(5, device="cuda"), torch.empty(0, 5, device="cuda"))
    assert sym.shape == (0, 5) and sym.dtype == torch.int32 and loss.shape == (0,)


@pytest.mark.parametrize("L,n", [(4, 33), (6, 47), (6, 48), (6, 49), (8, 700), (11, 1000), (16, 64), (16, 127), (16, 1100)])
@pytest.mark.parametrize("parted", [False, True])
def test_trace_back_in_pieces(L, n, parted):
    """Pieces of a row are walked from guessed states.  `parted`: two cheap paths that stay apart for good, the states 0 and M - 1 -- the
    guess follows the one, the cheapest path is the other, and every piece has to be walked again."""
    import rptc
    M = 1 << L
    g = torch.Generator().manual_seed(L * 1000 + n)
    weights = 0.5 + torch.rand(n, generator=g)
    if parted:
        alphabet = torch.full((M,), 100.0)
        alphabet[0], alphabet[-1] = 1.0, -1.0
        samples = torch.zeros(2, n)
        samples[0, 0], samples[1, -1] = 1e4, -1e4             # cheapest: 0 throughout; M - 1 in the end, and so all the way to it
    else:
        alphabet = torch.randn(M, generator=g)
        samples = torch.randn(2, n, generator=g)
    want, want_loss = rptc.quantize_rows(alphabet, weights, samples)
    got, loss = rptc.quantize_rows(alphabet.cuda(), weights.cuda(), samples.cuda())
    assert torch.equal(got.cpu(), want)
    torch.testing.assert_close(loss.cpu(), want_loss, rtol=1e-6, atol=0)


@pytest.mark.parametrize("L,n,rows", [(8, 159, 3), (8, 160, 3), (12, 239, 5), (12, 240, 5), (6, 1023, 1025), (6, 1024, 1025), (6, 130, 2049), (16, 320, 6)])
def test_trace_back_by_a_warp_and_in_pieces(L, n, rows):
    """Both sides of the lines between them (pieces of a row, rows), and rows that do not fill the last CTA of four."""
    import rptc
    g = torch.Generator().manual_seed(L + n + rows)
    alphabet, weights, samples = torch.randn(1 << L, generator=g), 0.5 + torch.rand(n, generator=g), torch.randn(rows, n, generator=g)
    got, loss = rptc.quantize_rows(alphabet.cuda(), weights.cuda(), samples.cuda())
    some = slice(None) if rows < 8 else torch.cat([torch.arange(3), torch.arange(rows - 5, rows)])
    want, want_loss = rptc.quantize_rows(alphabet, weights, samples[some])
    assert torch.equal(got[some].cpu(), want)
    torch.testing.assert_close(loss[some].cpu(), want_loss, rtol=1e-6, atol=0)
    # the rest against itself: rows encoded by eights take a few CTAs
    for r0 in range(0, rows, 512):
        assert torch.equal(rptc.quantize_rows(alphabet.cuda(), weights.cuda(), samples[r0:r0 + 8].cuda())[0], got[r0:r0 + 8])
