"""What the layers' native calls refuse: buffers of another type, size or place than the kernels read.  The checks come before anything
is launched, so that everything here but the tests of devices runs without a GPU."""
import pytest
import torch


def _packed(device="cpu", bias=True):
    import quantize_hf as q
    return q.FactorizedRPTCLinear(64, 128, 8, 2, bias, device=device)


def _linear(device="cpu"):
    from rptc_b200 import Format
    from rptc_b200.linear import RPTCLinear
    return RPTCLinear.random(256, 256, Format(), 0.02, 1, device=device)


PACKED = ["codes", "alphabets", "biases_out", "biases_in", "scales_out", "scales_in", "bias"]
LINEAR = ["codes", "lut", "signs_in", "signs_out"]
MAKE = {"packed": (_packed, 128, PACKED), "linear": (_linear, 256, LINEAR)}


@pytest.mark.parametrize("kind,cast,name", [("packed", torch.float16, "biases_out"), ("packed", torch.bfloat16, "alphabets"), ("packed", torch.float64, "alphabets"),
                                            ("linear", torch.float32, "lut"), ("linear", torch.bfloat16, "lut")])
def test_a_layer_that_was_cast_is_refused(kind, cast, name):
    make, n, _ = MAKE[kind]
    layer = make().to(cast)
    with pytest.raises(RuntimeError, match=f"{name} must have dtype"):
        layer(torch.zeros(1, n, dtype=torch.float16))


@pytest.mark.parametrize("kind,name", [(k, n) for k in MAKE for n in MAKE[k][2]])
def test_a_buffer_of_another_type_size_or_stride_is_refused(kind, name):
    make, n, _ = MAKE[kind]
    x = torch.zeros(3, n, dtype=torch.float16)
    good = make()
    t = getattr(good, name)
    for bad, what in ((t.to(torch.int16), "must have dtype"), (t.reshape(-1)[:-8].clone(), "elements, got"), (t.reshape(-1).repeat_interleave(2)[::2], "must be contiguous")):
        layer = make()
        layer._buffers[name] = bad
        with pytest.raises(RuntimeError, match=f"{name} .*{what}"):
            layer(x)


@pytest.mark.parametrize("kind", list(MAKE))
def test_a_layer_on_the_cpu_is_refused(kind):
    make, n, _ = MAKE[kind]
    with pytest.raises(RuntimeError, match="codes must be a CUDA tensor"):
        make()(torch.zeros(1, n, dtype=torch.float16))


@pytest.mark.gpu
@pytest.mark.parametrize("kind,name", [(k, n) for k in MAKE for n in MAKE[k][2]])
def test_a_buffer_that_does_not_fit_is_refused_on_the_gpu(kind, name):
    make, n, _ = MAKE[kind]
    x = torch.zeros(3, n, dtype=torch.float16, device="cuda")
    layer = make("cuda")
    t = getattr(layer, name)
    for bad, what in ((t.to(torch.int16), "must have dtype"), (t.reshape(-1)[:-8].clone(), "elements, got"), (t.reshape(-1).repeat_interleave(2)[::2], "must be contiguous"),
                      (t.cpu(), "must be a CUDA tensor")):
        layer._buffers[name] = bad
        with pytest.raises(RuntimeError, match=f"{name} .*{what}"):
            layer(x)
    layer._buffers[name] = t
    assert torch.isfinite(layer(x)).all()
    with pytest.raises(RuntimeError, match="x must be a CUDA tensor"):
        layer(x.cpu())


@pytest.mark.parametrize("kind", list(MAKE))
def test_an_attribute_that_is_missing_is_an_attribute_error(kind):
    make, n, names = MAKE[kind]
    layer = make()
    delattr(layer, names[1])
    with pytest.raises(AttributeError, match=names[1]):
        layer(torch.zeros(1, n, dtype=torch.float16))


@pytest.mark.gpu
def test_buffers_replaced_by_parameters_are_found():
    """Assigning an nn.Parameter to the name of a buffer moves it among the module's parameters (a bias that is to be trained)."""
    layer, x = _packed("cuda"), torch.ones(3, 128, device="cuda")
    layer.bias.copy_(torch.arange(64.0))
    want = layer(x)
    layer.bias = torch.nn.Parameter(layer.bias.clone())
    layer.scales_out = torch.nn.Parameter(layer.scales_out.clone())
    assert "bias" not in layer._buffers
    assert torch.equal(layer(x), want)


@pytest.mark.gpu
def test_a_cast_packed_layer_is_refused_on_the_gpu():
    x = torch.zeros(1, 128, dtype=torch.float16, device="cuda")
    for cast in (torch.float16, torch.bfloat16):
        with pytest.raises(RuntimeError, match="must have dtype"):
            _packed("cuda").to(cast)(x)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", list(MAKE))
def test_out_of_memory_is_torchs_own_exception(kind):
    import quantize_hf as q
    from rptc_b200 import Format
    from rptc_b200.linear import RPTCLinear
    layer = q.FactorizedRPTCLinear(8192, 256, 8, 2, device="cuda") if kind == "packed" else RPTCLinear.random(256, 8192, Format(), 0.02, 1)
    x = torch.zeros(60000, 256, dtype=torch.float16, device="cuda")               # a result of 1 GB
    torch.cuda.empty_cache()
    limit = (torch.cuda.memory_reserved() + (64 << 20)) / torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction(limit)
    try:
        with pytest.raises(torch.OutOfMemoryError):
            layer(x)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", list(MAKE))
def test_other_threads_run_while_a_layer_waits_for_room_in_the_stream(kind):
    """A stream holds about a thousand launches; a call that finds it full waits, and the interpreter does not wait with it."""
    import threading
    import time
    make, n, _ = MAKE[kind]
    layer, x = make("cuda"), torch.zeros(1, n, dtype=torch.float16, device="cuda")
    layer(x)
    torch.cuda.synchronize()
    start, stop = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    gaps, done = [0.0], threading.Event()

    def tick():
        last = time.perf_counter()
        while not done.is_set():
            time.sleep(0.001)
            now = time.perf_counter()
            gaps[0], last = max(gaps[0], now - last), now

    thread = threading.Thread(target=tick)
    thread.start()
    start.record()
    torch.cuda._sleep(1_500_000_000)                # the better part of a second
    for _ in range(1500):
        layer(x)
    stop.record()
    torch.cuda.synchronize()
    done.set()
    thread.join()
    busy = start.elapsed_time(stop) * 1e-3
    assert busy > 0.4 and gaps[0] < 0.5 * busy, (busy, gaps[0])


@pytest.mark.gpu
@pytest.mark.parametrize("kind", list(MAKE))
def test_buffers_written_right_in_front_of_a_call_are_the_ones_it_reads(kind):
    """Stream order holds for a layer's buffers: a product that fetches codes and table ahead of its activations does not run
    ahead of a copy into them."""
    import quantize_hf as q
    from rptc_b200 import CODE_LUT, LAYOUT_TILED, Format
    from rptc_b200.linear import RPTCLinear
    n, m = 1024, 4096
    g = torch.Generator(device="cuda").manual_seed(7)

    def make():
        if kind == "linear":
            return RPTCLinear.random(n, m, Format(CODE_LUT, 2, 16, 0, LAYOUT_TILED), 0.02, int(torch.randint(0, 1000, (1,))))
        rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
        return q.FactorizedRPTCLinear.from_parts(torch.randint(0, 4, (m, n), generator=g, device="cuda", dtype=torch.int32), rnd(8, 1 << 16), rnd(m), rnd(n),
                                                 rnd(m), rnd(n))
    sides = [make(), make()]
    x = torch.randn(12, n, generator=g, device="cuda").half()                  # nine rows and more: the same bits every time
    want = [side(x) for side in sides]
    layer = make()
    names = [k for k, v in layer._buffers.items() if v is not None]
    results = []
    for i in range(100):
        for name in names:
            layer._buffers[name].copy_(sides[i & 1]._buffers[name])
        results.append(layer(x))
    for i, y in enumerate(results):
        assert torch.equal(y, want[i & 1]), i
