"""The memory behind a matvec that its caller waits for: set up whole or not at all, and beside another thread's capture."""
import os
import subprocess
import sys
import threading

import pytest
import torch

HERE = os.path.dirname(os.path.abspath(__file__))


def test_timer_is_set_up_whole_or_not_at_all(tmp_path):
    """Every runtime call fails in turn: nothing is left allocated, the next call sets all of it up, and none of them is made in a capture
    mode in which another thread's capture forbids it."""
    exe = str(tmp_path / "waited_timer")
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"))), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-isystem", cuda, os.path.join(HERE, "waited_timer.cpp"), "-o", exe], check=True)
    assert subprocess.run([exe], capture_output=True, text=True).stdout == ""
    assert subprocess.run([exe]).returncode == 0


@pytest.mark.gpu
def test_first_timed_matvec_of_a_thread_while_another_captures():
    """In the default capture mode a thread's calls that allocate are refused while another captures, and spoil the capture.  A thread's first
    timed matvec sets its timer up, its end gives it back."""
    from rptc_b200 import CODE_HASH, LAYOUT_CHUNKED, LAYOUT_UNITMAJOR, Format, ops
    from rptc_b200._lib import native
    m = n = 2048
    g = torch.Generator(device="cuda").manual_seed(1)
    codes = torch.randint(-2**31, 2**31 - 1, (m * n // 16,), dtype=torch.int32, device="cuda", generator=g)
    x = torch.randn(n, dtype=torch.float16, device="cuda", generator=g)
    for layout in (LAYOUT_CHUNKED, LAYOUT_UNITMAJOR):
        fmt = Format(CODE_HASH, 2, 16, 8, layout)
        lut = torch.randn(fmt.lut_numel(), dtype=torch.float16, device="cuda", generator=g)
        acc, y = torch.zeros((1, m), device="cuda"), torch.empty(m, dtype=torch.float16, device="cuda")
        assert native().gemv_timed(codes, lut, x, acc, y, m, n, 0, 0, fmt) > 0
        want, done = y.clone(), []
        y.zero_()
        side, a = torch.cuda.Stream(), torch.zeros(64, device="cuda")
        torch.cuda.synchronize()

        def work():
            with torch.cuda.stream(side):
                done.append(native().gemv_timed(codes, lut, x, acc, y, m, n, 0, 0, fmt))

        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            a += 1
            thread = threading.Thread(target=work)
            thread.start()
            thread.join()
            a += 1
        graph.replay()
        torch.cuda.synchronize()
        assert done and type(done[0]) is float and done[0] > 0
        # UNITMAJOR adds its sums up in any order
        assert torch.equal(y, want) if layout == LAYOUT_CHUNKED else (y - want).float().norm() <= 1e-3 * want.float().norm()
        assert (a == 2).all()
    ops.device_status()


_UNDER_CAPTURE = """
import torch
from rptc_b200 import CODE_HASH, LAYOUT_CHUNKED, Format
from rptc_b200._lib import native
m = n = 2048
fmt = Format(CODE_HASH, 2, 16, 8, LAYOUT_CHUNKED)
codes, lut = torch.zeros(m * n // 16, dtype=torch.int32, device="cuda"), torch.ones(fmt.lut_numel(), dtype=torch.float16, device="cuda")
x, y, acc, a = torch.ones(n, device="cuda").half(), torch.zeros(m, device="cuda").half(), torch.zeros((1, m), device="cuda"), torch.zeros(1, device="cuda")
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
try:
    with torch.cuda.graph(graph):
        a += 1
        status = native().gemv_timed(codes, lut, x, acc, y, m, n, 0, 0, fmt)
    ended = False
except RuntimeError as e:
    ended = "capture" in str(e)
torch.cuda.synchronize()
assert ended and status == -5 and not a.any() and not y.any(), (ended, status)
assert native().gemv_timed(codes, lut, x, acc, y, m, n, 0, 0, fmt) > 0 and y.any()
print("refused")
"""


@pytest.mark.gpu
def test_timed_matvec_is_refused_on_a_stream_under_capture():
    """There is no result to wait for, and no graph may come of a capture that holds the kernel.  In a process of its own: torch's generators stay
    in the state of a capture that ended with an error."""
    env = dict(os.environ, PYTHONPATH=os.path.join(os.path.dirname(HERE), "let-it-slide_b200"))
    r = subprocess.run([sys.executable, "-c", _UNDER_CAPTURE], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "refused", r.stdout + r.stderr
