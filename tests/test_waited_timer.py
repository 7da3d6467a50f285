"""The memory behind a matvec that its caller waits for: set up whole or not at all."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_timer_is_set_up_whole_or_not_at_all(tmp_path):
    """Every runtime call fails in turn: nothing is left allocated, and the next call sets all of it up."""
    exe = str(tmp_path / "waited_timer")
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"))), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-isystem", cuda, os.path.join(HERE, "waited_timer.cpp"), "-o", exe], check=True)
    assert subprocess.run([exe], capture_output=True, text=True).stdout == ""
    assert subprocess.run([exe]).returncode == 0

