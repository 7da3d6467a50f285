"""Builds librptc_b200.so (the C-ABI library, include/rptc_b200.h) in-tree with nvcc for sm_100a.

    python let-it-slide_b200/build.py [--force] [--verbose]

Each .cu under csrc/ is compiled to an object (in parallel, skipped when up to date) and linked
into let-it-slide_b200/librptc_b200.so.  No torch headers are involved: the library is plain CUDA
runtime code with an extern "C" surface.  csrc/torch_ext.cpp, the layers' forward passes as the interpreter
calls them, becomes rptc_b200/_native.so against torch's headers and libraries.
"""
from __future__ import annotations

import concurrent.futures as cf
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "librptc_b200.so")
EXT = os.path.join(HERE, "rptc_b200", "_native.so")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-lineinfo", "-std=c++17", "-Xcompiler", "-fPIC",
         "--expt-relaxed-constexpr", "-Xptxas", "-v"]


def _newer(src: str, dst: str, deps: list[str]) -> bool:
    if not os.path.exists(dst):
        return True
    t = os.path.getmtime(dst)
    return any(os.path.getmtime(d) > t for d in [src] + deps)


def _ext_command() -> list[str]:
    import sysconfig
    from importlib.util import find_spec
    torch_dir = os.path.dirname(find_spec("torch").origin)
    inc = [sysconfig.get_paths()["include"], os.path.join(torch_dir, "include"), os.path.join(torch_dir, "include", "torch", "csrc", "api", "include"),
           os.path.join(os.path.dirname(os.path.dirname(NVCC)), "include")]
    libs = os.path.join(torch_dir, "lib")
    return ["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-DNDEBUG", os.path.join(CSRC, "torch_ext.cpp"), "-o", EXT] + [
        a for i in inc for a in ("-isystem", i)] + ["-L" + libs, "-Wl,-rpath," + libs, "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda"]


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(OBJ, exist_ok=True)
    srcs = sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cuh")]
    deps.append(os.path.join(HERE, "..", "include", "rptc_b200.h"))
    jobs = []
    for f in srcs:
        src, obj = os.path.join(CSRC, f), os.path.join(OBJ, f[:-3] + ".o")
        if force or _newer(src, obj, deps):
            jobs.append((src, obj))

    ext_src = os.path.join(CSRC, "torch_ext.cpp")
    if force or _newer(ext_src, EXT, [deps[-1]]):
        jobs.append((ext_src, None))

    def compile_one(job):
        src, obj = job
        cmd = _ext_command() if obj is None else [NVCC, "-c", src, "-o", obj] + FLAGS
        return src, subprocess.run(cmd, capture_output=True, text=True)

    with cf.ThreadPoolExecutor(max_workers=os.cpu_count() or 4) as ex:
        for src, r in ex.map(compile_one, jobs):
            if verbose or r.returncode != 0:
                sys.stderr.write(r.stdout + r.stderr)
            if r.returncode != 0:
                raise RuntimeError(f"the compiler failed on {src}")
            if src == ext_src:
                continue
            with open(os.path.join(OBJ, os.path.basename(src)[:-3] + ".ptxas.txt"), "w") as fh:
                fh.write(r.stderr)
    objs = [os.path.join(OBJ, f[:-3] + ".o") for f in srcs]
    if force or jobs or not os.path.exists(LIB):
        r = subprocess.run([NVCC, "-shared", "-o", LIB] + objs + ["-gencode", "arch=compute_100a,code=sm_100a",
                                                                   "-Xcompiler", "-fPIC", "-lcudart"],
                           capture_output=True, text=True)
        if r.returncode != 0:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("link failed")
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
