"""Build libturboquant_b200.so in-tree with nvcc for sm_100a.

    python turboquant-pytorch_b200/build.py [--force] [--verbose]

The library lands next to the Python package (turboquant/libturboquant_b200.so)
so that it is found without installation.  The CUDA runtime is linked
statically; the driver API is resolved at run time, so the library loads on a
machine without a GPU.
"""

from __future__ import annotations

import argparse
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUT = os.path.join(HERE, "turboquant", "libturboquant_b200.so")
SOURCES = ["tq_api.cu", "tq_simt.cu", "tq_few.cu", "tq_umma.cu", "tq_qjl_umma.cu", "tq_v2_umma.cu", "tq_score_static.cu", "tq_copy.cu", "tq_attn_mma.cu", "tq_qjl_packed.cu"]
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
HOST_SRC = os.path.join(CSRC, "tq_host.cpp")
HOST_OUT = os.path.join(HERE, "turboquant", "_tq_host.so")
HOST_STAMP = os.path.join(HERE, "turboquant", "_tq_host.built_for")


def nvcc_path() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; the CUDA extension cannot be built")
    return exe


def sources():
    return [os.path.join(CSRC, s) for s in SOURCES if os.path.exists(os.path.join(CSRC, s))]


def stale() -> bool:
    if not os.path.exists(OUT):
        return True
    t = os.path.getmtime(OUT)
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC)] + [os.path.join(HERE, "..", "include", "turboquant_b200.h")]
    return any(os.path.getmtime(d) > t for d in deps)


def host_built_for() -> str:
    """What the host extension has to be built for again: it is linked against torch and includes its headers."""
    import sysconfig

    import torch
    return f"torch {torch.__version__} {sysconfig.get_config_var('SOABI')}\n"


def build_host(force: bool = False) -> str:
    """Compile the Python extension that fills in and submits the jobs (no kernels in it).  What it was built for is
    written beside it: a module of another torch is rebuilt here and not loaded by the package."""
    deps = [HOST_SRC, os.path.join(HERE, "..", "include", "turboquant_b200.h")]
    want = host_built_for()
    if not force and os.path.exists(HOST_OUT) and all(os.path.getmtime(d) <= os.path.getmtime(HOST_OUT) for d in deps):
        if os.path.exists(HOST_STAMP) and open(HOST_STAMP).read() == want:
            return HOST_OUT
    import sysconfig

    import torch
    root = os.path.dirname(os.path.abspath(torch.__file__))
    cuda = os.path.join(os.path.dirname(nvcc_path()), "..", "include")
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}", "-I" + sysconfig.get_paths()["include"],
           "-I" + os.path.join(root, "include"), "-I" + os.path.join(root, "include", "torch", "csrc", "api", "include"),
           "-I" + cuda, "-o", HOST_OUT, HOST_SRC, "-L" + os.path.join(root, "lib"), "-lc10", "-lc10_cuda", "-ltorch_cpu",
           "-ltorch_python"]
    print(" ".join(cmd), flush=True)
    if os.path.exists(HOST_STAMP):
        os.remove(HOST_STAMP)
    subprocess.check_call(cmd)
    with open(HOST_STAMP, "w") as f:
        f.write(want)
    return HOST_OUT


def build(force: bool = False, verbose: bool = False, ablate: bool = False, out: str = OUT, defines=()) -> str:
    """Compile the library.  `ablate` adds -DTQ_ABLATION: the timing-only switches that skip parts of the
    tensor-core kernels (environment variable TQ_ABLATE) exist only in such a build; give it its own `out`
    path and load it through TURBOQUANT_B200_LIB, never as the in-tree library."""
    if ablate and os.path.abspath(out) == os.path.abspath(OUT):
        raise ValueError("an ablation build must not replace the in-tree library: pass --out")
    if out == OUT:
        build_host(force)
    if not force and out == OUT and not stale():
        return OUT
    # --fmad=false: products that the reference rounds before adding (k_mse before the
    # residual, for one) must not be contracted; the kernels call fmaf() where they want one.
    cmd = [nvcc_path(), *ARCH, "-lineinfo", "-O3", "-std=c++17", "--fmad=false", "--threads", "0", "-shared",
           "-Xcompiler", "-fPIC", "-Xcompiler", "-ffp-contract=off", "-o", out, *sources()]
    if ablate:
        cmd.insert(1, "-DTQ_ABLATION")
    for d in defines:
        cmd.insert(1, "-D" + d)
    if verbose:
        cmd.insert(1, "-Xptxas")
        cmd.insert(2, "-v")
    print(" ".join(cmd), flush=True)
    subprocess.check_call(cmd)
    return out


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    ap.add_argument("--ablate", action="store_true", help="profiling build with the TQ_ABLATE switches (needs --out)")
    ap.add_argument("--out", default=OUT)
    ap.add_argument("-D", dest="defines", action="append", default=[], help="extra preprocessor definitions")
    a = ap.parse_args()
    print(build(force=a.force or a.out != OUT, verbose=a.verbose, ablate=a.ablate, out=a.out, defines=a.defines))
