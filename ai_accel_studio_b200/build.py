"""Build ``libqgemv_b200.so`` in-tree with nvcc for sm_100a.

    python -m ai_accel_studio_b200.build [--force] [--verbose]
"""
from __future__ import annotations

import argparse
import os
import shutil
import subprocess
import sys
import sysconfig
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
LIB = PKG / "libqgemv_b200.so"
NATIVE = PKG / ("_native" + sysconfig.get_config_var("EXT_SUFFIX"))      # host side of eager calls, links the library above
# (source, extra defines, object name).  The tensor-core-assisted kernels are compiled in parts (per bit width; per
# path and activation type) so that the objects build in parallel.
UNITS = [
    ("qgemv_api.cu", [], "qgemv_api.o"),
    ("qgemv_simt.cu", [], "qgemv_simt.o"),
    ("qdequant.cu", [], "qdequant.o"),
    ("qpack.cu", [], "qpack.o"),
    ("qgemm.cu", [], "qgemm.o"),
    ("qcomm.cu", [], "qcomm.o"),
    ("qdecode.cu", [], "qdecode.o"),
    ("qgemv_mma.cu", ["-DQGEMV_INST_BITS=2"], "qgemv_mma_int2.o"),
    ("qgemv_mma.cu", ["-DQGEMV_INST_BITS=4"], "qgemv_mma_int4.o"),
    ("qgemv_pipe.cu", ["-DQGEMV_INST_BITS=2"], "qgemv_pipe_int2.o"),
    ("qgemv_pipe.cu", ["-DQGEMV_INST_BITS=4"], "qgemv_pipe_int4.o"),
    ("qgemv_plan.cu", [], "qgemv_plan.o"),
    *(("qgemv_stream.cu", [f"-DQGEMV_STREAM_MODE={m}", f"-DQGEMV_STREAM_BF16={b}"], f"qgemv_stream_{m}{b}.o") for m in range(3) for b in range(2)),
    ("qgemv_held_plan.cu", [], "qgemv_held_plan.o"),
    *(("qgemv_held.cu", [f"-DQGEMV_HELD_FMT={f}", f"-DQGEMV_HELD_BF16={b}"], f"qgemv_held_{f}{b}.o") for f in range(5) for b in range(2)),
]
OBJDIR = CSRC / "build"
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
]
# No --use_fast_math: the dequantisation kernels must round exactly like IEEE arithmetic.


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found; set NVCC or install the CUDA toolkit (12.8 or newer for sm_100a)")


def _stale(target: Path = LIB, patterns=("*.cu", "*.cuh")) -> bool:
    if not target.exists():
        return True
    t = target.stat().st_mtime
    deps = [d for pat in patterns for d in CSRC.glob(pat)] + list((PKG.parent / "include").glob("*.h"))
    return any(d.stat().st_mtime > t for d in deps)


def build_native(force: bool = False) -> Path:
    """The CPython extension with the host side of eager calls (csrc/qtorch.cpp); needs the library to link against."""
    if not force and not _stale(NATIVE, ("qtorch.cpp",)):
        return NATIVE
    import torch
    from torch.utils import cpp_extension
    libdir = Path(torch.__file__).parent / "lib"
    cuda_inc = Path(_nvcc()).resolve().parent.parent / "include"
    cmd = ["g++", "-O2", "-std=c++17", "-shared", "-fPIC", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           *[f"-I{p}" for p in cpp_extension.include_paths()], f"-I{cuda_inc}", f"-I{sysconfig.get_paths()['include']}",
           str(CSRC / "qtorch.cpp"), "-o", str(NATIVE), f"-L{PKG}", "-l:" + LIB.name, f"-L{libdir}", "-lc10", "-lc10_cuda", "-ltorch_cpu",
           "-ltorch", "-ltorch_python", "-Wl,-rpath,$ORIGIN"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"building {NATIVE.name} failed ({res.returncode}):\n{res.stdout}\n{res.stderr}")
    return NATIVE


def build(force: bool = False, verbose: bool = False, extra_flags: tuple = (), lib: Path = LIB) -> Path:
    """Compile the library if it is missing or older than its sources; return its path.

    ``extra_flags`` (e.g. ``("-DQGEMV_TRACE",)``) and ``lib`` let a measurement build sit beside the
    product build; objects of such a build go to their own directory."""
    if not force and not extra_flags and lib == LIB and not _stale():
        build_native()
        return lib
    nvcc = _nvcc()
    objdir = OBJDIR if not extra_flags else OBJDIR.with_name("build_" + "".join(c for c in "".join(extra_flags) if c.isalnum()))
    objdir.mkdir(parents=True, exist_ok=True)
    procs = []
    for src, defs, obj in UNITS:
        cmd = [nvcc, *NVCC_FLAGS, *defs, *extra_flags, "-c", str(CSRC / src), "-o", str(objdir / obj)]
        if verbose:
            cmd[1:1] = ["-Xptxas", "-v"]
            print(" ".join(cmd), flush=True)
        procs.append((cmd, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.PIPE, text=True)))
    failed = []
    for cmd, pr in procs:
        out, err = pr.communicate()
        if pr.returncode != 0:
            failed.append(f"{' '.join(cmd)}\n{out}\n{err}")
        elif verbose:
            print(err)
    if failed:
        raise RuntimeError("nvcc failed:\n" + "\n".join(failed))
    link = [nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-Xcompiler", "-fPIC", "-o", str(lib),
            *[str(objdir / obj) for _, _, obj in UNITS]]
    res = subprocess.run(link, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"link failed ({res.returncode}):\n{res.stdout}\n{res.stderr}")
    if lib == LIB:
        build_native(force)
    return lib


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    ap.add_argument("--define", action="append", default=[], help="extra -D flag for a measurement build, e.g. QGEMV_TRACE")
    ap.add_argument("--output", default=None, help="library path of a measurement build (default: the product library)")
    a = ap.parse_args()
    print(build(a.force, a.verbose, tuple("-D" + d for d in a.define), Path(a.output) if a.output else LIB))
    sys.exit(0)
