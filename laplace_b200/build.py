"""Builds liblaplace_cuda.so (sm_100a only) and _native.so, its torch binding, next to this file.

The shared library is the product; Python only loads it through ctypes. The
build is a plain nvcc invocation per source so that it works without a GPU
(nvcc cross-compiles) and leaves the .so in-tree.
"""
from __future__ import annotations

import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
ROOT = PKG.parent
LIB = PKG / "liblaplace_cuda.so"
NATIVE = PKG / "_native.so"

SOURCES = ["lp_api.cu", "lp_gemv.cu", "lp_quantize.cu", "lp_gemm_sa.cu", "lp_peak.cu", "lp_gguf.cu", "lp_types.cu", "lp_gemm_i8.cu", "lp_gemm_pair.cu", "lp_gemm_i8_tiles.cu"]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "--fmad=true",            # explicit __f*_rn intrinsics guard the quantizer's separate ops
    "-Xcompiler", "-fPIC",
    "-I", str(ROOT / "include"), "-I", str(CSRC),
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.sep not in cand or os.path.exists(cand)):
            return cand
    raise RuntimeError("nvcc not found")


def _stale(out: Path, deps: list[Path]) -> bool:
    if not out.exists():
        return True
    t = out.stat().st_mtime
    return any(d.stat().st_mtime > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compiles every source that is newer than its object, then links."""
    objdir = PKG / "build"
    objdir.mkdir(exist_ok=True)
    headers = list(CSRC.glob("*.cuh")) + [ROOT / "include" / "laplace_cuda.h"]
    nvcc = _nvcc()
    jobs = []
    for src in SOURCES:
        s = CSRC / src
        o = objdir / (s.stem + ".o")
        if force or _stale(o, [s] + headers):
            cmd = [nvcc, *NVCC_FLAGS, "-c", str(s), "-o", str(o)]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
            jobs.append(cmd)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("nvcc failed:\n" + " ".join(cmd) + "\n" + r.stdout + r.stderr)
        return r.stderr

    with ThreadPoolExecutor(max_workers=4) as ex:
        for log in ex.map(run, jobs):
            if verbose and log:
                print(log)
    objs = [objdir / (Path(s).stem + ".o") for s in SOURCES]
    if force or jobs or _stale(LIB, objs):
        cmd = [nvcc, "-shared", "-o", str(LIB), *map(str, objs), "-gencode", "arch=compute_100a,code=sm_100a"]
        run(cmd)
    build_native(force)
    return LIB


def _native_abi() -> str | None:
    """What _native.so is built against besides its sources: torch's headers and the interpreter. None: torch is not installed."""
    import sysconfig
    from importlib import metadata
    try:
        return f"torch {metadata.version('torch')}\npython {sysconfig.get_config_var('SOABI')}\n"
    except metadata.PackageNotFoundError:
        return None


def build_native(force: bool = False) -> Path | None:
    """The host side of the calls on torch tensors (lp_torch.cpp): a CPython module against torch's own headers. Built again when
    torch or the interpreter is another one; left out (device.py then makes its calls through ctypes) where torch is not installed."""
    src = CSRC / "lp_torch.cpp"
    abi, stamp = _native_abi(), PKG / "build" / "_native.abi"
    if abi is None:
        print("torch is not installed: _native.so is left out, the C library does not need it", file=sys.stderr)
        return None
    if force or _stale(NATIVE, [src, ROOT / "include" / "laplace_cuda.h"]) or not stamp.exists() or stamp.read_text() != abi:
        import sysconfig

        import torch
        t = Path(torch.__file__).resolve().parent
        cuda = Path(_nvcc()).resolve().parent.parent if os.path.sep in _nvcc() else Path("/usr/local/cuda")
        cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
               *(f"-I{d}" for d in (ROOT / "include", t / "include", t / "include" / "torch" / "csrc" / "api" / "include", cuda / "include", sysconfig.get_path("include"))),
               str(src), "-o", str(NATIVE), f"-L{t / 'lib'}", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python", f"-Wl,-rpath,{t / 'lib'}"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("the torch binding failed to build:\n" + " ".join(cmd) + "\n" + r.stdout + r.stderr)
        stamp.parent.mkdir(exist_ok=True)
        stamp.write_text(abi)
    return NATIVE


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(LIB)
