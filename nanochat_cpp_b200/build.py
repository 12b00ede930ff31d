"""Builds libmxb200.so (the C-ABI library, nvcc for sm_100a) and _torch_engine.so (the engine's native host path, a
torch extension over that C ABI) in-tree.

    python nanochat_cpp_b200/build.py          # rebuild when a source is newer than the library

nvcc cross-compiles without a GPU. The library links the CUDA runtime statically and takes the one driver
entry point it needs (cuTensorMapEncodeTiled) through cudaGetDriverEntryPoint, so it has no link-time
dependency beyond libc/libstdc++.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libmxb200.so")
ENGINE = os.path.join(HERE, "_torch_engine.so")
ENGINE_SOURCE = os.path.join(CSRC, "torch_engine.cpp")
SOURCES = ["capi.cu", "quantize_sm100.cu", "residual_norm_sm100.cu", "softcap_ce_sm100.cu", "gemm_sm100.cu"]
FLAGS = ["-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo",
         "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden", "--cudart", "static"]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; libmxb200.so cannot be built")


def have_nvcc() -> bool:
    try:
        _nvcc()
        return True
    except RuntimeError:
        return False


def _stale(target: str, deps: list) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps + [os.path.join(ROOT, "include", "mxb200.h"), __file__])


def _run(cmd: list, what: str, verbose: bool) -> None:
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if verbose or r.returncode != 0:
        sys.stderr.write(r.stdout)
    if r.returncode != 0:
        raise RuntimeError(f"{what} failed")


def _built_for() -> str:
    """What _torch_engine.so depends on beside its sources, as it is compiled into it: torch's and Python's C++ interfaces."""
    import torch
    return f"mxb200-engine-for torch {torch.__version__} {sysconfig.get_config_var('SOABI')};"


def _engine_stale() -> bool:
    if _stale(ENGINE, [ENGINE_SOURCE]):
        return True
    with open(ENGINE, "rb") as f:
        return _built_for().encode() not in f.read()


def build_engine(force: bool = False, verbose: bool = False) -> str:
    """The torch extension; needs libmxb200.so beside it (found again at run time through $ORIGIN)."""
    if not force and not _engine_stale():
        return ENGINE
    import torch
    tdir = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(_nvcc())))
    inc = [os.path.join(ROOT, "include"), os.path.join(tdir, "include"),
           os.path.join(tdir, "include", "torch", "csrc", "api", "include"), os.path.join(cuda, "include"),
           sysconfig.get_paths()["include"]]
    tmp = f"{ENGINE}.{os.getpid()}"
    _run(["g++", "-std=c++20", "-O2", "-fPIC", "-shared", "-fvisibility=hidden", "-DTORCH_EXTENSION_NAME=_torch_engine",
          "-DTORCH_API_INCLUDE_EXTENSION_H", f'-DMXB200_BUILT_FOR="{_built_for()}"',
          f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
          *(x for d in inc for x in ("-isystem" if d.startswith(tdir) else "-I", d)), ENGINE_SOURCE, "-o", tmp,
          "-L", HERE, "-l:libmxb200.so", "-L", os.path.join(tdir, "lib"), "-ltorch_python", "-ltorch", "-ltorch_cpu",
          "-ltorch_cuda", "-lc10", "-lc10_cuda", "-Wl,-rpath,$ORIGIN"], "build of _torch_engine.so", verbose)
    os.replace(tmp, ENGINE)
    return ENGINE


def build(force: bool = False, verbose: bool = False) -> str:
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if not f.endswith(".cpp")]
    if not force and not _stale(LIB, deps):
        build_engine(force, verbose)
        return LIB
    objs = []
    bdir = os.path.join(HERE, "build")
    os.makedirs(bdir, exist_ok=True)
    procs = []
    for src in SOURCES:
        obj = os.path.join(bdir, src.replace(".cu", ".o"))
        cmd = [_nvcc(), *FLAGS, "-I", os.path.join(ROOT, "include"), "-I", CSRC, "-c", os.path.join(CSRC, src), "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(obj)
    for src, p in procs:
        out, _ = p.communicate()
        if verbose or p.returncode != 0:
            sys.stderr.write(out)
        if p.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}")
    link = [_nvcc(), "-shared", "--cudart", "static", "-gencode", "arch=compute_100a,code=sm_100a", "-o", LIB, *objs]
    _run(link, "link of libmxb200.so", verbose)
    build_engine(force, verbose)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
