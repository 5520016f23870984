"""Build libfla_b200.so in-tree with nvcc for sm_100a.

Usage: python build.py [--force] [--verbose]
Each .cu under csrc/ is compiled to an object (in parallel, skipped when up to date) and the
objects are linked into fla_b200/lib/libfla_b200.so; the C++ sources under csrc/host/ become the
PyTorch binding fla_b200/lib/_host.so, which calls that library.  No GPU is needed to build.
"""
from __future__ import annotations

import concurrent.futures as cf
import os
import subprocess
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parent
CSRC = ROOT / "csrc"
OBJ = ROOT / "build"
HOST = CSRC / "host"
LIB = ROOT / "fla_b200" / "lib" / "libfla_b200.so"
BINDING = LIB.parent / "_host.so"

NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
CXX = os.environ.get("CXX", "g++")
FLAGS = [
    "-std=c++17", "-O3", "-lineinfo",
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
    "--expt-relaxed-constexpr",
    "-I", str(CSRC),
] + os.environ.get("FLA_B200_NVCC_FLAGS", "").split()


def _deps_mtime() -> float:
    hdrs = list(CSRC.rglob("*.cuh")) + [h for h in CSRC.rglob("*.h") if HOST not in h.parents] + list((ROOT.parent / "include").glob("*.h"))
    return max((h.stat().st_mtime for h in hdrs), default=0.0)


def _torch_flags():
    import sysconfig

    import torch
    from torch.utils import cpp_extension as ext
    cuda = Path(NVCC).resolve().parent.parent
    libdir = Path(torch.__file__).resolve().parent / "lib"
    cflags = [f"-I{p}" for p in (*ext.include_paths(), sysconfig.get_paths()["include"], cuda / "include")]
    cflags.append(f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}")
    return cflags, [f"-L{libdir}", "-ltorch_python", "-ltorch", "-ltorch_cuda", "-ltorch_cpu", "-lc10_cuda", "-lc10", "-ldl"]


def _build_binding(ex, force: bool) -> None:
    srcs = sorted(HOST.glob("*.cpp"))
    newest_header = max([h.stat().st_mtime for h in (*HOST.glob("*.h"), *(ROOT.parent / "include").glob("*.h"))], default=0.0)
    cflags, libs = _torch_flags()

    def compile_one(src: Path) -> Path:
        obj = OBJ / f"host_{src.stem}.o"
        if force or not obj.exists() or obj.stat().st_mtime <= max(src.stat().st_mtime, newest_header):
            _run([CXX, "-std=c++17", "-O2", "-fPIC", "-fvisibility=hidden", *cflags, "-c", str(src), "-o", str(obj)], src.name)
        return obj
    objs = list(ex.map(compile_one, srcs))
    if force or not BINDING.exists() or any(o.stat().st_mtime > BINDING.stat().st_mtime for o in objs):
        _run([CXX, "-shared", "-o", str(BINDING), *map(str, objs), *libs], BINDING.name)


def _run(cmd, what: str) -> str:
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"{Path(cmd[0]).name} failed for {what}:\n{res.stdout}\n{res.stderr}")
    return res.stderr


def _compile(src: Path, force: bool, verbose: bool, hdr_mtime: float) -> Path:
    obj = OBJ / (src.stem + ".o")
    if not force and obj.exists() and obj.stat().st_mtime > max(src.stat().st_mtime, hdr_mtime):
        return obj
    cmd = [NVCC, *FLAGS, "-c", str(src), "-o", str(obj)]
    if verbose:
        cmd.insert(1, "-Xptxas")
        cmd.insert(2, "-v")
    err = _run(cmd, src.name)
    if verbose:
        sys.stderr.write(err)
    return obj


def build(force: bool = False, verbose: bool = False) -> Path:
    OBJ.mkdir(exist_ok=True)
    LIB.parent.mkdir(parents=True, exist_ok=True)
    srcs = sorted(CSRC.glob("*.cu"))
    hdr_mtime = _deps_mtime()
    with cf.ThreadPoolExecutor(max_workers=min(8, len(srcs))) as ex:
        objs = list(ex.map(lambda s: _compile(s, force, verbose, hdr_mtime), srcs))
        _build_binding(ex, force)
    if force or not LIB.exists() or any(o.stat().st_mtime > LIB.stat().st_mtime for o in objs):
        _run([NVCC, "-shared", "-o", str(LIB), *map(str, objs), "-lcudart_static", "-lpthread", "-ldl", "-lrt"], LIB.name)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
