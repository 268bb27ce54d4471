"""In-tree build of the sm_100a kernel library ``libnpa_b200.so`` and of the torch binding ``_torch_ops.so``.

``python -m npa_b200.build`` (or :func:`build`) compiles every ``csrc/*.cu`` with
nvcc for ``sm_100a`` (one object per translation unit, in parallel) and links
them into ``npa_b200/libnpa_b200.so`` next to this file.  nvcc cross-compiles,
so no GPU is needed to build.  Objects are rebuilt only when a source or header
is newer than the object.  ``csrc/torch_ops.cpp`` (the autograd nodes) is compiled by the host compiler
against torch's headers and linked to the library next to it.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG_DIR = Path(__file__).resolve().parent
SRC_DIR = PKG_DIR / "csrc"
OBJ_DIR = PKG_DIR / "_build"
LIB_PATH = PKG_DIR / "libnpa_b200.so"
OPS_SRC = SRC_DIR / "torch_ops.cpp"
OPS_PATH = PKG_DIR / "_torch_ops.so"
INCLUDE_DIR = PKG_DIR.parent / "include"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-lineinfo", "-std=c++17",
    "-Xcompiler", "-fPIC",
    "--expt-relaxed-constexpr",
    "--compress-mode=size",  # the library is a hundred megabytes of sparse device code otherwise
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; the npa_b200 kernels cannot be built")
    return exe


def _headers_mtime() -> float:
    hdrs = list(SRC_DIR.glob("*.cuh")) + list(INCLUDE_DIR.glob("*.h"))
    return max(h.stat().st_mtime for h in hdrs)


def _compile(src: Path, verbose: bool, extra: list[str]) -> Path:
    obj = OBJ_DIR / (src.stem + ".o")
    newest = max(src.stat().st_mtime, _headers_mtime())
    if obj.exists() and obj.stat().st_mtime >= newest:
        return obj
    cmd = [_nvcc(), *NVCC_FLAGS, *extra, "-I", str(INCLUDE_DIR), "-c", str(src), "-o", str(obj)]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if verbose and (res.stdout or res.stderr):
        sys.stderr.write(f"--- {src.name}\n{res.stdout}{res.stderr}")
    if res.returncode != 0:
        raise RuntimeError(f"nvcc failed on {src.name}:\n{res.stdout}\n{res.stderr}")
    return obj


def _compile_ops(verbose: bool) -> Path:
    """The torch binding: object file only (it is linked once the kernel library exists)."""
    obj = OBJ_DIR / "torch_ops.o"
    newest = max(OPS_SRC.stat().st_mtime, max(h.stat().st_mtime for h in INCLUDE_DIR.glob("*.h")))
    if obj.exists() and obj.stat().st_mtime >= newest:
        return obj
    import torch
    from torch.utils.cpp_extension import include_paths

    includes = [arg for p in (*include_paths(), Path(_nvcc()).resolve().parent.parent / "include",
                              sysconfig.get_paths()["include"]) for arg in ("-isystem", str(p))]
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-DTORCH_EXTENSION_NAME=_torch_ops",
           "-DTORCH_API_INCLUDE_EXTENSION_H", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           *includes, "-c", str(OPS_SRC), "-o", str(obj)]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if verbose and (res.stdout or res.stderr):
        sys.stderr.write(f"--- {OPS_SRC.name}\n{res.stdout}{res.stderr}")
    if res.returncode != 0:
        raise RuntimeError(f"g++ failed on {OPS_SRC.name}:\n{res.stdout}\n{res.stderr}")
    return obj


def _link_ops(obj: Path) -> None:
    if OPS_PATH.exists() and OPS_PATH.stat().st_mtime >= obj.stat().st_mtime:
        return
    from torch.utils.cpp_extension import library_paths

    dirs = [arg for p in library_paths() for arg in (f"-L{p}", f"-Wl,-rpath,{p}")]
    cmd = ["g++", "-shared", "-o", str(OPS_PATH), str(obj), f"-L{PKG_DIR}", "-l:libnpa_b200.so", "-Wl,-rpath,$ORIGIN", *dirs,
           "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"link of {OPS_PATH.name} failed:\n{res.stdout}\n{res.stderr}")


def build(verbose: bool = False, force: bool = False, ptxas_info: bool = False) -> Path:
    """Compile and link the library; returns its path."""
    OBJ_DIR.mkdir(exist_ok=True)
    if force:
        for o in OBJ_DIR.glob("*.o"):
            o.unlink()
    sources = sorted(SRC_DIR.glob("*.cu"))
    if not sources:
        raise RuntimeError(f"no CUDA sources under {SRC_DIR}")
    extra = ["-Xptxas", "-v"] if ptxas_info else []
    workers = max(1, min(len(sources) + 1, os.cpu_count() or 1))
    with ThreadPoolExecutor(max_workers=workers) as pool:
        ops = pool.submit(_compile_ops, verbose)
        objs = list(pool.map(lambda s: _compile(s, verbose or ptxas_info, extra), sources))
        ops_obj = ops.result()
    if (not LIB_PATH.exists()) or any(o.stat().st_mtime > LIB_PATH.stat().st_mtime for o in objs):
        cmd = [_nvcc(), "-shared", "-gencode", "arch=compute_100a,code=sm_100a",
               "-cudart", "static", "-o", str(LIB_PATH), *map(str, objs)]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"link failed:\n{res.stdout}\n{res.stderr}")
    _link_ops(ops_obj)
    return LIB_PATH


if __name__ == "__main__":
    path = build(verbose=True, force="--force" in sys.argv, ptxas_info="--ptxas-info" in sys.argv)
    print(path)
