"""In-tree build of the sm_100a kernel library (``libb200rl.so``) and of its entry points that take tensors (``_host.so``).

Every ``csrc/*.cu`` is compiled with ``nvcc -gencode arch=compute_100a,code=sm_100a`` into an object file and
linked into one shared library next to this module, so the library travels with the source tree and is
loaded with ``ctypes``; no torch C++ headers are involved. ``csrc/host.cpp`` is one file against torch's headers and becomes a
Python extension beside it, built again when torch or Python change. A full rebuild takes well under a minute.
Run ``python -m cosmos_rl_b200.ops.build`` or call :func:`build`.
"""
from __future__ import annotations

import concurrent.futures
import hashlib
import os
import shutil
import subprocess
import sys
import sysconfig
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "csrc"
OUT_DIR = Path(__file__).resolve().parent
LIB_NAME = "libb200rl.so"
HOST_NAME = "_host.so"
OBJ_DIR = OUT_DIR / "build"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=default",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; set NVCC or put it on PATH")


def _digest(paths, flags) -> str:
    h = hashlib.sha256()
    for p in sorted(paths):
        h.update(p.name.encode())
        h.update(p.read_bytes())
    h.update(" ".join(flags).encode())
    return h.hexdigest()


def _fresh(target: Path, digest: str) -> bool:
    stamp = OUT_DIR / (target.name + ".sha256")
    return target.exists() and stamp.exists() and stamp.read_text().strip() == digest


def sources():
    return sorted(CSRC.glob("*.cu"))


def lib_path() -> Path:
    return OUT_DIR / LIB_NAME


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compile (if stale) and return the path of the shared library."""
    srcs = sources()
    headers = sorted(CSRC.glob("*.cuh")) + sorted(CSRC.glob("*.h"))
    stamp = OUT_DIR / (LIB_NAME + ".sha256")
    digest = _digest(srcs + headers, NVCC_FLAGS)
    lib = lib_path()
    if not force and _fresh(lib, digest):
        build_host(force)
        return lib
    OBJ_DIR.mkdir(exist_ok=True)
    nvcc = _nvcc()

    def compile_one(src: Path) -> Path:
        obj = OBJ_DIR / (src.stem + ".o")
        cmd = [nvcc, *NVCC_FLAGS, "-I", str(CSRC), "-c", str(src), "-o", str(obj)]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src.name}:\n{r.stdout}\n{r.stderr}")
        if verbose:
            sys.stderr.write(r.stderr)
        return obj

    with concurrent.futures.ThreadPoolExecutor(max_workers=min(8, len(srcs))) as ex:
        objs = list(ex.map(compile_one, srcs))
    cmd = [nvcc, "-shared", "-o", str(lib), *map(str, objs), "-lcudart"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    stamp.write_text(digest)
    build_host(force)
    return lib


def host_path() -> Path:
    return OUT_DIR / HOST_NAME


def build_host(force: bool = False) -> Path:
    """Compile (if stale) the extension of ``csrc/host.cpp``; the kernel library has been built."""
    import torch
    src, ext = CSRC / "host.cpp", host_path()
    root = Path(torch.__file__).resolve().parent
    flags = ["-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
             f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
    digest = _digest([src, CSRC / "api.h"], flags + [torch.__version__, sys.version])
    if not force and _fresh(ext, digest):
        return ext
    cuda = Path(_nvcc()).resolve().parent.parent
    include = [root / "include", root / "include/torch/csrc/api/include", sysconfig.get_paths()["include"], cuda / "include", CSRC]
    cmd = ["g++", *flags, *(f"-I{d}" for d in include), str(src), "-o", str(ext), f"-L{root / 'lib'}", "-ltorch_python",
           "-ltorch_cpu", "-ltorch", "-lc10", f"-L{OUT_DIR}", f"-l:{LIB_NAME}", "-Wl,-rpath,$ORIGIN"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"g++ failed for {src.name}:\n{r.stdout}\n{r.stderr}")
    (OUT_DIR / (HOST_NAME + ".sha256")).write_text(digest)
    return ext


if __name__ == "__main__":
    p = build(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(p)
