"""Builds libqlin_b200.so (the C-ABI library with every CUDA kernel of this package) and _qlin_host.so (the tensor-level
host code in C++, linked against it) in-tree.

The library is compiled for sm_100a only with plain ``nvcc``; nothing is JIT-compiled at run time.
``python -m fms_model_optimizer_b200.build_ext`` rebuilds it; ``build()`` is also what
``__graft_entry__.build()`` calls.  nvcc cross-compiles without a GPU.
"""

from __future__ import annotations

import hashlib
import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG_DIR = Path(__file__).resolve().parent
CSRC = PKG_DIR / "csrc"
LIB_DIR = PKG_DIR / "lib"
LIB_PATH = LIB_DIR / "libqlin_b200.so"
HOST_SRC = CSRC / "host" / "qlin_host.cpp"
HOST_PATH = LIB_DIR / "_qlin_host.so"
OBJ_DIR = LIB_DIR / "obj"

NVCC_FLAGS = [
    "-gencode",
    "arch=compute_100a,code=sm_100a",
    "-lineinfo",
    "-O3",
    "-std=c++17",
    "-Xcompiler",
    "-fPIC",
    "--expt-relaxed-constexpr",
]


HOST_FLAGS = ["-O2", "-std=c++17", "-fPIC", "-shared"]


def _build_host() -> None:
    """g++ for the host code: PyTorch's headers and libraries, libqlin_b200.so beside it at run time."""
    import torch

    root = Path(torch.__file__).resolve().parent
    includes = [root / "include", root / "include" / "torch" / "csrc" / "api" / "include", Path(sysconfig.get_path("include")), _cuda_include()]
    tmp = HOST_PATH.with_suffix(".so.tmp")
    cmd = ["g++", *HOST_FLAGS, f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
    for inc in includes:
        cmd += ["-isystem", str(inc)]
    cmd += [str(HOST_SRC), "-o", str(tmp), f"-L{LIB_DIR}", "-l:libqlin_b200.so", f"-L{root / 'lib'}", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python",
            "-Wl,-rpath,$ORIGIN"]  # fmt: skip
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"g++ failed for {HOST_SRC.name}:\n{res.stdout}\n{res.stderr}")
    os.replace(tmp, HOST_PATH)


def _cuda_include() -> Path:
    return Path(_nvcc()).resolve().parent.parent / "include"


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found: libqlin_b200.so cannot be built")
    return exe


def _sources() -> list[Path]:
    return sorted(CSRC.glob("*.cu"))


STAMP_PATH = LIB_DIR / "libqlin_b200.stamp"


def _host_environment() -> list[str]:
    """What the host library's binary interface depends on besides its source: PyTorch, its CUDA and C++ ABI, Python."""
    import torch

    return [str(v) for v in (torch.__version__, torch.version.cuda, torch._C._GLIBCXX_USE_CXX11_ABI, sysconfig.get_config_var("SOABI"))]


def source_digest(extra_flags: tuple = ()) -> str:
    """SHA-256 over the compiler flags, the name and content of every file the libraries are built from and the environment of
    the host library.  File times say nothing after a checkout or a copy to another machine, so staleness is decided by
    content."""
    files = sorted(list(CSRC.glob("*.cu")) + list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.h")))
    files += [PKG_DIR.parent / "include" / "qlin_b200.h", HOST_SRC]
    h = hashlib.sha256()
    h.update("\0".join([*NVCC_FLAGS, *HOST_FLAGS, *_host_environment(), *extra_flags]).encode())
    for f in files:
        h.update(f.name.encode() + b"\0")
        h.update(f.read_bytes())
    return h.hexdigest()


def is_stale() -> bool:
    """True unless the libraries exist and the digest stored beside them at build time equals the digest of the sources."""
    if not LIB_PATH.exists() or not HOST_PATH.exists() or not STAMP_PATH.exists():
        return True
    return STAMP_PATH.read_text().strip() != source_digest()


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compile every ``csrc/*.cu`` and link ``lib/libqlin_b200.so``, then the host code.  Returns the library path."""
    if not force and not is_stale():
        return LIB_PATH
    nvcc = _nvcc()
    OBJ_DIR.mkdir(parents=True, exist_ok=True)
    extra = ["-Xptxas", "-v"] if verbose else []

    def compile_one(src: Path) -> Path:
        obj = OBJ_DIR / (src.stem + ".o")
        cmd = [nvcc, *NVCC_FLAGS, *extra, "-c", str(src), "-o", str(obj)]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src.name}:\n{res.stdout}\n{res.stderr}")
        if verbose:
            sys.stderr.write(res.stderr)
        return obj

    with ThreadPoolExecutor(max_workers=4) as pool:
        objs = list(pool.map(compile_one, _sources()))
    tmp = LIB_PATH.with_suffix(".so.tmp")
    cmd = [nvcc, "-shared", "-o", str(tmp), *[str(o) for o in objs]]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"link failed:\n{res.stdout}\n{res.stderr}")
    os.replace(tmp, LIB_PATH)
    _build_host()
    STAMP_PATH.write_text(source_digest() + "\n")
    return LIB_PATH


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(path)
