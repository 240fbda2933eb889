"""Build of the native library ``tensor_parallel_b200/lib/libtpb200.so`` (sm_100a only).

Every ``csrc/*.cu`` is compiled with ``nvcc -gencode arch=compute_100a,code=sm_100a`` to an object
file (in parallel) and linked into one shared library with a C ABI, loaded through ``ctypes``.
``csrc/autograd.cpp`` becomes a Python module beside it (host code against torch's headers; it gets the library's entry points from
``ops.native``).  It fits one Python and one torch, which its file name names.
nvcc cross-compiles without a GPU, so the library can be built on a CPU-only machine and shipped.
``python -m tensor_parallel_b200.build`` rebuilds what is out of date.
"""
from __future__ import annotations

import fcntl
import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

import torch

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
LIB_DIR = PKG / "lib"
LIB_PATH = LIB_DIR / "libtpb200.so"
AUTOGRAD_MODULE = "tpb_autograd"
AUTOGRAD_PATH = LIB_DIR / f"{AUTOGRAD_MODULE}.{sysconfig.get_config_var('SOABI')}.torch-{torch.__version__}.so"
OBJ_DIR = PKG / "build" / "obj"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; set NVCC or add it to PATH")


def sources():
    return sorted(CSRC.glob("*.cu"))


def _newest_header_mtime() -> float:
    headers = list(CSRC.glob("*.h")) + list(CSRC.glob("*.cuh"))
    return max((h.stat().st_mtime for h in headers), default=0.0)


def build_autograd(force: bool = False) -> Path:
    """Builds the autograd module if it is missing or older than its sources.  Processes that come here at once take turns, and the file
    appears under its name when it is whole."""
    from torch.utils import cpp_extension

    source = CSRC / "autograd.cpp"
    newest = max(source.stat().st_mtime, (CSRC / "tpb_api.h").stat().st_mtime)

    def fresh():
        return AUTOGRAD_PATH.exists() and AUTOGRAD_PATH.stat().st_mtime >= newest

    if not force and fresh():
        return AUTOGRAD_PATH
    LIB_DIR.mkdir(parents=True, exist_ok=True)
    with open(LIB_DIR / f".{AUTOGRAD_MODULE}.lock", "w") as lock:
        fcntl.flock(lock, fcntl.LOCK_EX)
        if not force and fresh():  # (another process has built it meanwhile)
            return AUTOGRAD_PATH
        cuda_include = Path(_nvcc()).resolve().parent.parent / "include"
        includes = [*cpp_extension.include_paths(), sysconfig.get_paths()["include"], str(cuda_include), str(CSRC)]
        part = AUTOGRAD_PATH.with_name(f"{AUTOGRAD_PATH.name}.{os.getpid()}.part")
        # the host compiler that nvcc takes, and the C++ runtime that torch has loaded: in a module with a runtime of its own (a compiler that
        # links it statically), an exception that carries a message of torch's crashes the process
        cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-DTORCH_EXTENSION_NAME={AUTOGRAD_MODULE}",
               f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}", *(f"-I{i}" for i in includes), str(source),
               *(f"-L{d}" for d in cpp_extension.library_paths()), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch", "-ltorch_python", "-l:libstdc++.so.6",
               "-o", str(part)]
        try:
            proc = subprocess.run(cmd, capture_output=True, text=True)
            if proc.returncode != 0:
                raise RuntimeError(f"building {AUTOGRAD_PATH.name} failed: {' '.join(cmd)}\n{proc.stderr}")
            os.replace(part, AUTOGRAD_PATH)
        finally:
            part.unlink(missing_ok=True)
    return AUTOGRAD_PATH


def build(force: bool = False, verbose: bool = False, lib_path: Path = None, extra_flags=(), autograd: bool = True) -> Path:
    """Builds what is out of date.  ``lib_path`` / ``extra_flags`` make a variant of the library somewhere else (its
    objects live beside it), e.g. ``-DTPB_GEMM_TRACE`` for the kernel-internal phase trace or ``-DTPB_BOUNDS`` for the
    in-kernel bounds checks; ``TPB_LIB_PATH`` makes ``ops.native`` load such a variant.  ``autograd=False`` leaves the autograd module alone,
    which needs the headers of Python and torch."""
    nvcc = _nvcc()
    lib_path = Path(lib_path) if lib_path is not None else LIB_PATH
    obj_dir = OBJ_DIR if lib_path == LIB_PATH else lib_path.parent / (lib_path.stem + "_obj")
    obj_dir.mkdir(parents=True, exist_ok=True)
    lib_path.parent.mkdir(parents=True, exist_ok=True)
    header_time = _newest_header_mtime()
    flags = list(NVCC_FLAGS) + list(extra_flags) + os.environ.get("TPB_NVCC_FLAGS", "").split()
    jobs = []
    for src in sources():
        obj = obj_dir / (src.stem + ".o")
        stale = force or not obj.exists() or obj.stat().st_mtime < max(src.stat().st_mtime, header_time)
        if stale:
            jobs.append([nvcc, *flags, *( ["-Xptxas", "-v"] if verbose else []), "-c", str(src), "-o", str(obj)])

    def run(cmd):
        proc = subprocess.run(cmd, capture_output=True, text=True)
        if proc.returncode != 0:
            raise RuntimeError(f"nvcc failed: {' '.join(cmd)}\n{proc.stdout}\n{proc.stderr}")
        return proc.stderr

    if jobs:
        with ThreadPoolExecutor(max_workers=min(len(jobs), os.cpu_count() or 4)) as pool:
            for log in pool.map(run, jobs):
                if verbose and log:
                    print(log, file=sys.stderr)
    objs = [str(obj_dir / (src.stem + ".o")) for src in sources()]
    newest_obj = max(os.path.getmtime(o) for o in objs)
    if force or jobs or not lib_path.exists() or lib_path.stat().st_mtime < newest_obj:
        run([nvcc, "-shared", "-o", str(lib_path), *objs, "-gencode", "arch=compute_100a,code=sm_100a"])
    if autograd:
        build_autograd(force and lib_path == LIB_PATH)  # (it serves every variant of the library)
    return lib_path


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
