"""Builds the native library (``libtplr_b200.so``) in-tree with nvcc for sm_100a, and the autograd nodes
(``csrc_host/*.cpp`` -> ``tplr_host.so``) with the host compiler against PyTorch's headers.

``python -m templar_b200.ops.build`` (or :func:`build`) compiles every ``csrc/*.cu``
translation unit with ``-gencode arch=compute_100a,code=sm_100a -lineinfo`` and links
them into ``templar_b200/ops/_lib/libtplr_b200.so``.  nvcc cross-compiles without a GPU.
Objects are rebuilt only when a source or header is newer than the object, the library when an object is newer, the
extension module when its sources, its compiler call or PyTorch have changed.
"""

from __future__ import annotations

import os
import shutil
import subprocess
import sys
import zlib
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

HERE = Path(__file__).resolve().parent
CSRC = HERE / "csrc"
LIBDIR = HERE / "_lib"
LIBNAME = "libtplr_b200.so"
HOST_SRC = HERE / "csrc_host"
HOSTNAME = "tplr_host.so"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC,-fvisibility=hidden",
    "--expt-relaxed-constexpr",
]
HOST_FLAGS = ["-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden"]
# Approximate intrinsics and flush-to-zero only where the arithmetic is a softmax in base 2 (the flash
# attention kernels).  The loss, the norms, the optimizer, the quantiser and the compression kernels are
# compiled with IEEE division / square root and keep denormals; where they want a fast exponential they
# call __expf or its instruction explicitly.
FAST_MATH_SOURCES = {"attention.cu"}


def _nvcc() -> str:
    cand = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(cand).exists():
        raise RuntimeError("nvcc not found; set NVCC or install the CUDA toolkit")
    return cand


def lib_path() -> Path:
    return LIBDIR / LIBNAME


def host_path() -> Path:
    return LIBDIR / HOSTNAME


def sources() -> list[Path]:
    return sorted(CSRC.glob("*.cu"))


def host_sources() -> list[Path]:
    return sorted(HOST_SRC.glob("*.cpp"))


def headers() -> list[Path]:
    return sorted([*CSRC.glob("*.cuh"), *CSRC.glob("*.h")])


def _stale(out: Path, *made_from: Path) -> bool:
    return not out.exists() or any(p.stat().st_mtime > out.stat().st_mtime for p in made_from)


def _abi_flag() -> str:
    """The number that the library and the extension module must agree on: made from the declarations they share."""
    return f"-DTPLR_ABI={zlib.crc32((CSRC / 'entries.h').read_bytes()) & 0x7FFFFFFF}"


def _run(cmd: list[str]) -> str:
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("compiler failed: " + " ".join(cmd) + "\n" + r.stdout + r.stderr)
    return r.stderr


def _host_key() -> str:
    """What the extension module depends on beside its sources: a module of another PyTorch must not be loaded."""
    import torch

    return "\n".join([torch.__version__, sys.version, *HOST_FLAGS, _abi_flag()])


def _host_key_path() -> Path:
    return host_path().with_suffix(".key")


def host_usable() -> bool:
    """The extension module is there and not known to be of another PyTorch or Python."""
    key = _host_key_path()
    return host_path().exists() and (not key.exists() or key.read_text() == _host_key())


def build_host(force: bool = False) -> Path:
    """Compile the extension module of the autograd nodes (plain C++, no CUDA compiler involved); returns its path."""
    import sysconfig

    import torch

    srcs = host_sources()
    if not srcs:
        raise RuntimeError(f"no sources of the autograd nodes in {HOST_SRC}: the installed package is incomplete")
    out = host_path()
    if not force and host_usable() and _host_key_path().exists() and not _stale(out, *srcs):
        return out
    from torch.utils.cpp_extension import include_paths

    LIBDIR.mkdir(exist_ok=True)
    inc = [x for p in [*include_paths("cuda"), sysconfig.get_paths()["include"]] for x in ("-isystem", p)]
    tmp = out.with_suffix(f".{os.getpid()}.tmp")       # ranks that start together may all build
    _run([os.environ.get("CXX", "g++"), *HOST_FLAGS, _abi_flag(), *inc, *map(str, srcs), "-o", str(tmp),
          "-L" + str(Path(torch.__file__).parent / "lib"), "-lc10", "-ltorch_cpu", "-ltorch", "-ltorch_python", "-lc10_cuda"])
    os.replace(tmp, out)
    _host_key_path().write_text(_host_key())
    return out


def build_library(verbose: bool = False, force: bool = False) -> Path:
    """Compile and link the kernel library; returns its path."""
    nvcc = _nvcc()
    LIBDIR.mkdir(exist_ok=True)
    objs, jobs = [], []
    for src in sources():
        obj = LIBDIR / (src.stem + ".o")
        objs.append(obj)
        if force or _stale(obj, src, *headers()):
            extra = ["--use_fast_math"] if src.name in FAST_MATH_SOURCES else []
            cmd = [nvcc, *NVCC_FLAGS, *extra, _abi_flag(), "-I", str(CSRC), "-c", str(src), "-o", str(obj)]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
            jobs.append(cmd)
    if jobs:
        with ThreadPoolExecutor(max_workers=min(8, len(jobs))) as ex:
            for out in ex.map(_run, jobs):
                if verbose and out:
                    print(out, file=sys.stderr)
    lib = lib_path()
    # an object may be newer than the library without having been compiled here: a build that failed later leaves it
    if not lib.exists() or any(o.stat().st_mtime > lib.stat().st_mtime for o in objs):
        tmp = lib.with_suffix(f".{os.getpid()}.tmp")          # link beside the target, then rename: readers never see a partial file
        _run([nvcc, "-shared", "-o", str(tmp), *map(str, objs), "-lcudart"])
        os.replace(tmp, lib)
    return lib


def build(verbose: bool = False, force: bool = False) -> Path:
    """Build both, one beside the other; returns the kernel library's path.  The library is linked whether or not the
    extension module could be compiled."""
    with ThreadPoolExecutor(max_workers=1) as ex:
        host = ex.submit(build_host, force)
        lib = build_library(verbose, force)
        host.result()
    return lib


if __name__ == "__main__":
    print(build(verbose="-v" in sys.argv, force="-f" in sys.argv))
