"""Ahead-of-time build of the native code for sm_100a: ``python -m xqt_b200.build``.

Two in-tree binaries (so that they travel with the checkout): ``libxqt_b200.so``, the kernels behind their C ABI (every
``csrc/*.cu``, compiled one by one and linked), and ``_host.so``, the native call path of the bound layers
(``csrc/host.cpp``, a CPython extension against torch's headers).  xqt compiles its sm_89 sources just in time with a
cache key of flags + source hash (xqt/kernels/jit/utils/compile/spec.py:14-58, compile/cache.py:15-52); the same key
decides here, per source, whether it has to be compiled again, but the build itself happens once, offline.  nvcc
cross-compiles, so no GPU is needed to build.
"""

from __future__ import annotations

import concurrent.futures
import hashlib
import os
import pathlib
import shutil
import subprocess
import sys
import sysconfig

PACKAGE = pathlib.Path(__file__).resolve().parent
CSRC = PACKAGE / "csrc"
INCLUDE = PACKAGE.parent / "include"
OBJECTS = PACKAGE.parent / "build"
OUTPUT = PACKAGE / "libxqt_b200.so"
STAMP = PACKAGE / "libxqt_b200.so.key"
HOST_SOURCE = CSRC / "host.cpp"
HOST_OUTPUT = PACKAGE / "_host.so"
HOST_STAMP = PACKAGE / "_host.so.key"
ARCH_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a"]
# -fmad=false: no implicit multiply-add contraction, so fp32 results that the tests compare bit for
# bit (rotation, quantisation) do not depend on the compiler; the kernels spell out fmaf where they want it
NVCC_FLAGS = ["-O3", "-std=c++17", "-lineinfo", "-fmad=false", "-Xcompiler", "-fPIC"]
HOST_FLAGS = ["-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden"]


def sources() -> list[pathlib.Path]:
    return sorted(CSRC.glob("*.cu"))


def _digest(flags: list[str], paths: list[pathlib.Path]) -> str:
    digest = hashlib.sha256(" ".join(flags).encode())
    for path in paths:
        digest.update(path.name.encode())
        digest.update(path.read_bytes())
    return digest.hexdigest()


def _headers() -> list[pathlib.Path]:
    return sorted(list(CSRC.glob("*.cuh")) + list(INCLUDE.glob("*.h")))


def cache_key() -> str:
    return _digest(ARCH_FLAGS + NVCC_FLAGS, sources() + _headers())


def host_cache_key() -> str:
    import torch

    return _digest(HOST_FLAGS + [torch.__version__, sys.version], [HOST_SOURCE] + sorted(INCLUDE.glob("*.h")))


def _stamped(output: pathlib.Path, stamp: pathlib.Path, key: str) -> bool:
    return output.exists() and stamp.exists() and stamp.read_text().strip() == key


def up_to_date() -> bool:
    return _stamped(OUTPUT, STAMP, cache_key()) and _stamped(HOST_OUTPUT, HOST_STAMP, host_cache_key())


def _run(command: list[str], verbose: bool) -> None:
    result = subprocess.run(command, capture_output=True, text=True)
    if verbose or result.returncode != 0:
        sys.stderr.write(result.stdout + result.stderr)
    if result.returncode != 0:
        raise RuntimeError(f"{pathlib.Path(command[0]).name} failed with exit code {result.returncode}")


def _build_kernels(force: bool, verbose: bool) -> None:
    key = cache_key()
    if not force and _stamped(OUTPUT, STAMP, key):
        return
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not pathlib.Path(nvcc).exists():
        raise RuntimeError("nvcc not found; the sm_100a library cannot be built on this machine")
    OBJECTS.mkdir(exist_ok=True)

    def compile_one(path: pathlib.Path) -> pathlib.Path:
        target = OBJECTS / f"{path.stem}.{_digest(ARCH_FLAGS + NVCC_FLAGS, [path] + _headers())[:16]}.o"
        if force or verbose or not target.exists():
            for old in OBJECTS.glob(f"{path.stem}.*.o"):
                old.unlink()
            extra = ["-Xptxas", "-v"] if verbose else []
            _run([nvcc, *ARCH_FLAGS, *NVCC_FLAGS, *extra, "-I", str(INCLUDE), "-c", "-o", str(target), str(path)], verbose)
        return target

    with concurrent.futures.ThreadPoolExecutor(max_workers=max(2, os.cpu_count() or 2)) as pool:
        objects = list(pool.map(compile_one, sources()))
    _run([nvcc, *ARCH_FLAGS, "-shared", "-o", str(OUTPUT), *[str(o) for o in objects]], verbose)
    STAMP.write_text(key + "\n")


def _build_host(force: bool, verbose: bool) -> None:
    key = host_cache_key()
    if not force and _stamped(HOST_OUTPUT, HOST_STAMP, key):
        return
    import torch
    from torch.utils import cpp_extension

    includes = cpp_extension.include_paths() + [sysconfig.get_paths()["include"], "/usr/local/cuda/include"]
    command = [shutil.which("g++") or "g++", *HOST_FLAGS, f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
    for path in includes:
        command += ["-isystem", path]
    command += ["-o", str(HOST_OUTPUT), str(HOST_SOURCE), "-L", str(pathlib.Path(torch.__file__).parent / "lib")]
    command += ["-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python", "-lc10", "-lc10_cuda"]
    _run(command, verbose)
    HOST_STAMP.write_text(key + "\n")


def build(force: bool = False, verbose: bool = False) -> pathlib.Path:
    _build_kernels(force, verbose)
    _build_host(force, verbose)
    return OUTPUT


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(path)
