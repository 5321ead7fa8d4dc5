"""Ahead-of-time build of the sm_100a kernels into ``slinoss_b200/_C``.

``python -m slinoss_b200.build`` (or ``build()``) compiles every ``csrc/*.cu``
with nvcc for ``sm_100a`` and links one C-ABI shared library,
``_C/libslinoss_b200.so``, whose exports are declared in
``include/slinoss_b200.h``, then the host extension ``_C/_host.so`` (g++, ``csrc/host``)
that the Python ops call it through.  There is no JIT and no fallback: calling the ops
without these libraries raises.  ``build_selftest()`` builds ``csrc/selftest/*.cu`` into a
second, test-only library (``include/slinoss_b200_selftest.h``) that the product never loads.
"""

from __future__ import annotations

import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
OUT_DIR = PKG / "_C"
LIB = OUT_DIR / "libslinoss_b200.so"
HOST_LIB = OUT_DIR / "_host.so"
SELFTEST_LIB = OUT_DIR / "libslinoss_b200_selftest.so"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "--expt-relaxed-constexpr", "--extended-lambda", "-Xcompiler", "-fPIC",
]


def _nvcc() -> str:
    cand = os.environ.get("NVCC") or "/usr/local/cuda/bin/nvcc"
    return cand if Path(cand).exists() else "nvcc"


def _headers():
    inc = PKG.parent / "include"
    return (list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.inc")) + list(inc.glob("*.h")))


def _compile_and_link(sources, lib: Path, force: bool, verbose: bool) -> Path:
    OUT_DIR.mkdir(exist_ok=True)
    newest = max(f.stat().st_mtime for f in list(sources) + _headers())
    diag = os.environ.get("SLX_DIAG") == "1"
    marker = OUT_DIR / (lib.stem + ".flags")
    flags = "diag" if diag else "release"
    same_flags = marker.exists() and marker.read_text().strip() == flags
    if not force and same_flags and lib.exists() and lib.stat().st_mtime >= newest:
        return lib

    def compile_one(src: Path) -> Path:
        obj = OUT_DIR / (src.stem + ".o")
        cmd = [_nvcc(), *NVCC_FLAGS, "-c", str(src), "-o", str(obj)]
        if diag:  # SLX_DIAG=1: phase-clock stamps in the tensor-core kernels (never the shipped build)
            cmd.insert(1, "-DSLX_DIAG")
        if verbose:
            cmd.insert(1, "-Xptxas")
            cmd.insert(2, "-v")
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src.name}:\n{r.stdout}\n{r.stderr}")
        if verbose:
            sys.stderr.write(r.stderr)
        return obj

    with ThreadPoolExecutor(max_workers=min(8, len(sources))) as ex:
        objs = list(ex.map(compile_one, sources))
    tmp = OUT_DIR / f"{lib.stem}.{os.getpid()}.tmp.so"
    cmd = [_nvcc(), "-shared", "-o", str(tmp), *map(str, objs), "-gencode",
           "arch=compute_100a,code=sm_100a"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    os.replace(tmp, lib)
    marker.write_text(flags + "\n")
    return lib


def build_host(force: bool = False) -> Path:
    """The native host path (``csrc/host/*.cpp``): a Python extension module over libtorch and the product library,
    which it finds beside itself."""
    import sysconfig

    from torch.utils import cpp_extension

    sources = sorted((CSRC / "host").glob("*.cpp"))
    newest = max(f.stat().st_mtime for f in sources + list((PKG.parent / "include").glob("*.h")))
    if not force and HOST_LIB.exists() and HOST_LIB.stat().st_mtime >= newest:
        return HOST_LIB
    cuda = Path(_nvcc()).resolve().parents[1]
    includes = [*cpp_extension.include_paths(), sysconfig.get_paths()["include"], str(cuda / "include")]
    tmp = OUT_DIR / f"_host.{os.getpid()}.tmp.so"
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-DTORCH_EXTENSION_NAME=_host",
           *(f"-isystem{p}" for p in includes), *map(str, sources), "-o", str(tmp),
           *(f"-L{p}" for p in cpp_extension.library_paths()), f"-L{OUT_DIR}", f"-L{cuda / 'lib64'}",
           "-ltorch_python", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda", "-lslinoss_b200",
           "-Wl,-rpath,$ORIGIN"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"g++ failed for the host extension:\n{r.stdout}\n{r.stderr}")
    os.replace(tmp, HOST_LIB)
    return HOST_LIB


def build(force: bool = False, verbose: bool = False) -> Path:
    """The product library (every ``csrc/*.cu``) and the host extension over it."""
    lib = _compile_and_link(sorted(CSRC.glob("*.cu")), LIB, force, verbose)
    build_host(force)
    return lib


def build_selftest(force: bool = False, verbose: bool = False) -> Path:
    """The test-only library: every ``csrc/selftest/*.cu``."""
    return _compile_and_link(sorted((CSRC / "selftest").glob("*.cu")), SELFTEST_LIB, force, verbose)


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
    print(build_selftest(force="--force" in sys.argv, verbose="-v" in sys.argv))
