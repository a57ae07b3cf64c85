"""Compile the CUDA sources in ``csrc/`` into ``libgdn2_b200.so`` next to this file, and the native host
path (``csrc/host.cpp``, a CPython extension against PyTorch's headers) into ``_host.<Python>.<PyTorch>.so``:
another version of either finds no file of its own, and a build makes it.

``nvcc`` cross-compiles for sm_100a without a GPU, so this runs anywhere the CUDA
toolkit is installed.  The shared object is built in-tree (it is git-ignored) and is
rebuilt only when a source or header is newer than it.

    python -m gdn2_sm120_b200.build [--force] [--verbose]
"""

from __future__ import annotations

import concurrent.futures
import os
import pathlib
import shutil
import subprocess
import sys
import sysconfig
import tempfile

from . import _lib

PACKAGE_DIR = pathlib.Path(__file__).resolve().parent
CSRC = PACKAGE_DIR / "csrc"
INCLUDE = PACKAGE_DIR.parent / "include"
LIB_NAME = "libgdn2_b200.so"
LIB_PATH = PACKAGE_DIR / LIB_NAME
HOST_SOURCE = CSRC / "host.cpp"
HOST_PATH = _lib.host_path()

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC",
    "-Xcompiler", "-Wall",
]


def _nvcc() -> str:
    found = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(found):
        raise RuntimeError("nvcc not found; the gdn2_b200 kernels cannot be built")
    return found


def sources() -> list[pathlib.Path]:
    return sorted(CSRC.glob("*.cu"))


def _stale() -> bool:
    if not LIB_PATH.exists() or not HOST_PATH.exists():
        return True
    built = min(LIB_PATH.stat().st_mtime, HOST_PATH.stat().st_mtime)
    deps = list(CSRC.glob("*.cu")) + list(CSRC.glob("*.cuh")) + list(INCLUDE.glob("*.h")) + [HOST_SOURCE]
    return any(dep.stat().st_mtime > built for dep in deps)


def _host_command(output: str) -> list[str]:
    from torch.utils import cpp_extension

    includes = [*cpp_extension.include_paths("cuda"), sysconfig.get_paths()["include"]]
    return ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-Wall",
            *(flag for path in includes for flag in ("-isystem", path)), str(HOST_SOURCE), "-o", output,
            *(f"-L{path}" for path in cpp_extension.library_paths()),
            "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python"]


def build(force: bool = False, verbose: bool = False) -> pathlib.Path:
    """Compile the sources side by side (one nvcc per file) and link them."""

    if not force and not _stale():
        return LIB_PATH
    nvcc = _nvcc()
    common = [*NVCC_FLAGS, "-I", str(INCLUDE)] + (["-Xptxas", "-v"] if verbose else [])

    def run(cmd: list[str]) -> None:
        proc = subprocess.run(cmd, capture_output=True, text=True)
        if verbose or proc.returncode != 0:
            sys.stderr.write(proc.stdout + proc.stderr)
        if proc.returncode != 0:
            raise RuntimeError(f"{os.path.basename(cmd[0])} failed with exit code {proc.returncode}")

    with tempfile.TemporaryDirectory() as work:
        objects = [str(pathlib.Path(work) / (src.stem + ".o")) for src in sources()]
        jobs = [[nvcc, *common, "-c", str(src), "-o", obj] for src, obj in zip(sources(), objects)]
        host_tmp = HOST_PATH.with_suffix(".so.tmp")
        jobs.append(_host_command(str(host_tmp)))
        with concurrent.futures.ThreadPoolExecutor(max_workers=os.cpu_count() or 1) as pool:
            list(pool.map(run, jobs))
        tmp = LIB_PATH.with_suffix(".so.tmp")
        run([nvcc, *common, "-shared", *objects, "-o", str(tmp), "-lcudart", "-lcuda"])
    os.replace(tmp, LIB_PATH)
    os.replace(host_tmp, HOST_PATH)
    return LIB_PATH


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="--verbose" in sys.argv)
    print(path)
