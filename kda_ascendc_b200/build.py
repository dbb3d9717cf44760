"""In-tree build of libkda_b200.so (nvcc, sm_100a only) and of the host module _kda_host.so.

``python -m kda_ascendc_b200.build`` compiles the CUDA sources under ``csrc/`` into
``kda_ascendc_b200/libkda_b200.so`` and ``csrc/kda_host.cpp`` (the native host path of the
Python functions, linked against that library and PyTorch) into ``_kda_host.so`` beside it.
nvcc cross-compiles without a GPU, so the same command serves the build check on a CPU-only machine.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
from pathlib import Path

PKG_DIR = Path(__file__).resolve().parent
CSRC = PKG_DIR / "csrc"
LIB_PATH = PKG_DIR / "libkda_b200.so"
HOST_PATH = PKG_DIR / "_kda_host.so"
HOST_SOURCE = "kda_host.cpp"
SOURCES = ["kda_c_api.cu", "kda_k1_sm100.cu", "kda_k2_sm100.cu", "kda_k2la_sm100.cu", "kda_k2m_sm100.cu", "kda_k2t_sm100.cu", "kda_recurrent_sm100.cu", "kda_fold_sm100.cu", "kda_peer_sm100.cu",
           "kda_selftest.cu", "kda_static_scratch.cu"]
HEADERS = ["kda_common.cuh", "kda_tc.cuh", "kda_kernels.h", "../../include/kda_b200.h"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-shared", "-Xcompiler", "-fPIC",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found (set NVCC=/path/to/nvcc)")


def sources() -> list[Path]:
    return [CSRC / s for s in SOURCES if (CSRC / s).exists()]


def _older(target: Path, deps) -> bool:
    if not target.exists():
        return True
    built = target.stat().st_mtime
    return any(d.exists() and d.stat().st_mtime > built for d in deps)


def is_stale() -> bool:
    return _older(LIB_PATH, sources() + [(CSRC / h).resolve() for h in HEADERS])


def _run(cmd, out: Path, verbose: bool) -> None:
    """Run a compiler whose last argument pair is added here, then move the result into place."""
    tmp = out.with_suffix(".so.tmp%d" % os.getpid())
    proc = subprocess.run([*cmd, "-o", str(tmp)], cwd=str(CSRC), capture_output=True, text=True)
    if proc.returncode != 0:
        raise RuntimeError("%s failed:\n%s\n%s" % (cmd[0], " ".join(cmd), proc.stderr[-4000:]))
    if verbose:
        sys.stderr.write(proc.stderr)
    os.replace(tmp, out)


def build_host(force: bool = False, verbose: bool = False) -> Path:
    """Compile the host module if it is missing or older than its source or the C header."""
    src = CSRC / HOST_SOURCE
    if not force and not _older(HOST_PATH, [src, (CSRC / "../../include/kda_b200.h").resolve()]):
        return HOST_PATH
    import sysconfig

    import torch
    from torch.utils import cpp_extension as ext

    cxx = os.environ.get("CXX") or shutil.which("g++") or "g++"
    cuda_home = Path(_nvcc()).resolve().parents[1]
    cmd = [cxx, "-O2", "-std=c++17", "-fPIC", "-shared", "-D_GLIBCXX_USE_CXX11_ABI=%d" % torch._C._GLIBCXX_USE_CXX11_ABI,
           *["-I%s" % p for p in ext.include_paths()], "-I%s" % sysconfig.get_paths()["include"],
           "-I%s" % (cuda_home / "include"), str(src), *["-L%s" % p for p in ext.library_paths()],
           "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python", "-L%s" % PKG_DIR, "-l:%s" % LIB_PATH.name,
           "-Wl,-rpath,$ORIGIN"]
    _run(cmd, HOST_PATH, verbose)
    return HOST_PATH


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compile the library and the host module where they are missing or older than their sources."""
    if force or is_stale():
        cmd = [_nvcc(), *NVCC_FLAGS, *(["-Xptxas", "-v"] if verbose else []), *[str(s) for s in sources()]]
        _run(cmd, LIB_PATH, verbose)
    build_host(force, verbose)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
