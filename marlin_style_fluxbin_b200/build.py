"""Ahead-of-time build of the CUDA library (``libfluxbin_b200.so``) with nvcc for sm_100a, and of the extension
module behind eager calls (``_fb_calls``, tagged with Python's ABI) with the host compiler against torch's C++ interface.

Both are built in-tree, next to this file, so that they travel with the source tree.
``python -m marlin_style_fluxbin_b200.build`` rebuilds it; ``build()`` is incremental.
"""
from __future__ import annotations

import hashlib
import os
import shutil
import subprocess
import sys
import sysconfig
from pathlib import Path

PACKAGE = Path(__file__).resolve().parent
CSRC = PACKAGE / "csrc"
LIBRARY = PACKAGE / "libfluxbin_b200.so"
CALLS = PACKAGE / f"_fb_calls{sysconfig.get_config_var('EXT_SUFFIX')}"
STAMP = PACKAGE / "csrc" / ".build_stamp"

ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
COMMON = ["-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC", "-Xptxas", "-v"]
# Per-file extras.  The GEMV kernels keep separate multiply and add, as the reference
# builds its kernels (--fmad=false), so that products are rounded where it rounds them.
EXTRA = {"fb_w3_gemv.cu": ["--fmad=false"], "fb_w3_rows.cu": ["--fmad=false"], "fb_bb_gemv.cu": ["--fmad=false"]}


def _nvcc() -> str:
    for candidate in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if candidate and Path(candidate).exists():
            return candidate
    raise RuntimeError("nvcc not found; set NVCC or put it on PATH")


def sources() -> list[Path]:
    return sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cpp")])


def _fingerprint() -> str:
    import torch

    # the extension module reads tensor objects as this torch lays them out
    digest = hashlib.sha256(f"{torch.__version__} {torch._C._GLIBCXX_USE_CXX11_ABI} {CALLS.name}".encode())
    for path in sorted(sources() + list(CSRC.glob("*.cuh")) + list(CSRC.glob("python/*.cpp")) + [PACKAGE.parent / "include" / "fluxbin_b200.h", Path(__file__)]):
        digest.update(path.name.encode())
        digest.update(path.read_bytes())
    return digest.hexdigest()


def _build_calls(nvcc: str) -> str:
    import torch
    from torch.utils.cpp_extension import include_paths

    libraries = Path(torch.__file__).resolve().parent / "lib"
    headers = [*include_paths(), sysconfig.get_paths()["include"], str(Path(nvcc).resolve().parent.parent / "include")]
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", f'-DFB_TORCH_VERSION="{torch.__version__}"', f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           *(flag for path in headers for flag in ("-isystem", path)), str(CSRC / "python" / "fb_calls.cpp"), "-o", str(CALLS),
           f"-L{libraries}", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python"]
    done = subprocess.run(cmd, capture_output=True, text=True)
    if done.returncode != 0:
        raise RuntimeError(f"{cmd[0]} failed on fb_calls.cpp:\n{done.stdout}{done.stderr}")
    return f"$ {' '.join(cmd)}\n{done.stdout}{done.stderr}"


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compile every ``csrc/*.cu`` for sm_100a (and the host-only ``*.cpp``), link the shared library and build the extension."""
    fingerprint = _fingerprint()
    if not force and LIBRARY.exists() and CALLS.exists() and STAMP.exists() and STAMP.read_text() == fingerprint:
        return LIBRARY
    nvcc = _nvcc()
    objects = []
    logs = []
    for source in sources():
        obj = source.with_suffix(".o")
        cmd = [nvcc, *ARCH, *COMMON, *EXTRA.get(source.name, []), "-c", str(source), "-o", str(obj)]
        done = subprocess.run(cmd, capture_output=True, text=True)
        logs.append(f"$ {' '.join(cmd)}\n{done.stdout}{done.stderr}")
        if done.returncode != 0:
            raise RuntimeError(f"nvcc failed on {source.name}:\n{done.stdout}{done.stderr}")
        objects.append(obj)
    cmd = [nvcc, *ARCH, "-shared", "-o", str(LIBRARY), *map(str, objects)]
    done = subprocess.run(cmd, capture_output=True, text=True)
    if done.returncode != 0:
        raise RuntimeError(f"link failed:\n{done.stdout}{done.stderr}")
    logs.append(_build_calls(nvcc))
    (CSRC / "ptxas_report.txt").write_text("\n".join(logs))
    STAMP.write_text(fingerprint)
    if verbose:
        print("\n".join(logs))
    return LIBRARY


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose=True)
    print(LIBRARY)
