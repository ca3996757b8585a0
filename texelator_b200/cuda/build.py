"""Build libtexelator_b200.so in-tree with nvcc for sm_100a.

    python -m texelator_b200.cuda.build [--force] [--verbose]

The library is a plain C-ABI shared object (see include/texelator_b200.h); it links only the CUDA
runtime.  Reference counterpart: setup.py:9-36 / texelator/runtime.py:43-62, which build a torch
extension with no -gencode at all.
"""
from __future__ import annotations

import hashlib
import os
import shutil
import subprocess
import sys
from pathlib import Path

HERE = Path(__file__).resolve().parent
SOURCES = ["tx_api.cu", "tx_pack.cu", "tx_gemv.cu", "tx_stream.cu", "tx_prefill.cu", "tx_aux.cu", "tx_encode.cu"]
LIBRARY = HERE / "libtexelator_b200.so"
STAMP = HERE / ".build_stamp"
BINDING_SOURCE = HERE / "tx_torch.cpp"
BINDING = HERE / "_tx_torch.so"          # CPython module: the operator call without Python in between
BINDING_STAMP = HERE / ".binding_stamp"


def source_digest() -> str:
    digest = hashlib.sha256()
    for path in sorted(HERE.glob("*.cu")) + sorted(HERE.glob("*.cuh")) + [HERE.parent.parent / "include" / "texelator_b200.h"]:
        digest.update(path.name.encode())
        digest.update(path.read_bytes())
    return digest.hexdigest()


def nvcc_path() -> str:
    found = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(found).exists():
        raise RuntimeError("nvcc was not found; the CUDA library cannot be built")
    return found


def build(force: bool = False, verbose: bool = False) -> Path:
    digest = source_digest()
    if not force and LIBRARY.exists() and STAMP.exists() and STAMP.read_text().strip() == digest:
        return LIBRARY
    sources = [str(HERE / name) for name in SOURCES if (HERE / name).exists()]
    command = [
        nvcc_path(), "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo",
        "-Xptxas", "-v", "--shared", "-Xcompiler", "-fPIC", "--threads", "4",
        "-o", str(LIBRARY), *sources,
    ]
    result = subprocess.run(command, capture_output=True, text=True)
    (HERE / "build.log").write_text(" ".join(command) + "\n" + result.stdout + result.stderr)
    if verbose or result.returncode:
        sys.stderr.write(result.stdout + result.stderr)
    if result.returncode:
        raise RuntimeError(f"nvcc failed with exit code {result.returncode}; see {HERE / 'build.log'}")
    STAMP.write_text(digest + "\n")
    return LIBRARY


def binding_target() -> str:
    """What the binding is compiled for; the compiled module carries this text and the loader compares it."""
    import torch
    return f"torch {torch.__version__}, Python {sys.version_info.major}.{sys.version_info.minor}"


def binding_digest() -> str:
    return hashlib.sha256(BINDING_SOURCE.read_bytes() + binding_target().encode() + sys.version.encode()).hexdigest()


def binding_is_current() -> bool:
    """Whether the module on disk is the one this source and this torch would build (a prebuilt one without a stamp is
    left to the loader's check)."""
    if not BINDING.exists():
        return False
    return not (BINDING_STAMP.exists() and BINDING_SOURCE.exists()) or BINDING_STAMP.read_text().strip() == binding_digest()


def build_binding(force: bool = False, verbose: bool = False) -> Path:
    """The CPython module ``_tx_torch`` (host code only; g++ against the installed torch's headers)."""
    import sysconfig

    import torch
    digest = binding_digest()
    if not force and BINDING.exists() and BINDING_STAMP.exists() and BINDING_STAMP.read_text().strip() == digest:
        return BINDING
    root = Path(torch.__file__).resolve().parent
    cuda = Path(nvcc_path()).resolve().parent.parent
    include = [root / "include", root / "include" / "torch" / "csrc" / "api" / "include", sysconfig.get_paths()["include"], cuda / "include"]
    command = [shutil.which("g++") or "g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
               f'-DTX_BUILT_FOR="{binding_target()}"',
               *[f"-I{path}" for path in include], str(BINDING_SOURCE), "-o", str(BINDING), f"-L{root / 'lib'}", f"-Wl,-rpath,{root / 'lib'}",
               "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python"]
    result = subprocess.run(command, capture_output=True, text=True)
    if verbose or result.returncode:
        sys.stderr.write(result.stdout + result.stderr)
    if result.returncode:
        raise RuntimeError(f"g++ failed with exit code {result.returncode} on {BINDING_SOURCE.name}")
    BINDING_STAMP.write_text(digest + "\n")
    return BINDING


if __name__ == "__main__":
    build_binding(force="--force" in sys.argv, verbose="--verbose" in sys.argv)
    path = build(force="--force" in sys.argv, verbose="--verbose" in sys.argv)
    print(path, os.path.getsize(path), "bytes")
