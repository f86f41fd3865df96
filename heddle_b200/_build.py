"""Build the C-ABI shared library ``libheddle_b200.so`` in-tree with nvcc for sm_100a, and ``_native-*.so``, the host path
of the tensor-level calls (csrc/ops_native.cpp), with g++ against PyTorch's headers.

nvcc cross-compiles without a GPU, so this runs on a CPU-only host as well.
``python -m heddle_b200._build`` rebuilds; ``build(force=False)`` rebuilds only
when a source is newer than the library.
"""
from __future__ import annotations

import concurrent.futures
import os
import shutil
import subprocess
import sys
import sysconfig
import warnings
from pathlib import Path

PKG_DIR = Path(__file__).resolve().parent
CSRC = PKG_DIR / "csrc"
OBJ_DIR = CSRC / "build"
LIB_PATH = PKG_DIR / "libheddle_b200.so"
NATIVE_SRC = CSRC / "ops_native.cpp"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
    "-Xptxas", "-v",
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; the heddle_b200 kernels cannot be built")
    return exe


def sources() -> list[Path]:
    return sorted(CSRC.glob("*.cu"))


def _older(target: Path, deps: list[Path]) -> bool:
    return not target.exists() or any(d.stat().st_mtime > target.stat().st_mtime for d in deps)


def native_path() -> Path:
    """Where the native module for the running PyTorch and Python is: it is compiled against the headers of both, so that one built for
    others is neither fresh nor loaded."""
    import torch

    return PKG_DIR / f"_native-{torch.__version__}{sysconfig.get_config_var('EXT_SUFFIX')}"


def _header() -> Path:
    return PKG_DIR.parent / "include" / "heddle_b200.h"


def _stale() -> bool:
    return _older(LIB_PATH, [*CSRC.glob("*.cu"), *CSRC.glob("*.cuh"), *CSRC.glob("*.h"), _header()])


def _native_stale() -> bool:
    try:
        return _older(native_path(), [NATIVE_SRC, _header()])
    except ImportError:  # no PyTorch: _build_native() says so, and the library is built all the same
        return True


def _compile_one(src: Path) -> tuple[Path, str]:
    obj = OBJ_DIR / (src.stem + ".o")
    cmd = [_nvcc(), *NVCC_FLAGS, "-c", str(src), "-o", str(obj)]
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        raise RuntimeError(f"nvcc failed for {src.name}:\n{proc.stdout}\n{proc.stderr}")
    return obj, proc.stderr


def _compile_native() -> None:
    """PyTorch's libraries are the ones that ``import torch`` has loaded."""
    import torch

    torch_dir = Path(torch.__file__).resolve().parent
    cxx = shutil.which("g++") or "g++"
    cuda_include = Path(_nvcc()).resolve().parent.parent / "include"
    includes = [torch_dir / "include", torch_dir / "include/torch/csrc/api/include", cuda_include, sysconfig.get_paths()["include"]]
    cmd = [cxx, "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           *[f for d in includes for f in ("-isystem", str(d))], str(NATIVE_SRC), "-o", str(native_path()),
           f"-L{torch_dir / 'lib'}", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python"]
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        raise RuntimeError(f"g++ failed for {NATIVE_SRC.name}:\n{proc.stdout}\n{proc.stderr}")


def _build_native() -> None:
    """Without it (no g++, no headers of Python or PyTorch) the tensor-level calls do in Python what it does, at more host time."""
    try:
        native_path().unlink(missing_ok=True)  # one built from other sources may not stay behind
        _compile_native()
    except Exception as e:
        warnings.warn(f"heddle_b200._native was not built, its host path stays in Python: {e}", RuntimeWarning, stacklevel=2)


def build(force: bool = False, verbose: bool = False) -> Path:
    if force or _native_stale():
        _build_native()
    if not force and not _stale():
        return LIB_PATH
    OBJ_DIR.mkdir(parents=True, exist_ok=True)
    with concurrent.futures.ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as pool:
        results = list(pool.map(_compile_one, sources()))
    log = "".join(text for _, text in results)
    (OBJ_DIR / "ptxas.log").write_text(log)
    if verbose:
        sys.stderr.write(log)
    cmd = [_nvcc(), "-shared", "-cudart", "static", "-o", str(LIB_PATH), *[str(o) for o, _ in results], "-ldl"]
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        raise RuntimeError(f"link failed:\n{proc.stdout}\n{proc.stderr}")
    return LIB_PATH


if __name__ == "__main__":
    print(build(force=True, verbose="-v" in sys.argv))
