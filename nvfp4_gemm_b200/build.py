"""Ahead-of-time build of the CUDA library and the torch binding (``python -m nvfp4_gemm_b200.build``).

Compiles ``csrc/nvfp4_api.cu`` for sm_100a into ``libnvfp4_b200.so`` and ``csrc/torch_binding.cpp``
(host code only) into ``_native.so`` next to this file.  nvcc cross-compiles without a GPU.  The first
needs nvcc alone, the second g++ and the torch that it will run with.  Nothing is JIT-compiled at call
time (the reference builds at import with ``load_inline``, s_128t.py:587-602).
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
from pathlib import Path

PKG_DIR = Path(__file__).resolve().parent
SRC = PKG_DIR / "csrc" / "nvfp4_api.cu"
LIB = PKG_DIR / "libnvfp4_b200.so"
HEADER = PKG_DIR.parent / "include" / "nvfp4_b200.h"
BINDING_SRC = PKG_DIR / "csrc" / "torch_binding.cpp"
BINDING = PKG_DIR / "_native.so"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "--shared", "-Xcompiler", "-fPIC",
    "-cudart", "static",
]


def find_nvcc() -> str:
    nvcc = shutil.which("nvcc") or os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found (looked on PATH and in $CUDA_HOME/bin)")
    return nvcc


def sources() -> list[Path]:
    return [SRC, *sorted((PKG_DIR / "csrc").glob("*.cuh")), HEADER]


def _newer(target: Path, inputs: list[Path]) -> bool:
    return target.exists() and all(s.stat().st_mtime <= target.stat().st_mtime for s in inputs)


def binding_target() -> str:
    """What ``_native.so`` has to be built for: it holds layouts of torch's and Python's own types."""
    import torch
    return f"torch {torch.__version__}, C++11 ABI {int(torch._C._GLIBCXX_USE_CXX11_ABI)}, {sysconfig.get_config_var('SOABI')}"


def binding_built_for() -> str | None:
    """What the ``_native.so`` that is there was built for (the module carries it as a text)."""
    if not BINDING.exists():
        return None
    mark = b"nvfp4_native built for: "
    _, found, rest = BINDING.read_bytes().partition(mark)
    return rest.partition(b"\0")[0].decode() if found else None


def why_no_binding() -> str | None:
    """The binding serves callers with torch; why it cannot be built here, or None."""
    try:
        import torch
    except ImportError as e:
        return f"torch cannot be imported ({e})"
    if shutil.which("g++") is None:
        return "g++ was not found"
    if not (Path(torch.__file__).resolve().parent / "include" / "torch" / "csrc" / "autograd" / "python_variable.h").exists():
        return "this torch has no headers"
    if not (Path(sysconfig.get_paths()["include"]) / "Python.h").exists():
        return "Python's headers are not installed"
    return None


def _binding_current() -> bool:
    return _newer(BINDING, [BINDING_SRC, HEADER]) and binding_built_for() == binding_target()


def needs_build() -> bool:
    return not _newer(LIB, sources()) or (why_no_binding() is None and not _binding_current())


def _replace(target: Path, cmd: list[str], verbose: bool) -> None:
    tmp = target.with_suffix(".so.building")
    cmd = [*cmd, "-o", str(tmp)]
    if verbose:
        print(" ".join(cmd), file=sys.stderr)
    subprocess.check_call(cmd)
    os.replace(tmp, target)       # a reader never sees a half-written library


def _build_binding(verbose: bool) -> None:
    import torch
    torch_dir = Path(torch.__file__).resolve().parent
    cuda_home = Path(find_nvcc()).resolve().parent.parent
    includes = [torch_dir / "include", torch_dir / "include" / "torch" / "csrc" / "api" / "include", cuda_home / "include",
                Path(sysconfig.get_paths()["include"])]
    # (torch's own libraries are in the process when the module is loaded: torch is imported first)
    _replace(BINDING, ["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden",
                       f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f'-DNVFP4_BUILT_FOR="{binding_target()}"',
                       *[f for i in includes for f in ("-isystem", str(i))], str(BINDING_SRC),
                       f"-L{PKG_DIR}", "-l:libnvfp4_b200.so", f"-L{torch_dir / 'lib'}", "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10",
                       "-lc10_cuda", "-Wl,-rpath,$ORIGIN"], verbose)


def build(force: bool = False, verbose: bool = False) -> Path:
    """Builds what is out of date.  The C library needs nvcc alone; where the binding cannot be built, a
    caller of the C library is told so and gets it all the same (``_lib.native()`` refuses to go on without)."""
    if force or not _newer(LIB, sources()):
        _replace(LIB, [find_nvcc(), *(["-Xptxas", "-v"] if verbose else []), *NVCC_FLAGS, str(SRC)], verbose)
    why = why_no_binding()
    if why is not None:
        print(f"{BINDING.name} (calls on torch tensors) is not built: {why}", file=sys.stderr)
    elif force or not _binding_current():
        _build_binding(verbose)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
