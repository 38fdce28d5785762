"""Builds and loads the torch glue (csrc/torch_glue.cpp, sdpa_autograd.cpp, py_calls.cpp -> lib/libsdpa_b200_torch.so).

After ``load()``:
* ``torch.ops.b200_sdpa._scaled_dot_product_flash_attention`` (+ ``_backward``) and
  ``torch.ops.b200_sdpa._flash_attention_forward`` (+ ``_backward``) exist with the reference's
  schemas (codegen/mlu_functions.yaml:1313-1316) and differentiate through autograd.
* ``install_aten_overrides()`` additionally points the CUDA kernels of the same four ``aten``
  operators at this library, so ``F.scaled_dot_product_attention`` under the flash backend runs
  here. It is opt-in because it changes those operators for the whole process.
"""
from __future__ import annotations

import os
import subprocess
import sys

import torch

from . import _cabi, build as native_build

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
SOURCES = ["torch_glue.cpp", "sdpa_autograd.cpp", "py_calls.cpp"]
OBJ_DIR = os.path.join(HERE, "build")
LIB = os.path.join(_cabi.LIB_DIR, "libsdpa_b200_torch.so")
calls = None  # the module of csrc/py_calls.cpp, once load() has run
_load_error = None  # why calls_or_none() has none


def build(verbose: bool = False) -> str:
    """g++ the glue against the installed torch and the C-ABI library (no GPU needed)."""
    # A process that already holds the C-ABI library must not re-link it underneath itself: the glue would
    # then load the new file as a second copy with its own state (error text, launch counter).
    if _cabi._lib is None:
        native_build.build_native()
    headers = [os.path.join(CSRC, "torch_glue.h"), os.path.join(os.path.dirname(HERE), "include", "sdpa_b200.h")]
    newest = max(os.path.getmtime(p) for p in headers + [os.path.join(CSRC, f) for f in SOURCES])
    if os.path.exists(LIB) and os.path.getmtime(LIB) >= newest:
        return LIB
    import sysconfig
    from concurrent.futures import ThreadPoolExecutor
    from torch.utils import cpp_extension
    inc = [f"-I{p}" for p in cpp_extension.include_paths()]
    cuda_home = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    inc += [f"-I{cuda_home}/include", f"-I{sysconfig.get_paths()['include']}"]
    torch_lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    abi = int(torch._C._GLIBCXX_USE_CXX11_ABI)
    os.makedirs(OBJ_DIR, exist_ok=True)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        if verbose or r.returncode != 0:
            sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
        if r.returncode != 0:
            raise RuntimeError("building the torch glue failed")

    objs = [os.path.join(OBJ_DIR, f.replace(".cpp", ".glue.o")) for f in SOURCES]
    stale = [(f, o) for f, o in zip(SOURCES, objs) if not os.path.exists(o) or
             os.path.getmtime(o) < max(os.path.getmtime(p) for p in headers + [os.path.join(CSRC, f)])]
    with ThreadPoolExecutor(max_workers=len(SOURCES)) as ex:
        list(ex.map(lambda fo: run(["g++", "-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", f"-D_GLIBCXX_USE_CXX11_ABI={abi}",
                                    "-DTORCH_API_INCLUDE_EXTENSION_H", *inc, "-c", os.path.join(CSRC, fo[0]), "-o", fo[1]]), stale))
    run(["g++", "-shared", *objs, "-o", LIB, f"-L{_cabi.LIB_DIR}", "-lsdpa_b200", f"-L{torch_lib}", "-ltorch", "-ltorch_cpu", "-lc10",
         "-ltorch_cuda", "-lc10_cuda", "-ltorch_python", "-Wl,-rpath,$ORIGIN", f"-Wl,-rpath,{torch_lib}"])
    return LIB


def load():
    """Load the glue library (building it first if needed) and return its module of direct calls. Raises if it cannot
    be built."""
    global calls
    if calls is not None:
        return calls
    import importlib.machinery
    import importlib.util
    build()
    _cabi.load()
    torch.ops.load_library(LIB)
    loader = importlib.machinery.ExtensionFileLoader("libsdpa_b200_torch", LIB)
    module = importlib.util.module_from_spec(importlib.util.spec_from_loader("libsdpa_b200_torch", loader))
    loader.exec_module(module)
    module.set_status_error(_cabi.SdpaError)
    calls = module
    return calls


def calls_or_none():
    """The module of direct calls, loaded on first use; None where it cannot be built or loaded (no compiler or torch headers),
    which is said once. The C library and everything that needs only it work without the glue."""
    global _load_error
    if calls is not None:
        return calls
    if _load_error is None:
        try:
            return load()
        except Exception as e:  # a failed build, a library that does not fit this torch
            import warnings
            _load_error = e
            warnings.warn(f"the torch glue of torch_mlu_b200 is not available ({e}): calls go through ctypes, which costs some tens of "
                          "microseconds each", RuntimeWarning, stacklevel=3)
    return None


def install_aten_overrides() -> None:
    load()
    torch.ops.b200_sdpa._install_aten_overrides()


def remove_aten_overrides() -> None:
    if calls is not None:
        torch.ops.b200_sdpa._remove_aten_overrides()


if __name__ == "__main__":
    print(build(verbose="-v" in sys.argv))
