"""Ahead-of-time build of the C-ABI shared library and its Python binding (in-tree, sm_100a only).

    python -m xlstm_b200.build            # -> xlstm_b200/libxlstm_b200.so, xlstm_b200/_native.so

nvcc cross-compiles for sm_100a without a GPU.  The library has no link-time
dependency on libcuda (the one driver entry point it needs, the tensor-map
encoder, is looked up at run time) and links the CUDA runtime statically, so
it loads on a machine without a driver; only launching needs a B200.  The
binding (`csrc/binding.cpp`, the native host path of `ops.py`) is linked
against it and against the installed PyTorch.  Sources are compiled one by
one, in parallel, into `build/`, so a change recompiles only what it touches;
another PyTorch or interpreter than the last build's recompiles the binding.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "..", "build")
HEADER = os.path.join(HERE, "..", "include", "xlstm_b200.h")
LIB = os.path.join(HERE, "libxlstm_b200.so")
NATIVE = os.path.join(HERE, "_native.so")
STAMP = os.path.join(OBJ, "binding.stamp")
SOURCES = ["capi.cu", "mlstm_step.cu", "mlstm_recurrent.cu", "mlstm_chunkwise.cu", "mlstm_parts.cu", "slstm_fwd.cu", "slstm_bwd.cu", "slstm_wgrad.cu", "layer_adjacent.cu", "greedy_head.cu", "peer_reduce.cu", "headwise_proj.cu", "rows_linear.cu"]
BINDING = "binding.cpp"
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
NVCC_FLAGS = [*ARCH, "-lineinfo", "-O3", "-std=c++17", "-Xcompiler", "-fPIC"]


def _nvcc() -> str:
    cand = shutil.which("nvcc") or os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    if not os.path.exists(cand):
        raise RuntimeError("nvcc not found; set CUDA_HOME")
    return cand


def _run(cmd) -> str:
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"{cmd[0]} failed:\n" + res.stdout + res.stderr)
    return res.stderr


def _newer(deps, target) -> bool:
    return not os.path.exists(target) or any(os.path.getmtime(d) > os.path.getmtime(target) for d in deps)


def _headers():
    return [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))] + [HEADER]


def _binding_stamp() -> str:
    """What the binding is compiled against besides its sources: it is valid for this PyTorch and this interpreter only."""
    import torch
    return f"{torch.__version__} {os.path.dirname(torch.__file__)} {sys.version}"


def _binding_stale() -> bool:
    try:
        with open(STAMP) as fh:
            return fh.read() != _binding_stamp()
    except FileNotFoundError:
        return True


def needs_build() -> bool:
    cu = [os.path.join(CSRC, s) for s in SOURCES] + _headers()
    return _newer(cu, LIB) or _newer([os.path.join(CSRC, BINDING), HEADER], NATIVE) or _binding_stale()


def _binding_command(obj: str):
    import torch
    inc = os.path.join(os.path.dirname(torch.__file__), "include")
    cuda = os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "include")
    return ["g++", "-O2", "-std=c++17", "-fPIC", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            f'-DXL_BUILT_FOR="{torch.__version__}"', "-I", inc,
            "-I", os.path.join(inc, "torch", "csrc", "api", "include"), "-I", cuda, "-I", sysconfig.get_paths()["include"], "-c",
            os.path.join(CSRC, BINDING), "-o", obj]


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not needs_build():
        return LIB
    import torch
    os.makedirs(OBJ, exist_ok=True)
    extra = ["-Xptxas", "-v"] if verbose else []
    jobs, objs = [], []
    for s in SOURCES:
        src, obj = os.path.join(CSRC, s), os.path.join(OBJ, s + ".o")
        objs.append(obj)
        if force or _newer([src, *_headers()], obj):
            jobs.append([_nvcc(), *extra, *NVCC_FLAGS, "-c", src, "-o", obj])
    bobj = os.path.join(OBJ, BINDING + ".o")
    if force or _newer([os.path.join(CSRC, BINDING), HEADER], bobj) or _binding_stale():
        jobs.append(_binding_command(bobj))
    with ThreadPoolExecutor(max_workers=os.cpu_count() or 1) as pool:
        for log in pool.map(_run, jobs):
            if verbose:
                print(log)
    _run([_nvcc(), *ARCH, "--shared", "-Xlinker", "-soname=libxlstm_b200.so", "-o", LIB, *objs])
    tlib = os.path.join(os.path.dirname(torch.__file__), "lib")
    _run(["g++", "-shared", "-o", NATIVE, bobj, LIB, "-L", tlib, "-ltorch_python", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda",
          "-Wl,-rpath,$ORIGIN"])
    with open(STAMP, "w") as fh:
        fh.write(_binding_stamp())
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
