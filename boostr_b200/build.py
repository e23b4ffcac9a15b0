"""Compiles the CUDA sources into ``boostr_b200/libb200q.so`` for sm_100a with nvcc, and the Python entry points
(``host_ops.cpp``) into the extension module ``boostr_b200/_hostops`` against torch's headers.

No GPU is needed to build.  ``python -m boostr_b200.build`` (or ``build()``) recompiles only the translation units whose
sources changed, and the extension also when Python or torch did; ``-f`` recompiles everything.
"""
from __future__ import annotations

import concurrent.futures
import importlib.metadata
import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJDIR = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "libb200q.so")
HOST_LIB = os.path.join(HERE, "_hostops" + sysconfig.get_config_var("EXT_SUFFIX"))  # the name carries Python's ABI
HOST_STAMP = os.path.join(OBJDIR, "_hostops.stamp")
HOST_SOURCE = os.path.join(CSRC, "host_ops.cpp")
SOURCES = ["api.cu", "dequant.cu", "gemv.cu", "gemv_m1.cu", "gemv_m1_f32.cu", "kquant_few.cu", "kquant_i8.cu", "prefill.cu", "smallm_i8.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden", "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; set NVCC or add it to PATH")


def _newest_dep() -> float:
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    deps.append(os.path.join(HERE, "..", "include", "b200q.h"))
    return max(os.path.getmtime(d) for d in deps)


def _compile(src: str, verbose: bool) -> str:
    obj = os.path.join(OBJDIR, src.replace(".cu", ".o"))
    spath = os.path.join(CSRC, src)
    if os.path.exists(obj) and os.path.getmtime(obj) >= max(os.path.getmtime(spath), _newest_dep()):
        return obj
    cmd = [_nvcc(), *NVCC_FLAGS, "-c", spath, "-o", obj]
    if verbose:
        cmd.insert(1, "-Xptxas=-v")
    r = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or r.returncode:
        sys.stderr.write(r.stdout + r.stderr)
    if r.returncode:
        raise RuntimeError(f"nvcc failed on {src}")
    return obj


def _host_stamp() -> str:
    """What the extension is compiled against."""
    return f"{os.path.basename(HOST_LIB)} torch {importlib.metadata.version('torch')}"


def _host_current() -> bool:
    header = os.path.join(HERE, "..", "include", "b200q.h")
    if not (os.path.exists(HOST_LIB) and os.path.exists(HOST_STAMP)):
        return False
    with open(HOST_STAMP) as f:
        return f.read() == _host_stamp() and os.path.getmtime(HOST_LIB) >= max(os.path.getmtime(HOST_SOURCE), os.path.getmtime(header))


def _build_host() -> None:
    if _host_current():
        return
    import torch
    from torch.utils.cpp_extension import include_paths

    cuda = os.path.dirname(os.path.dirname(os.path.realpath(_nvcc())))
    incs = [*include_paths(), os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]
    tlib = os.path.join(os.path.dirname(torch.__file__), "lib")
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
           *[f"-I{i}" for i in incs], HOST_SOURCE, "-o", HOST_LIB, f"-L{tlib}", "-lc10", "-lc10_cuda", "-ltorch", "-ltorch_cpu", "-ltorch_cuda",
           "-ltorch_python", f"-L{HERE}", "-l:libb200q.so", "-Wl,-rpath,$ORIGIN"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode:
        sys.stderr.write(r.stdout + r.stderr)
        raise RuntimeError("g++ failed on host_ops.cpp")
    untagged = os.path.join(HERE, "_hostops.so")
    if os.path.exists(untagged):  # of a build without Python's ABI in the name
        os.remove(untagged)
    with open(HOST_STAMP, "w") as f:
        f.write(_host_stamp())


def build(verbose: bool = False, force: bool = False) -> str:
    os.makedirs(OBJDIR, exist_ok=True)
    if force:
        for f in os.listdir(OBJDIR):
            os.remove(os.path.join(OBJDIR, f))
    with concurrent.futures.ThreadPoolExecutor(max_workers=len(SOURCES)) as ex:
        objs = list(ex.map(lambda s: _compile(s, verbose), SOURCES))
    if not os.path.exists(LIB) or os.path.getmtime(LIB) < max(os.path.getmtime(o) for o in objs):
        cmd = [_nvcc(), "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a", "-lcudart"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("link failed")
    _build_host()
    return LIB


if __name__ == "__main__":
    print(build(verbose="-v" in sys.argv, force="-f" in sys.argv))
