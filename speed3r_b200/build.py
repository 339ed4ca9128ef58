"""Build recipe for the C-ABI library: every ``csrc/*.cu`` is compiled for sm_100a with nvcc and
linked into ``speed3r_b200/libspeed3r_b200.so`` (kept in-tree, next to the package).  The ``torch.library``
operators over it (``csrc/torch/*.cpp``, host C++ against the installed PyTorch) become
``libspeed3r_b200_torch.so``, which finds the C-ABI library beside itself.  The tests-only companion ``libspeed3r_b200_check.so`` (``csrc/check/*.cu`` plus the shared host plumbing) is built
beside it; the package never loads it.

    python -m speed3r_b200.build [-v] [--force]
"""
from __future__ import annotations

import concurrent.futures as cf
import glob
import os
import shutil
import subprocess
import sys

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
OBJ = os.path.join(PKG, "csrc", "build")
LIB = os.path.join(PKG, "libspeed3r_b200.so")
TORCH_LIB = os.path.join(PKG, "libspeed3r_b200_torch.so")
CHECK_LIB = os.path.join(PKG, "libspeed3r_b200_check.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
    "-Xptxas", "-v",
    "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    cand = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(cand):
        raise RuntimeError("nvcc not found: the CUDA library cannot be built")
    return cand


def _stale(target: str, deps) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def _compile(src: str, verbose: bool) -> str:
    obj = os.path.join(OBJ, os.path.basename(src)[:-3] + ".o")
    headers = glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(PKG, "..", "include", "*.h"))
    os.makedirs(OBJ, exist_ok=True)
    if _stale(obj, [src] + headers):
        cmd = [_nvcc()] + NVCC_FLAGS + ["-c", src, "-o", obj]
        r = subprocess.run(cmd, capture_output=True, text=True)
        log = os.path.join(OBJ, os.path.basename(src)[:-3] + ".ptxas.log")
        with open(log, "w") as f:
            f.write(r.stdout + r.stderr)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{r.stdout}\n{r.stderr}")
        if verbose:
            print(r.stderr)
    return obj


def _build_torch_lib() -> None:
    """The operators' library; recompiled when a source, the header or the PyTorch it was built for changes."""
    import torch
    inc = os.path.join(os.path.dirname(torch.__file__), "include")
    lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    srcs = sorted(glob.glob(os.path.join(CSRC, "torch", "*.cpp")))
    stamp = os.path.join(OBJ, "torch_version")
    built_for = open(stamp).read() if os.path.exists(stamp) else ""
    if built_for == torch.__version__ and not _stale(TORCH_LIB, srcs + glob.glob(os.path.join(PKG, "..", "include", "*.h"))):
        return
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        raise RuntimeError("no C++ compiler found: the operator library cannot be built")
    cmd = [cxx, "-O2", "-std=c++17", "-fPIC", "-shared", "-o", TORCH_LIB] + srcs + [
        f"-I{inc}", f"-I{inc}/torch/csrc/api/include", f"-I{cuda}/include",
        f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
        f"-L{PKG}", "-l:libspeed3r_b200.so", "-Wl,-rpath,$ORIGIN", f"-L{lib}", "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda",
        f"-L{cuda}/lib64", "-lcudart"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"{cxx} failed on the operator library:\n{r.stdout}\n{r.stderr}")
    with open(stamp, "w") as f:
        f.write(torch.__version__)


def build(verbose: bool = False, force: bool = False) -> str:
    os.makedirs(OBJ, exist_ok=True)
    if force:
        for f in glob.glob(os.path.join(OBJ, "*.o")):
            os.remove(f)
    srcs = sorted(glob.glob(os.path.join(CSRC, "*.cu")))
    check_srcs = sorted(glob.glob(os.path.join(CSRC, "check", "*.cu")))
    with cf.ThreadPoolExecutor(max_workers=min(8, len(srcs) + len(check_srcs))) as ex:
        all_objs = list(ex.map(lambda s: _compile(s, verbose), srcs + check_srcs))
    objs, check_objs = all_objs[:len(srcs)], all_objs[len(srcs):]
    api_obj = [o for o in objs if os.path.basename(o) == "api.o"]
    for lib, members in ((LIB, objs), (CHECK_LIB, check_objs + api_obj)):
        if _stale(lib, members):
            cmd = [_nvcc(), "-shared", "-o", lib] + members + ["-gencode", "arch=compute_100a,code=sm_100a", "-lcudart"]
            r = subprocess.run(cmd, capture_output=True, text=True)
            if r.returncode != 0:
                raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    _build_torch_lib()
    return LIB


if __name__ == "__main__":
    print(build(verbose="-v" in sys.argv, force="--force" in sys.argv))
