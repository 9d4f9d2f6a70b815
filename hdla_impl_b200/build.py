"""Build libhdla.so (the C-ABI CUDA library) in-tree with nvcc for sm_100a, and _binding.so (the host path between
PyTorch and that library) with g++.

    python -m hdla_impl_b200.build [--force] [--verbose]

Both land next to this file; each is rebuilt only when a source or header of it is newer, _binding.so also when it was
built for another PyTorch.  Processes that find one missing at the same time build it once: the others wait.
"""
from __future__ import annotations

import contextlib
import fcntl
import glob
import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libhdla.so")
BINDING = os.path.join(HERE, "_binding.so")
BINDING_SRC = os.path.join(CSRC, "binding.cpp")
ROOT = os.path.dirname(HERE)

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "--use_fast_math", "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
]


def _nvcc() -> str:
    cand = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(cand):
        raise RuntimeError("nvcc not found: libhdla.so cannot be built")
    return cand


def sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def _stale() -> bool:
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    deps = sources() + glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(ROOT, "include", "*.h"))
    return any(os.path.getmtime(f) > t for f in deps)


# In the file's own bytes, so that it says what it was built for before it is loaded into a process.
_BUILT_FOR = "hdla_impl_b200 _binding built for PyTorch "


def _torch_version() -> str:
    import torch
    return str(torch.__version__)


def binding_built_for(path: str) -> str:
    """The PyTorch version that the file was built for ("" if it does not say)."""
    with open(path, "rb") as f:
        _, found, rest = f.read().partition(_BUILT_FOR.encode())
    return rest.partition(b"\0")[0].decode(errors="replace") if found else ""


def _binding_sources():
    files = [BINDING_SRC, os.path.join(CSRC, "status_board.h"), os.path.join(ROOT, "include", "hdla.h")]
    return [f for f in files if os.path.exists(f)]


def _binding_stale() -> bool:
    if not os.path.exists(BINDING):
        return True
    t = os.path.getmtime(BINDING)
    return any(os.path.getmtime(f) > t for f in _binding_sources()) or binding_built_for(BINDING) != _torch_version()


@contextlib.contextmanager
def _one_builder(path: str):
    """Held by the process that builds ``path``."""
    with open(path + ".lock", "w") as f:
        fcntl.flock(f, fcntl.LOCK_EX)
        yield


def _compile(cmd, out: str, what: str) -> None:
    """Run ``cmd`` with its output going to a file of its own that then takes the place of ``out``: a process that opens
    ``out`` meanwhile finds a whole file, and one that has it mapped keeps what it has."""
    tmp = f"{out}.{os.getpid()}.tmp"
    try:
        r = subprocess.run([*cmd, "-o", tmp], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"{what}:\n{r.stdout}")
        os.replace(tmp, out)
    finally:
        if os.path.exists(tmp):
            os.remove(tmp)


def build_binding(force: bool = False) -> str:
    """Compile csrc/binding.cpp against the installed PyTorch (its headers and libraries)."""
    if not force and not _binding_stale():
        return BINDING
    with _one_builder(BINDING):
        if force or _binding_stale():
            import torch
            top = os.path.dirname(os.path.abspath(torch.__file__))
            cuda = os.path.dirname(os.path.dirname(_nvcc()))
            inc = [os.path.join(top, "include"), os.path.join(top, "include", "torch", "csrc", "api", "include"),
                   os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]
            cmd = [shutil.which("g++") or "g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
                   f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
                   f'-DHDLA_BUILT_FOR="{_BUILT_FOR}{_torch_version()}"', *[f"-I{d}" for d in inc], BINDING_SRC,
                   "-L" + os.path.join(top, "lib"), "-L" + os.path.join(cuda, "lib64"), "-ltorch", "-ltorch_cpu",
                   "-ltorch_cuda", "-ltorch_python", "-lc10", "-lc10_cuda", "-lcudart"]
            _compile(cmd, BINDING, f"g++ failed on {BINDING_SRC}")
    return BINDING


def build(force: bool = False, verbose: bool = False) -> str:
    build_binding(force)
    if not force and not _stale():
        return LIB
    with _one_builder(LIB):
        if force or _stale():
            _build_lib(verbose)
    return LIB


def _build_lib(verbose: bool) -> None:
    objdir = os.path.join(HERE, "build")
    os.makedirs(objdir, exist_ok=True)
    nvcc = _nvcc()
    objs = []
    procs = []
    for src in sources():
        obj = os.path.join(objdir, os.path.basename(src)[:-3] + ".o")
        extra = os.environ.get("HDLA_NVCC_EXTRA", "").split()        # e.g. -DHDLA_TIMELINE for the tracing build
        cmd = [nvcc, *NVCC_FLAGS, *extra, "-c", src, "-o", obj] + (["-Xptxas", "-v"] if verbose else [])
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(obj)
    for src, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{out}")
        if verbose and out:
            print(out)
    _compile([nvcc, "-shared", *objs, "-gencode", "arch=compute_100a,code=sm_100a", "-lcudart"], LIB, "link failed")


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
