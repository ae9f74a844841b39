"""Build recipe for libdmgs_gb300.so (sm_103a only).

Compiles every ``csrc/*.cu`` translation unit in parallel with nvcc and links
them into ``dmgs_gb300/libdmgs_gb300.so`` (in-tree, git-ignored); beside them
the host compiler builds ``csrc/autograd.cpp``, the native autograd nodes, into
``dmgs_gb300/_autograd.so``.  Objects go to ``dmgs_gb300/_build/``.  Rebuilds
only what changed.
"""
from __future__ import annotations

import concurrent.futures as cf
import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
BUILD = os.path.join(HERE, "_build")
LIB = os.path.join(HERE, "libdmgs_gb300.so")
EXT = os.path.join(HERE, "_autograd.so")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")

ARCH = ["-gencode", "arch=compute_103a,code=sm_103a"]
NVCC_FLAGS = ARCH + ["-O3", "-lineinfo", "-std=c++17", "-Xcompiler", "-fPIC",
                     "-Xptxas", "-warn-spills", "--expt-relaxed-constexpr"]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found: the CUDA toolkit is required to build libdmgs_gb300.so")


def _sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def _headers():
    hs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    hs.append(os.path.join(INCLUDE, "dmgs.h"))
    return hs


def _ext_commands():
    """(compile, link) commands of the autograd extension, its object."""
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    obj = os.path.join(BUILD, "autograd.cpp.o")
    inc = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
           os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]
    cxx = os.environ.get("CXX") or shutil.which("g++") or "c++"
    comp = [cxx, "-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-w",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            *[a for i in inc for a in ("-isystem", i)], "-c", os.path.join(CSRC, "autograd.cpp"), "-o", obj]
    link = [cxx, "-shared", "-o", EXT + ".tmp", obj, "-L", os.path.join(root, "lib"), "-ltorch", "-ltorch_cpu",
            "-ltorch_python", "-lc10", "-lc10_cuda", "-L", HERE, "-l:libdmgs_gb300.so", "-Wl,-rpath,$ORIGIN"]
    return comp, link, obj


def _stale(target: str, deps) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build(verbose: bool = False, force: bool = False, extra_flags=()) -> str:
    """Compile and link; returns the library path."""
    os.makedirs(BUILD, exist_ok=True)
    nvcc = _nvcc()
    headers = _headers()
    jobs = []
    objs = []
    for src in _sources():
        obj = os.path.join(BUILD, os.path.basename(src) + ".o")
        objs.append(obj)
        if force or _stale(obj, [src, *headers, __file__]):
            cmd = [nvcc, *NVCC_FLAGS, *extra_flags, "-I", INCLUDE, "-c", src, "-o", obj]
            jobs.append(cmd)

    ext_src = os.path.join(CSRC, "autograd.cpp")
    ext_compile, ext_link, ext_obj = _ext_commands()
    ext_stale = force or _stale(ext_obj, [ext_src, os.path.join(INCLUDE, "dmgs.h"), __file__])
    if ext_stale:
        jobs.insert(0, ext_compile)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        return cmd, r

    if jobs:
        with cf.ThreadPoolExecutor(max_workers=min(len(jobs), os.cpu_count() or 4)) as ex:
            for cmd, r in ex.map(run, jobs):
                if verbose or r.returncode != 0:
                    sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
                if r.returncode != 0:
                    raise RuntimeError(f"{os.path.basename(cmd[0])} failed for {cmd[-3]}")
    if force or jobs or _stale(LIB, objs):
        tmp = LIB + ".tmp"
        cmd = [nvcc, *ARCH, "-shared", "-cudart", "shared", "-o", tmp, *objs,
               "-Xlinker", "-rpath,/usr/local/cuda/lib64"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if verbose or r.returncode != 0:
            sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
        if r.returncode != 0:
            raise RuntimeError("link of libdmgs_gb300.so failed")
        os.replace(tmp, LIB)
    if ext_stale or _stale(EXT, [ext_obj]):
        r = subprocess.run(ext_link, capture_output=True, text=True)
        if verbose or r.returncode != 0:
            sys.stderr.write(" ".join(ext_link) + "\n" + r.stdout + r.stderr)
        if r.returncode != 0:
            raise RuntimeError("link of _autograd.so failed")
        os.replace(EXT + ".tmp", EXT)
    return LIB


if __name__ == "__main__":
    print(build(verbose="-v" in sys.argv, force="-f" in sys.argv))
