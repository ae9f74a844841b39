"""Build recipe for libdmgs_gb300.so (sm_103a only).

Compiles every ``csrc/*.cu`` translation unit in parallel with nvcc and links
them into ``dmgs_gb300/libdmgs_gb300.so`` (in-tree, git-ignored); beside them
the host compiler builds ``csrc/autograd.cpp``, the native autograd nodes, into
``dmgs_gb300/_autograd.so``.  Objects go to ``dmgs_gb300/_build/``.  Rebuilds
only what changed.

The library needs nvcc alone and is linked whatever becomes of the extension.
The extension needs the headers of a CUDA torch and is tied to the torch and
Python it was built with (recorded in ``_build/autograd.tag``); without a CUDA
torch it is not built, and a program that uses the library through its C
interface does not miss it.
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
TAG = os.path.join(BUILD, "autograd.tag")  # what EXT was built with
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
    """(compile command, link command, object, tag) of the autograd extension,
    the tag naming all that its build depends on besides the sources; None
    without a CUDA torch."""
    try:
        import torch
    except ImportError:
        return None
    if torch.version.cuda is None:
        return None
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
    return comp, link, obj, "\n".join([torch.__version__, sys.version, *comp, *link])


def _stale(target: str, deps) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def _read(path: str):
    try:
        with open(path) as f:
            return f.read()
    except OSError:
        return None


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

    ext = _ext_commands()
    ext_stale = False
    if ext is None:
        sys.stderr.write("no torch with CUDA: _autograd.so is not built\n")
    else:
        comp, link, ext_obj, tag = ext
        ext_src = os.path.join(CSRC, "autograd.cpp")
        ext_stale = (force or _stale(ext_obj, [ext_src, os.path.join(INCLUDE, "dmgs.h"), __file__])
                     or not os.path.exists(EXT) or _read(TAG) != tag)
        if ext_stale:
            jobs.insert(0, comp)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        if verbose or r.returncode != 0:
            sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
        return r.returncode == 0

    ext_failed = False
    if jobs:
        with cf.ThreadPoolExecutor(max_workers=min(len(jobs), os.cpu_count() or 4)) as ex:
            for cmd, ok in zip(jobs, ex.map(run, jobs)):
                if ok:
                    continue
                if ext_stale and cmd is comp:
                    ext_failed = True
                else:
                    raise RuntimeError(f"{os.path.basename(cmd[0])} failed for {cmd[-3]}")
    if force or jobs or _stale(LIB, objs):
        tmp = LIB + ".tmp"
        cmd = [nvcc, *ARCH, "-shared", "-cudart", "shared", "-o", tmp, *objs,
               "-Xlinker", "-rpath,/usr/local/cuda/lib64"]
        if not run(cmd):
            raise RuntimeError("link of libdmgs_gb300.so failed")
        os.replace(tmp, LIB)
    if ext_stale:
        if ext_failed:
            raise RuntimeError(f"{os.path.basename(comp[0])} failed for {comp[-3]} (libdmgs_gb300.so is built)")
        if not run(link):
            raise RuntimeError("link of _autograd.so failed (libdmgs_gb300.so is built)")
        os.replace(EXT + ".tmp", EXT)
        with open(TAG, "w") as f:
            f.write(tag)
    return LIB


if __name__ == "__main__":
    print(build(verbose="-v" in sys.argv, force="-f" in sys.argv))
