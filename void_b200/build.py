"""Builds the libraries of the SpMM path in-tree (void_b200/lib): the C-ABI library for sm_100a with nvcc, and the
native host path of the Python operators (a CPython extension on top of it) with the C++ compiler.

The host path is compiled against the headers of one torch and one Python, whose internals it uses.  Its file name carries
what it was built from and for, so that one made for another torch, Python or source is never found, let alone loaded.

nvcc cross-compiles for sm_100a without a GPU.  Run as ``python -m void_b200.build``.
"""
import hashlib
import os
import shutil
import subprocess
import sys
import sysconfig
import tempfile

import torch

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB_DIR = os.path.join(HERE, "lib")
LIB_PATH = os.path.join(LIB_DIR, "libvoid_b200.so")
SOURCES = ["spmm.cu", "rowacc_i8.cu", "rowacc_f8.cu", "rowacc_f16.cu", "rowacc_tf32.cu", "skinny.cu", "group.cu", "prep.cu", "plan.cu", "format.cu", "tile_grad.cu"]
HOST_SOURCE = os.path.join(CSRC, "host.cpp")
HEADERS = [os.path.join(CSRC, h) for h in ("ptx.cuh", "kinds.cuh", "epilogue.cuh", "launch.cuh", "pipeline.cuh", "rowacc.cuh", "skinny.cuh")] + [
    os.path.join(HERE, "..", "include", "void_b200.h")]

HOST_FLAGS = ["-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-D_GLIBCXX_USE_CXX11_ABI=%d" % int(torch._C._GLIBCXX_USE_CXX11_ABI)]
HOST_LIBS = ["-ltorch_python", "-ltorch", "-ltorch_cuda", "-ltorch_cpu", "-lc10_cuda", "-lc10"]


def native_path():
    """Where the host path for this torch, this Python and these sources lies."""
    h = hashlib.sha256()
    for text in (torch.__version__, str(torch.version.git_version), str(sysconfig.get_config_var("SOABI")), *HOST_FLAGS, *HOST_LIBS):
        h.update(text.encode() + b"\0")
    for f in (HOST_SOURCE, HEADERS[-1]):
        with open(f, "rb") as src:
            h.update(src.read() + b"\0")
    return os.path.join(LIB_DIR, "_native_%s.so" % h.hexdigest()[:16])


NVCC_FLAGS = [
    "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
]


def _nvcc():
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found: the void_b200 CUDA library cannot be built")
    return exe


def have_nvcc():
    return bool(shutil.which("nvcc")) or os.path.exists("/usr/local/cuda/bin/nvcc")


def needs_build():
    if not (os.path.exists(LIB_PATH) and os.path.exists(native_path())):
        return True
    t = os.path.getmtime(LIB_PATH)
    deps = [os.path.join(CSRC, s) for s in SOURCES if os.path.exists(os.path.join(CSRC, s))] + HEADERS
    return any(os.path.getmtime(d) > t for d in deps)


def _host_compile(obj):
    """Command that compiles host.cpp against the headers of this Python and of the installed torch."""
    from torch.utils import cpp_extension
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    inc = cpp_extension.include_paths() + [sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
    return ["g++"] + HOST_FLAGS + [f for d in inc for f in ("-isystem", d)] + ["-c", HOST_SOURCE, "-o", obj]


def _host_link(obj):
    from torch.utils import cpp_extension
    dirs = cpp_extension.library_paths()
    return ["g++", "-shared", "-o", native_path(), obj, LIB_PATH] + [f for d in dirs for f in ("-L" + d, "-Wl,-rpath," + d)] \
        + ["-Wl,-rpath,$ORIGIN"] + HOST_LIBS


def _run_all(cmds, verbose):
    """Runs the commands side by side; raises with the output of the first that failed."""
    procs = [(c, subprocess.Popen(c, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)) for c in cmds]
    outs = [(c, p.communicate()[0], p.returncode) for c, p in procs]
    for c, out, rc in outs:
        if rc != 0:
            raise RuntimeError("%s failed:\n%s" % (" ".join(c[:1]), out))
        if verbose:
            print(out)


def build(force=False, verbose=False):
    """Compile every source (in parallel) and link both libraries; returns the C-ABI library's path."""
    if not force and not needs_build():
        return LIB_PATH
    os.makedirs(LIB_DIR, exist_ok=True)
    srcs = [s for s in SOURCES if os.path.exists(os.path.join(CSRC, s))]
    with tempfile.TemporaryDirectory() as tmp:
        objs = [os.path.join(tmp, s + ".o") for s in srcs]
        extra = ["-Xptxas", "-v"] if verbose else []
        host_obj = os.path.join(tmp, "host.o")
        _run_all([[_nvcc()] + NVCC_FLAGS + extra + ["-c", os.path.join(CSRC, s), "-o", o] for s, o in zip(srcs, objs)]
                 + [_host_compile(host_obj)], verbose)
        # (by name, so that the host path finds the library beside it, not the place where both were linked)
        _run_all([[_nvcc()] + NVCC_FLAGS + ["-shared", "-Xlinker", "-soname=" + os.path.basename(LIB_PATH), "-o", LIB_PATH] + objs], verbose)
        _run_all([_host_link(host_obj)], verbose)
    for f in os.listdir(LIB_DIR):    # host paths of earlier sources
        if f.startswith("_native") and f.endswith(".so") and f != os.path.basename(native_path()):
            os.remove(os.path.join(LIB_DIR, f))
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
