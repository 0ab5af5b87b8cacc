"""Builds k2_b200/libk2b200.so from k2_b200/csrc/*.cu with nvcc for sm_100a, and
k2_b200/_host.so, the torch side of the host layer, from k2_b200/csrc/host/*.cc.

Both are built in-tree (next to this file) so that they travel with a snapshot of the
repository; nothing is JIT-compiled at import time.
"""
import glob
import os
import shutil
import subprocess
import sys
import sysconfig

_HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(_HERE, "csrc")
LIB_PATH = os.path.join(_HERE, "libk2b200.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-ccbin", "/usr/bin/g++", "-Xcompiler", "-fPIC",
    # no FMA contraction: sums that decide which states / arcs survive pruning
    # must be plain IEEE additions in the reference's order
    "-fmad=false",
]


def sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def _stale() -> bool:
    if not os.path.exists(LIB_PATH):
        return True
    t = os.path.getmtime(LIB_PATH)
    deps = sources() + glob.glob(os.path.join(CSRC, "*.cuh")) + \
        [os.path.join(_HERE, "..", "include", "k2b200.h"), os.path.abspath(__file__)]
    return any(os.path.getmtime(d) > t for d in deps)


HOST_PATH = os.path.join(_HERE, "_host.so")
HOST_SOURCE = os.path.join(CSRC, "host", "torch_host.cc")


# what _host.so was built for: it works with that Python and that torch only
HOST_KEY_PATH = os.path.join(_HERE, "_host.built_for")


def _host_key(command) -> str:
    import torch
    return "\n".join([sys.version, torch.__version__] + command) + "\n"


def _host_stale(command) -> bool:
    if not (os.path.exists(HOST_PATH) and os.path.exists(HOST_KEY_PATH)):
        return True
    with open(HOST_KEY_PATH) as f:
        if f.read() != _host_key(command):
            return True
    t = os.path.getmtime(HOST_PATH)
    deps = glob.glob(os.path.join(CSRC, "host", "*")) + \
        [os.path.join(_HERE, "..", "include", "k2b200.h"), os.path.abspath(__file__)]
    return any(os.path.getmtime(d) > t for d in deps)


def _host_command():
    """The C++ compiler on the one translation unit that includes torch's headers;
    libk2b200.so is found next to it, torch's libraries are loaded by `import torch`."""
    import torch
    torch_dir = os.path.dirname(torch.__file__)
    cuda = os.path.join(os.path.dirname(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")), "..")
    inc = os.path.join(torch_dir, "include")
    return [os.environ.get("CXX") or shutil.which("g++") or "c++", "-O2", "-std=c++17", "-fPIC",
            "-shared", "-fvisibility=hidden",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            "-DTORCH_EXTENSION_NAME=_host",
            "-isystem", inc, "-isystem", os.path.join(inc, "torch", "csrc", "api", "include"),
            "-isystem", os.path.join(cuda, "include"),
            "-isystem", sysconfig.get_paths()["include"], HOST_SOURCE, "-o", HOST_PATH,
            "-L" + _HERE, "-l:libk2b200.so", "-Wl,-rpath,$ORIGIN",
            "-L" + os.path.join(torch_dir, "lib"), "-lc10", "-lc10_cuda", "-ltorch_cpu",
            "-ltorch_cuda", "-ltorch", "-ltorch_python"]


def build(force: bool = False, verbose: bool = False) -> str:
    _build_library(force, verbose)
    command = _host_command()
    if force or _host_stale(command):
        subprocess.check_call(command)
        with open(HOST_KEY_PATH, "w") as f:
            f.write(_host_key(command))
    return LIB_PATH


def _build_library(force: bool, verbose: bool) -> str:
    if not force and not _stale():
        return LIB_PATH
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    objs = []
    procs = []
    for src in sources():
        obj = os.path.splitext(src)[0] + ".o"
        objs.append(obj)
        cmd = [nvcc] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", src, "-o", obj]
        procs.append((cmd, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT)))
    for cmd, p in procs:
        out, _ = p.communicate()
        if verbose or p.returncode != 0:
            sys.stderr.write(out.decode(errors="replace"))
        if p.returncode != 0:
            raise RuntimeError("nvcc failed: " + " ".join(cmd))
    subprocess.check_call([nvcc, "-shared", "-o", LIB_PATH] + objs +
                          ["-ccbin", "/usr/bin/g++", "-gencode", "arch=compute_100a,code=sm_100a",
                           "-ldl"])
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
