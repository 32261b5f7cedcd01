"""In-tree build of the CUDA library (sm_100a only).

    python -m difflogic_b200.build [--verbose]

compiles difflogic_b200/csrc/*.cu with nvcc into difflogic_b200/_lib/libdifflogic_b200.so.
The library has a plain C ABI (include/difflogic_b200.h) and links the CUDA runtime statically,
so it depends on nothing but the driver.  The training path's autograd nodes (csrc/autograd_nodes.cpp) are a Python
module of their own beside it, _lib/dl_autograd.so: host code that calls the library and links PyTorch.
"""
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
LIB_DIR = os.path.join(HERE, "_lib")
LIB_PATH = os.path.join(LIB_DIR, "libdifflogic_b200.so")
NODES_PATH = os.path.join(LIB_DIR, "dl_autograd.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
    "-cudart", "static",
]


def find_nvcc():
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; set NVCC or put it on PATH")


def sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def nodes_command():
    """Compiles and links the module of the autograd nodes against the library and the PyTorch that runs this."""
    import sysconfig
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(find_nvcc())))
    include = [os.path.join(ROOT, "include"), os.path.join(cuda, "include"), os.path.join(root, "include"),
               os.path.join(root, "include", "torch", "csrc", "api", "include"), sysconfig.get_paths()["include"]]
    return [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-ffunction-sections", "-fdata-sections",
            "-D_GLIBCXX_USE_CXX11_ABI=%d" % torch._C._GLIBCXX_USE_CXX11_ABI,
            *[flag for path in include for flag in ("-I", path)], os.path.join(CSRC, "autograd_nodes.cpp"), "-o", NODES_PATH,
            "-L", os.path.join(root, "lib"), "-ltorch", "-ltorch_cpu", "-ltorch_python", "-lc10", "-lc10_cuda",
            "-L", LIB_DIR, "-l:" + os.path.basename(LIB_PATH), "-Wl,-rpath,$ORIGIN", "-Wl,--gc-sections"]


def is_stale():
    if not (os.path.exists(LIB_PATH) and os.path.exists(NODES_PATH)):
        return True
    built = min(os.path.getmtime(LIB_PATH), os.path.getmtime(NODES_PATH))
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC)] + [os.path.join(ROOT, "include", "difflogic_b200.h")]
    return any(os.path.getmtime(d) > built for d in deps)


def build(verbose=False, force=False):
    """Compiles the library if it is missing or older than its sources; returns its path."""
    if not force and not is_stale():
        return LIB_PATH
    os.makedirs(LIB_DIR, exist_ok=True)
    nvcc = find_nvcc()
    objs = []
    procs = []
    for src in sources():
        obj = os.path.join(LIB_DIR, os.path.basename(src)[:-3] + ".o")
        cmd = [nvcc, *NVCC_FLAGS, "-I", os.path.join(ROOT, "include"), "-I", CSRC, "-c", src, "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas")
            cmd.insert(2, "-v")
        procs.append((cmd, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(obj)
    for cmd, p in procs:
        out, _ = p.communicate()
        if verbose or p.returncode != 0:
            sys.stderr.write(out)
        if p.returncode != 0:
            raise RuntimeError("nvcc failed: " + " ".join(cmd))
    link = [nvcc, "-shared", "-cudart", "static", "-gencode", "arch=compute_100a,code=sm_100a",
            "-Xcompiler", "-fPIC", "-o", LIB_PATH, *objs]
    for cmd, what in ((link, "link"), (nodes_command(), "g++")):
        r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
        if r.returncode != 0:
            sys.stderr.write(r.stdout)
            raise RuntimeError(what + " failed")
    return LIB_PATH


if __name__ == "__main__":
    print(build(verbose="--verbose" in sys.argv, force="--force" in sys.argv))
