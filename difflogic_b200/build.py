"""In-tree build of the CUDA library (sm_100a only).

    python -m difflogic_b200.build [--verbose]

compiles difflogic_b200/csrc/*.cu with nvcc into difflogic_b200/_lib/libdifflogic_b200.so.
The library has a plain C ABI (include/difflogic_b200.h) and links the CUDA runtime statically,
so it depends on nothing but the driver.  The training path's autograd nodes (csrc/autograd_nodes.cpp) are a Python
module of their own beside it, _lib/dl_autograd-<PyTorch>-<Python>.so: host code that calls the library and links PyTorch.
"""
import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
LIB_DIR = os.path.join(HERE, "_lib")
LIB_PATH = os.path.join(LIB_DIR, "libdifflogic_b200.so")

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


def nodes_path():
    """Where the module of the autograd nodes is for the PyTorch and Python that run this.  It has the layouts of their objects
    compiled in, so that one built for another version is another file, which is neither taken for this one nor loaded."""
    import torch
    return os.path.join(LIB_DIR, "dl_autograd-%s-%s-%s.so" % (torch.__version__, (torch.version.git_version or "")[:8],
                                                             sysconfig.get_config_var("SOABI")))


def nodes_command():
    """Compiles and links the module of the autograd nodes against the library and the PyTorch that runs this."""
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(find_nvcc())))
    include = [os.path.join(ROOT, "include"), os.path.join(cuda, "include"), os.path.join(root, "include"),
               os.path.join(root, "include", "torch", "csrc", "api", "include"), sysconfig.get_paths()["include"]]
    return [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-ffunction-sections", "-fdata-sections",
            "-D_GLIBCXX_USE_CXX11_ABI=%d" % torch._C._GLIBCXX_USE_CXX11_ABI,
            *[flag for path in include for flag in ("-I", path)], os.path.join(CSRC, "autograd_nodes.cpp"), "-o", nodes_path(),
            "-L", os.path.join(root, "lib"), "-ltorch", "-ltorch_cpu", "-ltorch_python", "-lc10", "-lc10_cuda",
            "-L", LIB_DIR, "-l:" + os.path.basename(LIB_PATH), "-Wl,-rpath,$ORIGIN", "-Wl,--gc-sections"]


def _older_than_sources(path):
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC)] + [os.path.join(ROOT, "include", "difflogic_b200.h")]
    return not os.path.exists(path) or any(os.path.getmtime(d) > os.path.getmtime(path) for d in deps)


def is_stale():
    return _older_than_sources(LIB_PATH) or _older_than_sources(nodes_path())


def _run(cmd, what):
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        sys.stderr.write(r.stdout)
        raise RuntimeError(what + " failed")


def build(verbose=False, force=False):
    """Compiles the library and the module of the autograd nodes, each if it is missing or older than its sources; returns the
    library's path."""
    if force or _older_than_sources(LIB_PATH):
        _build_library(verbose)
    if force or _older_than_sources(nodes_path()):
        _run(nodes_command(), "g++")
    return LIB_PATH


def _build_library(verbose):
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
    _run(link, "link")


if __name__ == "__main__":
    print(build(verbose="--verbose" in sys.argv, force="--force" in sys.argv))
