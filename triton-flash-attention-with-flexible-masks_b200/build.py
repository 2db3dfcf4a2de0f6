"""Builds the CUDA library in-tree: csrc/*.cu -> flash_b200/libfa_b200.so (sm_100a only), and the native part of its
torch binding on top of it: csrc/host.cpp -> flash_b200/_host.so.

Usage: python build.py [--force] [--library]. With --library, and where torch is not installed, the CUDA library alone is
built: it is all that users of the C ABI need, and links and includes nothing of torch's or Python's. nvcc cross-compiles without a GPU. The runtime is linked
statically and the driver API is resolved at run time, so the library loads on a machine
without a CUDA driver (its entry points then return an error instead of computing).
"""
import concurrent.futures
import importlib.util
import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUT = os.path.join(HERE, "flash_b200", "libfa_b200.so")
HOST_OUT = os.path.join(HERE, "flash_b200", "_host.so")
OBJ_DIR = os.path.join(HERE, "build")
HOST_TAG = os.path.join(OBJ_DIR, "host.tag")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xptxas", "-v",
]


def _sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def _deps():
    hdrs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cuh")]
    hdrs.append(os.path.join(HERE, "..", "include", "fa_b200.h"))
    return hdrs


def _stale(target, srcs):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(s) > t for s in srcs)


def _compile(src):
    obj = os.path.join(OBJ_DIR, os.path.basename(src)[:-3] + ".o")
    if not _stale(obj, [src] + _deps()):
        return obj, ""
    r = subprocess.run([NVCC, *FLAGS, "-c", src, "-o", obj], capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"nvcc failed on {src}:\n{r.stdout}\n{r.stderr}")
    return obj, r.stderr


def build(force=False, verbose=False, host=True):
    os.makedirs(OBJ_DIR, exist_ok=True)
    srcs = _sources()
    if force:
        for f in os.listdir(OBJ_DIR):
            if f.endswith(".o"):
                os.remove(os.path.join(OBJ_DIR, f))
    with concurrent.futures.ThreadPoolExecutor(max_workers=min(8, len(srcs))) as ex:
        results = list(ex.map(_compile, srcs))
    objs = [o for o, _ in results]
    if verbose:
        for _, log in results:
            for line in log.splitlines():
                if "registers" in line or "spill" in line or "Compiling entry" in line:
                    print(line)
    if force or _stale(OUT, objs):
        r = subprocess.run([NVCC, "-shared", "-o", OUT, *objs, "-gencode", "arch=compute_100a,code=sm_100a"],
                           capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    if host and importlib.util.find_spec("torch") is not None:
        _build_host(force)
    return OUT


def _cuda_include():
    """The toolkit's headers, beside the nvcc that NVCC names, by a path or by a name on PATH."""
    nvcc = os.path.realpath(shutil.which(NVCC) or NVCC)
    return os.path.join(os.path.dirname(os.path.dirname(nvcc)), "include")


def _host_tag():
    """What the host module is bound to besides its sources: this Python and the C++ interface of this torch."""
    import torch
    return f"{sysconfig.get_config_var('SOABI')} torch {torch.__version__} abi {int(torch._C._GLIBCXX_USE_CXX11_ABI)}\n"


def _host_stale():
    if _stale(HOST_OUT, [os.path.join(CSRC, "host.cpp"), OUT] + _deps()) or not os.path.exists(HOST_TAG):
        return True
    with open(HOST_TAG) as f:
        return f.read() != _host_tag()


def _build_host(force):
    if not force and not _host_stale():
        return
    import torch
    src = os.path.join(CSRC, "host.cpp")
    root = os.path.dirname(torch.__file__)
    include = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"), _cuda_include(),
               sysconfig.get_paths()["include"]]
    part = f"{HOST_OUT}.{os.getpid()}"  # moved into place when it is whole: another process may be loading the module
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", src, "-o", part, *("-I" + i for i in include),
                        f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
                        "-L" + os.path.join(root, "lib"), "-ltorch_python", "-ltorch_cpu", "-lc10", "-lc10_cuda",
                        "-L" + os.path.dirname(OUT), "-l:" + os.path.basename(OUT), "-Wl,-rpath,$ORIGIN"],
                       capture_output=True, text=True)
    if r.returncode != 0:
        if os.path.exists(part):
            os.remove(part)
        raise RuntimeError(f"g++ failed on {src}:\n{r.stdout}\n{r.stderr}")
    os.replace(part, HOST_OUT)
    with open(HOST_TAG, "w") as f:
        f.write(_host_tag())


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True, host="--library" not in sys.argv))
