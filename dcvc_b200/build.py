"""Build recipe for the native library libdcvc_b200.so (sm_100a only) and the Python entry points on top of it.

Compiles every .cu/.cpp under dcvc_b200/csrc with nvcc into one shared library placed next to
this file, so it ships with the source tree.  Objects are cached under dcvc_b200/_build and
rebuilt when a source or any header in csrc/ or include/ changes.  csrc/python/torch_calls.cpp, which
needs PyTorch's headers, becomes the extension module _torch_calls.so beside the library.
"""
import hashlib
import importlib.util
import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
INCLUDE = os.path.join(ROOT, "include")
BUILD = os.path.join(HERE, "_build")
LIB = os.path.join(HERE, "libdcvc_b200.so")
CALLS_SRC = os.path.join(CSRC, "python", "torch_calls.cpp")
CALLS = os.path.join(HERE, "_torch_calls.so")

NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
COMMON = ["-std=c++17", "-O3", "-lineinfo", "-Xcompiler", "-fPIC", "-Xcompiler", "-pthread",
          "-I" + CSRC, "-I" + INCLUDE]


def _sources():
    out = []
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cpp")):
            out.append(os.path.join(CSRC, name))
    return out


def _headers_digest():
    h = hashlib.sha1()
    for d in (CSRC, INCLUDE):
        for name in sorted(os.listdir(d)):
            if name.endswith((".h", ".cuh", ".hpp")):
                with open(os.path.join(d, name), "rb") as f:
                    h.update(name.encode())
                    h.update(f.read())
    return h.hexdigest()


def _compile(src, hdr_digest, verbose):
    with open(src, "rb") as f:
        key = hashlib.sha1(f.read() + hdr_digest.encode() + " ".join(COMMON + ARCH).encode()).hexdigest()[:16]
    obj = os.path.join(BUILD, os.path.basename(src) + "." + key + ".o")
    if os.path.exists(obj):
        return obj
    cmd = [NVCC] + ARCH + COMMON + ["-c", src, "-o", obj + ".tmp"]
    if src.endswith(".cpp"):
        cmd = [NVCC] + COMMON + ["-x", "c++", "-c", src, "-o", obj + ".tmp"]
    if verbose:
        print(" ".join(cmd), flush=True)
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"nvcc failed for {src}:\n{r.stdout}\n{r.stderr}")
    os.replace(obj + ".tmp", obj)
    return obj


def _build_calls(verbose):
    import torch
    torch_dir = os.path.dirname(importlib.util.find_spec("torch").origin)
    cuda = os.path.dirname(os.path.dirname(NVCC))
    flags = ["-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
             "-I" + INCLUDE, "-I" + sysconfig.get_paths()["include"], "-I" + os.path.join(torch_dir, "include"),
             "-I" + os.path.join(torch_dir, "include", "torch", "csrc", "api", "include"), "-I" + os.path.join(cuda, "include")]
    link = ["-L" + HERE, "-ldcvc_b200", "-Wl,-rpath,$ORIGIN", "-L" + os.path.join(torch_dir, "lib"), "-ltorch_python", "-ltorch",
            "-ltorch_cpu", "-lc10_cuda", "-lc10"]
    with open(CALLS_SRC, "rb") as f, open(os.path.join(INCLUDE, "dcvc_b200.h"), "rb") as h:
        text = f.read() + h.read()
    key = hashlib.sha1(text + " ".join(flags + link + [torch.__version__]).encode()).hexdigest()[:16]
    stamp = os.path.join(BUILD, "calls." + key)
    if os.path.exists(CALLS) and os.path.exists(stamp):
        return
    cmd = ["g++"] + flags + [CALLS_SRC, "-o", CALLS + ".tmp"] + link
    if verbose:
        print(" ".join(cmd), flush=True)
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"g++ failed for {CALLS_SRC}:\n{r.stdout}\n{r.stderr}")
    os.replace(CALLS + ".tmp", CALLS)
    for name in os.listdir(BUILD):
        if name.startswith("calls."):
            os.remove(os.path.join(BUILD, name))
    open(stamp, "w").close()


def build(verbose=False, jobs=None):
    lib = _build_lib(verbose, jobs)
    _build_calls(verbose)
    return lib


def _build_lib(verbose, jobs):
    os.makedirs(BUILD, exist_ok=True)
    digest = _headers_digest()
    srcs = _sources()
    jobs = jobs or min(len(srcs), os.cpu_count() or 4)
    with ThreadPoolExecutor(max_workers=jobs) as ex:
        objs = list(ex.map(lambda s: _compile(s, digest, verbose), srcs))
    link_flags = ["-shared", "-cudart", "static", "-lpthread"]
    link_key = hashlib.sha1(("".join(sorted(objs)) + " ".join(link_flags)).encode()).hexdigest()[:16]
    stamp = os.path.join(BUILD, "link." + link_key)
    if os.path.exists(LIB) and os.path.exists(stamp):
        return LIB
    cmd = [NVCC] + ARCH + ["-o", LIB + ".tmp"] + objs + link_flags
    if verbose:
        print(" ".join(cmd), flush=True)
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    os.replace(LIB + ".tmp", LIB)
    for name in os.listdir(BUILD):
        if name.startswith("link."):
            os.remove(os.path.join(BUILD, name))
    open(stamp, "w").close()
    return LIB


if __name__ == "__main__":
    print(build(verbose="-v" in sys.argv))
