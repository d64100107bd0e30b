"""Build libfsa_b200.so (sm_100a only) in-tree with nvcc, and the native launcher flash_sparse_attn/_host.so with g++.

Usage: ``python build.py [--force] [--verbose]``. The library has no dependency on libcuda at link
time (the one driver entry point it needs is resolved at run time), so it loads on machines without
a GPU; compute calls then fail with an error code.
"""

import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "libfsa_b200.so")
HOST_SRC = os.path.join(CSRC, "fsa_host.cpp")
HOST_LIB = os.path.join(HERE, "flash_sparse_attn", "_host.so")

SOURCES = [
    "fsa_api.cu",
    "fsa_aux.cu",
    "fsa_fwd_sm100.cu",
    "fsa_bwd_sm100.cu",
    "fsa_dec_sm100.cu",
    "fsa_static_scratch.cu",
    "fsa_quant.cu",
    "fsa_topk.cu",
    "fsa_kvcache.cu",
    "fsa_peer.cu",
]

NVCC_FLAGS = [
    "-gencode",
    "arch=compute_100a,code=sm_100a",
    "-O3",
    "-std=c++17",
    "-lineinfo",
    "-Xcompiler",
    "-fPIC",
    "-Xptxas",
    "-v",
    "--expt-relaxed-constexpr",
]


def _nvcc():
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    raise RuntimeError("nvcc not found")


def _newest_header():
    t = 0.0
    for root in (CSRC, os.path.join(HERE, "..", "include")):
        for f in os.listdir(root):
            if f.endswith((".h", ".cuh")):
                t = max(t, os.path.getmtime(os.path.join(root, f)))
    return t


def _compile(src, force, verbose):
    obj = os.path.join(OBJ, src.replace(".cu", ".o"))
    srcp = os.path.join(CSRC, src)
    if (
        not force
        and os.path.exists(obj)
        and os.path.getmtime(obj) >= max(os.path.getmtime(srcp), _newest_header())
    ):
        return obj, ""
    cmd = [_nvcc()] + NVCC_FLAGS + ["-c", srcp, "-o", obj]
    res = subprocess.run(cmd, capture_output=True, text=True)
    log = res.stdout + res.stderr
    if res.returncode != 0:
        raise RuntimeError(f"nvcc failed for {src}:\n{log}")
    with open(obj + ".log", "w") as f:
        f.write(log)
    if verbose:
        print(log)
    return obj, log


def build_host(force=False):
    """The native launcher: a CPython extension against the headers of the installed torch. It holds no device code
    and reaches the kernels through the addresses that the package hands it. Built again when its sources, the compile
    command, torch or the interpreter changed since (the key file beside the objects says what it was built with)."""
    import torch

    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(_nvcc())))
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}"]
    for inc in (sysconfig.get_paths()["include"], os.path.join(root, "include"),
                os.path.join(root, "include", "torch", "csrc", "api", "include"), os.path.join(cuda, "include")):
        cmd += ["-isystem", inc]
    cmd += [HOST_SRC, "-L" + os.path.join(root, "lib"), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch", "-ltorch_python"]
    key = "\n".join([torch.__version__, sys.version, *cmd])
    key_file = os.path.join(OBJ, "_host.key")
    header = os.path.join(HERE, "..", "include", "fsa_b200.h")
    newest = max(os.path.getmtime(HOST_SRC), os.path.getmtime(header))
    if not force and os.path.exists(HOST_LIB) and os.path.getmtime(HOST_LIB) >= newest and os.path.exists(key_file):
        with open(key_file) as f:
            if f.read() == key:
                return HOST_LIB
    part = HOST_LIB + ".part"
    res = subprocess.run(cmd + ["-o", part], capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("g++ failed for fsa_host.cpp:\n" + res.stdout + res.stderr)
    os.replace(part, HOST_LIB)
    os.makedirs(OBJ, exist_ok=True)
    with open(key_file, "w") as f:
        f.write(key)
    return HOST_LIB


def build(force=False, verbose=False):
    os.makedirs(OBJ, exist_ok=True)
    with ThreadPoolExecutor(max_workers=min(8, len(SOURCES))) as ex:
        results = list(ex.map(lambda s: _compile(s, force, verbose), SOURCES))
    objs = [o for o, _ in results]
    if (
        force
        or not os.path.exists(LIB)
        or any(os.path.getmtime(o) > os.path.getmtime(LIB) for o in objs)
    ):
        cmd = [_nvcc(), "-shared", "-o", LIB] + objs + ["-cudart", "static"]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError("link failed:\n" + res.stdout + res.stderr)
    build_host(force)  # last: the library needs neither torch nor its headers
    return LIB


if __name__ == "__main__":
    lib = build(force="--force" in sys.argv, verbose="--verbose" in sys.argv)
    print(lib)
