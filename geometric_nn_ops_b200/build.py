"""Build libtri_b200.so (nvcc, sm_100a) and the host extension _host.so (g++, torch's headers) in-tree.

Usage: ``python -m geometric_nn_ops_b200.build`` (or ``build_library()``).
Objects are cached by source mtime, so an unchanged tree rebuilds in no time.
"""

import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "libtri_b200.so")
HOST_SRC = os.path.join(CSRC, "torch_host.cpp")
HOST = os.path.join(HERE, "_host.so")
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr",
]


def _nvcc():
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    raise RuntimeError("nvcc not found")


def _stale(target, deps):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def _host_command():
    import sysconfig

    import torch
    from torch.utils.cpp_extension import include_paths, library_paths
    incs = [*include_paths(device_type="cuda"), sysconfig.get_paths()["include"]]
    libs = library_paths(device_type="cuda")
    return ["g++", "-shared", "-fPIC", "-O2", "-std=c++17", "-DTORCH_EXTENSION_NAME=_host", "-DTORCH_API_INCLUDE_EXTENSION_H",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}", *(f"-isystem{p}" for p in incs), HOST_SRC,
            "-o", HOST, *(f"-L{p}" for p in libs), *(f"-Wl,-rpath,{p}" for p in libs),
            "-lc10", "-lc10_cuda", "-ltorch", "-ltorch_cpu", "-ltorch_python", "-ldl"]


def build_library(verbose=False, force=False):
    os.makedirs(OBJ, exist_ok=True)
    sources = sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cuh")]
    headers.append(os.path.join(HERE, "..", "include", "tri_b200.h"))
    nvcc = _nvcc()
    jobs = []
    for src in sources:
        obj = os.path.join(OBJ, src[:-3] + ".o")
        if force or _stale(obj, [os.path.join(CSRC, src), *headers]):
            cmd = [nvcc, *NVCC_FLAGS, "-c", os.path.join(CSRC, src), "-o", obj]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
            jobs.append(cmd)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("compiler failed:\n" + " ".join(cmd) + "\n" + r.stdout + r.stderr)
        return r.stderr

    host_jobs = [_host_command()] if force or _stale(HOST, [HOST_SRC, headers[-1]]) else []
    with ThreadPoolExecutor(max_workers=min(8, max(1, len(jobs) + len(host_jobs)))) as ex:
        logs = list(ex.map(run, host_jobs + jobs))   # the host extension takes longest
    if verbose:
        print("\n".join(logs))
    objs = [os.path.join(OBJ, s[:-3] + ".o") for s in sources]
    if force or jobs or _stale(LIB, objs):
        run([nvcc, "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a"])
    return LIB


if __name__ == "__main__":
    print(build_library(verbose="-v" in sys.argv, force="-f" in sys.argv))
