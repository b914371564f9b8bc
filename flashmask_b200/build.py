"""Build libflashmask_b200.so in-tree with nvcc for sm_100a.

    python -m flashmask_b200.build [--force] [--verbose]

Every ``csrc/*.cu`` is compiled to an object under ``build/`` (in parallel,
skipped when the object is newer than all sources and headers) and linked into
``flashmask_b200/libflashmask_b200.so``.  The host C++ solver sources
(``csrc/*.cpp``) go through the same nvcc invocation.  ``csrc/torch/fm_torch.cpp``,
the native host path of the operator, is compiled against torch into
``flashmask_b200/_host.so`` and finds the library beside itself.
"""
from __future__ import annotations

import argparse
import concurrent.futures as cf
import glob
import os
import shutil
import subprocess
import sys

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(PKG, "csrc")
OUT = os.path.join(PKG, "libflashmask_b200.so")
HOST_SRC = os.path.join(CSRC, "torch", "fm_torch.cpp")
HOST_OUT = os.path.join(PKG, "_host.so")
OBJ = os.path.join(ROOT, "build", "obj")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
    "--expt-relaxed-constexpr", "-I", os.path.join(ROOT, "include"), "-I", CSRC,
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found (set NVCC=/path/to/nvcc)")


def _stale(obj: str, deps) -> bool:
    if not os.path.exists(obj):
        return True
    t = os.path.getmtime(obj)
    return any(os.path.getmtime(d) > t for d in deps)


def headers():
    """What an object depends on beside its own source: headers, sources that are included textually, this file."""
    return (glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(CSRC, "*.h")) +
            glob.glob(os.path.join(CSRC, "*.hpp")) + glob.glob(os.path.join(CSRC, "*.inc")) +
            glob.glob(os.path.join(ROOT, "include", "*.h")) + [os.path.abspath(__file__)])


def _host_command():
    """g++ invocation of the native host path (no device code, no pybind beyond torch's own)."""
    import sysconfig
    import torch
    from torch.utils import cpp_extension as ce
    lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    cmd = [shutil.which("g++") or "g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           "-DTORCH_API_INCLUDE_EXTENSION_H", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
    for d in ce.include_paths() + [sysconfig.get_paths()["include"], os.path.join(cuda, "include"),
                                   os.path.join(ROOT, "include")]:
        cmd += ["-isystem", d]
    return cmd + [HOST_SRC, "-o", HOST_OUT, f"-L{lib}", f"-L{PKG}", "-ltorch", "-ltorch_cpu", "-ltorch_python",
                  "-lc10", "-lc10_cuda", "-l:libflashmask_b200.so", "-Wl,-rpath,$ORIGIN"]


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(OBJ, exist_ok=True)
    srcs = sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cpp")))
    hdrs = headers()
    nvcc = _nvcc()
    jobs = []
    objs = []
    for s in srcs:
        o = os.path.join(OBJ, os.path.basename(s) + ".o")
        objs.append(o)
        if force or _stale(o, [s] + hdrs):
            cmd = [nvcc] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", s, "-o", o]
            if s.endswith(".cpp"):
                cmd.insert(1, "-x"); cmd.insert(2, "cu")
            jobs.append((s, cmd))

    def run(job):
        s, cmd = job
        r = subprocess.run(cmd, capture_output=True, text=True)
        return s, r

    if jobs:
        with cf.ThreadPoolExecutor(max_workers=min(8, len(jobs))) as ex:
            for s, r in ex.map(run, jobs):
                if verbose or r.returncode:
                    sys.stderr.write(f"--- {os.path.basename(s)}\n{r.stdout}{r.stderr}\n")
                if r.returncode:
                    raise RuntimeError(f"nvcc failed on {s}")
    if jobs or force or _stale(OUT, objs):
        cmd = [nvcc, "-shared", "-o", OUT] + objs + ["-gencode", "arch=compute_100a,code=sm_100a",
                                                      "-lcudart_static", "-lpthread", "-ldl", "-lrt"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("link failed")
    hdr = os.path.join(ROOT, "include", "flashmask_b200.h")
    if force or _stale(HOST_OUT, [HOST_SRC, hdr, os.path.abspath(__file__)]):
        r = subprocess.run(_host_command(), capture_output=True, text=True)
        if verbose or r.returncode:
            sys.stderr.write(r.stdout + r.stderr)
        if r.returncode:
            raise RuntimeError(f"g++ failed on {HOST_SRC}")
    return OUT


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(a.force, a.verbose))
