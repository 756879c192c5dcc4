"""Builds libcactus_b200.so (the CUDA kernels behind the C ABI) in-tree with nvcc for sm_100a.

    python -m cactus_b200.build [--force] [--verbose]
"""
from __future__ import annotations

import os
import re
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUT = os.path.join(HERE, "lib")
LIB = os.path.join(OUT, "libcactus_b200.so")
HOST_LIB = os.path.join(OUT, "_ops_host.so")   # the Python-facing host path (needs torch's headers)
SOURCES = ["abi.cu", "quantize.cu", "mmvq.cu", "mmq.cu", "mmq_stream.cu", "mmq_tc.cu", "mul_mat.cu", "fattn.cu", "rowops.cu", "kvops.cu", "fused.cu", "peer.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC,-fvisibility=hidden", "--fmad=true",
] + os.environ.get("B200_NVCC_EXTRA", "").split()


def nvcc() -> str:
    for c in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if c and (os.path.isabs(c) and os.path.exists(c) or not os.path.isabs(c)):
            return c
    raise RuntimeError("nvcc not found")


def _stale(target: str, deps: list[str]) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(OUT, exist_ok=True)
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    headers.append(os.path.join(os.path.dirname(HERE), "include", "cactus_b200.h"))
    objs, jobs = [], []
    for s in SOURCES:
        src = os.path.join(CSRC, s)
        obj = os.path.join(OUT, s.replace(".cu", ".o"))
        objs.append(obj)
        if force or _stale(obj, [src] + headers):
            cmd = [nvcc(), *NVCC_FLAGS, "-c", src, "-o", obj]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
            jobs.append(cmd)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("nvcc failed:\n" + " ".join(cmd) + "\n" + r.stdout + r.stderr)
        return r.stderr

    with ThreadPoolExecutor(max_workers=8) as ex:
        for log in ex.map(run, jobs):
            if verbose and log:
                print(log)
    if jobs or force or _stale(LIB, objs):
        run([nvcc(), "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a", "-lcudart"])
    build_host(force)
    return LIB


def host_abi() -> str:
    """What _ops_host.so binds besides its own source: torch's C++ classes and the interpreter's C API."""
    import sysconfig

    import torch
    return f"torch {torch.__version__} cuda {torch.version.cuda} cxx11abi {int(torch._C._GLIBCXX_USE_CXX11_ABI)} python {sysconfig.get_config_var('EXT_SUFFIX')}"


def built_host_abi(path: str) -> str:
    """What the library at `path` was built against: a string that the build leaves in it (b200_host_abi)."""
    with open(path, "rb") as f:
        m = re.search(rb"b200_host_abi\{([^}\0]*)\}", f.read())
    return m.group(1).decode() if m else "an unknown torch"


def host_stale() -> bool:
    """Older than its source, or built against another torch (whose classes may be laid out differently)."""
    deps = [os.path.join(CSRC, "host", "ops_host.cpp"), os.path.join(os.path.dirname(HERE), "include", "cactus_b200.h")]
    return _stale(HOST_LIB, deps) or built_host_abi(HOST_LIB) != host_abi()


def build_host(force: bool = False) -> str:
    if force or host_stale():
        import sysconfig

        import torch
        from torch.utils.cpp_extension import include_paths
        src = os.path.join(CSRC, "host", "ops_host.cpp")
        tlib = os.path.join(os.path.dirname(torch.__file__), "lib")
        cuda = os.path.dirname(os.path.dirname(nvcc())) if os.path.isabs(nvcc()) else "/usr/local/cuda"
        cmd = ["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
               f'-DB200_HOST_ABI="{host_abi()}"',
               *[f"-I{p}" for p in (*include_paths(), sysconfig.get_paths()["include"], os.path.join(cuda, "include"))], src, "-o", HOST_LIB,
               f"-L{OUT}", "-lcactus_b200", f"-L{tlib}", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python", "-Wl,-rpath,$ORIGIN"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("g++ failed:\n" + " ".join(cmd) + "\n" + r.stdout + r.stderr)
    return HOST_LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
