"""Build the CUDA library of the package in place (sm_100a only).

    python -m dev_field_efvm_b200.build

produces dev_field_efvm_b200/libefvm_b200.so from csrc/*.cu with nvcc.  The CUDA
runtime is linked statically so the library does not depend on the runtime
version torch ships.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUT = os.path.join(HERE, "libefvm_b200.so")
BUILD = os.path.join(HERE, "_build")
SOURCES = ["efvm_kernels.cu", "efvm_tile.cu", "efvm_api.cu", "efvm_batch.cu", "efvm_nn.cu", "efvm_noalloc.cu"]
HEADERS = ["efvm_internal.h", "efvm_plan.h", "efvm_math.cuh", "efvm_device.cuh", "efvm_kernels3d.cuh", "efvm_tc.cuh", "efvm_tma.cuh", "../../include/efvm.h"]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-lineinfo", "-std=c++17",
    "-Xcompiler", "-fPIC,-ffp-contract=off,-fvisibility=hidden",
    "-Xptxas", "-v",
]


def nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", shutil.which("nvcc")):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found")


def _newer(target: str, deps) -> bool:
    if not os.path.exists(target):
        return False
    t = os.path.getmtime(target)
    return all(os.path.getmtime(d) <= t for d in deps)


def build(verbose: bool = False, force: bool = False) -> str:
    deps = [os.path.join(CSRC, s) for s in SOURCES] + [os.path.normpath(os.path.join(CSRC, h)) for h in HEADERS]
    if not force and _newer(OUT, deps):
        return OUT
    os.makedirs(BUILD, exist_ok=True)
    objs = [os.path.join(BUILD, src.replace(".cu", ".o")) for src in SOURCES]

    def compile_one(src, obj):
        cmd = [nvcc(), *NVCC_FLAGS, "-c", os.path.join(CSRC, src), "-o", obj]
        return subprocess.run(cmd, capture_output=True, text=True)

    with ThreadPoolExecutor() as pool:  # the files are independent
        done = list(pool.map(compile_one, SOURCES, objs))
    log = [r.stdout + r.stderr for r in done]
    for src, r in zip(SOURCES, done):
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src}:\n{r.stderr}")
    tmp = OUT + ".tmp"
    cmd = [nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-cudart", "static",
           "-Xcompiler", "-fPIC", *objs, "-o", tmp]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stderr}")
    os.replace(tmp, OUT)
    with open(os.path.join(BUILD, "ptxas.log"), "w") as f:
        f.write("\n".join(log))
    if verbose:
        print("\n".join(log))
    return OUT


if __name__ == "__main__":
    print(build(verbose="-v" in sys.argv, force="-f" in sys.argv))
