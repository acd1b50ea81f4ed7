"""Ahead-of-time build of libb200q.so (sm_100a only, nvcc) and of the _native extension (g++).

The kernels are compiled here, in the source tree, not JIT-compiled at first use:
`python -m tilus_b200.build` (or `__graft_entry__.build()`) leaves
tilus_b200/libb200q.so and tilus_b200/_native.so next to the package.  nvcc cross-compiles
without a GPU.
"""
from __future__ import annotations

import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(CSRC, "_build")
LIB = os.path.join(HERE, "libb200q.so")
NATIVE = os.path.join(HERE, "_native.so")
NATIVE_STAMP = os.path.join(HERE, "_native.stamp")  # the interpreter and torch that NATIVE was built for
HEADER = os.path.join(os.path.dirname(HERE), "include", "b200q.h")
NPARTS = 8

# Extra -D definitions for experiments (e.g. B200Q_EXTRA_DEFS="-DB200Q_GPW=2") and an
# alternative output name (B200Q_LIB_NAME) so that several builds can sit side by side.
EXTRA_DEFS = os.environ.get("B200Q_EXTRA_DEFS", "").split()
if os.environ.get("B200Q_LIB_NAME"):
    LIB = os.path.join(HERE, os.environ["B200Q_LIB_NAME"])
    OBJ = OBJ + "_" + os.environ["B200Q_LIB_NAME"].replace(".", "_")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O3", "-lineinfo",
    "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    cand = os.environ.get("NVCC") or "/usr/local/cuda/bin/nvcc"
    return cand if os.path.exists(cand) else "nvcc"


def _jobs():
    jobs = []
    for part in range(NPARTS):
        jobs.append(("stream_kernel.cu", f"stream_part{part}.o", [f"-DB200Q_NPARTS={NPARTS}", f"-DB200Q_PART={part}"]))
    for part in range(NPARTS):
        jobs.append(("resident_kernel.cu", f"resident_part{part}.o", [f"-DB200Q_NPARTS={NPARTS}", f"-DB200Q_PART={part}"]))
    for part in range(NPARTS):
        jobs.append(("batch_kernel.cu", f"batch_part{part}.o", [f"-DB200Q_NPARTS={NPARTS}", f"-DB200Q_PART={part}"]))
    for part in range(NPARTS):
        jobs.append(("exact_kernel.cu", f"exact_part{part}.o", [f"-DB200Q_NPARTS={NPARTS}", f"-DB200Q_PART={part}"]))
    for part in range(NPARTS):
        jobs.append(("umma_kernel.cu", f"umma_part{part}.o", [f"-DB200Q_NPARTS={NPARTS}", f"-DB200Q_PART={part}"]))
    jobs.append(("dequant_kernel.cu", "dequant.o", []))
    jobs.append(("quantize_kernel.cu", "quantize.o", []))
    jobs.append(("cast_kernel.cu", "cast.o", []))
    jobs.append(("gather_kernel.cu", "gather.o", []))
    jobs.append(("fetch_kernel.cu", "fetch.o", []))
    jobs.append(("api.cu", "api.o", [f"-DB200Q_NPARTS={NPARTS}"]))
    return jobs


def build_native(force: bool = False) -> str:
    """The host path of QuantizedLinear (csrc/native.cpp) as a CPython extension against the installed torch."""
    import torch

    src = os.path.join(CSRC, "native.cpp")
    # what the binary fits: the interpreter's ABI, torch's C++ classes, the C ABI whose functions it calls by address
    stamp = f"{sysconfig.get_config_var('SOABI')} torch {torch.__version__} {os.path.dirname(torch.__file__)}"
    newest = max(os.path.getmtime(p) for p in (src, HEADER, os.path.abspath(__file__)))
    if (not force and os.path.exists(NATIVE) and os.path.getmtime(NATIVE) >= newest
            and os.path.exists(NATIVE_STAMP) and open(NATIVE_STAMP).read() == stamp):
        return NATIVE
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-w",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
           "-I" + os.path.join(root, "include"), "-I" + os.path.join(root, "include", "torch", "csrc", "api", "include"),
           "-I" + sysconfig.get_paths()["include"], "-I" + os.path.join(cuda, "include"), src, "-o", NATIVE,
           "-L" + os.path.join(root, "lib"), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"g++ failed for native.cpp:\n{r.stdout}\n{r.stderr}")
    with open(NATIVE_STAMP, "w") as f:
        f.write(stamp)
    return NATIVE


def _sources_mtime() -> float:
    paths = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh", ".h"))]
    paths.append(HEADER)
    paths.append(os.path.abspath(__file__))
    return max(os.path.getmtime(p) for p in paths)


def build(force: bool = False, verbose: bool = False, ptxas_info: bool = False) -> str:
    build_native(force)
    os.makedirs(OBJ, exist_ok=True)
    newest = _sources_mtime()
    if not force and os.path.exists(LIB) and os.path.getmtime(LIB) >= newest:
        return LIB
    nvcc = _nvcc()

    def compile_one(job):
        src, obj, defs = job
        out = os.path.join(OBJ, obj)
        if not force and os.path.exists(out) and os.path.getmtime(out) >= newest:
            return (obj, "")
        cmd = [nvcc, *NVCC_FLAGS, *EXTRA_DEFS, *defs, "-c", os.path.join(CSRC, src), "-o", out]
        if ptxas_info:
            cmd[1:1] = ["-Xptxas", "-v"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src} ({' '.join(defs)}):\n{r.stdout}\n{r.stderr}")
        return (obj, r.stderr)

    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as ex:
        results = list(ex.map(compile_one, _jobs()))
    if verbose or ptxas_info:
        for obj, log in results:
            if log.strip():
                print(f"--- {obj}\n{log}", file=sys.stderr)
    objs = [os.path.join(OBJ, j[1]) for j in _jobs()]
    cmd = [nvcc, "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a", "-cudart", "static"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True, ptxas_info="--ptxas" in sys.argv))
