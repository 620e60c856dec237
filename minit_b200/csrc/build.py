"""Ahead-of-time build of libminit_b200.so (sm_100a only) with nvcc.

    python minit_b200/csrc/build.py [--force]

(run as a script, or loaded by path: it must work while the library is missing or stale, so it
does not import the minit_b200 package, whose import binds the library's symbols)

Objects go to minit_b200/csrc/_obj/, the library to minit_b200/libminit_b200.so and the host-call extension (host.cc, built
with g++ against torch's headers) to minit_b200/_host<ABI tag>.so (in-tree, so they travel with the source tree; all are
git-ignored).  A source is recompiled when it or any header is newer than its object; the extension also when it was built
for another torch.
"""
from __future__ import annotations

import importlib.metadata
import importlib.util
import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

CSRC = os.path.dirname(os.path.abspath(__file__))
HERE = os.path.dirname(CSRC)
OBJ = os.path.join(CSRC, "_obj")
LIB = os.path.join(HERE, "libminit_b200.so")
HOST = os.path.join(HERE, "_host" + sysconfig.get_config_var("EXT_SUFFIX"))       # one Python's ABI, in its name
HOST_LOG = os.path.join(OBJ, "_host.torch")        # the torch that it was built for

NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC", "-Xptxas", "-v"]


def _nvcc() -> str:
    cand = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(cand):
        raise RuntimeError("nvcc not found: cannot build libminit_b200.so")
    return cand


def _units():
    units = [("dequant.cu", "dequant.o", []), ("api.cu", "api.o", []), ("qgemm_tc.cu", "qgemm_tc.o", []),
             ("qgemm_w8.cu", "qgemm_w8.o", []), ("qgemm_vec.cu", "qgemm_vec.o", []), ("repack.cu", "repack.o", []), ("qgemm_umma.cu", "qgemm_umma.o", []), ("qgemm_mid.cu", "qgemm_mid.o", []), ("qgemm_w8vec.cu", "qgemm_w8vec.o", []), ("decode_ops.cu", "decode_ops.o", []), ("attention.cu", "attention.o", []), ("noalloc.cu", "noalloc.o", []), ("nccl_shim.cc", "nccl_shim.o", [])]
    for bits in (4, 8):
        for bf in (0, 1):
            units.append(("qgemm_small_inst.cu", f"qgemm_small_i{bits}_{'bf16' if bf else 'f16'}.o",
                          [f"-DMT_INST_BITS={bits}", f"-DMT_INST_BF16={bf}"]))
    return [u for u in units if os.path.exists(os.path.join(CSRC, u[0]))]


def _headers_mtime() -> float:
    paths = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    paths.append(os.path.join(HERE, "..", "include", "minit_b200.h"))
    return max(os.path.getmtime(p) for p in paths)


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(OBJ, exist_ok=True)
    nvcc = _nvcc()
    hdr = _headers_mtime()
    jobs = []
    for src, obj, defs in _units():
        s, o = os.path.join(CSRC, src), os.path.join(OBJ, obj)
        if force or not os.path.exists(o) or os.path.getmtime(o) < max(os.path.getmtime(s), hdr):
            jobs.append((s, o, defs))

    def run(job):
        s, o, defs = job
        cmd = [nvcc, *NVCC_FLAGS, *defs, "-c", s, "-o", o]
        r = subprocess.run(cmd, capture_output=True, text=True)
        with open(o + ".log", "w") as f:
            f.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {s}:\n{r.stderr[-4000:]}")
        if verbose:
            print("compiled", os.path.basename(o))
        return o

    if jobs:
        with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as ex:
            list(ex.map(run, jobs))
    objs = [os.path.join(OBJ, u[1]) for u in _units()]
    if jobs or not os.path.exists(LIB) or any(os.path.getmtime(o) > os.path.getmtime(LIB) for o in objs):
        cmd = [nvcc, "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a", "-ldl"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("link failed:\n" + r.stderr[-4000:])
        if verbose:
            print("linked", LIB)
    _build_host(force, verbose)
    return LIB


def torch_version() -> str:
    return importlib.metadata.version("torch")


def host_command() -> list:
    torch_dir = os.path.dirname(importlib.util.find_spec("torch").origin)
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(_nvcc())))
    lib = os.path.join(torch_dir, "lib")
    return ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", os.path.join(CSRC, "host.cc"), "-o", HOST,
            f'-DMT_TORCH_VERSION="{torch_version()}"', "-I" + os.path.join(torch_dir, "include"),
            "-I" + os.path.join(torch_dir, "include", "torch", "csrc", "api", "include"), "-I" + os.path.join(cuda, "include"),
            "-I" + sysconfig.get_paths()["include"], "-L" + lib, "-lc10", "-lc10_cuda", "-ltorch", "-ltorch_cpu", "-ltorch_python",
            "-L" + HERE, "-l:libminit_b200.so", "-Wl,-rpath,$ORIGIN"]


def host_is_current() -> bool:
    deps = [os.path.join(CSRC, "host.cc"), os.path.join(HERE, "..", "include", "minit_b200.h"), os.path.abspath(__file__)]
    if not os.path.exists(HOST) or not os.path.exists(HOST_LOG) or os.path.getmtime(HOST) < max(os.path.getmtime(d) for d in deps):
        return False
    with open(HOST_LOG) as f:
        return f.read() == torch_version()


def _build_host(force: bool, verbose: bool) -> None:
    if not force and host_is_current():
        return
    cmd = host_command()
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("g++ failed for host.cc:\n" + r.stderr[-4000:])
    with open(HOST_LOG, "w") as f:
        f.write(torch_version())
    if verbose:
        print("compiled", HOST)


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
