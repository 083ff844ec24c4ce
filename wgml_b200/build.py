"""Builds libwgml_b200.so (sm_100a only) in-tree with nvcc, and the host module of the per-op calls with gcc.  Usage: python -m wgml_b200.build [-v]"""
from __future__ import annotations

import concurrent.futures as cf
import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "csrc", "build")
LIB = os.path.join(HERE, "libwgml_b200.so")
# CPython module, host path of the per-op calls (dispatch.c); named by the interpreter it is built for, whose C API it uses
EXT = os.path.join(HERE, "_dispatch" + sysconfig.get_config_var("EXT_SUFFIX"))

SOURCES = ["api.cpp", "gguf.cpp", "tokenizer.cpp", "quant.cu", "gemv.cu", "gemv_tc.cu", "attention.cu", "ops.cu", "sampler.cu", "prefill.cu", "prefill_q6k.cu", "prefill_q80.cu", "prefill_wide.cu", "llama2.cu", "gpt2.cu", "comm.cpp"]

ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
NVCC_FLAGS = ["-O3", "-std=c++17", "-lineinfo", "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC,-fvisibility=hidden",
              "-Xptxas", "-v" if os.environ.get("WGB_PTXAS_V") else "-warn-spills"]


def nvcc() -> str:
    path = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(path):
        raise RuntimeError("nvcc not found: the library has no other build route")
    return path


def _stale(target: str, deps: list[str]) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(OBJ, exist_ok=True)
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    headers.append(os.path.join(HERE, "..", "include", "wgml_b200.h"))
    headers.append(os.path.abspath(__file__))
    jobs = []
    objs = []
    for src in SOURCES:
        s = os.path.join(CSRC, src)
        o = os.path.join(OBJ, os.path.splitext(src)[0] + ".o")
        objs.append(o)
        if force or _stale(o, [s] + headers):
            cmd = [nvcc()] + ARCH + NVCC_FLAGS + ["-x", "cu", "-c", s, "-o", o]
            jobs.append(cmd)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        return cmd, r

    if jobs:
        with cf.ThreadPoolExecutor(max_workers=min(8, len(jobs))) as ex:
            for cmd, r in ex.map(run, jobs):
                if verbose or r.returncode != 0:
                    sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
                if r.returncode != 0:
                    raise RuntimeError("nvcc failed for " + cmd[-3])
    if jobs or force or _stale(LIB, objs):
        cmd = [nvcc(), "-shared", "-o", LIB] + objs + ["-lcudart", "-ldl"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if verbose or r.returncode != 0:
            sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
        if r.returncode != 0:
            raise RuntimeError("link failed")
    return LIB


def build_dispatch(force: bool = False, verbose: bool = False) -> str:
    """The module with the host path of the per-op calls (dispatch.c): a C compiler and Python's headers, no nvcc.  Apart from build():
    the library, the models and the C ABI do without it, and the per-op calls have the same path in Python."""
    src = os.path.join(CSRC, "dispatch.c")
    if force or _stale(EXT, [src, os.path.abspath(__file__)]):
        tmp = f"{EXT}.{os.getpid()}"   # renamed when whole: processes that start together load no half of it
        cmd = ["gcc", "-O2", "-Wall", "-shared", "-fPIC", "-I" + sysconfig.get_paths()["include"], src, "-o", tmp]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if verbose or r.returncode != 0:
            sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
        if r.returncode != 0:
            if os.path.exists(tmp):
                os.remove(tmp)
            raise RuntimeError("gcc failed for dispatch.c")
        os.replace(tmp, EXT)
    return EXT


if __name__ == "__main__":
    print(build(force="-f" in sys.argv, verbose="-v" in sys.argv))
    print(build_dispatch(force="-f" in sys.argv, verbose="-v" in sys.argv))
