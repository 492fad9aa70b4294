"""Builds libbitween_b200.so in-tree with nvcc for sm_100a (no JIT cache, no torch headers).

Beside it lands _host_forward, the native host side of the layer's forward (g++, torch's headers and libraries).  It
saves host time only: where it cannot be built, that is reported and the layers go without it.

Run as `python -m bitween_b200.csrc.build` or call build(); the library lands in
bitween_b200/_C/ next to the Python package so that it travels with the source tree.
"""
import concurrent.futures
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.dirname(HERE)
ROOT = os.path.dirname(PKG)
OUT_DIR = os.path.join(PKG, "_C")
OBJ_DIR = os.path.join(HERE, "build")
LIB = os.path.join(OUT_DIR, "libbitween_b200.so")

SOURCES = ["api.cu", "rtn_quantize.cu", "dequantize.cu", "qmatmul_smallm.cu", "qmatmul_rows.cu", "qmatmul_decode.cu", "qmatmul_tc.cu", "qmatmul_grad_input.cu", "fake_quant.cu", "peer_allreduce.cu"]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
    "-I", os.path.join(ROOT, "include"), "-I", HERE,
]
# BITWEEN_B200_TUNING=1 adds the experiment switches (bw_debug_*); the shipped build has none.
if os.environ.get("BITWEEN_B200_TUNING") == "1":
    NVCC_FLAGS.append("-DBW_TUNING")


def _nvcc():
    cand = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(cand):
        raise RuntimeError("nvcc not found; the CUDA extension cannot be built")
    return cand


def _stale(target, deps):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build_host(force=False, verbose=False):
    import sysconfig

    import torch
    from torch.utils import cpp_extension

    from ..kernels._lib import HOST_LIB_PATH as lib
    src = os.path.join(HERE, "host_forward.cpp")
    if not force and not _stale(lib, [src, os.path.join(ROOT, "include", "bitween_b200.h"), torch.__file__]):
        return
    os.makedirs(OUT_DIR, exist_ok=True)
    if os.path.exists(lib):
        os.remove(lib)                                   # (an outdated one is not left to be loaded)
    part = f"{lib}.{os.getpid()}"                        # (other processes load whole files only)
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(_nvcc())))
    includes = [os.path.join(ROOT, "include"), os.path.join(cuda, "include"), sysconfig.get_paths()["include"]] + cpp_extension.include_paths()
    libs = os.path.join(os.path.dirname(torch.__file__), "lib")
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"] + \
        [f"-I{d}" for d in includes] + [src, "-o", part, f"-L{libs}", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python",
                                               "-L" + os.path.join(cuda, "lib64"), "-lcudart"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or r.returncode != 0:
        sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
    if r.returncode != 0:
        raise RuntimeError("g++ failed for host_forward.cpp")
    os.replace(part, lib)


def build(force=False, verbose=False, ptxas_info=False):
    os.makedirs(OUT_DIR, exist_ok=True)
    os.makedirs(OBJ_DIR, exist_ok=True)
    headers = [os.path.join(HERE, f) for f in os.listdir(HERE) if f.endswith((".cuh", ".h"))]
    headers.append(os.path.join(ROOT, "include", "bitween_b200.h"))
    nvcc = _nvcc()
    jobs = []
    objs = []
    for src in SOURCES:
        s = os.path.join(HERE, src)
        o = os.path.join(OBJ_DIR, src.replace(".cu", ".o"))
        objs.append(o)
        if force or _stale(o, [s] + headers):
            cmd = [nvcc] + NVCC_FLAGS + (["-Xptxas", "-v"] if ptxas_info else []) + ["-c", s, "-o", o]
            jobs.append(cmd)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        return cmd, r

    host = concurrent.futures.ThreadPoolExecutor(max_workers=1).submit(build_host, force, verbose)
    if jobs:
        with concurrent.futures.ThreadPoolExecutor(max_workers=min(len(jobs), os.cpu_count() or 4)) as ex:
            for cmd, r in ex.map(run, jobs):
                if verbose or ptxas_info or r.returncode != 0:
                    sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
                if r.returncode != 0:
                    raise RuntimeError(f"nvcc failed for {cmd[-3]}")
    if jobs or _stale(LIB, objs):
        cmd = [nvcc, "-shared", "-o", LIB] + objs + ["-gencode", "arch=compute_100a,code=sm_100a",
                                                     "-lcudart_static" if False else "-lcudart"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("link failed")
    try:
        host.result()
    except Exception as e:  # noqa: BLE001
        sys.stderr.write(f"bitween_b200: the host side of the forward was not built ({e}); the layers run without it\n")
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv, ptxas_info="--ptxas" in sys.argv))
