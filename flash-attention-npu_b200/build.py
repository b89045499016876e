"""Builds libfa_b200.so (the C-ABI library, nvcc for sm_100a) and flash_b200/_native.so (the libtorch / CPython host path
above it, host compiler) in-tree.

    python flash-attention-npu_b200/build.py [--force]

Each .cu under csrc/ is compiled to an object in csrc/_obj/ (in parallel) and linked into
flash-attention-npu_b200/libfa_b200.so.  Objects are rebuilt when any source or header is newer.
"""
import concurrent.futures
import glob
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(CSRC, "_obj")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")
LIB = os.path.join(HERE, "libfa_b200.so")
NATIVE_SRC = os.path.join(CSRC, "torch_binding.cpp")
NATIVE = os.path.join(HERE, "flash_b200", "_native.so")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "--use_fast_math",
         "-Xcompiler", "-fPIC", "-I", INCLUDE, "-I", CSRC] + os.environ.get("FA_B200_NVCC_FLAGS", "").split()


def _newest(paths):
    return max(os.path.getmtime(p) for p in paths)


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(OBJ, exist_ok=True)
    sources = sorted(glob.glob(os.path.join(CSRC, "*.cu")))
    headers = glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(CSRC, "*.inc")) + \
        glob.glob(os.path.join(INCLUDE, "*.h"))
    dep_time = _newest(headers + [os.path.abspath(__file__)])
    jobs = []
    objs = []
    for src in sources:
        obj = os.path.join(OBJ, os.path.basename(src)[:-3] + ".o")
        objs.append(obj)
        if force or not os.path.exists(obj) or os.path.getmtime(obj) < max(dep_time, os.path.getmtime(src)):
            jobs.append((src, obj))

    def compile_one(job):
        src, obj = job
        cmd = [NVCC] + FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", src, "-o", obj]
        r = subprocess.run(cmd, capture_output=True, text=True)
        return src, r.returncode, r.stdout + r.stderr

    if jobs:
        with concurrent.futures.ThreadPoolExecutor(max_workers=min(8, len(jobs))) as ex:
            for src, rc, log in ex.map(compile_one, jobs):
                if verbose or rc != 0:
                    sys.stderr.write(log)
                if rc != 0:
                    raise RuntimeError(f"nvcc failed on {src}")
    if jobs or not os.path.exists(LIB):
        cmd = [NVCC, "-shared", "-o", LIB] + objs + ["-lcudart"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("link failed")
    build_native(force)
    return LIB


def build_native(force: bool = False) -> None:
    if not force and os.path.exists(NATIVE) and os.path.getmtime(NATIVE) >= max(
            os.path.getmtime(p) for p in (NATIVE_SRC, os.path.join(INCLUDE, "fa_b200.h"), os.path.abspath(__file__))):
        return
    import sysconfig

    import torch
    from torch.utils import cpp_extension
    libs = os.path.join(os.path.dirname(torch.__file__), "lib")
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-o", NATIVE, NATIVE_SRC, "-I", INCLUDE,
           "-I", sysconfig.get_path("include"), f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
    for path in cpp_extension.include_paths(device_type="cuda"):
        cmd += ["-isystem", path]
    cmd += ["-L", HERE, "-lfa_b200", "-Wl,-rpath,$ORIGIN/..", "-L", libs, "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda",
            "-ltorch", "-ltorch_python"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        sys.stderr.write(r.stdout + r.stderr)
        raise RuntimeError(f"host compiler failed on {NATIVE_SRC}")


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
