"""In-tree build of the x2dhf GB300 library (libx2dhf_gpu.so, sm_103a).

The CUDA sources under csrc/ are compiled with nvcc in parallel into one
shared library next to this file; no torch extension machinery is involved.
"""
import concurrent.futures as cf
import os
import shutil
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
BUILD = os.path.join(HERE, "_build")
LIB = os.path.join(HERE, "libx2dhf_gpu.so")
SOURCES = ["x2g_setup.cpp", "x2g_columns_plan.cpp", "x2g_tile_plan.cpp",
           "x2g_columns_a.cu", "x2g_columns_b.cu", "x2g_columns_c.cu",
           "x2g_columns_d.cu", "x2g_columns_e.cu", "x2g_columns_f.cu", "x2g_residual.cu",
           "x2g_kernels.cu", "x2g_capi.cu", "x2g_scf.cu", "x2g_compat.cu", "x2g_noalloc.cu"]
ARCH = ["-gencode", "arch=compute_103a,code=sm_103a"]


def nvcc():
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found")
    return exe


def _compile(src):
    obj = os.path.join(BUILD, os.path.splitext(src)[0] + ".o")
    path = os.path.join(CSRC, src)
    deps = [path] + [os.path.join(CSRC, h) for h in os.listdir(CSRC) if h.endswith((".h", ".cuh"))]
    deps.append(os.path.join(HERE, "..", "include", "x2dhf_gpu.h"))
    if os.path.exists(obj) and os.path.getmtime(obj) >= max(os.path.getmtime(d) for d in deps):
        return obj
    cmd = [nvcc(), "-c", "-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC,-O2,-ffp-contract=off",
           "-Xptxas", "-v" if os.environ.get("X2G_PTXAS_V") else "-O3"] + ARCH
    if src.endswith(".cpp"):
        cmd += ["-x", "cu"]
    cmd += [path, "-o", obj]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"nvcc failed for {src}:\n{r.stdout}\n{r.stderr}")
    if os.environ.get("X2G_PTXAS_V"):
        print(r.stderr)
    return obj


def build(force=False):
    os.makedirs(BUILD, exist_ok=True)
    if force:
        for f in os.listdir(BUILD):
            os.remove(os.path.join(BUILD, f))
    with cf.ThreadPoolExecutor(max_workers=len(SOURCES)) as ex:
        objs = list(ex.map(_compile, SOURCES))
    if not force and os.path.exists(LIB) and os.path.getmtime(LIB) >= max(os.path.getmtime(o) for o in objs):
        return LIB
    cmd = [nvcc(), "-shared", "-o", LIB] + objs + ARCH + ["-lcudart"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    return LIB


if __name__ == "__main__":
    print(build(force=True))
