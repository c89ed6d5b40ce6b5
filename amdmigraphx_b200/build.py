"""In-tree build of the native libraries.

  lib/libmgx_cuda_kernels.so  - sm_100a kernels behind the C ABI of include/mgx_cuda.h
                                (nvcc, cross-compiles without a GPU)
  lib/mgx_torch_ops.so        - the torch-tensor wrappers capi.py calls (C++ against torch's headers)
  lib/libmigraphx_cuda.so     - the MIGraphX `cuda` target plug-in (C++17 host code
                                compiled against the MIGraphX headers and linked to
                                libmigraphx.so); built only when those are available.

Run:  python -m amdmigraphx_b200.build [--verbose] [--force]
"""
import argparse
import concurrent.futures as cf
import os
import shutil
import subprocess
import sys
import sysconfig

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(PKG, "csrc")
LIB = os.path.join(PKG, "lib")
OBJ = os.path.join(PKG, "build")

KERNEL_SOURCES = ["runtime.cu", "quantize.cu", "qgemm.cu", "qgemm_split.cu", "qgemv.cu", "pointwise.cu", "reduce.cu", "layernorm.cu", "attention.cu", "kvcache.cu", "gqa_decode.cu", "gather.cu", "w4a16.cu", "w4a16_stream.cu", "w4a16_tc.cu", "w4a16_prefill.cu", "comm.cu"]
# qgemm_form.cu is compiled once for every form of the kernel: operand type, kind of tile, its columns
QGEMM_FORMS = [(t, k, bn) for t in ("i8", "f8", "f16")
               for k, widths in (("one", (64, 128, 256)), ("pair", (128, 192, 224, 256)), ("split", (64,))) for bn in widths]
KERNEL_LIB = os.path.join(LIB, "libmgx_cuda_kernels.so")
TORCH_OPS = os.path.join(LIB, "mgx_torch_ops.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
]


def nvcc_path():
    p = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(p):
        raise RuntimeError("nvcc not found: the CUDA kernels cannot be built")
    return p


def _newer(target, deps):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps if os.path.exists(d))


def _headers():
    hs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h", ".hpp"))]
    hs.append(os.path.join(ROOT, "include", "mgx_cuda.h"))
    return hs


def _jobs():
    """(source, object, definitions) of the kernel library, the longest to compile first."""
    forms = sorted(QGEMM_FORMS, key=lambda f: (f[1] == "one", -f[2]))
    jobs = [(os.path.join(CSRC, "qgemm_form.cu"), os.path.join(OBJ, f"qgemm_{t}_{k}_{bn}.o"),
             [f"-DMGX_FORM={t}_{k}_{bn}", f"-DMGX_FORM_TYPE={('i8', 'f8', 'f16').index(t)}",
              f"-DMGX_FORM_KIND=QGEMM_{k.upper()}", f"-DMGX_FORM_BN={bn}"]) for t, k, bn in forms]
    return jobs + [(os.path.join(CSRC, s), os.path.join(OBJ, s[:-3] + ".o"), []) for s in KERNEL_SOURCES]


def _compile(args):
    src, obj, defines, verbose, force = args
    if not force and not _newer(obj, [src] + _headers()):
        return src, 0, ""
    cmd = [nvcc_path(), "-c", src, "-o", obj] + defines + NVCC_FLAGS
    if verbose:
        cmd += ["-Xptxas", "-v"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    return src, r.returncode, (r.stdout + r.stderr)


def build_kernels(verbose=False, force=False):
    os.makedirs(LIB, exist_ok=True)
    os.makedirs(OBJ, exist_ok=True)
    jobs = [j + (verbose, force) for j in _jobs()]
    with cf.ThreadPoolExecutor(2 * (os.cpu_count() or 8)) as ex:
        for src, rc, out in ex.map(_compile, jobs):
            if verbose and out:
                print(out)
            if rc != 0:
                raise RuntimeError(f"nvcc failed for {src}:\n{out}")
    objs = [j[1] for j in jobs]
    if force or _newer(KERNEL_LIB, objs):
        cmd = [nvcc_path(), "-shared", "-o", KERNEL_LIB] + objs + [
            "-gencode", "arch=compute_100a,code=sm_100a", "-cudart", "static", "-ldl"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}{r.stderr}")
    return KERNEL_LIB


def build_torch_ops(force=False):
    """csrc/torch_ops.cpp against the installed torch, linked to the kernel library beside it."""
    import torch
    src = os.path.join(CSRC, "torch_ops.cpp")
    if not force and not _newer(TORCH_OPS, [src, os.path.join(ROOT, "include", "mgx_cuda.h"), torch.__file__]):
        return TORCH_OPS
    base = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(nvcc_path())))
    cmd = ["g++", "-O2", "-std=c++20", "-shared", "-fPIC", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           "-isystem", os.path.join(base, "include"),
           "-isystem", os.path.join(base, "include", "torch", "csrc", "api", "include"),
           "-isystem", os.path.join(cuda, "include"), "-isystem", sysconfig.get_paths()["include"], src, "-o", TORCH_OPS,
           "-L" + os.path.join(base, "lib"), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python",
           "-L" + LIB, "-lmgx_cuda_kernels", "-Wl,-rpath,$ORIGIN"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"building {TORCH_OPS} failed:\n{r.stdout}{r.stderr}")
    return TORCH_OPS


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--verbose", action="store_true")
    ap.add_argument("--force", action="store_true")
    a = ap.parse_args()
    print(build_kernels(a.verbose, a.force))
    print(build_torch_ops(a.force))
    try:
        from . import build_target
    except ImportError:
        build_target = None
    if build_target is not None:
        print(build_target.build_target(verbose=a.verbose, force=a.force))
    return 0


if __name__ == "__main__":
    sys.exit(main())
