"""Build the C-ABI shared library (sm_100a only) and the native wrapper module in-tree.

    python -m hexa_moe_b200.build            # builds hexa_moe_b200/libhexa_moe_b200.so and hexa_moe_b200/_host.so

nvcc cross-compiles without a GPU.  The library links the CUDA runtime statically-by-default
shared object (cudart) and resolves the one driver entry point it needs
(cuTensorMapEncodeTiled) at run time, so it does not link libcuda.  The wrapper module is a CPython extension over
torch's C++ API (g++, no device code); it finds the library's functions at run time.
"""
import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libhexa_moe_b200.so")
HOST = os.path.join(HERE, "_host.so")
SOURCES = ["route.cu", "rows.cu", "gemm_simt.cu", "gemm_tc.cu", "gemm_f32.cu", "ops_api.cu", "peer.cu", "gate.cu"]


def _nvcc():
    nv = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nv):
        raise RuntimeError("nvcc not found; the CUDA toolkit is required to build hexa_moe_b200")
    return nv


def _host_command():
    import torch
    root = os.path.dirname(os.path.abspath(torch.__file__))
    cuda = os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "include")
    include = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
               sysconfig.get_paths()["include"], cuda]
    cmd = [shutil.which("g++") or "g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
    for d in include:
        cmd += ["-isystem", d]
    lib = os.path.join(root, "lib")
    return cmd + [os.path.join(CSRC, "host.cpp"), "-o", HOST, "-L" + lib, "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch", "-ltorch_python"]


def needs_build():
    if not os.path.exists(LIB) or not os.path.exists(HOST):
        return True
    t = min(os.path.getmtime(LIB), os.path.getmtime(HOST))
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC)] + [os.path.join(HERE, "..", "include", "hexa_moe_b200.h")]
    return any(os.path.getmtime(d) > t for d in deps)


def build(force=False, verbose=False):
    if not force and not needs_build():
        return LIB
    objdir = os.path.join(HERE, "build")
    os.makedirs(objdir, exist_ok=True)
    flags = ["-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC"]
    if verbose:
        flags += ["-Xptxas", "-v"]
    objs = []
    procs = [("host.cpp", subprocess.Popen(_host_command(), stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True))]
    for src in SOURCES:
        obj = os.path.join(objdir, src.replace(".cu", ".o"))
        objs.append(obj)
        procs.append((src, subprocess.Popen([_nvcc(), *flags, "-c", os.path.join(CSRC, src), "-o", obj],
                                            stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    for src, p in procs:
        out, _ = p.communicate()
        if verbose or p.returncode:
            sys.stderr.write(out)
        if p.returncode:
            raise RuntimeError(f"compiling {src} failed")
    subprocess.check_call([_nvcc(), "-shared", "-o", LIB, *objs, "-cudart", "shared"])
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
