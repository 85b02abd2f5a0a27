"""Builds the native libraries of the package in-tree with nvcc for sm_100a.

    python -m litert_b200.build            # kernels + C ABI (+ delegate when the LiteRT headers are found)

Outputs go to litert_b200/lib/. Cross-compiles without a GPU.
"""
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "lib")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
COMMON = ["-lineinfo", "-O3", "-std=c++17", "-Xcompiler", "-fPIC,-fvisibility=hidden"]
COMMON += os.environ.get("B200_NVCC_FLAGS", "").split()  # e.g. -DB200_UMMA_KB=108 (shared-memory budget of a GEMV CTA)

KERNEL_SOURCES = ["pack.cu", "fc_umma.cu", "fc_w4_umma.cu", "fc_w4_gemv.cu", "sdpa_decode.cu", "sdpa_split.cu", "decoder_kernels.cu", "decoder.cu", "shim.cu", "sdpa_static.cu", "glue_abi.cu", "peak_probe.cu", "elementwise.cu"]


def _newer(target, deps):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps if os.path.exists(d))


def _all_deps():
    deps = []
    for root in (CSRC, os.path.join(os.path.dirname(HERE), "include")):
        for dirpath, _, files in os.walk(root):
            deps += [os.path.join(dirpath, f) for f in files]
    return deps


def build_kernels(force=False, verbose=False):
    os.makedirs(LIB, exist_ok=True)
    out = os.path.join(LIB, "liblitert_b200.so")
    srcs = [os.path.join(CSRC, s) for s in KERNEL_SOURCES if os.path.exists(os.path.join(CSRC, s))]
    if not force and not _newer(out, _all_deps()):
        return out
    objs = []
    procs = []
    for s in srcs:
        o = os.path.join(LIB, os.path.basename(s) + ".o")
        objs.append(o)
        cmd = [NVCC] + ARCH + COMMON + (["-Xptxas", "-v"] if verbose else []) + ["-c", s, "-o", o]
        procs.append((cmd, subprocess.Popen(cmd)))
    for cmd, p in procs:
        if p.wait() != 0:
            raise RuntimeError("nvcc failed: " + " ".join(cmd))
    cmd = [NVCC] + ARCH + ["-shared", "-o", out] + objs
    subprocess.check_call(cmd)
    for o in objs:
        os.remove(o)
    return out


def build_host_ops(force=False):
    """The CPython extension of the small calls (csrc/host_ops.cc), over the kernels' library and torch's C++ API, for this
    interpreter and this torch. None without torch: the calls then go through ctypes."""
    import glob
    import sysconfig

    try:
        import torch
    except ImportError:
        return None
    from ._lib import host_ops_path

    kernels = build_kernels()
    out = host_ops_path()
    src = os.path.join(CSRC, "host_ops.cc")
    if not force and not _newer(out, [src, os.path.join(os.path.dirname(HERE), "include", "litert_b200.h")]):
        return out
    for stale in glob.glob(os.path.join(glob.escape(LIB), "_host_ops*.so")):  # of another torch
        os.remove(stale)
    root = os.path.dirname(torch.__file__)
    inc = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
           sysconfig.get_paths()["include"], os.path.join(os.path.dirname(os.path.dirname(NVCC)), "include")]
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-shared", "-o", out, src,
                           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"] +
                          [f for d in inc for f in ("-isystem", d)] +
                          ["-L" + LIB, "-l:" + os.path.basename(kernels), "-Wl,-rpath,$ORIGIN", "-L" + os.path.join(root, "lib"),
                           "-ltorch_python", "-ltorch_cuda", "-ltorch_cpu", "-lc10_cuda", "-lc10"])
    return out


def build_all(force=False, verbose=False):
    paths = [p for p in (build_kernels(force, verbose), build_host_ops(force)) if p]
    try:
        from . import build_delegate
    except ImportError:
        build_delegate = None
    if build_delegate is not None:
        p = build_delegate.build(force)
        if p:
            paths.append(p)
        a = build_delegate.build_accelerator(force)
        if a:
            paths.append(a)
    return paths


if __name__ == "__main__":
    for p in build_all(force="--force" in sys.argv, verbose="-v" in sys.argv):
        print(p)
