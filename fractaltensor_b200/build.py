"""Builds libftb200.so (the C-ABI library) in-tree with nvcc for sm_100a, and _host.so, the
Python module in front of its short calls, with g++ against the installed torch.

Run as ``python -m fractaltensor_b200.build``.  The library links the CUDA
runtime statically and looks the driver's tensor-map encoder up at run time, so
it also loads on a machine that has no GPU driver (symbol checks only).
"""
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libftb200.so")
HOST_SRC = os.path.join(CSRC, "host_calls.cpp")
HOST = os.path.join(HERE, "_host.so")
SOURCES = ["tmap.cu", "pack.cu", "cell_gemm.cu", "cell_simt.cu", "lstm_simt_static.cu", "lstm_simt_flow.cu", "lstm_static.cu", "lstm_wmajor.cu", "lstm_flow.cu", "rnn_cluster.cu", "grid_flow.cu", "wavefront.cu", "b2b_gemm.cu", "flash_attn.cu", "flash_pair.cu",
           "online_softmax.cu", "project.cu", "embedding.cu", "sparse_attn.cu", "rnn_attention.cu", "rnn_chain.cu"]
NVCC_FLAGS = [
    "-std=c++17", "-O3", "-lineinfo",
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-Xcompiler", "-fPIC", "-Xptxas", "-v",
]


def _newer(a, b):
    return (not os.path.exists(b)) or os.path.getmtime(a) > os.path.getmtime(b)


def _host_flags():
    """Compile and link flags of _host.so (a plain CPython module that reads torch tensors)."""
    import sysconfig

    import torch
    root = os.path.dirname(torch.__file__)
    inc = [sysconfig.get_paths()["include"], os.path.join(root, "include"),
           os.path.join(root, "include", "torch", "csrc", "api", "include"), "/usr/local/cuda/include"]
    cflags = ["-std=c++17", "-O2", "-fPIC", "-fvisibility=hidden",
              "-D_GLIBCXX_USE_CXX11_ABI=%d" % int(torch._C._GLIBCXX_USE_CXX11_ABI)] + ["-I" + d for d in inc]
    ldflags = ["-L" + os.path.join(root, "lib"), "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda",
               "-L" + HERE, "-l:libftb200.so", "-Wl,-rpath,$ORIGIN"]
    return cflags, ldflags


def _host_object():
    """The object file of _host.so: named by the torch and the Python it is built against, so that with
    another of either there is none yet."""
    import torch
    return HOST_SRC.replace(".cpp", ".%s.%s.o" % (torch.__version__, sys.implementation.cache_tag))


def _host_is_stale(api):
    obj = _host_object()
    return _newer(HOST_SRC, obj) or _newer(api, obj) or _newer(obj, HOST)


def build(verbose=False, force=False):
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".h", ".cuh"))]
    api = os.path.join(HERE, "..", "include", "ftb200.h")
    headers.append(api)
    objs = []
    procs = []
    start = lambda name, cmd: procs.append(
        (name, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    for src in SOURCES:
        s = os.path.join(CSRC, src)
        if not os.path.exists(s):
            continue
        o = os.path.join(CSRC, src.replace(".cu", ".o"))
        objs.append(o)
        if force or _newer(s, o) or any(_newer(h, o) for h in headers):
            start(src, [nvcc] + NVCC_FLAGS + ["-c", s, "-o", o])
    link_lib = bool(procs) or not os.path.exists(LIB)
    host_obj = _host_object()
    build_host = force or _host_is_stale(api)
    if build_host:
        cflags, ldflags = _host_flags()
        start(os.path.basename(HOST_SRC), ["g++"] + cflags + ["-c", HOST_SRC, "-o", host_obj])
    failed = False
    for src, p in procs:
        out, _ = p.communicate()
        if verbose or p.returncode != 0:
            sys.stderr.write("== %s ==\n%s\n" % (src, out))
        failed = failed or p.returncode != 0
    if failed:
        raise RuntimeError("compilation failed")
    if link_lib:
        cmd = [nvcc, "-shared", "-Wno-deprecated-gpu-targets", "-o", LIB] + objs + ["-cudart", "static"]
        subprocess.check_call(cmd)
    if build_host:
        subprocess.check_call(["g++", "-shared", "-o", HOST, host_obj] + ldflags)
    return LIB


if __name__ == "__main__":
    print(build(verbose="-v" in sys.argv, force="-f" in sys.argv))
