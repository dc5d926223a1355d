"""Builds the sm_100a kernel library in-tree: relax_b200/libb200_q4f16.so.

nvcc cross-compiles without a GPU.  The library links the CUDA runtime statically and
resolves driver entry points (tensor-map encoding) at run time, so it has no link-time
dependency on libcuda and loads on a machine without a driver (the symbol-export test).

    python -m relax_b200.build [--force] [--verbose]
"""
from __future__ import annotations

import os
import subprocess
import sys
import sysconfig
import warnings

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libb200_q4f16.so")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")

SOURCES = ["capi.cu", "tmap.cu", "dequant.cu", "gemv.cu", "gemv_pipe.cu", "gemm_tcgen05.cu", "gemm_ws_tcgen05.cu", "decoder_ops.cu", "attn_decode.cu", "decode_layer.cu", "lm_head.cu"]
HEADERS = ["internal.h", "q4_common.cuh", "sm100_ptx.cuh", "tmap.h", "skinny_common.cuh", "smem_limit.h", "ws_plan.h"]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "--expt-relaxed-constexpr",
    "-Xcompiler", "-fPIC,-fvisibility=hidden",
    "-Xptxas", "-v",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def _stale() -> bool:
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    deps = [os.path.join(CSRC, f) for f in SOURCES + HEADERS if os.path.exists(os.path.join(CSRC, f))]
    deps += [os.path.join(INCLUDE, "b200_q4f16.h"), os.path.abspath(__file__)]
    return any(os.path.getmtime(d) > t for d in deps)


def torch_call_path(torch_version: str) -> str:
    """The CPython extension (torch tensors to the library's C ABI) for this interpreter and that torch.  It is compiled against
    the insides of torch's tensors, so one that was built for another torch or Python is never looked at."""
    return os.path.join(HERE, f"_torch_call.{sysconfig.get_config_var('SOABI')}.torch-{torch_version}.so")


def _torch_call_command(torch) -> list:
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc())) if os.path.isabs(_nvcc()) else "/usr/local/cuda"
    include = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
               sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
    lib = os.path.join(root, "lib")
    return ["/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *[f"-I{d}" for d in include],
            os.path.join(CSRC, "torch_call.cpp"), "-o", torch_call_path(torch.__version__), f"-L{lib}", f"-Wl,-rpath,{lib}",
            "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python"]


def _torch_call_stale(path: str) -> bool:
    deps = [os.path.join(CSRC, "torch_call.cpp"), os.path.join(INCLUDE, "b200_q4f16.h"), os.path.abspath(__file__)]
    return not os.path.exists(path) or any(os.path.getmtime(d) > os.path.getmtime(path) for d in deps)


def _start_torch_call(force: bool):
    """The compiler of the extension, started; None: it is there, or there is no torch to build it for.  Raises where it cannot run."""
    try:
        import torch
    except ImportError:
        return None
    if not force and not _torch_call_stale(torch_call_path(torch.__version__)):
        return None
    return subprocess.Popen(_torch_call_command(torch), stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)


def build(force: bool = False, verbose: bool = False) -> str:
    """The library, and the extension beside it.  The library needs nvcc only; without the extension the operators make
    its checks in Python, so what keeps it from being built is a warning."""
    compiler, why = None, ""
    try:
        compiler = _start_torch_call(force)
    except Exception as e:
        why = f"{type(e).__name__}: {e}"
    try:
        return _build_library(force, verbose)
    finally:
        if compiler is not None:
            out, _ = compiler.communicate()
            if compiler.returncode != 0:
                why = out
        if why:
            warnings.warn("torch_call.cpp was not built, operator calls on torch tensors take longer: " + why, RuntimeWarning, stacklevel=2)


def _build_library(force: bool, verbose: bool) -> str:
    if not force and not _stale():
        return LIB
    objs = []
    env = dict(os.environ)
    # the image exports CC/CXX pointing at a wrapper; nvcc should use the system g++
    ccbin = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"
    procs = []
    for src in SOURCES:
        obj = os.path.join(CSRC, src.rsplit(".", 1)[0] + ".o")
        cmd = [_nvcc(), "-ccbin", ccbin, *NVCC_FLAGS, "-I", INCLUDE, "-c", os.path.join(CSRC, src), "-o", obj]
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, env=env)))
        objs.append(obj)
    log = []
    for src, p in procs:
        out, _ = p.communicate()
        log.append(f"== {src}\n{out}")
        if p.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src}:\n{out}")
    cmd = [_nvcc(), "-ccbin", ccbin, "-shared", "-o", LIB, *objs, "-Xcompiler", "-fPIC", "-lcudart_static", "-ldl", "-lrt", "-lpthread"]
    r = subprocess.run(cmd, capture_output=True, text=True, env=env)
    if r.returncode != 0:
        raise RuntimeError("link failed:\n" + r.stdout + r.stderr)
    with open(os.path.join(HERE, "build.log"), "w") as f:
        f.write("\n".join(log))
    if verbose:
        print("\n".join(log))
    return LIB


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="--verbose" in sys.argv)
    print(path)
