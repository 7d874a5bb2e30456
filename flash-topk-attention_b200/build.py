"""Build libftk_sm100.so in-tree with nvcc for sm_100a.

    python flash-topk-attention_b200/build.py [--force]

Each csrc/*.cu is compiled to an object under build/ and the objects are
linked into lib/libftk_sm100.so (CUDA runtime linked statically; the driver
API is reached through cudaGetDriverEntryPoint, so the library also loads on
a machine without a GPU driver).  What ptxas says of the kernels (registers,
spills) stays beside the objects.  csrc/host/torch_ops.cpp, the native layer
between the Python operators and that library, becomes
flash_topk_attn_v2/_native.so (host code only: g++ against PyTorch's headers).
"""

from __future__ import annotations

import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "build")
LIBDIR = os.path.join(HERE, "lib")
LIB = os.path.join(LIBDIR, "libftk_sm100.so")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")

FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
    "-lineinfo", "-Xcompiler", "-fPIC", "-Xptxas", "-v",
]


def _sources():
    return sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))


def ptxas_log(src: str) -> str:
    return os.path.join(OBJ, src[:-3] + ".ptxas")


def _headers_mtime():
    include = os.path.join(os.path.dirname(HERE), "include")
    hs = [os.path.join(d, f) for d in (CSRC, include) for f in os.listdir(d)
          if f.endswith((".cuh", ".h"))]
    return max(os.path.getmtime(h) for h in hs) if hs else 0.0


def _compile(src: str, force: bool) -> str:
    obj = os.path.join(OBJ, src[:-3] + ".o")
    log = ptxas_log(src)
    spath = os.path.join(CSRC, src)
    newest = max(os.path.getmtime(spath), _headers_mtime())
    if (not force and os.path.exists(obj) and os.path.exists(log)
            and os.path.getmtime(obj) >= newest):
        return obj
    cmd = [NVCC, *FLAGS, "-c", spath, "-o", obj]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"nvcc failed for {src}:\n{r.stdout}\n{r.stderr}")
    with open(log, "w") as f:
        f.write(r.stderr)
    return obj


def build(force: bool = False) -> str:
    os.makedirs(OBJ, exist_ok=True)
    os.makedirs(LIBDIR, exist_ok=True)
    srcs = _sources()
    with ThreadPoolExecutor(max_workers=min(8, len(srcs))) as ex:
        objs = list(ex.map(lambda s: _compile(s, force), srcs))
    if (not force and os.path.exists(LIB)
            and os.path.getmtime(LIB) >= max(os.path.getmtime(o) for o in objs)):
        return LIB
    cmd = [NVCC, "-shared", "-o", LIB, *objs, "-gencode",
           "arch=compute_100a,code=sm_100a", "-cudart", "static"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    return LIB


HOST_SRC = os.path.join(CSRC, "host", "torch_ops.cpp")
NATIVE = os.path.join(HERE, "flash_topk_attn_v2", "_native.so")
NATIVE_STAMP = os.path.join(OBJ, "native.stamp")   # what NATIVE was built against
CXX = os.environ.get("CXX", "g++")


def built_for() -> str:
    """The PyTorch and the interpreter that _native.so is tied to: it uses the C++
    interfaces of both, which another version does not have to keep."""
    import torch
    return f"torch {torch.__version__}, {sys.implementation.cache_tag}"


def native_is_current() -> bool:
    """Whether NATIVE is there, newer than its sources and built for this PyTorch."""
    include = os.path.join(os.path.dirname(HERE), "include")
    newest = max(os.path.getmtime(p) for p in
                 [HOST_SRC] + [os.path.join(include, f) for f in os.listdir(include)])
    if not os.path.exists(NATIVE) or os.path.getmtime(NATIVE) < newest:
        return False
    if not os.path.exists(NATIVE_STAMP):
        return False
    with open(NATIVE_STAMP) as f:
        return f.read() == built_for()


def build_native(force: bool = False) -> str:
    """flash_topk_attn_v2/_native.so; links lib/libftk_sm100.so (built first)."""
    if not force and native_is_current():
        return NATIVE
    import sysconfig

    import torch
    from torch.utils import cpp_extension as ext

    cuda = os.path.dirname(os.path.dirname(NVCC))
    dirs = [*ext.include_paths(), os.path.join(cuda, "include"), sysconfig.get_path("include")]
    torch_lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    cmd = [CXX, "-O2", "-std=c++17", "-fPIC", "-shared", "-DTORCH_EXTENSION_NAME=_native",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
           f'-DFTK_BUILT_FOR="{built_for()}"',
           *[x for d in dirs for x in ("-isystem", d)], HOST_SRC, "-o", NATIVE,
           "-L", LIBDIR, "-l:libftk_sm100.so", "-Wl,-rpath,$ORIGIN/../lib",
           "-L", torch_lib, "-lc10", "-lc10_cuda", "-ltorch", "-ltorch_cpu", "-ltorch_cuda",
           "-ltorch_python", f"-Wl,-rpath,{torch_lib}"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"{CXX} failed for torch_ops.cpp:\n{r.stdout}\n{r.stderr}")
    os.makedirs(OBJ, exist_ok=True)
    with open(NATIVE_STAMP, "w") as f:
        f.write(built_for())
    return NATIVE


PROBE_SRC = os.path.join(os.path.dirname(HERE), "tests", "native", "wait_probe.cu")
PROBE_LIB = os.path.join(os.path.dirname(HERE), "tests", "native", "libftk_wait_probe.so")


def build_wait_probe(force: bool = False) -> str:
    """Test-only library: the bounded waits of csrc/ftk_sm100.cuh compiled with a
    wait limit of 200 000 clock ticks (tests/native/wait_probe.cu)."""
    if not os.path.exists(PROBE_SRC):
        return ""
    newest = max(os.path.getmtime(PROBE_SRC), _headers_mtime())
    if not force and os.path.exists(PROBE_LIB) and os.path.getmtime(PROBE_LIB) >= newest:
        return PROBE_LIB
    cmd = [NVCC, *FLAGS, "-DFTK_WAIT_CYCLES=200000LL", "-ftz=true", "-I", CSRC, "-shared", "-cudart", "static",
           PROBE_SRC, "-o", PROBE_LIB]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"nvcc failed for wait_probe.cu:\n{r.stdout}\n{r.stderr}")
    return PROBE_LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv))
    print(build_native(force="--force" in sys.argv))
    print(build_wait_probe(force="--force" in sys.argv))
