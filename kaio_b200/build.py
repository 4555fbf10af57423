"""Builds ``libkaio_b200.so`` (sm_100a) in place with nvcc.

Run as ``python -m kaio_b200.build`` or through ``__graft_entry__.build()``.  nvcc
cross-compiles without a GPU.  Each ``csrc/*.cu`` is compiled to an object in parallel and
linked into ``kaio_b200/lib/libkaio_b200.so``; the CUDA runtime is linked statically and the
driver API is reached through the runtime's entry-point lookup, so the library loads on a
machine without ``libcuda.so`` (where every op then reports a CUDA error).  ``csrc/bindings.cpp``
(the argument unpacking of ``kaio_b200.ops``) becomes the extension module ``kaio_b200/_native``,
linked against that library; it is built again when the Python or the torch it was built for has changed.
"""
from __future__ import annotations

import concurrent.futures as cf
import glob
import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB_DIR = os.path.join(HERE, "lib")
OBJ_DIR = os.path.join(HERE, "build")
LIB = os.path.join(LIB_DIR, "libkaio_b200.so")
# tagged with the Python ABI, so that another interpreter does not load it
NATIVE = os.path.join(HERE, "_native" + (sysconfig.get_config_var("EXT_SUFFIX") or ".so"))
NATIVE_STAMP = os.path.join(OBJ_DIR, "native.txt")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC,-fvisibility=hidden", "--expt-relaxed-constexpr",
    "-Xptxas", "-v", "-Xptxas", "-warn-spills",
]


def _nvcc() -> str:
    for cand in (shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found: cannot build libkaio_b200.so")


def _newest_header_mtime() -> float:
    hdrs = glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(CSRC, "*.h"))
    hdrs += glob.glob(os.path.join(os.path.dirname(HERE), "include", "*.h"))
    return max(os.path.getmtime(h) for h in hdrs)


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(LIB_DIR, exist_ok=True)
    os.makedirs(OBJ_DIR, exist_ok=True)
    nvcc = _nvcc()
    srcs = sorted(glob.glob(os.path.join(CSRC, "*.cu")))
    hdr_m = _newest_header_mtime()
    jobs = []
    for src in srcs:
        obj = os.path.join(OBJ_DIR, os.path.basename(src)[:-3] + ".o")
        stale = force or not os.path.exists(obj) or os.path.getmtime(obj) < max(os.path.getmtime(src), hdr_m)
        jobs.append((src, obj, stale))

    def compile_one(job):
        src, obj, stale = job
        if not stale:
            return src, ""
        extra = os.environ.get("KAIO_B200_NVCC_EXTRA", "").split()
        r = subprocess.run([nvcc, *NVCC_FLAGS, *extra, "-c", src, "-o", obj], capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{r.stdout}\n{r.stderr}")
        return src, r.stderr

    with cf.ThreadPoolExecutor(max_workers=min(8, len(jobs))) as ex:
        logs = list(ex.map(compile_one, jobs))
    usage = os.path.join(OBJ_DIR, "resource_usage.txt")
    with open(usage, "a" if not force else "w") as f:
        for src, log in logs:
            if log:
                f.write(f"==== {os.path.basename(src)}\n{log}\n")
                if verbose:
                    print(log)
    objs = [j[1] for j in jobs]
    if force or any(j[2] for j in jobs) or not os.path.exists(LIB):
        r = subprocess.run([nvcc, "-shared", "-o", LIB, *objs, "-cudart", "static", "-ldl",
                            "-gencode", "arch=compute_100a,code=sm_100a"], capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    build_native(force)
    return LIB


NATIVE_FLAGS = ["-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden"]


def _native_key() -> str:
    """What the extension module depends on beside its sources."""
    import torch
    return "\n".join([f"torch {torch.__version__}", f"python {sysconfig.get_config_var('EXT_SUFFIX')}", *NATIVE_FLAGS])


def native_is_current() -> bool:
    if not os.path.exists(NATIVE) or not os.path.exists(NATIVE_STAMP):
        return False
    srcs = [os.path.join(CSRC, "bindings.cpp"), os.path.join(os.path.dirname(HERE), "include", "kaio_b200.h")]
    if os.path.getmtime(NATIVE) < max(os.path.getmtime(f) for f in srcs):
        return False
    with open(NATIVE_STAMP) as f:
        return f.read() == _native_key()


def build_native(force: bool = False) -> str:
    """Compiles ``csrc/bindings.cpp`` against the installed torch and this library."""
    if not force and native_is_current():
        return NATIVE
    import torch
    os.makedirs(OBJ_DIR, exist_ok=True)
    untagged = os.path.join(HERE, "_native.so")
    if untagged != NATIVE and os.path.exists(untagged):
        os.remove(untagged)  # an earlier build's, which any Python would load
    src = os.path.join(CSRC, "bindings.cpp")
    torch_dir = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    inc = [os.path.join(torch_dir, "include"), os.path.join(torch_dir, "include/torch/csrc/api/include"),
           sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
    r = subprocess.run([shutil.which("g++") or "g++", *NATIVE_FLAGS, f'-DKAIO_TORCH_VERSION="{torch.__version__}"',
                        *[f"-I{d}" for d in inc], src, "-o", NATIVE, f"-L{LIB_DIR}", "-lkaio_b200",
                        f"-L{os.path.join(torch_dir, 'lib')}", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python",
                        "-Wl,-rpath,$ORIGIN/lib"], capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"g++ failed on {src}:\n{r.stdout}\n{r.stderr}")
    with open(NATIVE_STAMP, "w") as f:
        f.write(_native_key())
    return NATIVE


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
