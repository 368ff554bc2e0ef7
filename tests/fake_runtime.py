"""The library's host code on a CUDA runtime that runs nothing (fake_cuda/cudart.cpp): what it does where device memory or
threads run out, shown without a GPU.

The sources are those of the library, compiled for the host with their kernels left as unoptimised PTX, except the fused
passes' translation units (their kernels are only named)."""
import concurrent.futures
import ctypes
import importlib.util
import os

import build as pkg_build

HERE = os.path.dirname(os.path.abspath(__file__))
SOURCES = ["gsb_engine.cu", "gsb_batch.cu", "gsb_grad.cu", "gsb_dp.cu", "gsb_probe.cu", "gsb_plan.cpp", "gsb_order.cpp",
           "gsb_fuse.cpp"]
DIR = os.path.join(pkg_build.ROOT, "_build", "fake")
LIB = os.path.join(DIR, "libgsb_fake.so")


def build():
    headers = [os.path.join(pkg_build.CSRC, f) for f in pkg_build.LIB_DEPS if not f.endswith((".cu", ".cpp"))]
    headers.append(os.path.join(pkg_build.INCLUDE, "gsb.h"))
    os.makedirs(DIR, exist_ok=True)
    runtime = os.path.join(HERE, "fake_cuda", "cudart.cpp")
    cmds, objs = [], []
    for src in [os.path.join(pkg_build.CSRC, f) for f in SOURCES] + [runtime]:
        obj = os.path.join(DIR, os.path.basename(src) + ".o")
        objs.append(obj)
        if pkg_build._stale(obj, [src] + headers):
            cmds.append([pkg_build._nvcc(), "-gencode", "arch=compute_100a,code=compute_100a", "-Xcicc", "-O0", "-std=c++17",
                         "-Xcompiler", "-fPIC", "-c", "-I" + pkg_build.INCLUDE, "-I" + pkg_build.CSRC, "-o", obj, src])
    with concurrent.futures.ThreadPoolExecutor(max_workers=max(1, min(len(cmds), os.cpu_count() or 1))) as ex:
        list(ex.map(pkg_build._run, cmds))
    if cmds or pkg_build._stale(LIB, objs):
        # its own runtime, whatever else of CUDA the process has loaded
        pkg_build._run(["g++", "-shared", "-Wl,-Bsymbolic", "-o", LIB] + objs + ["-lpthread"])
    return LIB


def load():
    """(gsb, device): a copy of the package's gsb module on the fake runtime, and that runtime's controls."""
    path = build()
    cdll = ctypes.CDLL
    ctypes.CDLL = lambda name, *a, **k: cdll(path)
    try:
        spec = importlib.util.spec_from_file_location("gsb_on_fake_runtime", os.path.join(pkg_build.HERE, "gsb.py"))
        gsb = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(gsb)
    finally:
        ctypes.CDLL = cdll
    dev = cdll(path)
    for f in ("fake_used", "fake_largest"):
        getattr(dev, f).restype = ctypes.c_size_t
    dev.fake_count.restype = ctypes.c_long
    dev.fake_set_capacity.argtypes = [ctypes.c_size_t]
    dev.fake_fail.argtypes = [ctypes.c_long]
    return gsb, dev


(MALLOCS, FAILED, LAUNCHES, ATTRIBUTES, NULL_TABLES, STALE_REPLAYS, REPLAYS, FUSED_ONE, FUSED_SEVERAL,
 FUSED_WRONG) = range(10)
