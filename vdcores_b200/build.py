"""Builds libvdcores_b200.so in-tree with nvcc for sm_100a:  python -m vdcores_b200.build"""
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
LIB = os.path.join(HERE, "libvdcores_b200.so")
SOURCES = [os.path.join(HERE, "csrc", f) for f in ("megakernel.cu", "stage_kernels.cu", "wide_kernels.cu", "step_kernel.cu", "capi.cu")]
# VDC_NO_STREAMER: the optional HBM->L2 streamer warp stays out of the build (it did not pay for
# the registers it costs: 13 warps cap the kernel at 128 registers per thread instead of 168).
FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "-shared",
         "-Xcompiler", "-fPIC", "-DVDC_NO_STREAMER"]
OBJ_DIR = os.path.join(HERE, "build")


def needs_build() -> bool:
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    csrc = os.path.join(HERE, "csrc")
    deps = [os.path.join(csrc, f) for f in os.listdir(csrc)] + [os.path.join(HERE, "..", "include", "vdcores.h")]
    return any(os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> str:
    """One object per source (compiled side by side, kept while neither it nor a header changes), then the library."""
    if not (force or needs_build()):
        return LIB
    nvcc = os.environ.get("NVCC", "nvcc")
    os.makedirs(OBJ_DIR, exist_ok=True)
    csrc = os.path.join(HERE, "csrc")
    headers = [os.path.join(csrc, f) for f in os.listdir(csrc) if not f.endswith(".cu")]
    headers += [os.path.join(HERE, "..", "include", "vdcores.h"), os.path.abspath(__file__)]
    objs, running = [], []
    for src in SOURCES:
        obj = os.path.join(OBJ_DIR, os.path.basename(src)[:-3] + ".o")
        objs.append(obj)
        if force or not os.path.exists(obj) or any(os.path.getmtime(d) > os.path.getmtime(obj) for d in [src, *headers]):
            cmd = [nvcc, *(f for f in FLAGS if f != "-shared"), *(["-Xptxas", "-v"] if verbose else []), "-c", "-o", obj, src]
            running.append((cmd, subprocess.Popen(cmd)))
    failed = [cmd for cmd, p in running if p.wait() != 0]
    if failed:
        raise subprocess.CalledProcessError(1, failed[0])
    subprocess.check_call([nvcc, *FLAGS, "-o", LIB, *objs])
    return LIB


def build_trace(define: str) -> str:
    """A second library with one of the tracing switches compiled in (VDC_TRACE_ATTN: stamps inside the attention
    task, VDC_TRACE_GEMV: inside the GEMV task, VDC_TRACE_CHUNKS: life of SM 0's ring entries); select it with
    VDCORES_LIB=<path>.  The stamps go into the launch's profile rows (vdcores_b200.stage_trace prints them)."""
    assert define in ("VDC_TRACE_ATTN", "VDC_TRACE_GEMV", "VDC_TRACE_CHUNKS")
    out = os.path.join(HERE, f"libvdcores_b200_{define.lower()}.so")
    subprocess.check_call([os.environ.get("NVCC", "nvcc"), *FLAGS, f"-D{define}", "-o", out, *SOURCES])
    return out


if __name__ == "__main__":
    if "--trace" in sys.argv:
        print(build_trace(sys.argv[sys.argv.index("--trace") + 1]))
    else:
        print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
