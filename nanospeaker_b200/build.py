"""Build the CUDA library in-tree, nanospeaker_b200/libmoe_b200.so (sm_100a only), and the pybind
shim over it, nanospeaker_b200/_moe_shim.so (host code; it launches through the library's C ABI).

Run as `python -m nanospeaker_b200.build`. nvcc cross-compiles without a GPU present.
"""
import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libmoe_b200.so")
SHIM = os.path.join(HERE, "_moe_shim.so")
SHIM_SOURCE = "shim.cpp"
SOURCES = ["api.cu", "routing.cu", "router_fused.cu", "router_front.cu", "movement.cu", "norm.cu", "gemm.cu", "ep.cu", "block.cu", "stack.cu",
           "muon.cu"]
HEADERS = ["act.cuh", "agree.cuh", "wgrad_order.cuh", "stack_shape.cuh", "stages.cuh", "tma_map.cuh", "ptx.cuh", "pdl.cuh", "gemm.cuh", "gemm_rows.cuh", "gemm_rows2.cuh", "gemm_wgrad2.cuh", "gemm_wgrad.cuh", "routing.cuh", "dispatch_scatter.cuh", "route_token.cuh", "per_device.cuh", os.path.join("..", "..", "include", "moe_b200.h")]


def _stale(out: str, files) -> bool:
    if not os.path.exists(out):
        return True
    built = os.path.getmtime(out)
    deps = [os.path.join(CSRC, f) for f in files]
    return any(os.path.getmtime(d) > built for d in deps if os.path.exists(d))


def _shim_command():
    import torch
    from torch.utils.cpp_extension import include_paths
    lib_dir = os.path.join(os.path.dirname(torch.__file__), "lib")
    cuda_home = os.path.dirname(os.path.dirname(
        shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"))
    cmd = [shutil.which("g++") or "c++", "-shared", "-fPIC", "-std=c++20", "-O2", "-g0",
           "-fvisibility=hidden", "-DTORCH_EXTENSION_NAME=_moe_shim",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
    for p in [*include_paths(), os.path.join(cuda_home, "include"),
              sysconfig.get_path("include")]:
        cmd += ["-isystem", p]
    cmd += [os.path.join(CSRC, SHIM_SOURCE), "-o", SHIM, f"-L{lib_dir}", "-lc10", "-lc10_cuda",
            "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python", f"-Wl,-rpath,{lib_dir}"]
    return cmd


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every .cu for sm_100a into one shared library, and the shim; returns the library's
    path."""
    jobs = []
    if force or _stale(LIB, SOURCES + HEADERS):
        nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
        cmd = [
            nvcc, "-shared", "-Xcompiler", "-fPIC", "-std=c++17", "-O3", "-lineinfo",
            "-gencode", "arch=compute_100a,code=sm_100a",
            "-t", "0",
            "-o", LIB,
        ] + [os.path.join(CSRC, s) for s in SOURCES]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        jobs.append(cmd)
    if force or _stale(SHIM, [SHIM_SOURCE, HEADERS[-1]]):
        jobs.append(_shim_command())
    running = [(c, subprocess.Popen(c, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True))
               for c in jobs]
    outputs = [(c, p.communicate()[0], p.returncode) for c, p in running]
    for cmd, out, rc in outputs:
        if rc != 0:
            raise RuntimeError(f"build failed:\n{' '.join(cmd)}\n{out}")
        if verbose:
            print(out)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
