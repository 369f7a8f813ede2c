"""Builds stages.cu against the built libgpt.so (nvcc, for the GPU tests that look at one stage of a batch)."""
import ctypes
import os
import shutil
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(os.path.dirname(HERE)), "gpu-pcg-tracking_b200")


def build(folder):
    out = os.path.join(str(folder), "libstages.so")
    nvcc = shutil.which("nvcc") or os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-O2",
                    "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-shared", "-I", os.path.join(PKG, "csrc"),
                    os.path.join(HERE, "stages.cu"), "-o", out, "-L", PKG, "-lgpt", "-Xlinker", "-rpath=" + PKG],
                   check=True)
    return ctypes.CDLL(out)
