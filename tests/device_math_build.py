"""Builds tests/device_math.cu (host entries to the kernels' headers) with nvcc."""
import ctypes
import importlib
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def load(outdir: str) -> ctypes.CDLL:
    b = importlib.import_module("0buf_b200.build")
    so = os.path.join(outdir, "device_math.so")
    cmd = [b.nvcc(), "-std=c++17", "-O1", "-shared", "-Xcompiler", "-fPIC,-ffp-contract=off", "-I", b.INCLUDE, "-I",
           b.CSRC] + b.ARCH + [os.path.join(ROOT, "tests", "device_math.cu"), "-o", so]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"nvcc failed:\n{r.stdout}\n{r.stderr}")
    return ctypes.CDLL(so)
