"""Shared libraries of the sources in tests/cuda, built with the library's own flags."""
import ctypes
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def load(name, folder):
    from ysim_b200 import build
    out = os.path.join(str(folder), name + ".so")
    subprocess.run([build.nvcc(), *build.ARCH, *build.FLAGS, "-shared", "-I", build.SRC, "-I",
                    os.path.join(build.ROOT, "include"), os.path.join(HERE, "cuda", name + ".cu"), "-o", out], check=True)
    return ctypes.CDLL(out)
