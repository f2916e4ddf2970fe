"""The library's host code built against a fake CUDA runtime (tests/host/):
failures and sizes that a test sets, with no GPU."""
import ctypes as C
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def build_host(name, out_dir):
    """tests/host/<name>.cu as a shared library, loaded"""
    from gpuseed_gb300 import build as gbuild
    so = os.path.join(str(out_dir), f"lib{name}.so")
    subprocess.run([gbuild._nvcc(), *gbuild.ARCH, "-O1", "-std=c++17", "-cudart", "none", "-shared",
                    "-Xcompiler", "-fPIC,-Wall,-Wno-unused-function", "-Xlinker", "-Bsymbolic", "-I",
                    gbuild.INCLUDE, os.path.join(HERE, "host", name + ".cu"), "-o", so], check=True)
    return C.CDLL(so)
