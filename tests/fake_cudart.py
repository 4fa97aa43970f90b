"""Runs a program against libdlgpu.so and the CUDA runtime of
fake_cudart.cpp, in a process of its own."""
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
REPO = os.path.dirname(HERE)

PROLOGUE = """
import ctypes as C, sys
import numpy as np
sys.path.insert(0, %r)
from drawlab_gb300 import abi, api, scenes
api.lib()
fake = C.CDLL("libcudart.so.13")
fake.fake_log.restype = C.c_char_p
fake.fake_fail_kernel.argtypes = [C.c_char_p, C.c_int]
log = lambda: fake.fake_log().decode().split("\\n")[:-1]
""" % REPO


def run(code, tmp_path):
    from drawlab_gb300 import build
    build.build()
    lib = tmp_path / "libcudart.so.13"
    subprocess.run([build.CXX, "-std=c++17", "-O1", "-shared", "-fPIC", "-Wl,-soname,libcudart.so.13",
                    "-I", str(build.CUDA_HOME / "include"), os.path.join(HERE, "fake_cudart.cpp"), "-o", str(lib)],
                   check=True, timeout=300)
    env = dict(os.environ, LD_LIBRARY_PATH=str(tmp_path))
    r = subprocess.run([sys.executable, "-c", PROLOGUE + code], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    return r.stdout
