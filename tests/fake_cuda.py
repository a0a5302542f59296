"""Runs a piece of Python against the library with fake_cudart.cpp in place of the CUDA runtime (no device)."""
import os
import subprocess
import sys
import textwrap

from skirt7_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))
PRELUDE = """
import ctypes as C, os, sys
sys.path[:0] = [%r, %r]
fake = C.CDLL(os.environ["LD_PRELOAD"])
fake.fake_log.restype = C.c_char_p
fake.fake_memory.argtypes = [C.c_size_t]
fake.fake_used.restype = C.c_size_t
def log(what=""):
    return [l for l in fake.fake_log().decode().splitlines() if what in l]
from skirt7_b200 import _abi as A, models, runtime
from helpers import cell_center_density
def oligo(N=(6, 5, 4), **kw):
    m = models.oligo_disk(N=N, npix=8, **kw)
    m.rho = cell_center_density(m)
    return m
"""


def compile_fake(folder):
    """The fake runtime as a shared library in `folder`."""
    out = os.path.join(str(folder), "libfakecudart.so")
    params = os.path.join(str(folder), "fake_params.o")
    subprocess.run([os.environ.get("NVCC", "nvcc"), "-c", "-O1", "-std=c++17", "-Xcompiler", "-fPIC",
                    "--expt-relaxed-constexpr"] + build.ARCH + ["-o", params, os.path.join(HERE, "fake_params.cu")], check=True)
    subprocess.run(["g++", "-shared", "-fPIC", "-O1", "-std=c++17", "-I" + build.CUDA_INC, "-o", out,
                    os.path.join(HERE, "fake_cudart.cpp"), params], check=True)
    return out


def run(fake, code):
    """Runs `code` (after PRELUDE) in a process of its own; its asserts are the test's."""
    env = dict(os.environ, LD_PRELOAD=fake)
    r = subprocess.run([sys.executable, "-c", PRELUDE % (os.path.dirname(HERE), HERE) + textwrap.dedent(code)], env=env,
                       capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    return r.stdout
