"""Runs a script against the library on a CUDA runtime without a GPU
(tests/cpp/fake_cudart.cpp): the host code runs, kernels are only counted."""
import os
import subprocess
import sys
import textwrap

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
OUT = os.path.join(ROOT, "_build", "cpp")

HEAD = r"""
import ctypes, sys
sys.path.insert(0, %r)
fake = ctypes.CDLL(%r)
import numpy as np
import paxpro_b200 as pxp
from paxpro_b200 import _capi
from paxpro_b200 import workloads as wl
lib = _capi.lib()


def spec(kind, n, nsteps=64, prec=0, save_every=0):
    dx = wl.step_for_nodes(-250.0, 250.0, n)
    x = pxp.Disc(-250.0, 250.0, dx)
    return pxp.ProblemSpec(kind=kind, x=x, y=x, z=pxp.Disc(0.0, nsteps * 500.0, 500.0), wavenumber=wl.K,
                           precision=prec, save_every=save_every)
"""


def run(script: str, timeout: int = 120) -> str:
    os.makedirs(OUT, exist_ok=True)
    so = os.path.join(OUT, "fake_cudart.so")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["/usr/bin/g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I" + cuda + "/include",
                    os.path.join(ROOT, "tests", "cpp", "fake_cudart.cpp"), "-o", so], check=True)
    r = subprocess.run([sys.executable, "-c", HEAD % (ROOT, so) + textwrap.dedent(script)],
                       env=dict(os.environ, LD_PRELOAD=so), capture_output=True, text=True, timeout=timeout)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout
