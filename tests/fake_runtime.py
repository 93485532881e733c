"""Runs a test's script in a process with a C file preloaded over the CUDA
runtime: fake_cudart.c in its place, for the library's host code with calls that
can be made to fail on any machine, or limit_pool.c on a GPU."""
import os
import shutil
import subprocess
import sys
import textwrap

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PREAMBLE = """
import ctypes
import numpy as np
from goma_gb300 import _lib
from goma_gb300 import problem as pb
from goma_gb300.newton import GomaNewton
fake = ctypes.CDLL(None)
ll = lambda name: ctypes.c_longlong.in_dll(fake, name)
integer = lambda name: ctypes.c_int.in_dll(fake, name)
cavity = lambda nx, ny: pb.lid_cavity_2d(0, mesh=pb.box_mesh(2, nx, ny))
"""


def run(script, tmp_path, source="fake_cudart.c"):
    """The script's output; a failure of the script fails the test."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    inc = os.path.join(os.path.dirname(os.path.realpath(nvcc)), "..", "include")
    so = os.path.join(str(tmp_path), "preloaded.so")
    subprocess.run(["gcc", "-std=c11", "-O1", "-Wall", "-Werror", "-shared", "-fPIC", "-I", inc,
                    os.path.join(ROOT, "tests", source), "-o", so, "-ldl"], check=True)
    env = dict(os.environ, LD_PRELOAD=so, PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", PREAMBLE + textwrap.dedent(script)], env=env,
                       cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.returncode, r.stdout + r.stderr)
    return r.stdout
