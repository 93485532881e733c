"""The host tables of the line sweeps, on which their progress rests: every line
after all lines it depends on, the nodes of a line consecutive, every off-node
unknown of a node's triangle exactly once among its far or near columns with the
place of its entry in every row, and no values shared by two tasks.  On meshes
with lines of one node to whole planes, nodes of 2 to 10 unknowns, independent
problems, renumbered nodes and the multicoloured order."""
import ctypes
import os
import shutil
import subprocess

import pytest

from goma_gb300 import problem as pb
from tests.test_gpu_line_sweeps import CASES

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "goma_gb300", "csrc")


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    so = os.path.join(tmp_path_factory.mktemp("tables"), "check.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC, "-I",
                    os.path.join(os.path.dirname(os.path.realpath(nvcc)), "..", "include"),
                    os.path.join(ROOT, "tests", "line_tables_check.cpp"),
                    os.path.join(CSRC, "gb_sweep_tables.cpp"), os.path.join(CSRC, "gb_layout.cpp"),
                    "-o", so], check=True)
    return ctypes.CDLL(so)


@pytest.mark.parametrize("ordering", [0, 1], ids=["natural", "multicoloured"])
@pytest.mark.parametrize("name", list(CASES))
def test_tables(name, ordering, library):
    desc, keep = pb.make_desc(CASES[name][0]())
    msg = ctypes.create_string_buffer(256)
    assert library.line_tables_check(ctypes.byref(desc), ordering, msg) == 0, msg.value
    del keep
