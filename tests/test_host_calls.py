"""What the library's host code asks of the CUDA runtime, on a machine without a
GPU: libbmfp.so runs over a stand-in runtime (cxx/fake_cudart.cpp) in a child
process, whose calls can be counted and made to fail."""
import os
import shutil
import subprocess
import sys

import pytest

from conftest import ROOT
from block_matrix_format_performance_gb300.build import cuda_home

pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")

PRELUDE = """
import ctypes
import numpy as np
import block_matrix_format_performance_gb300 as bm
fake = ctypes.CDLL(FAKE)
fake.fake_pending.argtypes = [ctypes.c_void_p]
STREAM = 0x1000
def grid_matrix(n):
    rp, c, v, _ = bm.gen_q4_elasticity(n, n)
    return bm.Matrix.from_bcsr(rp, c, v, 2, stream=STREAM)
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory, lib):
    out = tmp_path_factory.mktemp("fake") / "libfakecudart.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", f"{ROOT}/include",
                    "-I", f"{ROOT}/block_matrix_format_performance_gb300/csrc", "-I", f"{cuda_home()}/include",
                    f"{ROOT}/tests/cxx/fake_cudart.cpp", "-o", str(out)], check=True)
    return str(out)


def run(fake, code):
    p = subprocess.run([sys.executable, "-c", f"FAKE = {fake!r}\n" + PRELUDE + code], cwd=ROOT, text=True,
                       capture_output=True, env={**os.environ, "LD_PRELOAD": fake})
    assert p.returncode == 0, p.stdout + p.stderr


@pytest.mark.parametrize("precision", ["fp64", "fp32", "mixed"])
@pytest.mark.parametrize("mode", ["auto", "graph", "persistent"])
def test_solver_creation_leaves_nothing_on_its_stream(fake, mode, precision):
    """The header promises that creation synchronises the stream: a solver may
    then be used on another one. Without the FP64 fallback no probe waits."""
    run(fake, f"""
A = grid_matrix(40)
s = bm.Solver(A, {precision!r}, stream=STREAM, launch_mode={mode!r}, fallback_fp64=0)
assert fake.fake_pending(STREAM) == 0, fake.fake_pending(STREAM)
""")
