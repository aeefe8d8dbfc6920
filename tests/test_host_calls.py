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


@pytest.mark.parametrize("bs", [16, 32])
def test_autotuner_can_pick_the_default(fake, bs):
    """FP64 at block sizes 16 and 32: no explicit lane count names the default
    kernel, so the autotuner has to time it beside them. Each candidate in turn
    is made the fastest."""
    run(fake, f"""
m = bm.Matrix.from_bcsr(np.array([0, 1], np.int32), np.array([0], np.int32), np.ones({bs * bs}), {bs}, stream=STREAM)
fake.fake_fast_intervals(-1, -1)
m.autotune(0x10000, 0x20000, stream=STREAM)
n, reps = fake.fake_intervals(), 5
picked = []
for k in range(0, n, reps):
    fake.fake_fast_intervals(k, k + reps)
    picked.append(m.autotune(0x10000, 0x20000, stream=STREAM))
assert 0 in picked and len(set(picked)) == len(picked) == n // reps, picked
""")


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_no_room_for_the_resident_kernel_leaves_the_graphs(fake, precision):
    """Each allocation of a solver's creation fails in turn. The ones that only
    the auto mode makes (the sliced copy, and the words, flags and published
    vectors of its kernel) are not needed for a solve."""
    run(fake, f"""
A = grid_matrix(40)
def create(mode, fail):
    fake.fake_fail_malloc(fail)
    s = bm.Solver(A, {precision!r}, stream=STREAM, launch_mode=mode)
    s.close()
    return fake.fake_mallocs()
def survives(mode, k):
    graphs = fake.fake_graphs()
    try:
        create(mode, k)
    except bm.BmfpError:
        return False
    assert fake.fake_graphs() == graphs + 1, (mode, k)
    return True
counts = {{mode: create(mode, -1) for mode in ("auto", "graph")}}
extra = counts["auto"] - counts["graph"]
assert extra >= 1, counts
spare = {{mode: sum(survives(mode, k) for k in range(counts[mode])) for mode in counts}}
assert spare["auto"] == spare["graph"] + extra, (counts, spare)
""")


def test_auto_mode_returns_to_the_graphs_after_a_timeout(fake):
    """A cooperative kernel whose waits give up: the auto mode solves again with
    the graphs and stays with them; a caller who asked for the kernel is told."""
    run(fake, """
b, x = np.zeros(3200), np.empty(3200)
A = grid_matrix(40)
fake.fake_cooperative_fault(1)
s = bm.Solver(A, "fp64", stream=STREAM)
graphs = fake.fake_graphs()
for _ in range(2):
    assert s.solve(b, x, stream=STREAM)["status"] == bm.SUCCESS
    assert fake.fake_graphs() == graphs + 1
p = bm.Solver(A, "fp64", stream=STREAM, launch_mode="persistent")
try:
    p.solve(b, x, stream=STREAM)
    assert False
except bm.BmfpError as e:
    assert e.status == bm.ERROR_TIMEOUT, e
""")
