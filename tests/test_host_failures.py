"""What the engine's host code does after an error, and what it asks of its kernels: the engine's objects linked with a CUDA runtime that
keeps device memory on the host, launches nothing and fails on request (tests/cpp/fake_cudart.cpp), each
case in a process of its own."""
import os
import shutil
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROLOGUE = """
import ctypes as C
import sys
import numpy as np
from rampack_gb300 import _lib
lib = _lib.load(sys.argv[1])
lib.fake_launched.restype = C.c_char_p
lib.fake_fail.argtypes = [C.c_char_p, C.c_int]
from rampack_gb300 import workloads as W
from rampack_gb300.packing import GpuPacking

def fails(call, after, f):
    lib.fake_fail(call.encode(), after)
    try:
        f()
    except _lib.EngineError:
        return True
    finally:
        lib.fake_fail(b"", -1)
    return False

def kernels(f):
    lib.fake_launched()
    f()
    return lib.fake_launched().decode()

def spheres(n=6):
    return GpuPacking(W.SPHERE, np.array([0.5]), W.lattice((n,) * 3, (1.5,) * 3), W.aligned_rotations(n ** 3),
                      W.diag_box(1.5 * n, 1.5 * n, 1.5 * n))
"""


@pytest.fixture(scope="module")
def fake(engine, tmp_path_factory):
    from rampack_gb300 import build as B
    objects = [os.path.join(B.HERE, "_build", s.replace(".cu", ".o")) for s in B.SOURCES]
    if not all(os.path.exists(o) for o in objects):
        B.build(force=True)
    lib = str(tmp_path_factory.mktemp("fake") / "librampack_fake.so")
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(shutil.which(B.nvcc())))), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-I", include, "-I", B.CSRC,
                    "-I", os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "cpp", "fake_cudart.cpp"), *objects, "-o", lib], check=True)
    return lib


def run(fake, code):
    p = subprocess.run([sys.executable, "-c", PROLOGUE + code, fake], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr[-3000:]


SHAPES = {
    "convex": 'GpuPacking(W.CONVEX, "cuboid 1 1 2; sphere 0.1; sum", W.lattice((5, 5, 5), (4.0,) * 3),'
              ' W.aligned_rotations(125), W.diag_box(20.0, 20.0, 20.0))',
    "soft": "spheres()",
}


@pytest.mark.parametrize("shape", sorted(SHAPES))
def test_refused_rototranslations_leave_the_grid(fake, shape):
    run(fake, f"""
g = {SHAPES[shape]}
if {shape!r} == "soft":
    g.set_soft(_lib.SOFT_REPULSIVE_LJ, 1.0, 1.0, False)
g.set_grid((0.25, 0.5, 0.75))
before = g.grid()[2]
assert fails("", -1, lambda: g.sweep(0.1, 0.1, seed=3, counter=0, rototranslation=True))
# the lists are the grid's that was set: nothing rebuilt them, so its bounds must stand
rebuilt = "k_scatter" in kernels(lambda: g.grid())
assert rebuilt or np.array_equal(before, g.grid()[2])
""")


@pytest.mark.parametrize("call", ["cudaMalloc", "cudaMemsetAsync", "k_rot_table", "k_cluster_sweep"])
def test_a_failed_small_sweep_leaves_no_grid_behind(fake, call):
    run(fake, f"""
g = spheres()
g.set_grid()
assert "k_cluster_sweep" in kernels(lambda: g.sweep(0.1, 0.0, seed=3, counter=0))
reads = [g.count_total_overlaps, lambda: fails("", -1, lambda: g.try_move(0, 0, (0.1, 0.0, 0.0))), g.grid]
for counter, read in enumerate(reads):
    assert fails({call!r}, 0, lambda: g.sweep(0.1, 0.1, seed=3, counter=counter, log=True))
    assert "k_scatter" in kernels(read), counter
""")


@pytest.mark.parametrize("call,after", [("cudaMalloc", 0), ("cudaMalloc", 1), ("cudaMalloc", 2), ("cudaHostAlloc", 0)])
def test_a_single_move_after_a_failed_allocation_has_its_buffers(fake, call, after):
    run(fake, f"""
def buffers(after):
    g = spheres()
    g.set_grid()
    lib.fake_allocations()
    if after >= 0:
        assert fails({call!r}, after, lambda: g.try_move(0, 0, (0.1, 0.0, 0.0)))
    # (the kernel does nothing here: its answer is missed, not looked for at a null address)
    assert "k_try_single" in kernels(lambda: fails("", -1, lambda: g.try_move(0, 0, (0.1, 0.0, 0.0))))
    return lib.fake_allocations()

assert buffers({after}) == buffers(-1) > 3
""")


@pytest.mark.parametrize("kind", ["W.SPHERE, np.array([0.5])", "W.SPHEROCYLINDER, np.array([0.3, 0.5])"])
def test_fp64_only_reaches_the_hard_pairs_of_soft_sweeps(fake, kind):
    run(fake, f"""
g = GpuPacking({kind}, W.lattice((6, 6, 6), (1.9,) * 3), W.aligned_rotations(216), W.diag_box(11.4, 11.4, 11.4))
g.set_soft(_lib.SOFT_SQUARE_INVERSE_CORE, 1.0, 1.2, True)
for only in (True, False, True):
    k = kernels(lambda: g.sweep(0.1, 0.1, seed=3, counter=0, fp64_only=only))
    assert "k_soft_sweep" in k or not only
    assert "k_soft_sweep" not in k or lib.fake_soft_fp64_only() == only
""")


CONVEX = 'GpuPacking(W.CONVEX, "cuboid 1 1 2; sphere 0.1; sum", W.lattice(({0}, {0}, {0}), ({1},) * 3), W.aligned_rotations({0} ** 3),' \
         ' W.diag_box({0} * {1}, {0} * {1}, {0} * {1}))'


@pytest.mark.parametrize("side,cell,counting,warps", [(6, 2.8, False, 1), (6, 2.8, True, 8), (6, 1.1, False, 8)])
def test_warps_of_a_convex_single_move(fake, side, cell, counting, warps):
    run(fake, f"""
g = {CONVEX.format(side, cell)}
g.set_counting({counting})
assert "k_try_singleILi3ELi{warps}E" in kernels(lambda: fails("", -1, lambda: g.try_move(0, 0, (0.1, 0.0, 0.0))))
""")


@pytest.mark.parametrize("shape,fp64_only,cluster", [
    ("spheres()", False, True), ("spheres()", True, True),
    ('GpuPacking(W.POLYSPHEROCYLINDER, W.polyspherocylinder_params(W.BENT_ROD), W.lattice((5, 5, 5), (2.0,) * 3),'
     ' W.aligned_rotations(125), W.diag_box(10.0, 10.0, 10.0))', False, True),
    ('GpuPacking(W.POLYSPHEROCYLINDER, W.polyspherocylinder_params(W.BENT_ROD), W.lattice((5, 5, 5), (2.0,) * 3),'
     ' W.aligned_rotations(125), W.diag_box(10.0, 10.0, 10.0))', True, False)])
def test_small_sweeps_in_fp64_alone_spread_multi_centre_bodies_over_the_chip(fake, shape, fp64_only, cluster):
    run(fake, f"""
g = {shape}
assert ("k_cluster_sweep" in kernels(lambda: g.sweep(0.1, 0.1, seed=1, counter=0, fp64_only={fp64_only}))) == {cluster}
""")
