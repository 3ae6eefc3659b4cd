"""The FP64 step's branch-free quotients where their remainder is no number: an
infinite, zero or NaN operand (tests/native/quotient_edges.cu), and the calls
that reach it -- an infinite turbulent Prandtl number, which switches the
subgrid heat flux off (nu_t / Pr_t = 0)."""
import os
import shutil
import subprocess

import numpy as np
import pytest

import oracle
from cfd_cavity_b200 import CavityBatch, CavitySolver
from cfd_cavity_b200.octree import OctreeSolver

pytestmark = pytest.mark.gpu

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))
INF = float("inf")


def test_zero_infinite_and_nan_operands(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    exe = tmp_path / "quotient_edges"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17",
                    "--expt-relaxed-constexpr", "-I", os.path.join(ROOT, "cfd_cavity_b200", "csrc"),
                    os.path.join(ROOT, "tests", "native", "quotient_edges.cu"), "-o", str(exe)],
                   check=True, capture_output=True, timeout=300)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "err 0 differing 0" in r.stdout, r.stdout + r.stderr


# 128 x 445 takes the 128-register build of the step
@pytest.mark.parametrize("nx,ny,steps", [(16, 40, 120), (33, 70, 90), (128, 445, 12)])
def test_uniform_infinite_turbulent_prandtl_number(nx, ny, steps):
    args = (nx, ny, 1.0e5, 0.71, 0.12, INF, 0.02, 42)
    g, o = CavitySolver(*args, precision="f64"), oracle.OracleSolver(*args)
    g.step(steps)
    o.step(steps)
    fg, fo = g.fields(), o.fields()
    for k in ("rho", "ux", "uy", "temperature", "nu_t"):
        np.testing.assert_array_equal(fg[k], fo[k], err_msg=k)
    for pg, po in zip(g.populations(), o.populations()):
        np.testing.assert_array_equal(pg, po)
    assert g.diag()["finite"] == 1


@pytest.mark.parametrize("kernel", [0, 2, 3])
def test_batch_infinite_turbulent_prandtl_number(kernel):
    sizes = [(16, 40), (37, 61)]
    b = CavityBatch([dict(nx=nx, ny=ny, ra=1e5, cs=0.12, seed=5) for nx, ny in sizes], precision="f64", pr_t=INF)
    b.set_tuning(4, 3, kernel=kernel)
    b.step(90)
    for i, (nx, ny) in enumerate(sizes):
        o = oracle.OracleSolver(nx, ny, 1e5, 0.71, 0.12, INF, 0.02, 5, init_mode=oracle.INIT_ZERO, noise_amp=1e-4)
        o.step(90)
        for pb, po in zip(b.populations(i), o.populations()):
            np.testing.assert_array_equal(pb, po)


@pytest.mark.parametrize("precision", ["f64", "f32"])
def test_octree_infinite_turbulent_prandtl_number(precision):
    """With the fixed-Cs model on the levels: nu_t / 1e300 is lost beside alpha, so
    that run has the bits an infinite number must give."""
    a, b = (OctreeSolver(32, 64, 4, 1.0e6, 0.71, 0.02, 42, levels=3, precision=precision, cs=0.1, pr_t=pr_t)
            for pr_t in (INF, 1e300 if precision == "f64" else 1e30))
    a.step_cavity(20)
    b.step_cavity(20)
    for lvl in range(5):
        la, lb = a.level(lvl, pops=True), b.level(lvl, pops=True)
        for k in ("rho", "ux", "uy", "temp", "f", "g"):
            assert np.isfinite(la[k]).all()
            np.testing.assert_array_equal(la[k], lb[k], err_msg="level %d %s" % (lvl, k))
