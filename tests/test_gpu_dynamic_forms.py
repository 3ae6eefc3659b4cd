"""The dynamic model's forms against the FP64 oracle: the unrolled two-node
test filter (eta 2, fused kernels in the uniform solver) and the general one
(eta 1, 3), the square-root form of the mixed powers (alpha 1/2) and the general
one, on odd and ragged grids, over launches and graph replays of 16 steps.

Tolerances as in test_gpu_dynamic.py: the powers differ from the C library's
by at most a few ulp (CUDA's pow, or one square root of the product), which 40
steps leave below a relative 1e-10."""
import numpy as np
import pytest

import oracle
from cfd_cavity_b200 import CavitySolver
from cfd_cavity_b200.octree import OctreeSolver

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.max(np.abs(a - b)) / max(np.max(np.abs(b)), 1e-300)


@pytest.mark.parametrize("nx,ny,alpha,eta", [(16, 40, 0.5, 2.0), (33, 67, 0.3, 2.0), (31, 66, 0.5, 1.0),
                                             (17, 41, 0.5, 3.0), (35, 50, 1.0, 3.4), (32, 49, 0.0, 2.0), (5, 9, 0.5, 2.0)])
def test_uniform_forms_match_the_oracle(nx, ny, alpha, eta):
    args = (nx, ny, 1.0e5 if ny > 20 else 1.0e3, 0.71, 0.1, 0.9, 0.02, 42)
    g, o = CavitySolver(*args, precision="f64"), oracle.OracleSolver(*args)
    for s in (g, o):
        s.set_dynamic_sgs(True, alpha, -0.1, eta)
        s.step(40)
    fg, fo = g.fields(), o.fields()
    for k in ("rho", "ux", "uy", "temperature", "nu_t"):
        assert rel(fg[k], fo[k]) <= 1e-10, (k, rel(fg[k], fo[k]))


def test_uniform_graph_replays_equal_single_steps():
    """Past the 200-step ramp, 16 steps replay as one graph; the per-step Nu
    sums and the model's constants changed on the way included."""
    args = (33, 70, 1.0e5, 0.71, 0.1, 0.9, 0.02, 5)
    a, b = (CavitySolver(*args, precision="f16sr") for _ in range(2))
    for s in (a, b):
        s.set_dynamic_sgs(True)
    a.step(190)
    b.step(190)
    for s in (a, b):
        s.nu_accumulate(True)
    a.step(61)
    for _ in range(61):
        b.step(1)
    assert a.nu_accumulated() == b.nu_accumulated()
    for s in (a, b):
        s.set_dynamic_sgs(True, 0.4, -0.05, 2.0)
    a.step(37)
    for _ in range(37):
        b.step(1)
    fa, fb = a.fields(), b.fields()
    for k in fa:
        np.testing.assert_array_equal(fa[k], fb[k])
    np.testing.assert_array_equal(a.populations()[0], b.populations()[0])


@pytest.mark.parametrize("alpha,eta", [(0.5, 3.0), (0.3, 2.0)])
def test_octree_forms_match_the_oracle(alpha, eta):
    args = (24, 48, 4, 1.0e6, 0.71, 0.02, 3)
    g = OctreeSolver(*args, levels=3, precision="f64")
    o = oracle.OracleOctree(*args, levels=3)
    for s in (g, o):
        s.set_dynamic_sgs(True, alpha, -0.1, eta)
        s.step_cavity(20)
    for lvl in range(5):
        lg, lo = g.level(lvl), o.level(lvl)
        for k in ("rho", "ux", "uy", "temp"):
            assert np.max(np.abs(lg[k] - lo[k])) <= 1e-11, (lvl, k)


def test_octree_graphs_equal_single_steps():
    """A replayed graph of 16 coarse steps advances the step index once; the
    stochastic rounding follows it step by step."""
    a, b = (OctreeSolver(24, 60, 4, 1e6, 0.71, 0.02, 3, levels=3, precision="f32_f16") for _ in range(2))
    a.step_cavity(37)
    for _ in range(37):
        b.step_cavity(1)
    for lvl in range(5):
        la, lb = a.level(lvl, pops=True), b.level(lvl, pops=True)
        for k in ("rho", "ux", "uy", "temp", "f", "g"):
            np.testing.assert_array_equal(la[k], lb[k])
