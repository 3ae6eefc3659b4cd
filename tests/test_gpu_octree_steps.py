"""Inside a call the octree's L0 steps write the reference state and the moments
only where the couplings read them, and past the viscosity ramp the level
steps take their constants with the launch.  Both must leave what a caller
sees unchanged: the state after any call length equals that of single steps
(whose every step is a call's last), with and without a ramp, over launches
and both kinds of graphs, and stays so when diagnostics, couplings and
restarts come in between."""
import numpy as np
import pytest

from cfd_cavity_b200.octree import OctreeSolver

pytestmark = pytest.mark.gpu


def same(a, b, levels):
    for lvl in range(3 if levels == 2 else 5):
        la, lb = a.level(lvl, pops=True), b.level(lvl, pops=True)
        for k in ("rho", "ux", "uy", "temp", "f", "g"):
            np.testing.assert_array_equal(la[k], lb[k], err_msg="level %d %s" % (lvl, k))


@pytest.mark.parametrize("precision,levels,ramp,size", [
    ("f64", 2, 1.0, (24, 61, 3)), ("f32", 3, 1.0, (33, 64, 5)), ("f32_f16", 3, 1.05, (25, 60, 4)),
    ("f32_f16g", 2, 1.0, (40, 50, 2)), ("f64", 3, 1.02, (20, 40, 9))])
def test_call_lengths_do_not_change_the_state(precision, levels, ramp, size):
    args = (*size, 1e5, 0.71, 0.02, 3)
    a, b = (OctreeSolver(*args, levels=levels, precision=precision, nu_start_mult=ramp) for _ in range(2))
    for n in (1, 16, 5, 37):
        a.step_cavity(n)
        for _ in range(n):
            b.step_cavity(1)
        same(a, b, levels)
        assert a.diag() == b.diag()
    for s in (a, b):
        s.couple(0)
        s.couple(1)
    a.step_cavity(18)
    for _ in range(18):
        b.step_cavity(1)
    same(a, b, levels)


def test_steps_across_the_end_of_the_ramp():
    """The ramp's constants converge bit for bit some 40 000 steps in (2000 for
    the buoyancy): from a set time step just before, graphs and launches with
    the table's constants and with the steady ones give one trajectory."""
    args = (24, 60, 4, 1e5, 0.71, 0.02, 3)
    a, b = (OctreeSolver(*args, levels=3, precision="f32", nu_start_mult=2.0) for _ in range(2))
    for s in (a, b):
        s.set_time_step(36_000)
    n = 1500
    a.step_cavity(n)
    for _ in range(n // 10):
        b.step_cavity(10)
    same(a, b, 3)
