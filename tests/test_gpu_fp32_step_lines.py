"""FP32's step kernel on both sides of each line of its rule (one node per thread,
the same with its loads in rounds, node pairs): narrow grids whose pairs would lie
beyond the wall, pairs in one wave and just past it.  Same bits as the one-node
batch kernel; odd sizes; the per-step Nusselt sums of the rounds form."""
import numpy as np
import pytest

from cfd_cavity_b200 import CavityBatch, CavitySolver
from cfd_cavity_b200 import _lib as L

pytestmark = pytest.mark.gpu

# 148 SMs: one-node CTAs (32 x 4) of 444 | 445 .. 666 | 667 ..; pairs (64 x 2) 1480; one-node 1924
SIZES = [(128, 444), (129, 356), (193, 377), (96, 888), (97, 667), (33, 1336),  # rounds
         (31, 2700), (32, 2701), (95, 891), (65, 893),                          # one node: 1 or 3 columns of 32
         (255, 739), (256, 741), (511, 479), (512, 482)]                        # the pairs' wave, level again


@pytest.mark.parametrize("nx,ny", SIZES)
def test_each_side_of_a_line_gives_the_same_bits(nx, ny):
    args = dict(nx=nx, ny=ny, ra=1e6, cs=0.11, seed=9)
    s = CavitySolver(nx, ny, 1e6, 0.71, 0.11, 0.9, 0.02, 9, precision="f32", init_mode=L.CAV_INIT_ZERO, noise_amp=1e-4)
    b = CavityBatch([args], precision="f32")
    b.set_tuning(4, 8, kernel=3)
    for n in (1, 12):
        s.step(n)
        b.step(n)
    for p, q in zip(s.populations(), b.populations(0)):
        np.testing.assert_array_equal(p, q)
    fs, fb = s.fields(), b.fields(0)
    for k in fs:
        np.testing.assert_array_equal(fs[k], fb[k])


def test_nusselt_sums_of_the_rounds_form():
    nx, ny = 129, 357
    s, t = (CavitySolver(nx, ny, 1e6, 0.71, 0.1, 0.9, 0.02, 3, precision="f32") for _ in range(2))
    s.step(5)
    t.step(5)
    s.nu_accumulate(True)
    s.step(6)
    hot, cold, n = s.nu_accumulated()
    assert n == 6
    want = np.zeros(2)
    for _ in range(6):
        t.step(1)
        p = t.temperature.reshape(ny, nx)
        want += [np.abs(p[:, 1] - p[:, 2]).mean(), np.abs(p[:, -2] - p[:, -3]).mean()]
    # FP64 sums of the same FP32 temperatures, in another order
    assert np.allclose([hot, cold], want / 6 * (ny - 1), rtol=1e-12, atol=0)


@pytest.mark.parametrize("nx,ny", [(129, 356), (255, 739)])  # rounds, pairs
def test_one_node_per_thread_when_the_caller_sets_it(nx, ny):
    s, t = (CavitySolver(nx, ny, 1e6, 0.71, 0.1, 0.9, 0.02, 3, precision="f32") for _ in range(2))
    s.step(280)  # past the ramp: graphs of the rule's kernel
    s.set_step_kernel(L.CAV_STEP_NODE)
    assert s.step_kernel() == L.CAV_STEP_NODE
    s.step(90)
    t.step(370)
    for p, q in zip(s.populations(), t.populations()):
        np.testing.assert_array_equal(p, q)
