"""A batch larger than the L2 is stepped group of cavities by group: every
cavity still equals the same cavity alone, for calls of any length (single
launches, graph replays, remainders, the spin-up rows of the scalar table)
and whichever kernel runs, at the first and last cavity of a group."""
import numpy as np
import pytest

from cfd_cavity_b200 import CavityBatch, CavitySolver
from cfd_cavity_b200 import _lib as L

pytestmark = pytest.mark.gpu

# FP32: 148 B per node, f16: 76 B; groups hold 75 MB
CFG = [dict(nx=nx, ny=ny, ra=ra, cs=0.1, seed=70 + i) for i, (nx, ny, ra) in enumerate(
    [(257, 1030, 1e7), (64, 256, 1e6), (255, 1024, 1e7), (130, 514, 1e6), (256, 1027, 3e7), (33, 90, 1e5),
     (512, 1024, 1e7), (96, 384, 1e6)])]


@pytest.mark.parametrize("precision,kernels", [("f32", (3, 5, 0, 2)), ("f16", (6, 5, 1))])
def test_grouped_batch_equals_single_cavities(precision, kernels):
    b = CavityBatch(CFG, precision=precision)
    calls = (1, 90, 64, 2, 131)
    done = 0
    for j, n in enumerate(calls):
        b.set_tuning(4, 3, kernel=kernels[j % len(kernels)])
        b.step(n)
        done += n
    assert b.info()["time_step"] == done
    b.sync()
    for i, c in enumerate(CFG):
        s = CavitySolver(c["nx"], c["ny"], c["ra"], 0.71, c["cs"], 0.9, 0.02, c["seed"], precision=precision,
                         init_mode=L.CAV_INIT_ZERO, noise_amp=1e-4)
        s.step(done)
        fb, fs = b.fields(i), s.fields()
        for k in fb:
            np.testing.assert_array_equal(fb[k], fs[k])
        pb, ps = b.populations(i), s.populations()
        np.testing.assert_array_equal(pb[0], ps[0])
        np.testing.assert_array_equal(pb[1], ps[1])
        s.close()
