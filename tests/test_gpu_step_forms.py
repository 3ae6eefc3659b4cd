"""FP32 and FP64 pick their step kernel by the grid's size (one node per
thread, node pairs, pairs split over two warps; FP64 at full or at 128
registers).  Every form gives a node the same bits: a cavity stepped alone
equals the same cavity in a batch stepped by the one-node kernel (3) and, for
FP32, by the node-pair kernel (5), populations and fields, at sizes on both
sides of each line and with odd widths and heights."""
import numpy as np
import pytest

from cfd_cavity_b200 import CavityBatch, CavitySolver

pytestmark = pytest.mark.gpu

SIZES = {
    "f32": [(4, 4), (33, 70), (96, 499), (97, 496), (128, 512), (101, 694), (129, 543), (130, 640),
            (128, 546), (128, 547), (33, 1455), (33, 1500),
            (128, 443), (128, 445), (98, 470), (20, 1100)],
    "f64": [(5, 4), (31, 63), (64, 32), (64, 33), (64, 443), (128, 443), (128, 445), (65, 593), (97, 601)],
}


@pytest.mark.parametrize("precision,nx,ny", [(p, *s) for p in SIZES for s in SIZES[p]])
def test_forms_give_the_same_bits(precision, nx, ny):
    ra = 1e4 if ny < 50 else 1e6
    cfg = dict(nx=nx, ny=ny, ra=ra, cs=0.11, seed=9)
    alone = CavitySolver(nx, ny, ra, 0.71, 0.11, 0.9, 0.02, 9, precision=precision, init_mode=1, noise_amp=1e-4)
    alone.step(23)
    f, g = alone.populations()
    fields = alone.fields()
    for kernel in (3, 5):
        b = CavityBatch([cfg], precision=precision)
        b.set_tuning(4, 8, kernel=kernel)
        b.step(23)
        fb, gb = b.populations(0)
        np.testing.assert_array_equal(f, fb)
        np.testing.assert_array_equal(g, gb)
        other = b.fields(0)
        for k in fields:
            np.testing.assert_array_equal(fields[k], other[k])


@pytest.mark.parametrize("nx,ny", [(96, 499), (101, 499), (128, 600)])
def test_fp32_nusselt_accumulation_in_every_form(nx, ny):
    """The per-step Nu sums of a form that accumulates inside its step kernel
    equal the wall gradients of the fields read after every step."""
    s = CavitySolver(nx, ny, 1e6, 0.71, 0.1, 0.9, 0.02, 3, precision="f32")
    t = CavitySolver(nx, ny, 1e6, 0.71, 0.1, 0.9, 0.02, 3, precision="f32")
    s.step(5)
    t.step(5)
    s.nu_accumulate(True)
    s.step(7)
    hot, cold, n = s.nu_accumulated()
    assert n == 7
    want = np.zeros(2)
    for _ in range(7):
        t.step(1)
        p = t.temperature.reshape(ny, nx)
        want += [np.abs(p[:, 1] - p[:, 2]).mean(), np.abs(p[:, -2] - p[:, -3]).mean()]
    # FP64 sums of the same FP32 temperatures, in another order
    assert np.allclose([hot, cold], want / 7 * (ny - 1), rtol=1e-12, atol=0)
