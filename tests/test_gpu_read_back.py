"""Fields of a large cavity read back into arrays whose pages have no memory yet
(populate_pages in solver.cuh): fresh, off the page grid, mapped from a file, with
memory already; the same values, and nothing written beside them."""
import mmap

import numpy as np
import pytest

from cfd_cavity_b200 import CavitySolver
from cfd_cavity_b200 import _lib as L

pytestmark = pytest.mark.gpu

NX, NY = 511, 701  # 2.9 MB a field, no whole number of pages
N = NX * NY
KEYS = ("rho", "ux", "uy", "temperature", "nu_t", "fy_node")


def read(s, arrays):
    s._ck(L.load().cav_get_fields(s._h, *[a.ctypes.data_as(L.load().cav_get_fields.argtypes[1]) for a in arrays]))


def test_fields_into_any_kind_of_array(tmp_path):
    s = CavitySolver(NX, NY, 1e6, 0.71, 0.1, 0.9, 0.02, 3, precision="f32")
    s.step(20)
    want = s.fields()
    resident = [np.zeros(N) for _ in KEYS]
    anonymous = mmap.mmap(-1, 8 * (N + 1024))
    fresh = np.frombuffer(anonymous, dtype=np.float64)
    guarded = np.full(N + 2, 7.5)
    with open(tmp_path / "field", "wb+") as fh:
        fh.truncate(8 * N)
        mapped = np.memmap(fh, dtype=np.float64, mode="r+", shape=N)
    cases = {
        "resident": resident,
        "fresh": [fresh[37:37 + N]] + resident[1:],  # neither end on a page
        "guarded": [resident[0], guarded[1:-1]] + resident[2:],
        "mapped": [mapped] + resident[1:],
    }
    for name, arrays in cases.items():
        read(s, arrays)
        for key, a in zip(KEYS, arrays):
            np.testing.assert_array_equal(a, want[key], err_msg=name + " " + key)
    assert not fresh[:37].any() and not fresh[37 + N:].any()
    assert guarded[0] == 7.5 and guarded[-1] == 7.5
