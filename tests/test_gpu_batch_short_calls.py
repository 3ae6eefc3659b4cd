"""A call of a few steps advances a batch of any size with one launch per step
over all cavities, a longer one group of cavities by group where the kernel gains
from it; either gives the same bits, at the last length of one and the first of
the other, and in the graphs of a kernel that is never grouped."""
import numpy as np
import pytest

from cfd_cavity_b200 import CavityBatch

pytestmark = pytest.mark.gpu

# 150 MB in 16 bits, 290 MB in FP32
CFG = [dict(nx=nx, ny=ny, ra=1e6, cs=0.1, seed=7 + i) for i, (nx, ny) in enumerate(
    [(257, 1030), (64, 256), (255, 1024), (130, 514), (256, 1027), (33, 90), (512, 1024), (96, 384)])]
NEVER = 10**9
# format, kernel, the longest call that is one launch per step
LINES = [("f32", 0, 16), ("f32", 1, NEVER), ("f32", 2, 6), ("f32", 3, 2), ("f32", 4, 2), ("f32", 5, 2),
         ("f64", 3, 2), ("f64", 1, NEVER),
         ("f16", 0, 16), ("f16", 2, NEVER), ("f16", 3, NEVER), ("bf16", 4, 4), ("f16", 5, 2), ("f16", 6, NEVER)]


@pytest.mark.parametrize("precision,kernel,line", LINES)
def test_short_calls(precision, kernel, line):
    b = CavityBatch(CFG, precision=precision)
    b.set_tuning(4, 3, kernel=kernel)
    b.step(1)  # from the initial state: a collision per cavity
    done = 1
    for n in (1, 2, 3) if line == NEVER else (1, line, line + 1, 1):
        before = b.launch_count()
        b.step(n)
        done += n
        launches = b.launch_count() - before
        assert launches == n if n <= line else launches % n == 0 and launches > n, (n, launches)
    if line == NEVER:
        before = b.launch_count()
        b.step(130)  # 64 steps twice as a graph and two singly
        done += 130
        assert b.launch_count() - before == 130 + 2 + 1
    want = CavityBatch(CFG, precision=precision)
    want.set_tuning(4, 3, kernel=3)
    for n in (1, done - 2, 1):
        want.step(n)
    for i in range(len(CFG)):
        for p, q in zip(b.populations(i), want.populations(i)):
            np.testing.assert_array_equal(p, q)
        fb, fw = b.fields(i), want.fields(i)
        for k in fb:
            np.testing.assert_array_equal(fb[k], fw[k])
