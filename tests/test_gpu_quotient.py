"""The FP64 step's branch-free reciprocals, quotients and square roots (rcp_rn,
quot_rn, sqrt_nr in lattice.cuh) against the division and sqrt() on 2^28
operand pairs: every result the same bits, the hardware's approximation within the 2^-19 that the Newton steps
assume (tests/native/quotient_check.cu)."""
import os
import re
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))


def test_quotients_round_like_the_division(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    exe = tmp_path / "quotient_check"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17",
                    "--expt-relaxed-constexpr", "-I", os.path.join(ROOT, "cfd_cavity_b200", "csrc"),
                    os.path.join(ROOT, "tests", "native", "quotient_check.cu"), "-o", str(exe)],
                   check=True, capture_output=True, timeout=300)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    m = re.search(r"err (\d+) reciprocals (\d+) quotients (\d+) approx (\d+) infinite (\d+) roots (\d+)", r.stdout)
    assert r.returncode == 0 and m, r.stdout + r.stderr
    assert [int(x) for x in m.groups()][:3] == [0, 0, 0], r.stdout
    assert int(m.group(4)) <= 1 and int(m.group(5)) == 0 and int(m.group(6)) == 0, r.stdout
