"""The digit products by themselves (csrc/fp64tc.cu, tests/fp64tc_dev.cu, built with nvcc): every number
of digits, real and complex, K at and beside multiples of its blocks and of a read-out, split over
CTAs or not, tiles at their edges, against long double sums within the stated bound for that many
digits. Rows beyond the result and the other half stay as they are."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    from vecjac_gb300 import build
    out = str(tmp_path_factory.mktemp("fp64tc") / "fp64tc_dev")
    nvcc = build.nvcc()
    assert shutil.which(nvcc)
    r = subprocess.run([nvcc] + build.ARCH + ["-O2", "-std=c++17", "--fmad=false",
                                              "-I" + os.path.join(os.path.dirname(HERE), "include"),
                                              os.path.join(HERE, "fp64tc_dev.cu"), "-o", out],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return out


@pytest.mark.parametrize("kind", ["d", "z"])
@pytest.mark.parametrize("nd", [3, 4, 5, 6, 7, 8])
def test_products(exe, kind, nd):
    for k, n1, n2 in [(1, 1, 1), (31, 65, 63), (128, 128, 64), (129, 129, 65), (520, 40, 24), (1000, 130, 24)]:
        r = subprocess.run([exe, kind, str(nd), str(k), str(n1), str(n2), str(k + nd)], capture_output=True, text=True,
                           timeout=120)
        assert r.returncode == 0, r.stdout + r.stderr
        rows = [x.split() for x in r.stdout.splitlines()]
        assert len(rows) == 3
        for mode, worst, kept in rows:
            assert float(worst) <= 1.0 and kept == "1", (kind, nd, k, n1, n2, mode, worst, kept)
