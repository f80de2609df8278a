"""The paired arithmetic of csrc/exact_pair.cuh against sqrtf, IEEE division and scalar rounding, bit for bit, and
steps at the ends of the radius range that uses it."""
import os
import subprocess

import pytest

from novaphy_gb300 import _build
from test_gpu_walk_forms import block, check

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def counts(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("pair") / "exact_pair_check")
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "exact_pair_check.cu")
    subprocess.run([_build.nvcc(), *_build.NVCC_COMMON, *_build.CU_FLAGS["pbf_exact.cu"], src, "-o", exe],
                   check=True, capture_output=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    print(out)
    return {name: (int(n), int(wrong)) for name, n, wrong in (line.split() for line in out.splitlines())}


@pytest.mark.parametrize("name", ["roots", "quotients_of_inexact_inverses", "quotients", "sums"])
def test_rounding(counts, name):
    assert counts[name][0] > 0 and counts[name][1] == 0, counts


def test_few_inverses_are_an_ulp_off(counts):
    # Two significands of the root are, in each octave; every dividend is checked with each of them.
    assert counts["inverses"][1] < 1 << 20, counts


# h = 1e-3 and 100, the ends of the range, and one float outside on either side.
@pytest.mark.parametrize("n", [3000, 140000])
@pytest.mark.parametrize("r", [0.00025, 0.000249999, 25.0, 25.00001])
def test_ends_of_the_radius_range(port_mt, n, r):
    check(port_mt, block(n, seed=13, r=r, vorticity=1e-4), 1)
