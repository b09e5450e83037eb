"""FP64 operations on the integer pipes (scream_gb300/csrc/p3x_intfp64.cuh),
compiled for the host.  The device code is the same integer arithmetic (the
division's seed is the hardware's FP32 reciprocal there; p3x_selftest compares
it on the GPU).

Bounds.  Division: IEEE's result, bit for bit.  Functions, in units of 2^-52
of the result: one rounding (0.5) plus the error before it, 2^-57 of log2
through the power 0.54 (0.04, and its Q56 product 2^-56 ln 2 = 0.05) or the
cube root and the exponential (2^-58 and 2^-60), plus the check's own extended
precision; a log2 in Q57 is off by its last unit and 2^-57.  Ice table: the
coordinates' error, 2^-54, times the table's slope (neighbouring entries
within a factor of 8, three axes), the products' 28 units of a stored
coefficient's last place (2^-60 of the cell's largest), and one rounding.  Rain table: the
coordinate is at most 80 with a relative error of 2^-57, in Q53."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "scream_gb300" / "csrc"
FAMILIES = ["ordinary", "edge significands", "exact quotients", "small integers", "any bits", "zero numerators",
            "quotients near the smallest normal", "quotients near one"]
BOUND = {"log2": 2.0 ** -4, "exp2": 0.51, "cbrt": 0.53, "pow": 0.62, "fix": 0.5001, "ice": 2.0 ** -49, "rain": 2.0 ** -48}


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    exe = tmp_path_factory.mktemp("intfp64") / "check"
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", f"-I{CSRC}", f"-I{ROOT / 'include'}",
                    str(ROOT / "tests" / "intfp64_check.cpp"), str(CSRC / "p3x_fixtables.cpp"), "-o", str(exe)],
                   check=True)
    return lambda *a: float(subprocess.run([str(exe), *map(str, a)], capture_output=True, text=True, check=True).stdout)


@pytest.mark.parametrize("family", range(len(FAMILIES)), ids=FAMILIES)
def test_integer_division_is_ieee_division(checker, family):
    assert checker("div", family, 1000000) == 0


@pytest.mark.parametrize("family", range(3))
@pytest.mark.parametrize("what", sorted(BOUND))
def test_fixed_point_functions(checker, what, family):
    assert checker(what, family, 200000) <= BOUND[what]
