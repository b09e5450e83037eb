"""FP64 operations on the integer pipes (scream_gb300/csrc/p3x_intfp64.cuh),
compiled for the host: the division is IEEE's, bit for bit, on every operand
family.  The device code is the same integer arithmetic with the hardware's
FP32 reciprocal as its seed; p3x_selftest compares it on the GPU."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
FAMILIES = ["ordinary", "edge significands", "exact quotients", "small integers", "any bits", "zero numerators",
            "quotients near the smallest normal", "quotients near one"]


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    exe = tmp_path_factory.mktemp("intfp64") / "check"
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", f"-I{ROOT / 'scream_gb300' / 'csrc'}",
                    str(ROOT / "tests" / "intfp64_check.cpp"), "-o", str(exe)], check=True)
    return exe


@pytest.mark.parametrize("family", range(len(FAMILIES)), ids=FAMILIES)
def test_integer_division_is_ieee_division(checker, family):
    out = subprocess.run([str(checker), str(family), "1000000"], capture_output=True, text=True, check=True).stdout
    assert int(out) == 0
