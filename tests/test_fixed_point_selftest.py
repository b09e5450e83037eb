"""The host's side of the self-test that compares the fixed-point functions of
the device with the host's, word for word (p3x_fixtest.hpp; p3x_selftest runs
both): its rows reach what they are meant to reach, and a high product that is
wrong in its last places changes them."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "scream_gb300" / "csrc"
PROGRAM = r"""
#include <cstdio>
#include <set>
#include "p3x_fixtables.hpp"
#include "p3x_fixtest.hpp"
using namespace p3x;
int main() {
  const auto w = fix_test_words(fix_test_coefficients());
  uint64_t sum = 0;
  for (uint64_t v : w) sum = sum * 6364136223846793005ull + v;
  std::set<uint64_t> cells, rows;
  bool below = false, above = false, odd = false;
  for (size_t i = 0; i < w.size(); i += kFixTestWords) {
    cells.insert(uint32_t(w[i + 7]));
    rows.insert(uint32_t(w[i + 19]));
    below |= int32_t(w[i + 19] >> 32) < 0;
    above |= int32_t(w[i + 19] >> 32) > 0;
    odd |= w[i + 7] >> 32;
  }
  std::printf("%llu %zu %zu %d %d %d\n", (unsigned long long)sum, cells.size(), rows.size(), below, above, odd);
}
"""


def run(tmp_path, header):
    d = tmp_path / "csrc"
    d.mkdir(exist_ok=True)
    for n in ("p3x_fixtables.cpp", "p3x_fixtables.hpp", "p3x_fixtables.inc", "p3x_fixtest.hpp", "p3x_internal.hpp"):
        (d / n).write_text((CSRC / n).read_text())
    (d / "p3x_intfp64.cuh").write_text(header)
    (d / "main.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O2", f"-I{d}", f"-I{ROOT / 'include'}", str(d / "main.cpp"),
                    str(d / "p3x_fixtables.cpp"), "-o", str(d / "main")], check=True)
    return list(map(int, subprocess.run([str(d / "main")], capture_output=True, text=True, check=True).stdout.split()))


def test_rows_cover_the_tables_and_notice_a_wrong_product(tmp_path):
    header = (CSRC / "p3x_intfp64.cuh").read_text()
    want = run(tmp_path, header)
    assert want[1] > 500 and want[2] > 70 and want[3:5] == [1, 1]
    right = "return acc + int64_t(ah) * bh + 2 * int64_t(mulhi_s32(ah, bl) + mulhi_s32(bh, al));"
    assert right in header
    assert run(tmp_path, header.replace(right, right.replace("mulhi_s32(bh, al)", "mulhi_s32(bh, al + 1)")))[0] != want[0]


@pytest.mark.gpu
def test_device_agrees_with_the_host(gpu_ctx):
    import ctypes as C
    n = C.c_uint64(1)
    assert gpu_ctx.lib.p3x_selftest(C.byref(n)) == 0
    assert n.value == 0
