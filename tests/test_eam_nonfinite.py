"""EAM's use of the P3 results where a field holds an infinity or a NaN of
either sign (components/eam/src/physics/p3/scream/micro_p3_interface.F90:
1182-1431): every threshold, maximum and minimum is an IEEE comparison, so a
NaN passes no threshold.  The comparisons themselves run on the host too."""
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parent.parent / "scream_gb300" / "csrc"
ODD = np.array([0x7ff8000000000000, 0xfff8000000000000, 0x7fffffffffffffff, 0xffffffffffffffff, 0x7ff0000000000000,
                0xfff0000000000000, 0x8000000000000000, 0, 1, 0x8000000000000001], dtype=np.uint64).view(np.float64)

COMPARE = r"""
#include <cstdio>
#include <limits>
#include <random>
#include "p3x_intfp64.cuh"
using namespace p3x::dev;
int main() {
  std::mt19937_64 g(5);
  const uint64_t odd[] = {ODD};
  const double limits[] = {1e-14, 1e-7, 1e-6, 5e-5, 1e-4, 0.005, 0.01, 1.0, 4.9e-324, 1.7e308};
  long bad = 0;
  for (double c : limits)
    for (long i = 0; i < 200000; ++i) {
      uint64_t u = g();
      if (i % 4 == 1) u = odd[g() % (sizeof(odd) / 8)];
      if (i % 4 == 2) u = d_bits(c) + g() % 5 - 2;
      if (i % 4 == 3) u = (d_bits(c) + g() % 5 - 2) ^ kSignPattern;
      const double x = d_from_bits(u);
      bad += ieee_gt(x, c) != (x > c);
      bad += ieee_ge(x, c) != (x >= c);
      bad += ieee_lt(x, c) != (x < c);
      bad += ieee_neg(x) != (x < 0);
    }
  std::printf("%ld\n", bad);
}
"""


def test_integer_comparisons_are_ieee_comparisons(tmp_path):
    src = tmp_path / "compare.cpp"
    src.write_text(COMPARE.replace("ODD", ", ".join(f"{u:#x}ull" for u in ODD.view(np.uint64))))
    subprocess.run(["g++", "-std=c++17", "-O2", f"-I{CSRC}", str(src), "-o", str(tmp_path / "compare")], check=True)
    assert int(subprocess.run([str(tmp_path / "compare")], capture_output=True, text=True, check=True).stdout) == 0


def literal_post(e, f, dt):
    """The outputs that thresholds decide, each comparison as written."""
    from oracle import eam_driver as E
    def top(a, b): return np.where(a > b, a, b)
    def low(a, b): return np.where(a < b, a, b)
    w = {s: f[E.P3_NAME[s]] * (e["pdeldry"] / e["pdel"]) for s in E.SPECIES}
    cl, ci, cr, pmid, t = f["cld_frac_l"], f["cld_frac_i"], f["cld_frac_r"], e["pmid"], e["t"]
    out = {"ptend_" + s: (top(0.0, w[s]) - e[s]) / dt for s in E.SPECIES}
    out["icimrst"] = low(e["cldice"] / top(E.MINCLD, ci), 0.005)
    out["icwmrst"] = low(e["cldliq"] / top(E.MINCLD, cl), 0.005)
    out["icinc"] = e["numice"] / top(E.MINCLD, ci) * pmid / (287.15 * t)
    out["icwnc"] = e["numliq"] / top(E.MINCLD, cl) * pmid / (287.15 * t)
    clear = e["ast"] < 1e-4
    out["mu"] = np.where(clear, E.MUCON, 0.0)
    out["dei"] = np.where(clear, E.DEICON, f["diag_eff_radius_qi"] * 1e6 * 2.0)
    tot = w["rain"] + w["cldice"] + w["cldliq"]
    out["nfice"] = np.where((w["cldice"] > E.QSMALL) & (tot > E.QSMALL), low(w["cldice"] / tot, 1.0), 0.0)
    liq = (cl > 0.01) & (out["icwmrst"] > 5e-5)
    ice = (ci > 0.01) & (out["icimrst"] > 1e-6)
    out["freql"], out["ncout"] = np.where(liq, cl, 0.0), np.where(liq, out["icwnc"] * cl, 0.0)
    out["freqi"], out["niout"] = np.where(ice, ci, 0.0), np.where(ice, out["icinc"] * ci, 0.0)
    out["efcout"] = np.where(liq, f["diag_eff_radius_qc"] * 1e6 * cl, 0.0)
    out["efiout"] = np.where(ice, f["diag_eff_radius_qi"] * 1e6 * ci, 0.0)
    rain = w["rain"] >= 1e-7
    out["freqr"], out["aqrain"] = np.where(rain, cr, 0.0), np.where(rain, w["rain"] * cr, 0.0)
    out["anrain"] = np.where(rain, w["numrain"] * cr, 0.0)
    out["reff_rain"] = np.where(rain, f["diag_eff_radius_qr"] * 1e6, f["diag_eff_radius_qr"])
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["qi", "qr", "qc", "qv", "cld_frac_l", "cld_frac_i", "cld_frac_r", "ast", "cldice",
                                  "cldliq"])
def test_device_post_with_nonfinite_values(gpu_ctx, name):
    """`name`: the P3 result or the EAM state field that holds the odd values."""
    import torch
    import scream_gb300 as p3
    from oracle import eam_driver as E
    from test_eam_driver import NCOL, NLEV, DT, _alloc_outputs, _device_state, eam_case
    inp, e = eam_case(1009)
    f = p3.P3Fields.from_inputs(inp)
    pre = E.eam_pre(e)
    rng = np.random.default_rng(3)
    for n in ("qc", "qr", "qi"):  # condensate on every level, so that the thresholds pass on most
        pre[n] = 10.0 ** rng.uniform(-9, -3, pre[n].shape)
    for n in ("cldice", "cldliq"):
        e[n] = 10.0 ** rng.uniform(-7, -3, e[n].shape)
    for n in ("cld_frac_l", "cld_frac_i", "cld_frac_r"):
        pre[n] = rng.uniform(0.005, 1.0, pre[n].shape)
    for n in ("diag_eff_radius_qc", "diag_eff_radius_qi", "diag_eff_radius_qr"):
        pre[n] = rng.uniform(1e-6, 1e-4, pre["qc"].shape)
    at = (e if name in e and name not in ("qv",) else pre)[name]
    at.flat[5::7] = np.resize(ODD, at.flat[5::7].size)
    for n, v in pre.items():
        f.t[n].copy_(torch.from_numpy(np.ascontiguousarray(v)))
    eam = _device_state(e, torch)
    _alloc_outputs(eam, NCOL, NLEV, torch)
    gpu_ctx.eam_tend_post(eam, f, DT)
    torch.cuda.synchronize()
    with np.errstate(all="ignore"):
        want = literal_post(e, pre, DT)
    for n, w in want.items():
        np.testing.assert_array_equal(eam[n].cpu().numpy(), w, err_msg=n)
