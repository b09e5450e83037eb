"""Part1+2 sorts the levels of a column (with a hydrometeor, near ice
nucleation, neither) and evaluates saturation only where it is read; and
the kernels have launch shapes of their own for calls that fill the GPU and
for calls that leave most of it idle.  Both are checked where the choice
changes."""
import numpy as np
import pytest

from conftest import oracle_state, rel_l2

pytestmark = pytest.mark.gpu
DT = 300.0
CCN = {"prescribed": (True, True), "predicted": (True, False), "fixed": (False, False)}
# temperatures around the classes' limits (150 K, the nucleation threshold
# Tmelt - 15, Tmelt) and supersaturations over ice around -0.05 (the early
# exit), 0.05 (nucleation) and the margins of the FP32 estimate
TEMPS = [149.5, 150.5, 200.0, 230.0, 258.1, 258.149, 258.2, 258.3, 273.1, 273.2]
SS = [-0.4, -0.0515, -0.0505, -0.05 - 1e-9, -0.05 + 1e-9, -0.0495, -0.0485, 0.0, 0.0485, 0.0495, 0.05 - 1e-9,
      0.05 + 1e-9, 0.06, 0.5]


def svp_ice(t):
    return np.exp(9.550426 - 5723.265 / t + 3.53068 * np.log(t) - 0.00728332 * t)


def dry_columns(extra_qi=0.0):
    """One column per (temperature, supersaturation): level 1 of 5 holds the
    pair, the others are warm and dry, so that the pair alone decides."""
    import scream_gb300 as p3
    T, ss = (a.ravel() for a in np.meshgrid(TEMPS, SS, indexing="ij"))
    inp = {k: v for k, v in p3.generate_inputs(0, 5, T.size, 5).items()}
    for n in ("qc", "nc", "qr", "nr", "qi", "qm", "ni", "bm"):
        inp[n][:] = 0.0
    p = 30000.0
    inp["pres"][:] = p
    inp["inv_exner"][:] = 1.0
    inp["th"][:] = 290.0
    inp["th"][:, 1] = T
    inp["qv"][:] = 1e-4
    inp["qv"][:, 1] = (1.0 + ss) * (18.016 / 28.966) * svp_ice(T) / p
    inp["qi"][:, 1] = extra_qi
    inp["qv_prev"][:], inp["t_prev"][:] = inp["qv"], inp["th"]
    return inp, ss


@pytest.mark.parametrize("ccn", sorted(CCN))
@pytest.mark.parametrize("qi", [0.0, 3e-15, 2e-14], ids=["dry", "below qsmall", "above qsmall"])
def test_dry_levels_at_the_class_limits(gpu_ctx, tables, ccn, qi):
    """FP64 part1+2 against the oracle's, and the FP32-bulk form away from the
    thresholds by more than FP32 resolves."""
    import scream_gb300 as p3
    from oracle import p3_oracle as O
    predict, prescribed = CCN[ccn]
    inp, ss = dry_columns(qi)
    inp["ni_activated"][:] = 1e4
    o = oracle_state(inp)
    err, rows, cflag = O.p3_main_part12(o, tables, DT, predictNc=predict, prescribedCCN=prescribed)
    assert err == 0
    ncol, nlev = inp["qc"].shape
    for prec in (p3.P3X_FP64, p3.P3X_FP32_BULK):
        f = p3.P3Fields.from_inputs(inp)
        ho = gpu_ctx.allocate_handover(ncol, nlev)
        gpu_ctx.p3_main_stages(f, DT, p3.P3X_STAGE_PART12, ho, prec, predictNc=predict, prescribedCCN=prescribed)
        g = f.to_host()
        g_rows, g_cf = (x.cpu().numpy() for x in gpu_ctx.handover_views(ho, ncol, nlev))
        sure = np.ones(ncol, bool) if prec == p3.P3X_FP64 else (np.abs(ss + 0.05) > 1e-6) & (np.abs(ss - 0.05) > 1e-6)
        np.testing.assert_array_equal(g_cf[sure], cflag[sure])
        for n in ("qi", "ni", "qv", "th", "qm", "bm", "qc", "qr", "qv2qi_depos_tend", "vap_ice_exchange"):
            # FP64: round-off; FP32-bulk: a tendency of a few FP32 operations
            bound = 1e-10 if prec == p3.P3X_FP64 else 1e-5
            assert rel_l2(g[n][sure], o[n][sure]) <= bound, (prec, n, rel_l2(g[n][sure], o[n][sure]))
        if prec == p3.P3X_FP64:
            on = cflag == 1
            for h in range(5):
                assert rel_l2(g_rows[h][on], rows[h][on]) <= 1e-12, h


@pytest.mark.parametrize("precision", ["fp64", "bulk"])
@pytest.mark.parametrize("nlev", [1, 31, 32, 33, 72, 128, 129, 164, 170, 257])
def test_launch_shapes_agree(gpu_ctx, nlev, precision):
    """A call that fills every SM with columns (FP32-bulk sedimentation: tables
    in shared memory, where the columns leave room) against the same columns
    in smaller calls, the smallest of which share a column's levels among
    warps: columns are independent, so every field is bitwise the same."""
    import torch
    import scream_gb300 as p3
    prec = p3.P3X_FP64 if precision == "fp64" else p3.P3X_FP32_BULK
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = 20 * sms + 3
    half = 10 * sms
    inp = p3.generate_inputs(0, 77, n, nlev)
    whole = p3.P3Fields.from_inputs(inp)
    gpu_ctx.p3_main(whole, DT, prec)
    whole = whole.to_host()
    for a, b in ((0, 1), (1, 8), (8, 2 * sms), (2 * sms, half), (half, n)):
        part = p3.P3Fields.from_inputs({k: np.ascontiguousarray(v[a:b]) for k, v in inp.items()})
        gpu_ctx.p3_main(part, DT, prec)
        for k, v in part.to_host().items():
            np.testing.assert_array_equal(v, whole[k][a:b], err_msg=f"{k} {a}:{b}")
