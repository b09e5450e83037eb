"""A work list's order decides how part1+2 pools its columns and nothing else:
lists whose items are not an instance's columns in a row give the same bits as one
call per instance.  The library's own lists are in a row, so this calls its
internal launch with lists of other orders."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
DT = 300.0
LAUNCH_WORK = "_ZN3p3x11launch_workEP11p3x_contextRK11p3x_runtimeiPKNS_3dev4InstEPKNS5_8WorkItemEiiPjP11CUstream_std"
FIELDS = ["qc", "nc", "qr", "nr", "qi", "qm", "ni", "bm", "qv", "th", "nc_nuceat_tend", "nccn", "ni_activated",
          "inv_qc_relvar", "cld_frac_i", "cld_frac_l", "cld_frac_r", "pres", "dz", "dpres", "inv_exner", "qv_prev",
          "t_prev", "qv2qi_depos_tend", "precip_liq_surf", "precip_ice_surf", "diag_eff_radius_qc",
          "diag_eff_radius_qi", "diag_eff_radius_qr", "rho_qi", "precip_liq_flux", "precip_ice_flux",
          "precip_total_tend", "nevapr", "liq_ice_exchange", "vap_liq_exchange", "vap_ice_exchange", "scr", "cflag"]
SIZES = [(311, 40), (7, 72), (402, 72), (1, 33), (260, 9)]


class Inst(C.Structure):
    _fields_ = ([(n, C.c_void_p) for n in FIELDS] +
                [("ld", C.c_int64), ("ld_int", C.c_int64), ("ncol", C.c_int32), ("nlev", C.c_int32), ("dt", C.c_double),
                 ("predictNc", C.c_int32), ("prescribedCCN", C.c_int32), ("precision", C.c_int32), ("pad_", C.c_int32)])


def order(kind):
    items = np.array([(i, c) for i, (n, _) in enumerate(SIZES) for c in range(n)], dtype=np.int32)
    rng = np.random.default_rng(17)
    if kind == "reversed":
        return items[::-1]
    if kind == "interleaved":
        return items[np.lexsort((items[:, 0], items[:, 1]))]
    if kind == "shuffled":
        return items[rng.permutation(len(items))]
    if kind == "shuffled runs":
        cut = np.sort(rng.choice(np.arange(1, len(items)), 200, replace=False))
        runs = np.split(items, cut)
        return np.concatenate([runs[i] for i in rng.permutation(len(runs))])
    return items


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("kind", ["in a row", "reversed", "interleaved", "shuffled", "shuffled runs"])
def test_any_order_gives_the_same_bits(gpu_ctx, precision, kind):
    import torch
    import scream_gb300 as p3
    from scream_gb300 import _lib as L
    fields = [p3.P3Fields.from_inputs(p3.generate_inputs(0, 60 + i, n, k)) for i, (n, k) in enumerate(SIZES)]
    keep, insts = [], (Inst * len(SIZES))()
    for f, (n, k), d in zip(fields, SIZES, insts):
        size = C.c_int64()
        assert gpu_ctx.lib.p3x_handover_bytes(n, k, C.byref(size)) == 0
        scr = torch.empty(size.value, dtype=torch.uint8, device="cuda")
        keep.append(scr)
        for name in FIELDS[:-2]:
            setattr(d, name, f.t[name].data_ptr())
        d.scr, d.cflag = scr.data_ptr(), scr.data_ptr() + 5 * n * k * 8
        d.ld, d.ld_int, d.ncol, d.nlev, d.dt = k, k + 1, n, k, DT
        d.predictNc = d.prescribedCCN = 1
        d.precision = precision
    insts_d = torch.frombuffer(bytearray(insts), dtype=torch.uint8).cuda()
    work_d = torch.from_numpy(np.ascontiguousarray(order(kind))).cuda()
    assert work_d.shape[0] == sum(n for n, _ in SIZES)
    launch = getattr(gpu_ctx.lib, LAUNCH_WORK)
    launch.argtypes = [C.c_void_p, C.c_void_p, C.c_int, C.c_void_p, C.c_void_p, C.c_int, C.c_int, C.c_void_p,
                       C.c_void_p, C.c_double]
    torch.cuda.synchronize()
    assert launch(gpu_ctx.h, C.byref(L.default_runtime()), precision, insts_d.data_ptr(), work_d.data_ptr(),
                  work_d.shape[0], max(k for _, k in SIZES), None, None, 1.0) == 0
    torch.cuda.synchronize()
    gpu_ctx.check()
    for i, (f, (n, k)) in enumerate(zip(fields, SIZES)):
        one = p3.P3Fields.from_inputs(p3.generate_inputs(0, 60 + i, n, k))
        gpu_ctx.p3_main(one, DT, precision)
        got = f.to_host()
        for name, v in one.to_host().items():
            np.testing.assert_array_equal(got[name], v, err_msg=f"{i} {name}")
