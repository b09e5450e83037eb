"""Performance cases of the P3 microphysics step and the interfaces around it.

Each case is one call (or the short sequence of calls) that a host model makes
per physics step, through the package's public entry points, on device data
unless the path works on host data:

  step       P3Context.p3_main on device fields (Functions::p3_main)
  process    P3Microphysics.run_process: preamble, step, postamble (EAMxx)
  interface  P3Context.preamble and P3Context.postamble by themselves
  eam        P3Context.eam_micro_p3_tend with every diagnostic (EAM's driver)
  batch      P3Batch.run: many instances of uneven size, as a CUDA graph
  host       P3Context.p3_main_host on page-locked host arrays

The step changes its state in place and the host model hands it a new one at
the next call, so every pass begins by copying the state in (one copy per set
of fields, as the dynamics or the other processes leave it) and then calls the
framework.  Columns are the seeded standard-atmosphere columns of the
package's own configurations: one cloud layer of 1-4 km with log-uniform
condensate, relative humidity U(0.3, 1.05), or U(0.9, 1.05) in every second
column ("moist").  `ccn` says how the cloud droplet number is treated:
"prescribed" (EAMxx's default), "predicted" (activation tendencies, EAM) or
"fixed".
"""
import math

import numpy as np
import torch

import scream_gb300 as p3
from scream_gb300 import _lib as L

DT = 300.0
PRECISION = {"fp64": p3.P3X_FP64, "bulk": p3.P3X_FP32_BULK}
CCN = {"prescribed": (True, True), "predicted": (True, False), "fixed": (False, False)}

RD, G, CP, P0 = 287.042, 9.80616, 1004.64, 100000.0
EP2 = 18.016 / 28.966
WET = ["qc", "nc", "qr", "nr", "qi", "qm", "ni", "bm", "qv"]  # the nine wet mixing ratios


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------
def listed():
    return [
        # a single-column model: one column, the caller reads the result of every step
        {"name": "column_1x72_fp64", "kind": "step", "ncol": 1, "nlev": 72, "precision": "fp64",
         "ccn": "prescribed", "moist": False, "wait": True},
        # the smallest configuration: a rank's handful of columns, FP64 and FP32-bulk
        {"name": "step_64x72_fp64", "kind": "step", "ncol": 64, "nlev": 72, "precision": "fp64",
         "ccn": "prescribed", "moist": False, "wait": False},
        {"name": "step_64x72_bulk", "kind": "step", "ncol": 64, "nlev": 72, "precision": "bulk",
         "ccn": "prescribed", "moist": False, "wait": False},
        # odd sizes: neither the columns nor the levels are a multiple of a warp; predicted droplets
        {"name": "step_1537x97_fp64", "kind": "step", "ncol": 1537, "nlev": 97, "precision": "fp64",
         "ccn": "predicted", "moist": False, "wait": False},
        # ne30 on one GPU at 128 levels, the plain FP64 form and the FP32-bulk form
        {"name": "step_21600x128_fp64", "kind": "step", "ncol": 21600, "nlev": 128, "precision": "fp64",
         "ccn": "prescribed", "moist": False, "wait": False},
        {"name": "step_21600x128_bulk", "kind": "step", "ncol": 21600, "nlev": 128, "precision": "bulk",
         "ccn": "prescribed", "moist": False, "wait": False},
        # the headline workload: ne120-sized, FP32-bulk, half the columns near saturation
        {"name": "step_345600x128_bulk", "kind": "step", "ncol": 345600, "nlev": 128, "precision": "bulk",
         "ccn": "prescribed", "moist": True, "wait": False},
        # one EAMxx atmosphere-process step: preamble, P3, postamble
        {"name": "process_21601x128_bulk", "kind": "process", "ncol": 21601, "nlev": 128, "precision": "bulk",
         "ccn": "prescribed", "moist": False},
        # the process interface by itself, as a host model that calls the step separately uses it
        {"name": "interface_65536x128", "kind": "interface", "ncol": 65536, "nlev": 128, "moist": False},
        # EAM's driver on an ne30 rank of a four-GPU node, with every diagnostic the physics buffer holds
        {"name": "eam_5400x72_fp64", "kind": "eam", "ncol": 5400, "nlev": 72, "precision": "fp64",
         "ccn": "predicted", "moist": False},
        # an ensemble: 256 instances of uneven size advanced by one captured graph
        {"name": "batch_256_bulk", "kind": "batch", "instances": 256, "max_ncol": 2048, "precision": "bulk",
         "ccn": "prescribed", "moist": False},
        # a host model whose state lives in host memory
        {"name": "host_21600x72_fp64", "kind": "host", "ncol": 21600, "nlev": 72, "precision": "fp64",
         "ccn": "prescribed", "moist": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "process", "interface", "eam", "batch", "host"])
    precision = rng.choice(["fp64", "bulk"])
    nlev = rng.choice([72, 128, rng.randint(33, 160)])
    case = {"kind": kind, "ccn": rng.choice(["prescribed", "predicted", "fixed"]), "moist": rng.random() < 0.5}
    if kind == "batch":
        most = 2048 if precision == "bulk" else 256
        return dict(case, instances=rng.randint(16, 256), max_ncol=_log(rng, 16, most), precision=precision)
    # most column-levels of a pass, so that none costs more than the largest listed case
    most = {"step": {"fp64": 2.2e6, "bulk": 3.0e7}[precision], "process": {"fp64": 2.0e6, "bulk": 1.0e7}[precision],
            "interface": 1.6e7, "eam": {"fp64": 1.8e6, "bulk": 4.0e6}[precision],
            "host": {"fp64": 1.6e6, "bulk": 3.0e6}[precision]}[kind]
    least = 256 if kind in ("interface", "host") else 1
    case.update(ncol=_log(rng, least, most / nlev), nlev=nlev)
    if kind == "interface":
        del case["ccn"]
        return case
    case["precision"] = precision
    if kind == "step":
        case["wait"] = rng.random() < 0.3
    return case


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
def _qsat_liq(T, p):
    logt = torch.log(T)
    e = torch.exp(54.842763 - 6763.22 / T - 4.210 * logt + 0.000367 * T +
                  torch.tanh(0.0415 * (T - 218.8)) * (53.878 - 1331.22 / T - 9.44523 * logt + 0.014025 * T))
    return EP2 * e / p


def _columns(ncol, nlev, moist, predicted, partial, seed, device="cuda"):
    """The 23 P3 inputs of seeded standard-atmosphere columns, (ncol, nlev) each.
    `partial`: cloud fractions below one inside the cloud."""
    g = torch.Generator(device=device)
    g.manual_seed(seed)

    def uni(lo, hi, *shape):
        return lo + (hi - lo) * torch.rand(*shape, generator=g, dtype=torch.float64, device=device)

    def normal(sd, *shape):
        return sd * torch.randn(*shape, generator=g, dtype=torch.float64, device=device)

    top = 200.0
    ps = P0 + normal(500.0, ncol, 1)
    eta = (torch.arange(nlev + 1, dtype=torch.float64, device=device) / nlev) ** 1.5
    pint = top + (P0 - top) * eta[None, :] + torch.clamp((eta - 0.2) / 0.8, min=0.0)[None, :] * (ps - P0)
    pint[:, 0] = top
    pint[:, nlev:] = ps
    pmid = 0.5 * (pint[:, :-1] + pint[:, 1:])
    dp = pint[:, 1:] - pint[:, :-1]
    Ts, lapse, T11 = 288.15, 6.5e-3, 216.65
    expo = G / (RD * lapse)
    p11 = ps * (T11 / Ts) ** expo
    z = torch.where(pmid >= p11, (Ts / lapse) * (1.0 - (pmid / ps) ** (1.0 / expo)),
                    11000.0 + (RD * T11 / G) * torch.log(p11 / pmid))
    T = torch.where(z <= 11000.0, Ts - lapse * z, torch.full_like(z, T11)) + normal(2.0, ncol, nlev)
    rh = uni(0.3, 1.05, ncol, nlev)
    if moist:
        rh[::2] = 0.9 + 0.15 * (rh[::2] - 0.3) / 0.75
    qv = rh * _qsat_liq(T, pmid)
    inv_exner = (P0 / pmid) ** (RD / CP)
    thick = uni(1000.0, 4000.0, ncol, 1)
    base = 1000.0 + (9000.0 - thick) * uni(0.0, 1.0, ncol, 1)
    cloudy = ((z >= base) & (z <= base + thick)).to(torch.float64)

    def condensate():
        return cloudy * 10.0 ** uni(-7.0, -3.0, ncol, nlev)

    f = {"qc": condensate(), "nc": cloudy * uni(5.0e7, 2.0e8, ncol, nlev),
         "qr": condensate(), "nr": cloudy * uni(1.0e3, 1.0e5, ncol, nlev),
         "qi": condensate(), "ni": cloudy * uni(1.0e3, 1.0e6, ncol, nlev)}
    f["qm"] = f["qi"] * uni(0.0, 0.5, ncol, nlev)
    f["bm"] = f["qm"] / uni(100.0, 900.0, ncol, nlev)
    f["qv"], f["th"] = qv, T * inv_exner
    f["nc_nuceat_tend"] = cloudy * uni(0.0, 1.0e4, ncol, nlev) if predicted else torch.zeros_like(T)
    f["nccn"] = torch.full_like(T, 1.0e8)
    f["ni_activated"] = torch.zeros_like(T)
    f["inv_qc_relvar"] = torch.ones_like(T)
    frac = cloudy * uni(0.2, 1.0, ncol, nlev) if partial else cloudy
    cl = torch.clamp(frac, min=1.0e-4)
    cr = cl.clone()
    cr[:, 1:] = torch.maximum(cr[:, 1:], frac[:, :-1])
    f["cld_frac_l"], f["cld_frac_i"], f["cld_frac_r"] = cl, cl.clone(), cr
    f["pres"], f["dpres"], f["inv_exner"] = pmid, dp, inv_exner
    f["dz"] = (RD / G) * dp * T * (1.0 + (1.0 / EP2 - 1.0) * qv) / pmid
    f["qv_prev"], f["t_prev"] = qv.clone(), T.clone()
    return f, {"cloud": frac, "T": T}


def _fields(inputs, device="cuda", host=False):
    """P3Fields of the inputs whose prognostic state is one block of memory, and
    that block's initial values."""
    ncol, nlev = inputs["qc"].shape
    kw = {"dtype": torch.float64, "pin_memory": True} if host else {"dtype": torch.float64, "device": device}
    f = p3.P3Fields(ncol, nlev)
    block = torch.empty(len(L.PROG_FIELDS), ncol, nlev, **kw)
    for i, n in enumerate(L.PROG_FIELDS):
        block[i].copy_(inputs.pop(n))
        f.t[n] = block[i]
    for n in L.DIAG_IN_FIELDS:
        f.t[n] = torch.empty(ncol, nlev, **kw)
        f.t[n].copy_(inputs.pop(n))
    for n in L.OUTPUT_FIELDS:
        shape = (ncol,) if n in L.SURFACE_FIELDS else (ncol, nlev + 1) if n in L.INTERFACE_FIELDS else (ncol, nlev)
        f.t[n] = torch.zeros(*shape, **kw)
    return f, block, block.clone()


_CONTEXT = []


def _context():
    """The lookup tables on the device: a program creates them once."""
    if not _CONTEXT:
        _CONTEXT.append(p3.P3Context())
    return _CONTEXT[0]


def prepare(case, seed):
    return {"step": _prepare_step, "process": _prepare_process, "interface": _prepare_interface,
            "eam": _prepare_eam, "batch": _prepare_batch, "host": _prepare_host}[case["kind"]](case, seed)


def run(state):
    return state["run"](state)


def _options(case):
    predict, prescribed = CCN[case["ccn"]]
    return {"precision": PRECISION[case["precision"]], "predictNc": predict, "prescribedCCN": prescribed}


def _prepare_step(case, seed):
    inputs, _ = _columns(case["ncol"], case["nlev"], case["moist"], case["ccn"] == "predicted", False, seed)
    f, block, start = _fields(inputs)
    return {"run": _run_step, "ctx": _context(), "f": f, "block": block, "start": start,
            "options": dict(_options(case), sync=case["wait"])}


def _step_outputs(f):
    return {n: f.t[n] for n in L.PROG_FIELDS + L.OUTPUT_FIELDS}


def _run_step(s):
    s["block"].copy_(s["start"])
    s["ctx"].p3_main(s["f"], DT, **s["options"])
    return _step_outputs(s["f"])


def _prepare_host(case, seed):
    inputs, _ = _columns(case["ncol"], case["nlev"], case["moist"], case["ccn"] == "predicted", False, seed)
    f, block, start = _fields(inputs, host=True)
    return {"run": _run_host, "ctx": _context(), "f": f, "block": block, "start": start, "options": _options(case)}


def _run_host(s):
    s["block"].copy_(s["start"])
    s["ctx"].p3_main_host(s["f"], DT, **s["options"])
    return _step_outputs(s["f"])


def _host_model(case, seed):
    """Fields of an EAMxx host model (wet mixing ratios) around the step."""
    inputs, more = _columns(case["ncol"], case["nlev"], case["moist"], case.get("ccn") == "predicted", True, seed)
    pdd = inputs["dpres"]
    h = {"pmid": inputs["pres"].clone(), "pseudo_density_dry": pdd.clone(),
         "pseudo_density": pdd * (1.0 + inputs["qv"]), "cld_frac_t": more["cloud"]}
    return inputs, h, more["T"]


def _prepare_process(case, seed):
    ncol, nlev = case["ncol"], case["nlev"]
    inputs, h, T = _host_model(case, seed)
    # what a pass changes: the ten prognostics, qv_prev, t_prev, T and the two precipitation masses
    names = L.PROG_FIELDS + ["qv_prev", "t_prev"]
    n = ncol * nlev
    block = torch.empty((len(names) + 1) * n + 2 * ncol, dtype=torch.float64, device="cuda")
    proc = p3.P3Microphysics({"precision": PRECISION[case["precision"]], "do_predict_nc": CCN[case["ccn"]][0],
                              "do_prescribed_CCN": CCN[case["ccn"]][1]})
    proc.set_grids(ncol, nlev)
    proc.ctx = _context()
    f = p3.P3Fields(ncol, nlev)
    for i, name in enumerate(names):
        f.t[name] = block[i * n:(i + 1) * n].view(ncol, nlev)
        f.t[name].copy_(inputs.pop(name))
    h["T_atm"] = block[len(names) * n:(len(names) + 1) * n].view(ncol, nlev)
    h["T_atm"].copy_(T)
    h["T_prev"] = f.t["t_prev"]
    h["precip_liq_surf_mass"] = block[-2 * ncol:-ncol]
    h["precip_ice_surf_mass"] = block[-ncol:]
    block[-2 * ncol:] = 0.25
    for name in list(inputs):
        f.t[name] = inputs.pop(name)
    for name in L.OUTPUT_FIELDS:
        shape = (ncol,) if name in L.SURFACE_FIELDS else (ncol, nlev + 1) if name in L.INTERFACE_FIELDS else (ncol, nlev)
        f.t[name] = torch.zeros(*shape, dtype=torch.float64, device="cuda")
    for name in ("vapor_flux", "water_flux", "ice_flux", "heat_flux"):
        h[name] = torch.zeros(ncol, dtype=torch.float64, device="cuda")
    proc.fields = f
    return {"run": _run_process, "proc": proc, "h": h, "block": block, "start": block.clone()}


def _run_process(s):
    s["block"].copy_(s["start"])
    s["proc"].run_process(s["h"], DT)
    f, h = s["proc"].fields, s["h"]
    out = _step_outputs(f)
    for n in ("qv_prev", "inv_exner", "dz", "cld_frac_l", "cld_frac_i", "cld_frac_r"):
        out[n] = f.t[n]
    for n in ("T_atm", "T_prev", "precip_liq_surf_mass", "precip_ice_surf_mass", "water_flux", "ice_flux"):
        out[n] = h[n]
    return out


# The interface by itself: the preamble on one set of fields (a wet state), the
# postamble on another (a dry state with radii and precipitation after a step).
PRE_STATE = WET + ["qv_prev"]
PRE_OUT = PRE_STATE + ["th", "inv_exner", "dz", "cld_frac_l", "cld_frac_i", "cld_frac_r"]
POST_STATE = WET + ["diag_eff_radius_qc", "diag_eff_radius_qi", "diag_eff_radius_qr"]
POST_OUT = POST_STATE + ["qv_prev"]
POST_HOST = ["T_atm", "T_prev", "precip_liq_surf_mass", "precip_ice_surf_mass", "vapor_flux", "water_flux",
             "ice_flux", "heat_flux"]


def _interface_inputs(case, seed):
    ncol, nlev = case["ncol"], case["nlev"]
    a, h, T = _host_model(case, seed)
    g = torch.Generator(device="cuda")
    g.manual_seed(seed + 1)

    def uni(lo, hi, *shape):
        return lo + (hi - lo) * torch.rand(*shape, generator=g, dtype=torch.float64, device="cuda")

    b = {n: a[n] * uni(0.5, 1.0, ncol, nlev) for n in WET}
    b["th"] = a["th"] + uni(-1.0, 1.0, ncol, nlev)
    b["diag_eff_radius_qc"] = uni(5e-6, 2e-5, ncol, nlev)
    b["diag_eff_radius_qi"] = uni(1e-5, 1e-4, ncol, nlev)
    b["diag_eff_radius_qr"] = uni(1e-4, 5e-4, ncol, nlev)
    surf = {"precip_liq_surf": uni(0.0, 1e-6, ncol), "precip_ice_surf": uni(0.0, 1e-7, ncol)}
    mass = {"precip_liq_surf_mass": uni(0.0, 1.0, ncol), "precip_ice_surf_mass": uni(0.0, 1.0, ncol)}
    return a, b, h, T, surf, mass


def _prepare_interface(case, seed):
    ncol, nlev = case["ncol"], case["nlev"]
    a, b, h, T, surf, mass = _interface_inputs(case, seed)
    n, rows = ncol * nlev, len(PRE_STATE) + len(POST_STATE) + 1
    block = torch.empty(rows * n + 2 * ncol, dtype=torch.float64, device="cuda")
    at = 0

    def placed(v):
        nonlocal at
        view = block[at:at + v.numel()].view(v.shape)
        view.copy_(v)
        at += v.numel()
        return view

    def empty(*shape):
        return torch.zeros(*shape, dtype=torch.float64, device="cuda")

    pre, post = p3.P3Fields(ncol, nlev), p3.P3Fields(ncol, nlev)
    for name in PRE_STATE:
        pre.t[name] = placed(a[name])
    for name in POST_STATE:
        post.t[name] = placed(b[name])
    h_pre = dict(h, T_atm=T)
    h_post = dict(h, T_atm=placed(T), T_prev=empty(ncol, nlev))
    for name, v in mass.items():
        h_post[name] = placed(v)
    for name in ("vapor_flux", "water_flux", "ice_flux", "heat_flux"):
        h_post[name] = empty(ncol)
    post.t.update(surf, th=b["th"])
    for fields in (pre, post):
        for name in L.ALL_FIELDS:
            if name in fields.t:
                continue
            if name in ("th", "inv_exner", "dz", "cld_frac_l", "cld_frac_i", "cld_frac_r", "qv_prev"):
                fields.t[name] = empty(ncol, nlev)
            else:  # not touched by the interface: any device array does
                fields.t[name] = h["pmid"]
    return {"run": _run_interface, "ctx": _context(), "pre": pre, "post": post, "h_pre": h_pre, "h_post": h_post,
            "block": block, "start": block.clone()}


def _run_interface(s):
    s["block"].copy_(s["start"])
    s["ctx"].preamble(s["h_pre"], s["pre"])
    s["ctx"].postamble(s["h_post"], s["post"], DT)
    return {"pre": {n: s["pre"].t[n] for n in PRE_OUT},
            "post": {n: s["post"].t[n] for n in POST_OUT} | {n: s["h_post"][n] for n in POST_HOST}}


def _prepare_eam(case, seed):
    ncol, nlev = case["ncol"], case["nlev"]
    inputs, more = _columns(ncol, nlev, case["moist"], case["ccn"] == "predicted", True, seed)
    names = ["qv", "qc", "nc", "qr", "nr", "qi", "ni", "qm", "bm"]  # in the order of L.EAM_SPECIES
    dry = inputs["dpres"].clone()
    wet = dry * (1.0 + inputs["qv"])
    z = torch.zeros(ncol, nlev + 1, dtype=torch.float64, device="cuda")
    z[:, :nlev] = torch.flip(torch.cumsum(torch.flip(inputs["dz"], [1]), 1), [1])
    eam = {"pmid": inputs["pres"].clone(), "pmiddry": inputs["pres"] / (1.0 + inputs["qv"]), "pdel": wet,
           "pdeldry": dry, "zi": z, "t": more["T"], "ast": more["cloud"], "npccn": inputs["nc_nuceat_tend"].clone(),
           "ni_activated": inputs["ni_activated"].clone(), "relvar": inputs["inv_qc_relvar"].clone(),
           "cmeliq": 1e-8 * (inputs["qv"] - inputs["qv"].mean())}
    for s, n in zip(L.EAM_SPECIES, names):
        eam[s] = inputs[n] * dry / wet
    block = torch.empty(2, ncol, nlev, dtype=torch.float64, device="cuda")
    block[0], block[1] = inputs["t_prev"], inputs["qv_prev"]
    eam["t_prev"], eam["qv_prev"] = block[0], block[1]
    column = ("prec_pcw", "snow_pcw", "prec_str", "snow_str", "cdnumc")
    out = ["ptend_s"] + ["ptend_" + s for s in L.EAM_SPECIES] + L.EAM_DIAG
    for n in out:
        shape = (ncol,) if n in column else (ncol, nlev + 1) if n in ("flxprc", "flxsnw") else (ncol, nlev)
        eam[n] = torch.zeros(*shape, dtype=torch.float64, device="cuda")
    f, _, _ = _fields(inputs)
    return {"run": _run_eam, "ctx": _context(), "eam": eam, "f": f, "block": block, "start": block.clone(),
            "out": out + ["t_prev", "qv_prev"], "options": _options(case)}


def _run_eam(s):
    s["block"].copy_(s["start"])
    s["ctx"].eam_micro_p3_tend(s["eam"], s["f"], DT, **s["options"])
    return {n: s["eam"][n] for n in s["out"]}


def _batch_shapes(case):
    """(ncol, nlev, dt) of the instances: the case alone decides them."""
    r = np.random.RandomState(case["instances"] * 100003 + case["max_ncol"])
    ncol = np.exp(r.uniform(0.0, math.log(case["max_ncol"] + 1), case["instances"])).astype(int)
    return [(int(max(1, min(case["max_ncol"], c))), int(r.choice([72, 128])), float(r.choice([300.0, 120.0])))
            for c in ncol]


def _prepare_batch(case, seed):
    shapes = _batch_shapes(case)
    whole = {}
    for nlev in sorted({s[1] for s in shapes}):
        ncol = sum(s[0] for s in shapes if s[1] == nlev)
        inputs, _ = _columns(ncol, nlev, case["moist"], case["ccn"] == "predicted", False, seed + nlev)
        whole[nlev] = _fields(inputs)
    at = dict.fromkeys(whole, 0)
    fields = []
    for ncol, nlev, _ in shapes:
        f = p3.P3Fields(ncol, nlev)
        f.t = {n: v[at[nlev]:at[nlev] + ncol] for n, v in whole[nlev][0].t.items()}
        at[nlev] += ncol
        fields.append(f)
    predict, prescribed = CCN[case["ccn"]]
    batch = p3.P3Batch(_context(), fields, [s[2] for s in shapes], PRECISION[case["precision"]],
                       predictNc=predict, prescribedCCN=prescribed)
    stream = torch.cuda.Stream()
    batch.capture_graph(stream)
    stream.synchronize()
    return {"run": _run_batch, "batch": batch, "whole": whole}


def _run_batch(s):
    for _, block, start in s["whole"].values():
        block.copy_(start)
    s["batch"].run()
    return {str(nlev): _step_outputs(w[0]) for nlev, w in s["whole"].items()}


# --------------------------------------------------------------------------
# work and values in 64 bits
# --------------------------------------------------------------------------
def _step_bytes(ncol, nlev):
    # 23 inputs read, 10 + 7 fields and 2 interface fluxes and 3 history fields written, per level
    return 8.0 * ncol * (45 * nlev + 4)


def work(case):
    """Bytes of the fields that a pass reads and writes.  The step's arithmetic
    (process rates, table lookups, sedimentation substeps) depends on the data
    and has no closed count, so none is given for it."""
    kind = case["kind"]
    if kind == "batch":
        return {"bytes": sum(_step_bytes(c, k) for c, k, _ in _batch_shapes(case)), "flops": 0.0}
    ncol, nlev = case["ncol"], case["nlev"]
    n = 8.0 * ncol * nlev
    pre, post = 31 * n, 32 * n
    if kind == "interface":
        return {"bytes": pre + post, "flops": 0.0}
    b = _step_bytes(ncol, nlev)
    if kind == "process":
        b += pre + post
    if kind == "eam":
        b = n * (6 + 9 + 5 + 2) + n * (2 + 10 + 25)
    return {"bytes": b, "flops": 0.0}


def exact(case, seed):
    """The interface's formulas in plain float64 tensors on the CPU
    (eamxx_p3_process_interface.hpp:63-269).  The step itself has no such
    value: one restatement of its ~45 process rates and its sedimentation
    differs from another by their roundings, which ice sedimentation carries
    far."""
    if case["kind"] != "interface":
        return None
    a, b, h, T, surf, mass = _interface_inputs(case, seed)
    a, b, h, surf, mass = ({k: v.cpu() for k, v in d.items()} for d in (a, b, h, surf, mass))
    T = T.cpu()
    pd, pdd, pmid, ct = h["pseudo_density"], h["pseudo_density_dry"], h["pmid"], h["cld_frac_t"]
    exner = (pmid / P0) ** (RD / CP)
    pre = {n: a[n] * pd / pdd for n in PRE_STATE}
    pre["th"], pre["inv_exner"] = T / exner, 1.0 / exner
    pre["dz"] = (RD / G) * pd * (T * (1.0 + (1.0 / EP2 - 1.0) * a["qv"])) / pmid
    cl = torch.clamp(ct, min=1e-4)
    cr = cl.clone()
    cr[:, 1:] = torch.maximum(cr[:, 1:], ct[:, :-1])
    pre["cld_frac_l"], pre["cld_frac_i"], pre["cld_frac_r"] = cl, cl, cr
    post = {n: b[n] * pdd / pd for n in WET}
    for n in POST_STATE[len(WET):]:
        post[n] = b[n] * 1e6
    post["qv_prev"] = post["qv"]
    post["T_atm"] = (b["th"] * exner - T) * pdd / pd + T
    post["T_prev"] = post["T_atm"]
    liq, ice = surf["precip_liq_surf"], surf["precip_ice_surf"]
    post["precip_liq_surf_mass"] = mass["precip_liq_surf_mass"] + liq * 1000.0 * DT
    post["precip_ice_surf_mass"] = mass["precip_ice_surf_mass"] + ice * 1000.0 * DT
    post["vapor_flux"], post["heat_flux"] = torch.zeros_like(liq), torch.zeros_like(liq)
    post["water_flux"], post["ice_flux"] = liq + ice, ice
    return {"pre": pre, "post": post}
