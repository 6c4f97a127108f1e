"""The work a user of this framework has it do, as measurable cases.

Kinds (``case["kind"]``):

  lucy    one Lucy iteration without peel-off: the temperature field goes in
          (``set_tdust``), the tallies are zeroed, the packets run, the tallies
          are read back and the temperatures are solved -- one call of the
          reference's ``disk()`` in its Lucy loop
  peel    the peeled iteration: packets with their peel-off rays, then the SED,
          the peeled SED and the images read back
  batch   the Lucy iteration of several models of a grid in one launch
          (``run_batch``), then each model's tallies and temperatures
  serve   model runs through the server: requests submitted together, each a
          Lucy iteration and a peeled one, their SEDs returned
  update  the Lucy temperature solve alone on device buffers the caller owns
          (``hc3d_lucy_update_noalloc``)

Models, grids, packet counts and options are those of
``hochunk3d_gb300/configs.py`` and of the model-grid distribution of
``bench.py`` (disk mass 1e-4..0.1 Msun, infall 1e-7..1e-4 Msun/yr, cavity
5..45 deg, stars of 3000..10000 K, grids 100x99x1, 200x199x1, 200x199x32).
The temperature field is the warm profile 1600 K (r/Rsub)^-0.45 of the tests
and the benchmark.  MAXINT, the cap on a packet's interactions, is set where
the disk is so thick that single packets would walk for seconds.

The tallies are int64 fixed point and are compared whole; Monte Carlo tallies
have no value in 64 bits that could be had without the packets' streams, so
``exact`` answers for the temperature solve only.
"""
from __future__ import annotations

import ctypes as C
import math
import tempfile

import numpy as np
import torch

from hochunk3d_gb300 import configs, hc3d

_MODELS: dict = {}  # the last models built: a model depends on its case, not on the seed


def listed():
    return [
        # the smallest grid of the tests: launch, copy and single-packet latency
        {"name": "lucy_tiny", "kind": "lucy", "model": "tiny", "np": 2000, "fp64": False, "maxint": 1000000},
        # the plain small model as configured (0.01 Msun disk): long walks in an optically thick disk
        {"name": "lucy_plain_thick", "kind": "lucy", "model": "plain", "np": 100000, "fp64": False, "maxint": 60000},
        # a low-mass model of the model grid: many crossings, few interactions
        {"name": "lucy_plain_thin", "kind": "lucy", "model": "plain", "np": 1000000, "fp64": False,
         "maxint": 1000000, "massd": 1e-4, "rate": 5e-7},
        # a three-dimensional grid of the model grid, 1.3e6 cells
        {"name": "lucy_3d", "kind": "lucy", "model": "plain", "np": 300000, "fp64": False, "maxint": 20000,
         "massd": 1e-3, "rate": 5e-6, "npg": 33},
        # peel-off with few directions and packets
        {"name": "peel_tiny3d", "kind": "peel", "model": "tiny3d", "np": 5000, "fp64": False, "maxint": 1000000},
        # the peeled iteration of the plain model: 10 inclinations, 149^2 images
        {"name": "peel_plain", "kind": "peel", "model": "plain", "np": 200000, "fp64": False, "maxint": 20000},
        # the full three-dimensional workload: 80 directions, 301^2 Stokes images, 5e6 cells
        {"name": "peel_full3d", "kind": "peel", "model": "full3d", "np": 200000, "fp64": False, "maxint": 10000},
        # requests of models of the grid, served together: model set-up, load, Lucy iteration, peeled iteration
        {"name": "serve_grid", "kind": "serve", "model": "plain", "np": 20000, "fp64": False, "maxint": 20000,
         "massd": 1e-3, "rate": 5e-6, "models": 4, "slots": 4},
        # the all-FP64 form, both directions
        {"name": "lucy_fp64", "kind": "lucy", "model": "plain", "np": 5000, "fp64": True, "maxint": 20000,
         "massd": 1e-4, "rate": 5e-7},
        {"name": "peel_fp64", "kind": "peel", "model": "tiny3d", "np": 20000, "fp64": True, "maxint": 20000},
        # the Lucy iteration of four models of a grid in one launch
        {"name": "batch_grid", "kind": "batch", "model": "plain", "np": 20000, "fp64": False, "maxint": 20000,
         "massd": 1e-3, "rate": 5e-6, "models": 4},
        # the temperature solve of the full three-dimensional grid, 20 million (cell, species) pairs
        {"name": "update_full3d", "kind": "update", "nrg": 400, "ntg": 199, "npg": 65, "ndg": 4},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["lucy", "lucy", "peel", "peel", "fp64", "batch", "serve", "update"])
    if kind == "update":
        return {"kind": "update", "nrg": rng.randint(60, 400), "ntg": rng.randint(31, 199), "npg": rng.randint(2, 65),
                "ndg": 4}
    if kind == "serve":
        return {"kind": "serve", "model": rng.choice(["tiny", "tiny3d", "plain"]), "np": _logint(rng, 1000, 20000),
                "fp64": False, "maxint": 20000, "massd": 10 ** rng.uniform(-4, -2.5), "rate": 10 ** rng.uniform(-7, -5),
                "models": rng.randint(2, 5), "slots": rng.randint(1, 4)}
    if kind == "fp64":
        return {"kind": rng.choice(["lucy", "peel"]), "model": rng.choice(["tiny", "tiny3d", "tiny_isrf"]),
                "np": _logint(rng, 500, 10000), "fp64": True, "maxint": 10000}
    if kind == "batch":
        return {"kind": "batch", "model": "plain", "np": _logint(rng, 1000, 20000), "fp64": False, "maxint": 20000,
                "massd": 10 ** rng.uniform(-4, -2), "rate": 10 ** rng.uniform(-7, -5), "models": rng.randint(2, 4)}
    model = rng.choice(["plain", "plain", "tiny", "tiny3d", "tiny_isrf", "tiny_acc", "tiny_sg"])
    c = {"kind": kind, "model": model, "np": _logint(rng, 1000, 200000), "fp64": False,
         "maxint": _logint(rng, 5000, 20000)}
    if model == "plain":
        nrg, ntg, npg = rng.choice([(100, 99, 2), (200, 199, 2), (150, 121, 17), (200, 199, 33)])
        c.update(nrg=nrg, ntg=ntg, npg=npg, massd=10 ** rng.uniform(-4, -1), rate=10 ** rng.uniform(-7, -4),
                 cavity=rng.uniform(5.0, 45.0), tstar=rng.uniform(3000.0, 10000.0))
    if kind == "peel":
        c["npeel"] = rng.choice([1, 3, 7, 10, 37])
        c["nx"] = rng.choice([31, 149, 150])
    return c


# ---- what a user's program has in hand ---------------------------------------


def _overrides(case, k=0):
    o = {"MAXINT": case["maxint"]}
    if "massd" in case:
        o["MASSD"] = case["massd"] * (1.0 + 0.7 * k)
    if "rate" in case:
        o["RATE"] = case["rate"]
    if "cavity" in case:
        o["THET1"] = o["THET2"] = case["cavity"]
    if "tstar" in case:
        o["TSTAR"] = case["tstar"]
    for key in ("nrg", "ntg", "npg"):
        if key in case:
            o[key.upper()] = case[key]
    if "nx" in case:
        o["NXIMG"] = case["nx"]
    if "npeel" in case:
        n = case["npeel"]
        o["NPEEL"] = n
        o["THETE"] = ",".join("%.3f" % math.degrees(math.acos(1.0 - (j + 0.5) * 1.9 / n)) for j in range(n))
        o["PHIE"] = ",".join("%.1f" % (j * 47.0 % 360.0) for j in range(n))
    return o


def _warm(model):
    """T = 1600 K (r/Rsub)^-0.45, floored at 10 K, in K/11605."""
    rave = np.sqrt(model.rarr[:-1] * model.rarr[1:])
    t = np.clip(1600.0 * (rave / model.info.rminsub) ** -0.45, 10.0, 1600.0) / 11605.0
    td = np.full(model.shape4, 0.1 / 11605.0, order="F")
    td[:-1] = t[:, None, None, None]
    return np.asfortranarray(td)


def _model(case, k=0):
    key = (case["model"], tuple(sorted(_overrides(case, k).items())))
    if key not in _MODELS:
        if len(_MODELS) >= 6:
            _MODELS.pop(next(iter(_MODELS)))
        with tempfile.TemporaryDirectory() as d:
            m = hc3d.Model(configs.write_par(d, case["model"], **_overrides(case, k)))
        m.set_tdust(_warm(m))
        _MODELS[key] = m
    return _MODELS[key]


def _params(model, case, seed, k=0):
    # iteration 1 of a model with small grains needs no mean intensity of the one before
    p = model.run_params(np=case["np"], iter=1 if model.sg else 3, ipeel=1 if case["kind"] == "peel" else 0)
    p.seed = (1000003 * seed + 7919 * k + 17) & 0xFFFFFFFFFFFF
    return p


def _context(case, model):
    return hc3d.Context(hc3d.PREC_FP64 if case["fp64"] else hc3d.PREC_MIXED).load(model)


def _update_state(case, seed):
    """Device buffers of a grid whose absorbed-path tallies belong to temperatures of 10..1500 K."""
    dev = torch.device("cuda", 0)
    base = _model({"kind": "lucy", "model": "tiny", "maxint": 1000000})
    shape = (case["ndg"], case["npg"], case["ntg"], case["nrg"])  # Fortran (nrg,ntg,npg,ndg)
    gen = torch.Generator(device=dev).manual_seed(seed)

    def uniform(lo, hi):
        return lo + (hi - lo) * torch.rand(shape, generator=gen, device=dev, dtype=torch.float64)

    r = torch.linspace(0.0, 1.0, case["nrg"], device=dev, dtype=torch.float64)
    t = 1500.0 * torch.pow(150.0, -r) * torch.pow(10.0, uniform(-0.3, 0.1))  # K, falling outwards
    t = torch.clamp(t, 10.0, 1500.0) / 11605.0
    dens = torch.where(uniform(0.0, 1.0) < 0.2, 0.0, torch.pow(10.0, uniform(-22.0, -12.0)))
    mass = torch.pow(dens * torch.pow(10.0, uniform(36.0, 40.0)), 0.25)
    n_packets, ltot = 100000000, float(base.info.ltot)
    b = hc3d.LucyBuffers()
    keep = {"lTint": torch.from_numpy(base.lTint).to(dev), "kappap": torch.from_numpy(base.kappap).to(dev)}
    s = {"kappav": [float(base.kappav[j]) for j in range(case["ndg"])], "ltot": ltot, "np": n_packets, "nT": base.nT,
         "lTint": keep["lTint"], "kappap": keep["kappap"], "path_scale": 2.0 ** 21}
    na = torch.empty_like(t)
    for j in range(case["ndg"]):
        kp = _kapp(s, j, t[j])
        na[j] = torch.pow(t[j] * 11605.0 * mass[j], 4) * (4.0 * 5.6704e-5 * n_packets * s["kappav"][j] * kp) / ltot
    s["dtauabs"] = torch.clamp(torch.round(na * s["path_scale"]), 0.0, 9.0e15).to(torch.int64)
    s["densarr"], s["massarr"] = dens, mass
    s["tdust_in"] = torch.clamp(t * uniform(0.7, 1.3), 0.1 / 11605.0, 1600.0 / 11605.0)
    s["tdust_out"] = torch.empty_like(t)
    b.device, b.nrg, b.ntg, b.npg, b.ndg = 0, case["nrg"], case["ntg"], case["npg"], case["ndg"]
    for name in ("dtauabs", "densarr", "massarr", "tdust_in", "tdust_out", "lTint", "kappap"):
        setattr(b, name, s[name].data_ptr())
    b.path_scale, b.nT, b.ltot, b.np = s["path_scale"], s["nT"], ltot, n_packets
    for j in range(case["ndg"]):
        b.kappav[j] = s["kappav"][j]
    s["buffers"] = b
    return s


def prepare(case, seed):
    if case["kind"] == "update":
        return dict(_update_state(case, seed), kind="update")
    if case["kind"] == "serve":
        d = tempfile.TemporaryDirectory()
        pars = []
        for k in range(case["models"]):
            o = dict(_overrides(case, k), NP=case["np"], NPMIN=min(case["np"], 1000), I1=-(1 + (seed * 31 + k) % 1000000))
            pars.append(configs.write_par(d.name + "/m%d" % k, case["model"], **o))
        return {"kind": "serve", "server": hc3d.Server(slots=case["slots"]), "pars": pars, "np": case["np"], "dir": d}
    n = case["models"] if case["kind"] == "batch" else 1
    models = [_model(case, k) for k in range(n)]
    return {"kind": case["kind"], "models": models, "contexts": [_context(case, m) for m in models],
            "params": [_params(m, case, seed, k) for k, m in enumerate(models)], "np": case["np"],
            "tdust": [m.tdust for m in models]}


# ---- one pass -----------------------------------------------------------------


def run(s):
    if s["kind"] == "update":
        b = s["buffers"]
        b.stream = torch.cuda.current_stream().cuda_stream
        rel, conv = C.c_double(0.0), C.c_int(0)
        rc = hc3d.lib().hc3d_lucy_update_noalloc(C.byref(b), C.byref(rel), C.byref(conv))
        if rc != 0:
            raise hc3d.Hc3dError(rc, "hc3d_lucy_update_noalloc")
        return {"tdust": s["tdust_out"], "max_rel_change": rel.value, "converged": bool(conv.value)}
    if s["kind"] == "serve":
        tickets = [s["server"].submit(p, n_lucy=1, np_lucy=s["np"], np_=s["np"]) for p in s["pars"]]
        out = {}
        for k, t in enumerate(tickets):
            r = s["server"].wait(t)
            out.update({"%s_%d" % (n, k): r[n] for n in ("si", "nums", "ti", "numt", "max_rel_change")})
        return out
    if s["kind"] == "peel":
        c, p = s["contexts"][0], s["params"][0]
        c.zero()
        c.run(p)
        return c.tallies(p, grid=False)
    for c, td in zip(s["contexts"], s["tdust"]):
        c.set_tdust(td)
        c.zero()
    if s["kind"] == "batch":
        hc3d.run_batch(s["contexts"], s["params"])
    else:
        s["contexts"][0].run(s["params"][0])
    outs = []
    for c, p, m in zip(s["contexts"], s["params"], s["models"]):
        t = c.tallies(p)
        t["tdust"], t["max_rel_change"], t["converged"] = c.lucy_update(m.info.ltot, s["np"])
        outs.append(t)
    if len(outs) == 1:
        return outs[0]
    return {k: np.concatenate([np.ravel(np.asarray(t[k]), order="F") for t in outs]) for k in outs[0]}


# ---- what a pass cannot do without ----------------------------------------------


#: cell crossings and interactions of a packet on its way out, counted on these models
_PER_PACKET = {"tiny": (61, 8), "tiny3d": (62, 8), "tiny_isrf": (36, 4), "tiny_acc": (210, 150), "tiny_sg": (60, 8),
               "plain": (550, 190), "full3d": (750, 150)}


def work(case):
    if case["kind"] == "update":
        n = case["nrg"] * case["ntg"] * case["npg"] * case["ndg"]
        # tally, density, mass and temperature in, temperature out; about six fixed-point steps of a log and a power
        return {"bytes": 40.0 * n, "flops": 0.8 * n * 6 * 60.0}
    cfg = dict(configs.BASE)
    cfg.update(configs.CONFIGS[case["model"]])
    cfg.update(_overrides(case))
    cells = float((int(cfg["NRG"]) - 1) * (int(cfg["NTG"]) - 1) * (int(cfg["NPG"]) - 1))
    models = case.get("models", 1)
    crossings, events = _PER_PACKET[case["model"]]
    if case["model"] == "plain" and case.get("massd", 0.01) < 1e-3:
        crossings, events = 300, 10
    packets = float(case["np"]) * models
    rho = 8 if case["fp64"] else 4
    sed = 9 * int(cfg["NFREQ"]) * int(cfg["NMU"]) * int(cfg["NPH"]) * int(cfg["NAP"]) * 8 * 8
    b = models * (cells * 4 * rho + sed)
    f = packets * (crossings * 60.0 + events * 300.0)
    if case["kind"] in ("lucy", "batch"):
        # temperatures and masses in, temperatures and the absorption, path and count tallies out
        b += models * cells * (2 * 4 * 8 + 4 * 8 + 2 * 4 * 8 + 8 + 8)
    else:
        npeel, nx = int(cfg["NPEEL"]), int(cfg["NXIMG"])
        b += models * npeel * (9 * int(cfg["NFREQ"]) * int(cfg["NAP"]) * 8 * 8 + 4 * nx * nx * 8)
        f += packets * npeel * min(events, 40) * 50 * 30.0
        if case["kind"] == "serve":
            f += packets * crossings * 60.0
    return {"bytes": b, "flops": f}


# ---- the same in 64 bits -----------------------------------------------------------


def _kapp(s, j, t):
    """Planck-mean opacity of species j at t, linear in log t."""
    lt, n = s["lTint"], s["nT"]
    kp = s["kappap"][j * n:(j + 1) * n]
    k = ((n - 1) * (torch.log(t) - lt[0]) / (lt[n - 1] - lt[0])).to(torch.int64) + 1
    i = torch.clamp(k, 1, n - 1)
    f = (torch.log(t) - lt[i - 1]) / (lt[i] - lt[i - 1])
    v = (1.0 - f) * kp[i - 1] + f * kp[i]
    return torch.where(k < 1, kp[0], torch.where(k > n - 1, kp[n - 1], v))


def exact(case, seed):
    if case["kind"] != "update":
        return None
    s = _update_state(case, seed)
    na = s["dtauabs"].to(torch.float64) / s["path_scale"]
    out = s["tdust_in"].clone()
    worst = 0.0
    lo, hi = 0.1 / 11605.0, 1600.0 / 11605.0
    for j in range(case["ndg"]):
        t0, mass = s["tdust_in"][j], s["massarr"][j]
        t, old = t0.clone(), 0.5 * t0
        busy = torch.ones_like(t, dtype=torch.bool)
        for _ in range(1000):
            busy = busy & ((t - old).abs() > 1e-5 * t)
            if not bool(busy.any()):
                break
            new = torch.pow(na[j] * s["ltot"] / (4.0 * 5.6704e-5 * s["np"] * s["kappav"][j] * _kapp(s, j, t)), 0.25) / 11605.0
            new = torch.clamp(torch.where(mass > 0.0, new / mass, torch.full_like(new, lo)), lo, hi)
            old = torch.where(busy, t, old)
            t = torch.where(busy, new, t)
        live = s["densarr"][j] > 0.0
        live[-1, :, :] = False
        live[:, -1, :] = False
        live[:, :, -1] = False
        out[j] = torch.where(live, t, t0)
        counted = live & (na[j] >= 1.0e4)
        if bool(counted.any()):
            worst = max(worst, float(((t - t0).abs() / t)[counted].max()))
    return {"tdust": out, "max_rel_change": worst, "converged": None}
