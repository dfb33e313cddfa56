"""The work a reionization run gives this library, as cases that can be timed and compared.

A run of Meraxes calls, per snapshot: the source deposit, ComputeTs, find_HII_bubbles, the
brightness temperature and its power spectrum.  The cases call the public entry points of
include/rg_b200.h for these, on seeded synthetic inputs with the distributions of the package's
``workloads`` module (made here on the GPU).  Persistent state (z_at_ionization, T_K, x_e, N_rec,
the cumulative outputs) is put back at the start of a pass, so every pass is the same snapshot.

The snapshot list, the cosmology and the reionization parameters are those of
``workloads.CONFIGS``; ReionEfficiency follows ``workloads.batch_efficiency`` (a partly ionised
box), except where a case sets ``efficiency``.
"""

import ctypes as C
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "meraxes-devs_qyxnew_b200"))

import rg_b200 as rg  # noqa: E402
import workloads as wl  # noqa: E402

SIZES = (64, 96, 128, 192, 256)          # find_HII_bubbles: powers of two and 3 times a power of two
POW2 = (32, 64, 128, 256)                # ComputeTs takes powers of two
XH_TOL = float(np.float32(1e-5))         # REL_TOL of the reference
ABS_TOL = float(np.float32(1e-8))


def listed():
    return [
        # the smallest box of the batch runs: launches and latencies count
        dict(name="hii_64", kind="hii", n=64, z=8.0, filter=0, spin=0, bh=0),
        # the ordinary single-box call, real-space top-hat
        dict(name="hii_256", kind="hii", n=256, z=7.0, filter=0, spin=0, bh=0),
        # a size that is not a power of two, Gaussian filter, black-hole feedback on
        dict(name="hii_192_bh", kind="hii", n=192, z=6.5, filter=2, spin=0, bh=1),
        # inhomogeneous recombinations with the temperature-dependent rates
        dict(name="rec_128", kind="rec", n=128, z=8.0, filter=0, tdep=1),
        # several independent small boxes in one call (a parameter scan)
        dict(name="batch_96", kind="batch", n=96, units=6, z=9.0, filter=1),
        # spin temperature of a small box with both AGN X-ray bands
        dict(name="ts_64_agn", kind="ts", n=64, z=12.0, filter=1, shells=40, agn=1, xe=2e-4, spread=0.3),
        # spin temperature early (dark ages ending) and later, when the gas is partly ionised by X-rays
        dict(name="ts_128", kind="ts", n=128, z=15.0, filter=1, shells=40, agn=0, xe=2e-4, spread=0.3),
        dict(name="ts_256", kind="ts", n=256, z=9.0, filter=1, shells=40, agn=0, xe=1e-2, spread=0.5),
        # the whole snapshot on grids resident in HBM: the production size, at the efficiency of that workload
        dict(name="step_512", kind="step", n=512, z=8.0, agn=0, xe=2e-4, spread=0.3, rmax=1000.0, efficiency=1.0),
        # the whole snapshot from and to the caller's pinned host arrays, as Meraxes' C code calls it
        dict(name="host_128", kind="host", n=128, z=12.0, agn=0, xe=2e-4, spread=0.3, rmax=50.0),
        # 21-cm map with redshift-space distortions, then its power spectrum
        dict(name="map_256", kind="map", n=256, z=8.0, vel=3),
        # source grids of a snapshot from the galaxies
        dict(name="deposit_128", kind="deposit", n=128, galaxies=1_000_000, props=4),
    ]


def draw(rng):
    kind = rng.choice(["hii", "hii", "rec", "batch", "ts", "ts", "step", "host", "map", "deposit"])
    z = round(rng.uniform(6.0, 13.0), 2)
    if kind == "hii":
        return dict(kind=kind, n=rng.choice(SIZES), z=z, filter=rng.choice([0, 0, 1, 2]), spin=rng.choice([0, 1]),
                    bh=rng.choice([0, 0, 1]))
    if kind == "rec":
        return dict(kind=kind, n=rng.choice([64, 96, 128, 192]), z=z, filter=rng.choice([0, 1, 2]),
                    tdep=rng.choice([0, 1]))
    if kind == "batch":
        return dict(kind=kind, n=rng.choice([64, 96, 128]), units=rng.randint(2, 8), z=z, filter=rng.choice([0, 1, 2]))
    if kind == "map":
        return dict(kind=kind, n=rng.choice([64, 96, 128, 192, 256]), z=z, vel=rng.choice([0, 1, 2, 3]))
    if kind == "deposit":
        return dict(kind=kind, n=rng.choice(SIZES), galaxies=int(10 ** rng.uniform(4.5, 6.7)), props=rng.randint(1, 8))
    zt = round(rng.uniform(6.5, 20.0), 2)
    xe = round(10 ** rng.uniform(-3.8, -1.5), 6)
    spread = round(rng.uniform(0.05, 0.6), 2)
    if kind == "ts":
        return dict(kind=kind, n=rng.choice(POW2), z=zt, filter=rng.choice([1, 1, 1, 0, 2]), shells=rng.randint(15, 40),
                    agn=rng.choice([0, 0, 1, 2, 3]), xe=xe, spread=spread)
    return dict(kind=kind, n=rng.choice([64, 128, 256] if kind == "step" else [64, 128]), z=zt, agn=rng.choice([0, 0, 1]),
                xe=xe, spread=spread, rmax=rng.choice([20.34, 50.0, 1000.0]))


# ---------------------------------------------------------------------------
# inputs

def _box(n):
    """About 1 Mpc/h a cell, as the package's configurations have it."""
    return float(n) if n < 256 else n * 250.0 / 256.0


def _rand(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _normal(shape, gen):
    return torch.randn(shape, generator=gen, device="cuda")


def _lognormal(shape, sigma, gen):
    return torch.randn(shape, generator=gen, device="cuda").mul_(sigma).exp_()


def _gaussian_field(n, box, gen, smooth=0.0):
    """workloads.gaussian_field on the GPU: P(k) ~ k^-2 with a Gaussian cut at half the Nyquist wavenumber
    (and, with smooth, at so many cells)."""
    wk = torch.fft.rfftn(_normal((n, n, n), gen))
    f = 2.0 * math.pi / box
    kx = torch.fft.fftfreq(n, d=1.0 / n, device="cuda") * f
    kz = torch.fft.rfftfreq(n, d=1.0 / n, device="cuda") * f
    k2 = kx[:, None, None] ** 2 + kx[None, :, None] ** 2 + kz[None, None, :] ** 2
    kc = 0.5 * math.pi * n / box
    amp = torch.exp(-k2 * (0.25 / kc ** 2 + 0.5 * (smooth * box / n) ** 2)) / torch.sqrt(k2.clamp_min(1e-30))
    amp[0, 0, 0] = 0.0
    g = torch.fft.irfftn(wk.mul_(amp), s=(n, n, n))
    g -= g.mean()
    return g


def _pad(a):
    """An [n][n][n] field in the padded layout [n][n][2 (n/2 + 1)]."""
    n = a.shape[0]
    out = torch.zeros(wl.padded_shape(n), device="cuda")
    out[:, :, :n] = a
    return out


def _sources(n, seed):
    """deltax, stars, sfr and X-ray luminosity of workloads.make_sources."""
    gen = _rand(seed)
    shape = (n, n, n)
    g = _gaussian_field(n, _box(n), gen)
    g *= 0.8 / g.std()
    delta = torch.exp(g - 0.32) - 1.0
    msun = wl.COSMO["Hubble_h"] / 1e10
    per_year = wl.UNITS["UnitLength_in_cm"] / wl.UNITS["UnitVelocity_in_cm_per_s"] / wl.SEC_PER_YEAR
    stars = (1.0 + delta).square_().mul_(1e7 * msun) * _lognormal(shape, 0.5, gen)
    stars[torch.rand(shape, generator=gen, device="cuda") < 0.8] = 0.0
    sfr = stars * _lognormal(shape, 0.3, gen) * (1e-8 * per_year)
    xray = sfr * (3.16 * wl.UNITS["UnitMass_in_g"] / wl.SOLAR_MASS / per_year)
    return {"deltax": _pad(delta), "stars": _pad(stars), "weighted_sfr": _pad(sfr), "sfr": None,
            "xray_luminosity": _pad(xray)}


def _params(case):
    n = case["n"]
    kind = case["kind"]
    z = case.get("z", 8.0)
    kw = dict(Flag_EvolvingReionRBubbleMax=0, ReionRBubbleMax=case.get("rmax", 50.0),
              ReionEfficiency=case.get("efficiency", wl.batch_efficiency(min(max(z, 6.0), 16.0))))
    if kind in ("hii", "rec", "batch"):
        kw.update(ReionFilterType=case["filter"], Flag_IncludeSpinTemp=case.get("spin", 0),
                  Flag_BHFeedback=case.get("bh", 0))
    if kind == "rec":
        kw.update(Flag_IncludeRecombinations=1, ReionRBubbleMaxRecomb=33.9, ReionUVBFlag=2,
                  Flag_TemperatureDependentRec=case["tdep"])
    if kind in ("ts", "step", "host"):
        kw.update(Flag_IncludeSpinTemp=1, TsHeatingFilterType=case.get("filter", 1),
                  TsNumFilterSteps=case.get("shells", 40), Flag_IncludeAGNXray=case["agn"])
    if kind == "map":
        kw.update(Flag_IncludeSpinTemp=1, Flag_IncludePecVelsFor21cm=case["vel"])
    return rg.make_params(n, _box(n), **kw)


def _inputs(case, seed):
    """The device grids that the case's calls read."""
    n, kind = case["n"], case["kind"]
    gen = _rand(seed + 77)
    if kind == "deposit":
        # galaxies cluster: nine in ten sit in one of 4096 groups a few cells wide
        m, box = case["galaxies"], _box(n)
        centre = torch.rand((4096, 3), generator=gen, device="cuda") * box
        at = torch.randint(0, 4096, (m,), generator=gen, device="cuda")
        pos = centre[at] + _normal((m, 3), gen) * (2.0 * box / n)
        field = torch.rand((m,), generator=gen, device="cuda") < 0.1
        pos[field] = torch.rand((int(field.sum()), 3), generator=gen, device="cuda") * box
        vals = _lognormal((case["props"], m), 1.0, gen)
        return {"pos": torch.remainder(pos, box), "vals": vals}
    t = _sources(n, seed)
    shape = (n, n, n)
    if kind == "map":
        xH = torch.rand(shape, generator=gen, device="cuda")
        xH[torch.rand(shape, generator=gen, device="cuda") < 0.2] = 0.0
        # coherent over a few cells, displacements of up to a few cells, |dv/dz| / H well below 1
        vel = _gaussian_field(n, _box(n), gen, smooth=3.0)
        vel *= 8.0 / vel.std()
        return {"deltax": t["deltax"], "xH": xH, "TS_box": 20.0 + 80.0 * torch.rand(shape, generator=gen, device="cuda"),
                "vel": _pad(vel)}
    if kind in ("ts", "step", "host"):
        t["sfr"] = t["weighted_sfr"].clone()
        t["x_e_box_prev"] = _pad(_lognormal(shape, case["spread"], gen) * case["xe"])
        t["Tk_box"] = (t["deltax"][:, :, :n] * 0.3 + 1.0).mul_(12.0).clamp_min_(2.0)
        zz, snap = wl.snapshot_redshifts(case["z"])
        p = _params(case)
        # the history slots that the shells use
        coef = rg.ts_tables(p, zz, snap, snap + 1, 2e-4, 1e-3, np.zeros(len(zz)), with_freq=False)[2]
        nh = max(1, int(np.nonzero(np.any(coef != 0, axis=0))[0].max()))
        bands = [b for b, on in (("soft", case["agn"] in (1, 3)), ("hard", case["agn"] in (1, 2))) if on]
        for b in bands:
            # sparse emissivity: one cell in ten
            a = t["xray_luminosity"] * _lognormal(t["xray_luminosity"].shape, 1.0, gen) * 3e-4
            a[torch.rand(a.shape, generator=gen, device="cuda") > 0.1] = 0.0
            t["bh_xray_" + b] = a
        pairs = [("sfr", "sfr_histories"), ("xray_luminosity", "xray_luminosity_histories")]
        pairs += [("bh_xray_" + b, "bh_xray_histories_" + b) for b in bands]
        hist = {h: torch.empty((nh,) + wl.padded_shape(n), device="cuda") for _, h in pairs}
        for h in range(nh):
            # older slots fainter, each with a modulation of its own that the kinds share
            mod = _lognormal(wl.padded_shape(n), 0.2, gen) if h else 1.0
            amp = math.exp(-0.4 * (zz[snap - h] - zz[snap]))
            for cur, name in pairs:
                torch.mul(t[cur], mod if torch.is_tensor(mod) else 1.0, out=hist[name][h])
                hist[name][h] *= amp
        t.update(hist)
        return t
    if case.get("spin"):
        t["x_e_box"] = _pad(torch.rand(shape, generator=gen, device="cuda") * 0.2)
        t["Tk_box"] = 10.0 + 990.0 * torch.rand(shape, generator=gen, device="cuda")
    if case.get("bh"):
        t["effective_bhm"] = t["stars"] * torch.rand(t["stars"].shape, generator=gen, device="cuda") * 0.05
        t["effective_bhar"] = t["effective_bhm"] * 1e-3
    if kind == "rec":
        t["N_rec"] = _pad(torch.rand(shape, generator=gen, device="cuda") * 0.3)
        t["Gamma12"] = torch.rand(shape, generator=gen, device="cuda") * 0.5
    return t


# ---------------------------------------------------------------------------
# state and passes

class _Program:
    """What one run of Meraxes (one configuration) on this GPU keeps: a context and a stream."""
    ctx = None
    case = None
    stream = None

    @classmethod
    def context(cls, case):
        if cls.stream is None:
            cls.stream = torch.cuda.Stream()
        if cls.case != case:
            cls.ctx, cls.case = None, None
            cls.ctx, cls.case = rg.Context(case["n"]), dict(case)
            cls.ctx.call("rg_set_stream", C.c_void_p(cls.stream.cuda_stream))
            if case["kind"] == "rec":
                cls.ctx.set_recombination_tables(*wl.rec_stand_in_tables())
        return cls.ctx


HII_OUT = ("xH", "r_bubble", "z_at_ionization", "J_21_at_ionization", "temp_kinetic_all_gas")
REC_OUT = ("residual_xH", "clumping_factor", "t_resp")
TS_OUT = ("x_e_box_prev", "x_e_box", "Tk_box", "TS_box")
FRESH = {"z_at_ionization": -1.0, "J_21_at_ionization": 0.0, "temp_kinetic_all_gas": 0.0}


def _grids(t, n_hist=0):
    g = rg.rg_grids()
    for k, v in t.items():
        if v is not None and hasattr(rg.rg_grids, k):
            setattr(g, k, v.data_ptr())
    g.n_hist = n_hist
    return g


def _unit(case, seed):
    """One snapshot: inputs, outputs, the initial value of what a pass updates, and the ABI structs."""
    n, kind = case["n"], case["kind"]
    t = _inputs(case, seed)
    cell = (n, n, n)
    out, first = [], {}
    if kind in ("ts", "step", "host"):
        first.update({k: t[k].clone() for k in ("x_e_box_prev", "Tk_box")})
        t["x_e_box"] = torch.zeros(wl.padded_shape(n), device="cuda")
        t["TS_box"] = torch.zeros(cell, device="cuda")
        out += TS_OUT
    if kind in ("hii", "rec", "batch", "step", "host"):
        for k in HII_OUT:
            t[k] = torch.zeros(cell, device="cuda")
        first.update(FRESH)
        out += HII_OUT
    if kind == "rec":
        first.update({k: t[k].clone() for k in ("N_rec", "Gamma12")})
        for k in REC_OUT:
            t[k] = torch.zeros(cell, device="cuda")
        out += REC_OUT + ("N_rec", "Gamma12")
    if kind in ("step", "host", "map"):
        t["delta_T"] = torch.zeros(cell, device="cuda")
        out.append("delta_T")
    zz, snap = wl.snapshot_redshifts(case["z"])
    fcoll = np.zeros(len(zz))
    fcoll[snap - 1] = 1e-5
    nh = t["sfr_histories"].shape[0] if "sfr_histories" in t else 0
    if kind == "host":
        t = {k: v.cpu().pin_memory() for k, v in t.items()}
        first = {k: v.cpu() if torch.is_tensor(v) else v for k, v in first.items()}
    return dict(p=_params(case), s=rg.snapshot(zz, snap, fcoll), t=t, g=_grids(t, nh), first=first, out=out,
                hii=rg.rg_hii_scalars(), ts=rg.rg_ts_scalars(), tb=C.c_double())


def prepare(case, seed):
    kind, n = case["kind"], case["n"]
    ctx = _Program.context(case)
    if kind == "deposit":
        t = _inputs(case, seed)
        grids = [torch.zeros(wl.padded_shape(n), device="cuda") for _ in range(case["props"])]
        st = dict(ctx=ctx, kind=kind, t=t, grids=grids, box=_box(n), divisors=[1.0] * (case["props"] - 1) + [3.7e-2])
    elif kind == "batch":
        # one redshift bin of a scan: the same radii, an efficiency of its own for each box
        units = [_unit(case, seed * 101 + u) for u in range(case["units"])]
        for i, u in enumerate(units):
            u["p"].ReionEfficiency *= 1.0 + 0.05 * i
        st = dict(ctx=ctx, kind=kind, units=units)
    else:
        st = dict(ctx=ctx, kind=kind, units=[_unit(case, seed)])
    torch.cuda.synchronize()
    return st


def _results(u, kind):
    r = {k: u["t"][k] for k in u["out"]}
    if kind in ("ts", "step", "host"):
        r.update(u["ts"].as_dict())
    if kind in ("hii", "rec", "batch", "step", "host"):
        r.update(u["hii"].as_dict())
    if kind in ("step", "host", "map"):
        r["volume_ave_Tb"] = u["tb"].value
    return r


def run(state):
    ctx, kind = state["ctx"], state["kind"]
    with torch.cuda.stream(_Program.stream):
        if kind == "deposit":
            t = state["t"]
            ctx.deposit_ngp(state["box"], t["pos"].shape[0], t["pos"].data_ptr(), t["vals"].data_ptr(),
                            [g.data_ptr() for g in state["grids"]], state["divisors"])
            return state["grids"]
        for u in state["units"]:
            for k, v in u["first"].items():
                u["t"][k].copy_(v) if torch.is_tensor(v) else u["t"][k].fill_(v)
        if kind == "batch":
            outs = ctx.find_hii_batch(*([u[k] for u in state["units"]] for k in ("p", "s", "g")))
            for u, o in zip(state["units"], outs):
                u["hii"] = o
            # the averages as one array each over the units
            scal = {k: np.array([getattr(o, k) for o in outs], np.float32) for k in outs[0].as_dict()}
            return {"grids": [{k: u["t"][k] for k in u["out"]} for u in state["units"]], "averages": scal}
        u = state["units"][0]
        snap = (C.byref(u["p"]), C.byref(u["s"]), C.byref(u["g"]))
        if kind == "host":
            ctx.call("rg_reion_step_host", *snap, C.byref(u["ts"]), C.byref(u["hii"]), C.byref(u["tb"]))
            return _results(u, kind)
        if kind in ("ts", "step"):
            ctx.call("rg_compute_Ts", *snap, C.byref(u["ts"]))
        if kind in ("hii", "rec", "step"):
            ctx.call("rg_find_HII_bubbles", *snap, C.byref(u["hii"]))
        if kind in ("step", "map"):
            ctx.call("rg_delta_T", *snap, C.byref(u["tb"]))
        r = _results(u, kind)
        if kind == "map":
            r["PS_k"], r["PS_data"], r["PS_error"] = ctx.power_spectrum(u["p"], u["t"]["delta_T"].data_ptr())
        return r


# ---------------------------------------------------------------------------
# what a pass cannot do without

def work(case):
    n, kind = case["n"], case["kind"]
    n3, npad = float(n) ** 3, float(n) * n * 2 * (n // 2 + 1)
    fft = 2.5 * n3 * 3.0 * math.log2(n)          # operations of one real 3-D transform
    if kind == "deposit":
        m = case["galaxies"]
        return {"bytes": 12.0 * m + 4.0 * case["props"] * (m + npad), "flops": float(m * case["props"])}
    p = _params(case)
    if kind == "map":
        vel = case["vel"] > 0
        return {"bytes": 4.0 * (n3 * 3 + npad * (2 if vel else 1)), "flops": fft * (3 if vel else 1)}
    nbytes = flops = 0.0
    if kind in ("hii", "rec", "batch", "step", "host"):
        grids = 2 + (p.Flag_IncludeSpinTemp != 0) + (p.Flag_BHFeedback != 0) + (2 if kind == "rec" else 0)
        nr = len(rg.radius_schedule(p, case["z"]))
        b = 4.0 * npad * (grids + (kind != "rec")) + 4.0 * n3 * (5 + p.Flag_IncludeSpinTemp)
        if kind == "rec":
            b += 4.0 * (npad + 4 * n3)
        nbytes += b * case.get("units", 1)
        flops += fft * grids * (1 + nr) * case.get("units", 1)
    if kind in ("ts", "step", "host"):
        zz, snap = wl.snapshot_redshifts(case["z"])
        coef = rg.ts_tables(p, zz, snap, snap + 1, 2e-4, 1e-3, np.zeros(len(zz)), with_freq=False)[2]
        used = int(np.count_nonzero(np.any(coef != 0, axis=0)))
        kinds = 2 + (0, 2, 1, 1)[case["agn"]]
        nbytes += 4.0 * npad * (used * kinds + 4) + 4.0 * n3 * 3
        flops += fft * kinds * (used + p.TsNumFilterSteps)
    if kind in ("step", "host"):
        nbytes += 4.0 * n3
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------
# the same in 64 bits

def _window(case, p, n, R):
    """filter() of the reference in double (real-space top-hat, sharp-k, Gaussian)."""
    dk = 2.0 * math.pi / p.BoxSize
    i = torch.fft.fftfreq(n, d=1.0 / n, device="cuda", dtype=torch.float64)
    h = torch.arange(n // 2 + 1, device="cuda", dtype=torch.float64)
    kR = torch.sqrt(i[:, None, None] ** 2 + i[None, :, None] ** 2 + h[None, None, :] ** 2) * (dk * R)
    if case["filter"] == 0:
        w = 3.0 * (torch.sin(kR) / kR ** 3 - torch.cos(kR) / kR ** 2)
        return torch.where(kR > 1e-4, w, torch.ones_like(w))
    if case["filter"] == 1:
        return (kR * 0.413566994 <= 1.0).to(torch.float64)
    return torch.exp(-(kR * 0.643) ** 2 / 2.0)


def _exact_hii(case, seed, scale=1.0):
    """The excursion set in FP64 (no temperatures: they need the RECFAST table)."""
    n, z = case["n"], case["z"]
    p = _params(case)
    t = _inputs(case, seed)
    names = ["deltax", "stars"] + (["x_e_box"] if case.get("spin") else []) + (["effective_bhm"] if case.get("bh") else [])
    f64 = torch.float64
    spec = {k: torch.fft.rfftn(t[k][:, :, :n].to(f64)) for k in names}
    unit_t = p.UnitLength_in_cm / p.UnitVelocity_in_cm_per_s
    hub = 3.2407789e-18 * unit_t
    G = 6.672e-8 / p.UnitLength_in_cm ** 3 * p.UnitMass_in_g * unit_t ** 2
    rho = p.OmegaM * 3 * hub * hub / (8 * math.pi * G)
    sfr_time = p.ReionSfrTimescale / (hub * math.sqrt(p.OmegaM * (1 + z) ** 3 + p.OmegaK * (1 + z) ** 2 + p.OmegaLambda))
    pix = (p.BoxSize / n) ** 3
    eff = p.ReionEfficiency * scale
    xH = torch.ones((n, n, n), device="cuda", dtype=f64)
    zion = torch.full_like(xH, -1.0)
    J21 = torch.zeros_like(xH)
    # the schedule: from the largest radius down in steps of ReionDeltaRFactor to the cell's own
    R, f, cell = min(p.ReionRBubbleMax, 0.620350491 * p.BoxSize), p.ReionDeltaRFactor, p.BoxSize / n
    cell *= 1.0 if cell < 1.0 else 0.620350491
    radii = []
    while R / f > cell and R / f > p.ReionRBubbleMin:
        radii.append(R)
        R /= f
    radii.append(cell)
    for i, R in enumerate(radii):
        last = i == len(radii) - 1
        w = None if last else _window(case, p, n, R)
        f = {k: torch.fft.irfftn(s if w is None else s * w, s=(n, n, n)) for k, s in spec.items()}

        def source(v):
            v = v.clamp_min(0.0)
            return torch.where(v < ABS_TOL, torch.zeros_like(v), v)
        dom = 1.0 + f["deltax"].clamp_min(float(np.float32(-1.0) + np.float32(1e-5)))
        stars = source(f["stars"])
        bhm = source(f["effective_bhm"]) if case.get("bh") else 0.0
        nf = 1.0 - source(f["x_e_box"]).clamp_max(float(np.float32(0.999))) if case.get("spin") else 1.0
        pref = eff * (4.0 / 3.0) * math.pi / pix / ((4.0 / 3.0) * math.pi * R ** 3 * rho) * R ** 3
        gam = (1 + z) ** 2 * R * p.UnitLength_in_cm / pix * p.UnitLength_in_cm ** -3.0
        gam *= p.UnitMass_in_g / unit_t / 1.6726e-24 * p.ReionNionPhotPerBary
        j = gam * 6.6262e-27 * 1e21 / (4.0 * math.pi) * p.ReionGammaHaloBias / sfr_time
        frac = (stars + bhm) / dom * pref
        ion = frac > nf
        xH[ion] = 0.0
        if last:
            xH = torch.where(~ion & (xH > XH_TOL), (nf - frac).clamp(0.0, 1.0), xH)
        new = (xH < XH_TOL) & (zion < 0)
        zion[new] = float(np.float32(z))
        J21[new] = (stars * (j * p.ReionAlphaUV) + bhm * (j * p.ReionAlphaUVBH))[new]
    dom = 1.0 + t["deltax"][:, :, :n].to(f64)
    return {"xH": xH, "r_bubble": torch.zeros_like(xH), "z_at_ionization": zion, "J_21_at_ionization": J21,
            "volume_weighted_global_xH": float(xH.mean()), "volume_weighted_global_r_bubble": 0.0,
            "mass_weighted_global_xH": float((xH * dom).sum() / dom.sum())}


def _exact_map(case, seed):
    """delta_T (without the line-of-sight re-binning) and its power spectrum in FP64."""
    n = case["n"]
    p = _params(case)
    t = {k: v.to(torch.float64) for k, v in _inputs(case, seed).items()}
    z = float(np.float32(case["z"]))
    cf = 27.0 * (p.OmegaM * p.BaryonFrac * p.Hubble_h ** 2 / 0.023) * math.sqrt(0.15 / p.OmegaM / p.Hubble_h ** 2 *
                                                                               (1 + z) / 10.0)
    d = cf * t["xH"] * (1.0 + t["deltax"][:, :, :n])
    trad = 2.728 * (1 + z)
    if case["vel"] < 2:
        d = d * (1.0 - trad / t["TS_box"])
    else:
        d = d * (1 + z) / (1000.0 * t["TS_box"])
    if case["vel"]:
        H = 3.2407789e-18 * p.Hubble_h * math.sqrt(p.OmegaM * (1 + z) ** 3 + p.OmegaLambda)
        v = t["vel"][:, :, :n] * ((1 + z) * (1e5 / 3.086e24) * (1 + z))
        kz = torch.arange(n // 2 + 1, device="cuda", dtype=torch.float64) * (2.0 * math.pi / p.BoxSize)
        g = torch.fft.irfftn(torch.fft.rfftn(v) * (p.Hubble_h * 1j * kz), s=(n, n, n)) / H
        if case["vel"] == 1:
            d = d / (g.clamp(-float(np.float32(0.2)), float(np.float32(0.2))) + 1.0)
        else:
            gc = (g + 1.0).abs()
            d = (1.0 - torch.exp(-d / gc)) * 1000.0 * (t["TS_box"] - trad) / (1 + z)
    return {"delta_T": d, "volume_ave_Tb": float(d.mean())}


def exact(case, seed):
    """None where a restatement would be a second framework: ComputeTs (and the steps that hold it)
    needs the frequency integrals of the 21cmFAST tables, the recombination branch the MHR splines,
    and the line-of-sight re-binning moves 50 sub-cells per cell by float displacements."""
    kind = case["kind"]
    if kind == "hii":
        return _exact_hii(case, seed)
    if kind == "batch":
        units = [_exact_hii(case, seed * 101 + u, 1.0 + 0.05 * u) for u in range(case["units"])]
        scal = [k for k, v in units[0].items() if not torch.is_tensor(v)]
        return {"grids": [{k: v for k, v in u.items() if k not in scal} for u in units],
                "averages": {k: np.array([u[k] for u in units]) for k in scal}}
    if kind == "map" and case["vel"] < 3:
        return _exact_map(case, seed)
    if kind == "deposit":
        n, t = case["n"], _inputs(case, seed)
        ind = torch.round(t["pos"].to(torch.float64) / _box(n) * n).to(torch.int64)
        ind[ind > n - 1] = 0
        at = (ind[:, 0] * n + ind[:, 1]) * wl.padded_shape(n)[2] + ind[:, 2]
        div = [1.0] * (case["props"] - 1) + [3.7e-2]
        grids = [torch.zeros(n * n * wl.padded_shape(n)[2], device="cuda", dtype=torch.float64) for _ in div]
        return [g.index_add_(0, at, v.to(torch.float64)).div_(d).view(wl.padded_shape(n))
                for g, v, d in zip(grids, t["vals"], div)]
    return None
