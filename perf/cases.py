"""The library's measured work: what its users have it compute, case by case.

Each case is one call (or the short fixed sequence of calls) a program makes
through the ``wltube`` binding of the C ABI: single evaluations, scans, whole
(rho, T) grids, the proper-time integral, the effective action, the lattice,
uneven batches and the reference driver's own caller chain.  Ensembles are
closed Brownian bridges of unit proper time with their mean removed, float32
``[Nl][ppl][4]``; proper times and fluxes are those of the library's
configurations (T in [1e-3, 1e3], F in [0.1, 10], groups of 128 loops).
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "worldline-flux-tube-lattice_gb300"))

import wltube  # noqa: E402

E_CHARGE = 0.30282212


def listed():
    return [
        # one centre and proper time at the reference's 50 intervals: an
        # interactive query, what one EV() of the reference's driver asks for
        {"name": "one_point", "kind": "eval", "profile": "smooth", "fermion": 0, "nint": 50,
         "lambda2": 1.0, "a": 1.0, "Nl": 1024, "ppl": 1024, "group": 128, "ninst": 1, "nF": 1,
         "F": 1.0, "T0": 0.05, "T1": 5.0, "rmax": 2.0},
        # the reference's driver: integrateT -> Tfunc -> EV at one radius, its
        # main()'s ensemble, 40 panels, 50 intervals
        {"name": "driver_chain", "kind": "chain", "profile": "smooth", "fermion": 0, "nint": 50,
         "lambda2": 1.0, "a": 1.0, "Nl": 5120, "ppl": 1024, "group": 128, "nF": 1, "F": 1.0,
         "panels": 40, "rmax": 2.0},
        # proper-time scan at a few centres, three fluxes, arrays on the device
        {"name": "T_scan", "kind": "device", "profile": "smooth", "fermion": 1, "nint": 4,
         "lambda2": 1.0, "a": 1.0, "Nl": 5120, "ppl": 2048, "group": 128, "ninst": 96, "nF": 3,
         "F": 0.1, "T0": 1e-2, "T1": 1e2, "rmax": 8.0},
        # the scalar configuration: 64 T x 16 rho on 1024 loops of 1024 points
        {"name": "scalar_grid", "kind": "device", "profile": "smooth", "fermion": 0, "nint": 4,
         "lambda2": 1.0, "a": 1.0, "Nl": 1024, "ppl": 1024, "group": 128, "ninst": 1024, "nF": 1,
         "F": 1.0, "T0": 1e-2, "T1": 1e2, "rmax": 5.0},
        # odd sizes throughout, an interval count between the two usual ones
        {"name": "gaussian_ragged", "kind": "eval", "profile": "gaussian", "fermion": 1, "nint": 16,
         "lambda2": 0.5, "a": 1.0, "Nl": 1500, "ppl": 516, "group": 100, "ninst": 333, "nF": 2,
         "F": 0.3, "T0": 2e-2, "T1": 2e1, "rmax": 3.0},
        # the spinor configuration: L_eff(rho) from 64 rho x 128 T, three fluxes
        {"name": "spinor_leff", "kind": "tint", "profile": "smooth", "fermion": 1, "nint": 4,
         "lambda2": 1.0, "a": 1.0, "Nl": 5120, "ppl": 2048, "group": 128, "nrho": 64, "nT": 128,
         "nbins": 20, "nF": 3, "F": 0.1, "T0": 1e-3, "T1": 1e3, "rmax": 8.0},
        # the reference driver's effective action in one call
        {"name": "action", "kind": "action", "profile": "smooth", "fermion": 0, "nint": 50,
         "lambda2": 0.01, "a": 1.0, "Nl": 5120, "ppl": 1024, "group": 128, "nrho": 20,
         "panels": 40, "nF": 1, "F": 1.0},
        # square lattice of tubes, centres over the unit cell
        {"name": "lattice", "kind": "device", "profile": "lattice", "fermion": 1, "nint": 4,
         "lambda2": 1.0, "a": 5.0, "Nl": 1024, "ppl": 1024, "group": 128, "ninst": 512, "nF": 1,
         "F": 1.0, "T0": 1e-2, "T1": 1e2, "rmax": 5.0},
        # the reference's two lattice-of-tubes models, at its 50 intervals
        {"name": "periodic", "kind": "eval", "profile": "periodic", "fermion": 0, "nint": 50,
         "lambda2": 0.04, "a": 1.0, "Nl": 1024, "ppl": 512, "group": 128, "ninst": 128, "nF": 1,
         "F": 1.0, "T0": 1e-2, "T1": 5.0, "rmax": 0.5},
        {"name": "fixflux", "kind": "eval", "profile": "fixflux", "fermion": 1, "nint": 50,
         "lambda2": 0.25, "a": 1.0, "Nl": 512, "ppl": 512, "group": 128, "ninst": 64, "nF": 1,
         "F": 0.5, "T0": 1e-2, "T1": 5.0, "rmax": 0.5},
        # an uneven batch: jobs of different ensembles, profiles and sizes
        {"name": "uneven_batch", "kind": "batch", "fermion": 1, "nint": 4, "jobs": 6, "Nl": 2048,
         "ppl": 2048, "group": 128, "ninst": 1500, "nF": 1, "F": 1.0, "T0": 1e-2, "T1": 1e2},
        # an ensemble named by its seed: generated, evaluated once, released
        {"name": "fresh_ensemble", "kind": "fresh", "profile": "smooth", "fermion": 1, "nint": 4,
         "lambda2": 1.0, "a": 1.0, "Nl": 2048, "ppl": 1024, "group": 128, "ninst": 256, "nF": 1,
         "F": 1.0, "T0": 1e-2, "T1": 1e2, "rmax": 5.0},
    ]


# ------------------------------------------------------------- drawn cases --
# node evaluations of a case, weighted by the profile's cost per node
WEIGHT = {"smooth": 1.0, "step": 1.2, "quadratic": 1.3, "gaussian": 2.5, "lattice": 30.0,
          "spline": 12.0, "periodic": 45.0, "fixflux": 170.0}
MOST = 1.0e11  # spinor_leff is 4.3e11


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["eval", "eval", "device", "device", "tint", "action", "lattice", "cell",
                       "batch", "fresh", "chain"])
    fermion = rng.randrange(2)
    group = rng.choice([128, 128, 128, 64, 100, 30])
    Nl = group * max(2, round(_log(rng, 256, 5120) / group))
    ppl = 4 * round(_log(rng, 64, 4096) / 4)
    profile = rng.choice(["smooth", "smooth", "gaussian", "gaussian", "step", "quadratic"])
    # half of the users keep one of the two usual interval counts
    nint = rng.choice([4, 4, 50, 2 * rng.randint(2, 16)])
    lam2 = float("%.3g" % _log(rng, 0.05, 4.0))
    a = 1.0
    nF = rng.choice([1, 1, 2, 3, 4])
    F = 10.0 ** (1 - nF) if nF > 1 else float("%.3g" % _log(rng, 0.05, 3.0))
    c = {"kind": kind, "profile": profile, "fermion": fermion, "nint": nint, "lambda2": lam2,
         "a": a, "Nl": Nl, "ppl": ppl, "group": group, "nF": nF, "F": F, "T0": 1e-2,
         "T1": float("%.3g" % _log(rng, 5.0, 100.0)), "rmax": float("%.3g" % _log(rng, 0.5, 8.0))}
    if profile in ("step", "quadratic"):
        c["fermion"] = 0  # their f' jumps or kinks at the edge: any rounding moves a node over it
    if c["fermion"]:  # spin exponents of some tens, as the configurations have
        c["T1"] = float("%.3g" % max(0.1, min(c["T1"], 20.0 * lam2 / (F * 10.0 ** (nF - 1)))))
    if kind in ("eval", "device", "fresh"):
        c["ninst"] = round(_log(rng, 1, 4000))
        if kind == "fresh":
            c["profile"], c["ninst"] = "smooth", round(_log(rng, 32, 1000))
    elif kind == "lattice":
        lam = math.sqrt(lam2)
        c.update(kind="device", profile="lattice", nint=4, a=float("%.3g" % (lam * rng.uniform(2, 10))),
                 ninst=round(_log(rng, 16, 1000)), nF=1, F=1.0, T1=20.0)
        c["rmax"] = c["a"]
    elif kind == "cell":
        p = rng.choice(["periodic", "periodic", "spline", "fixflux", "fixflux"])
        c.update(kind="eval", profile=p, nint=rng.choice([8, 20, 50]), a=1.0,
                 lambda2=float("%.3g" % _log(rng, 0.02, 0.5)), nF=1, F=0.5, T1=5.0, rmax=0.5,
                 ninst=round(_log(rng, 1, 500)))
    elif kind == "tint":
        c.update(nrho=rng.randint(2, 40), nT=rng.randint(9, 120), nbins=2)
        if c["profile"] != "smooth":
            c["profile"], c["fermion"] = "gaussian", fermion
        c["Nl"] = c["group"] * 2 * max(1, Nl // (2 * c["group"]))
    elif kind == "action":
        c.update(nrho=rng.randint(2, 20), panels=rng.randint(5, 40), nF=1, F=1.0,
                 profile=rng.choice(["smooth", "gaussian"]), nint=rng.choice([4, 50]))
        del c["T0"], c["T1"], c["rmax"]
    elif kind == "chain":
        c.update(profile="smooth", nint=50, group=128, Nl=128 * rng.randint(2, 40), nF=1,
                 F=1.0, panels=rng.randint(5, 40), rmax=3.0)
        del c["T0"], c["T1"]
    elif kind == "batch":
        c = {"kind": "batch", "fermion": fermion, "nint": 4, "jobs": rng.randint(2, 8),
             "Nl": 128 * rng.randint(2, 16), "ppl": ppl, "group": 128,
             "ninst": round(_log(rng, 30, 3000)), "nF": 1, "F": 1.0, "T0": 1e-2, "T1": 1e2}
    # bounded: fewer loops where the case would cost more than the largest
    while _nodes(c) > MOST:
        c["Nl"] = c["group"] * 2 * max(1, c["Nl"] // (4 * c["group"]))
        if _nodes(c) > MOST:
            c["ppl"] = 4 * max(16, c["ppl"] // 8)
    return c


def _ninst(c):
    if c["kind"] == "tint":
        return c["nrho"] * c["nT"]
    if c["kind"] == "action":
        return 2 * c["nrho"] * (2 * c["panels"] - 1)
    if c["kind"] == "chain":
        return 2 * c["panels"] - 1
    return c["ninst"]


def _nodes(c):
    n = sum(_nodes(j) for j in _jobs(c)) if c["kind"] == "batch" else \
        float(c["Nl"]) * c["ppl"] * _ninst(c) * (c["nint"] + 1) * WEIGHT[c["profile"]]
    return n


def _jobs(c):
    """The jobs of an uneven batch, from its sizes: smooth, Gaussian and lattice
    tubes of different widths on ensembles of different shapes."""
    out = []
    for k in range(c["jobs"]):
        prof = ("smooth", "gaussian", "smooth", "lattice")[k % 4]
        lam2 = (1.0, 0.5, 0.2, 1.0, 4.0)[k % 5]
        j = {"kind": "eval", "profile": prof, "fermion": c["fermion"], "nint": c["nint"],
             "lambda2": lam2, "a": 5.0 * math.sqrt(lam2), "group": c["group"],
             "Nl": c["group"] * max(1, c["Nl"] // (1 + k % 3) // c["group"]),
             "ppl": 4 * max(4, c["ppl"] // (1 + k % 2) // 4),
             "ninst": max(1, c["ninst"] // (1 + 2 * (k % 3))), "nF": 1,
             "F": (1.0, 0.3, 2.0)[k % 3], "T0": c["T0"], "T1": c["T1"],
             "rmax": 5.0 * math.sqrt(lam2)}
        if prof == "lattice":
            j["ninst"], j["T1"] = max(1, j["ninst"] // 8), 10.0
        out.append(j)
    return out


# -------------------------------------------------------------- the inputs --
def _ensemble(Nl, ppl, seed):
    """Closed Brownian bridges of unit proper time (step variance 2/ppl per
    component), mean removed."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    w = torch.randn((Nl, ppl, 4), generator=g, device="cuda", dtype=torch.float32)
    w *= math.sqrt(2.0 / ppl)
    y = torch.cumsum(w.double(), dim=1)
    k = torch.arange(1, ppl + 1, device="cuda", dtype=torch.float64)[None, :, None] / ppl
    y -= k * y[:, -1:, :].clone()
    y -= y.mean(dim=1, keepdim=True)
    return y.float().contiguous()


def _field(c):
    return wltube.field(c["profile"], fermion=c["fermion"], nint=c["nint"], lambda2=c["lambda2"],
                        tubedist=c["a"])


def _fluxes(c):
    return [c["F"] * 10.0 ** j for j in range(c["nF"])]


def _instances(c, seed):
    """Centres and proper times: radii on the x axis (the lattice: anywhere in
    the unit cell), T log-uniform with a float32 square root."""
    rng = np.random.default_rng([seed, 7])
    n = c["ninst"]
    cx = rng.uniform(0.0, c["rmax"], n)
    cy = rng.uniform(0.0, c["rmax"], n) if c["profile"] == "lattice" else np.zeros(n)
    rt = np.exp(0.5 * rng.uniform(math.log(c["T0"]), math.log(c["T1"]), n)).astype(np.float32)
    return (cx.astype(np.float32).astype(np.float64), cy.astype(np.float32).astype(np.float64),
            rt.astype(np.float64) ** 2)


def _rho_T(c, seed):
    rng = np.random.default_rng([seed, 8])
    rho = np.linspace(0.0, c["rmax"] * rng.uniform(0.9, 1.0), c["nrho"])
    return rho.astype(np.float32).astype(np.float64), np.geomspace(c["T0"], c["T1"], c["nT"])


def prepare(case, seed):
    c = case
    s = {"case": c, "seed": seed, "ctx": wltube.Context(0)}
    if c["kind"] == "batch":
        jobs = []
        for k, j in enumerate(_jobs(c)):
            loops = _ensemble(j["Nl"], j["ppl"], seed * 64 + k)
            cx, cy, T = _instances(j, seed * 64 + k)
            jobs.append({"handle": s["ctx"].wrap(loops.data_ptr(), j["Nl"], j["ppl"]),
                         "field": _field(j), "cx": cx, "cy": cy, "T": T, "F": _fluxes(j),
                         "group": j["group"], "loops": loops})
        s["jobs"] = jobs
        torch.cuda.synchronize()
        return s
    s["field"], s["F"] = _field(c), _fluxes(c)
    if c["kind"] != "fresh":
        s["loops"] = _ensemble(c["Nl"], c["ppl"], seed)
        s["h"] = s["ctx"].wrap(s["loops"].data_ptr(), c["Nl"], c["ppl"])
    if c["kind"] in ("eval", "device", "fresh"):
        s["cx"], s["cy"], s["T"] = _instances(c, seed)
    if c["kind"] == "device":
        s["dev"] = [torch.from_numpy(v).cuda() for v in (s["cx"], s["cy"], s["T"])]
        n, nF, ng = c["ninst"], c["nF"], c["Nl"] // c["group"]
        s["out"] = [torch.zeros(sh, dtype=torch.float64, device="cuda")
                    for sh in ((n, nF, ng), (n, nF), (n, nF))]
    elif c["kind"] == "tint":
        s["rho"], s["T"] = _rho_T(c, seed)
    elif c["kind"] == "chain":
        wltube.legacy_configure(c["profile"], nint=c["nint"])
        Nl = c["Nl"]
        s["dev"] = [torch.zeros(Nl * 4, device="cuda") for _ in range(2)]
        s["host"] = [np.zeros((Nl, 4), np.float32) for _ in range(2)]
        p = wltube.Wparams()
        p.Nl, p.Nppl, p.F, p.l2 = Nl, c["ppl"], c["F"], c["lambda2"]
        p.fermion, p.ng = c["fermion"], Nl // 128
        p.worldlines = s["loops"].data_ptr()
        p.Wsscal_d, p.Wsferm_d = (d.data_ptr() for d in s["dev"])
        p.Wsscal_h, p.Wsferm_h = (h.ctypes.data for h in s["host"])
        p.xcm.x = _chain_rho(c, seed)
        s["params"] = p
    torch.cuda.synchronize()
    return s


def _chain_rho(c, seed):
    return float(np.float32(np.random.default_rng([seed, 9]).uniform(0.0, c["rmax"])))


def run(state):
    s, c = state, state["case"]
    ctx, kind = s["ctx"], c["kind"]
    if kind == "eval":
        return ctx.eval(s["h"], s["field"], s["cx"], s["cy"], s["T"], s["F"], c["group"])
    if kind == "device":
        ctx.eval_device(s["h"], s["field"], c["ninst"], *(d.data_ptr() for d in s["dev"]), s["F"],
                        c["group"], *(o.data_ptr() for o in s["out"]))
        return s["out"]
    if kind == "tint":
        return ctx.tint(s["h"], s["field"], s["rho"], s["T"], s["F"], c["group"], c["nbins"])
    if kind == "action":
        return ctx.effective_action(s["h"], s["field"], c["F"], None, c["group"], c["nrho"],
                                    c["panels"])
    if kind == "batch":
        return ctx.batch_eval(s["jobs"])
    if kind == "chain":
        return wltube.integrateT(c["panels"], s["params"])
    h = ctx.generate(s["seed"], c["Nl"], c["ppl"])
    try:
        return ctx.eval(h, s["field"], s["cx"], s["cy"], s["T"], s["F"], c["group"])
    finally:
        ctx.release(h)


def work(case):
    """The ensemble read once and the outputs written once; per segment the
    polynomial (14) and its combination (8), per node 4 operations and the
    profile's own (a reciprocal or an exponential counted as one)."""
    if case["kind"] == "batch":
        parts = [work(j) for j in _jobs(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    c, n = case, _ninst(case)
    segs = float(c["Nl"]) * c["ppl"] * n
    per = {"smooth": 2, "step": 2, "quadratic": 4, "gaussian": 5, "lattice": 12, "spline": 20,
           "periodic": 60, "fixflux": 100}[c["profile"]]
    node = 4 + per + 2 * c["fermion"]
    ng = c["Nl"] // c["group"]
    return {"bytes": 16.0 * c["Nl"] * c["ppl"] + 8.0 * n * c["nF"] * (ng + 2),
            "flops": segs * (22 + (c["nint"] + 1) * node)}


# ----------------------------------------------------- the same in 64 bits --
# Written from the formulas (Idt, WilsonLoop, EVMean, Tfunc of the reference;
# the lattice as the sum of its Gaussian tubes) on torch tensors.
EXACT_MOST = 6.0e10  # node evaluations that take a few seconds


def _ei_cf(x):
    """Ei(x), x < -1: -E1(-x) by its continued fraction (Abramowitz and Stegun
    5.1.22), evaluated backwards."""
    z = -x
    t = torch.zeros_like(z)
    for k in range(50, 0, -1):
        t = k / (1.0 + k / (z + t))
    return -torch.exp(-z) / (z + t)


def _bump(x):
    return torch.where(x * x < 1.0, torch.exp(-1.0 / (1.0 - x * x).clamp_min(1e-300)), 0.0 * x)


def _profile(c, r2):
    """f / rho^2 and f' at rho^2."""
    l2, a, p = c["lambda2"], c["a"], c["profile"]
    l2 = float(np.float32(l2))
    if p == "smooth":
        g = 1.0 / (l2 + r2)
        return g, l2 * g * g
    if p == "step":
        inside = r2 < l2
        return torch.where(inside, torch.full_like(r2, 1.0 / l2), 1.0 / r2), inside.double() / l2
    if p == "quadratic":
        inside, u = r2 < l2, r2 / l2
        return (torch.where(inside, (2.0 - u) / l2, 1.0 / r2),
                torch.where(inside, 2.0 / l2 * (1.0 - u), 0.0 * u))
    if p in ("gaussian", "lattice"):
        x = r2 / l2
        return -torch.expm1(-x) / r2.clamp_min(1e-300), torch.exp(-x) / l2
    if p == "periodic":
        lam, ln2 = math.sqrt(l2), math.log(2.0)
        rho = torch.sqrt(r2)
        fl = torch.floor(rho / a)
        f = torch.where(fl > 2, 0.5 * (fl - 3.0) * (fl - 2.0), 0.0 * fl)
        d = torch.zeros_like(rho)
        axis = fl <= 2
        ex = torch.exp(-rho / lam)
        f = torch.where(axis, -rho / a * ex / (1 + ex) - lam / a * torch.log1p(ex), f)
        d = torch.where(axis, ex / (a * (1 + ex) ** 2), d)
        for k in range(-2, 3):
            i = fl + k
            e = torch.exp((-(rho - i * a) / lam).clamp_max(600.0))
            on = i > 0
            f = f + torch.where(on, i / (1 + e), 0.0 * e)
            d = d + torch.where(on, i / rho * e / (1 + e) ** 2, 0.0 * e)
        return (a / (lam * ln2) * f + 1.0) / r2, a / (2.0 * l2 * ln2) * d
    # fixflux (intEV.cu's fits)
    lam, lmin = math.sqrt(l2), 0.1 * a
    lml, aml = (lam - lmin) / (a - lmin), (a - lam) / (a - lmin)
    q1, q2 = 0.443991, 0.0742478
    rho = torch.sqrt(r2)
    n = torch.floor((rho + 0.5 * a) / a)
    first = r2 <= 0.25 * a * a
    x = torch.where(first, 2.0 * rho / lam, 2.0 * (rho - n * a) / lam)
    bump = x * x < 0.999
    o = torch.where(bump, 1.0 - x * x, torch.full_like(x, 0.5))
    ei = _ei_cf(-1.0 / o)
    phi = torch.where(x < 0.999, 1.0 - 0.5 / q2 * (o * torch.exp(-1.0 / o) + ei), 1.0 + 0.0 * x)
    xs = torch.where(bump, x, 0.0 * x)
    s = 3.31 * xs + 5.25 * xs ** 3 * torch.sin(xs) * torch.cos(-0.907 * xs ** 2 - 1.29 * xs ** 8)
    chi = 0.5 * (-o * torch.exp(-1.0 / o) - ei) + \
        2.0 * n * a / lam * 0.444 / (1.0 + torch.exp(-s / torch.cos(xs)))
    chi = torch.where(bump, chi, torch.where(x < 0, 0.0 * x, 2.0 * n * a * q1 / lam))
    f_in = (1.0 - 0.75 * lml) * phi + 3.0 * r2 / (a * a) * lml
    f_out = 1.0 + 0.75 * (4.0 * r2 / (a * a) - 1.0) * lml + 3.0 * n * (n - 1.0) * aml + \
        3.0 * lam / (q1 * a) * aml * chi
    bg = 3.0 / (a * a) * lml
    xb = x * x < 0.999
    b = torch.where(xb, _bump(torch.where(xb, x, 0.0 * x)), 0.0 * x)
    fp = torch.where(first, bg + 2.0 / (l2 * q2) * (1.0 - 0.75 * lml) * b,
                     bg + 6.0 / (q1 * lam * a) * aml * b)
    return torch.where(first, f_in, f_out) / r2, fp


def _simpson(c, zx, zy, nx, ny, clamp):
    """Per segment: the phase at F = 1 and the integral of f'."""
    dx, dy = nx - zx, ny - zy
    a, b, cc = zx * zx + zy * zy, zx * dx + zy * dy, dx * dx + dy * dy
    cross = zx * ny - zy * nx
    if clamp:
        a, b, cc = a.clamp_min(1e-8), b.clamp_min(1e-8), cc.clamp_min(1e-8)
    n = c["nint"]
    t = torch.arange(n + 1, dtype=torch.float64, device=zx.device) / n
    w = torch.full_like(t, 2.0)
    w[1::2] = 4.0
    w[0] = w[n] = 1.0
    G = H = 0.0
    some = max(1, 8_000_000 // max(1, zx.numel()))  # nodes at a time
    for j in range(0, n + 1, some):
        tj, wj = (v[j:j + some, None, None] for v in (t, w))
        g, f = _profile(c, a + tj * (2.0 * b + cc * tj))
        G = G + (wj * g).sum(0)
        if c["fermion"]:
            H = H + (wj * f).sum(0)
    return cross * G / (3.0 * n), (H / (3.0 * n) if c["fermion"] else None)


def _sums(c, x, y, cx, cy, s):
    """Per loop: phases and f' integrals of the sub-loops N/2, N/4 (2 mod 4),
    N/4 (0 mod 4) of the loops s x + cx, s y + cy."""
    zx, zy = s * x + cx, s * y + cy
    box = None
    if c["profile"] == "lattice":
        a, l2, lim = c["a"], c["lambda2"], 12
        cut = math.sqrt(18.0 * l2)
        box = torch.stack([zx.min(1).values, zx.max(1).values, zy.min(1).values,
                           zy.max(1).values])
        x0, y0 = box[0].min().item() - cut, box[2].min().item() - cut
        x1, y1 = box[1].max().item() + cut, box[3].max().item() + cut
        imgs = [(m * a, n * a)
                for m in range(max(-lim, math.ceil(x0 / a)), min(lim, math.floor(x1 / a)) + 1)
                for n in range(max(-lim, math.ceil(y0 / a)), min(lim, math.floor(y1 / a)) + 1)
                if m * m + n * n <= lim * lim]
    ph, sp = [], []
    for first, step in ((1, 2), (2, 4), (0, 4)):
        px, py = zx[:, first::step], zy[:, first::step]
        if box is None:
            g, f = _simpson(c, px, py, px.roll(-1, 1), py.roll(-1, 1), True)
            g, f = g.sum(1), (f.sum(1) if f is not None else None)
        else:
            g = f = torch.zeros(px.shape[0], dtype=torch.float64, device=px.device)
            for rx, ry in imgs:
                on = ((rx >= box[0] - cut) & (rx <= box[1] + cut) & (ry >= box[2] - cut) &
                      (ry <= box[3] + cut)).nonzero()[:, 0]
                if not len(on):
                    continue
                ux, uy = px[on] - rx, py[on] - ry
                gi, fi = _simpson(c, ux, uy, ux.roll(-1, 1), uy.roll(-1, 1), False)
                g = g.index_add(0, on, gi.sum(1))
                if fi is not None:
                    f = f.index_add(0, on, fi.sum(1))
        ph.append(g)
        sp.append(f)
    return ph, sp


def _groups(c, loops, cx, cy, T, F):
    """<W> per group [ninst][nF][ng] (Richardson 8/3, -2, 1/3)."""
    x, y = loops[:, :, 0].double(), loops[:, :, 1].double()
    Nl, ppl = x.shape
    ng = Nl // c["group"]
    out = torch.empty((len(T), len(F), ng), dtype=torch.float64, device=x.device)
    for i in range(len(T)):
        s = float(np.float32(math.sqrt(T[i])))
        ph, sp = _sums(c, x, y, float(np.float32(cx[i])), float(np.float32(cy[i])), s)
        for j, f in enumerate(F):
            p = [f * v for v in ph]
            n4 = p[1] + p[2]
            w = [torch.cos(0.5 * p[0] + 0.25 * n4), torch.cos(p[0]), torch.cos(0.5 * n4)]
            if c["fermion"]:
                q = [f * 2.0 * s * s / (ppl / d) * v for d, v in zip((2, 4, 4), sp)]
                n4 = q[1] + q[2]
                over = (n4.abs() >= 601.0) | (q[0].abs() >= 601.0)  # EVMean's sentinel
                w = [u * torch.where(over, 1e10, torch.cosh(v)) for u, v in
                     zip(w, (0.5 * q[0] + 0.25 * n4, q[0], 0.5 * n4))]
            r = 8.0 / 3.0 * w[0] - 2.0 * w[1] + w[2] / 3.0
            out[i, j] = r.reshape(ng, -1).mean(1)
    return out


def _stats(g):
    ng = g.shape[2]
    sem = g.std(2) / math.sqrt(ng) if ng > 1 else torch.zeros_like(g[:, :, 0])
    return [g.cpu().numpy(), g.mean(2).cpu().numpy(), sem.cpu().numpy()]


def _igrand(c, rho, T, F, W):
    """Tfunc's integrand of the groups at one (rho, T, F)."""
    l2, e = c["lambda2"], E_CHARGE
    r2 = rho * rho
    if c["profile"] == "smooth":
        B, small = l2 / (l2 + r2) ** 2, 0.5 * (l2 + r2)
    else:
        B, small = (math.exp(-r2 / l2) / l2 if r2 < 100.0 * l2 else 0.0), l2
    B *= 2.0 * F / e
    tb, pre = e * T * B, math.exp(-T) / T ** 3
    b2 = (e * B) ** 2
    b4, b6 = b2 * b2, b2 ** 3
    if T < 0.1 and T < 0.01 * small:
        if c["fermion"]:
            v = b4 * T * (T - 1) / 45 + (2 * b6 / 945 - b4 / 90) * T ** 3 + \
                (7 * b4 - 4 * b6) / 1890 * T ** 4
        else:
            v = 7 / 360 * b4 * T * (1 - T) + (147 * b4 - 31 * b6) / 15120 * T ** 3 + \
                (31 * b6 - 49 * b4) / 15120 * T ** 4
        return torch.full_like(W, v)
    if T < 0.01 * small:
        if tb <= 1e-6 or B < 1e-40:
            return torch.zeros_like(W)
        if c["fermion"]:
            v = tb / math.tanh(tb) - 1 - tb * tb / 3
        else:
            v = (tb / math.sinh(tb) if tb < 50 else 0.0) - 1 + tb * tb / 6
        return torch.full_like(W, pre * v)
    if T > 49.0:
        return torch.full_like(W, (-1 / 3 if c["fermion"] else 1 / 6) * math.exp(-T) / T * b2)
    return pre * (W - 1 + (-tb * tb / 3 if c["fermion"] else tb * tb / 6))


def _integrals(c, loops, rhos, Ts, ws, F):
    """The proper-time integral per (rho, F, group)."""
    out = []
    for rho in rhos:
        W = _groups(c, loops, [rho] * len(Ts), [0.0] * len(Ts), Ts, F)
        out.append(torch.stack([sum(w * _igrand(c, rho, T, f, W[k, j])
                                    for k, (T, w) in enumerate(zip(Ts, ws)))
                                for j, f in enumerate(F)]))
    return torch.stack(out)


def _log_weights(T):
    """Simpson in ln T (3/8 on the last three intervals of an odd count)."""
    n, du = len(T), math.log(T[1] / T[0])
    w = np.zeros(n)
    m = n - 1 if (n - 1) % 2 == 0 else n - 4
    for k in range(0, m, 2):
        w[k:k + 3] += du / 3 * np.array([1.0, 4.0, 1.0])
    if m < n - 1:
        w[m:] += 3 * du / 8 * np.array([1.0, 3.0, 3.0, 1.0])
    return w * T


def _subst(n):
    """integrateT's nodes: T = (1 - t)/t, n Simpson panels in t; t = 1 adds 0."""
    h, T, w = 1.0 / n, [], []
    for i in range(n):
        for t, k in ((h * (i + 0.5), 4.0), (h * (i + 1), 2.0)):
            if t < 1.0 - 1e-12:
                T.append((1 - t) / t)
                w.append(k * h / 6 / t ** 2)
    return T, w


def _philox(seed, k, l):
    """Philox4x32-10 at counter (k, l, tag, 0): four uint32 as int64 tensors."""
    m32 = 0xFFFFFFFF
    k0, k1 = seed & m32, (seed >> 32) & m32
    c0, c1 = k.clone(), l.clone()
    c2, c3 = torch.full_like(k, 0x764C6F6F), torch.zeros_like(k)
    for r in range(10):
        if r:
            k0, k1 = (k0 + 0x9E3779B9) & m32, (k1 + 0xBB67AE85) & m32
        p0, p1 = c0 * 0xD2511F53, c2 * 0xCD9E8D57  # wraps in 64 bits as unsigned does
        h0, h1 = (p0 >> 32) & m32, (p1 >> 32) & m32
        c0, c1, c2, c3 = h1 ^ c1 ^ k0, p1 & m32, h0 ^ c3 ^ k1, p0 & m32
    return c0, c1, c2, c3


def _generated(seed, Nl, ppl):
    """The seeded ensemble: Box-Muller steps of variance 2/ppl, bridged."""
    k = torch.arange(ppl, device="cuda")[None, :].expand(Nl, ppl).contiguous()
    l = torch.arange(Nl, device="cuda")[:, None].expand(Nl, ppl).contiguous()
    r = [(v.double() + 0.5) / 4294967296.0 for v in _philox(seed, k, l)]
    rad, ang = torch.sqrt(-2.0 * torch.log(r[0])), 2.0 * math.pi * r[1]
    out = []
    for n in (rad * torch.cos(ang), rad * torch.sin(ang)):
        d = n * math.sqrt(2.0 / ppl)
        y = torch.cumsum(d, 1)
        x = y - d - k / ppl * y[:, -1:]
        out.append((x - x.mean(1, keepdim=True)).float())
    return torch.stack(out, 2)


def exact(case, seed):
    c = case
    if c["kind"] == "batch":
        jobs = _jobs(c)
        if sum(_cost(j) for j in jobs) > EXACT_MOST:
            return None
        return [_stats(_groups(j, _ensemble(j["Nl"], j["ppl"], seed * 64 + k),
                               *_instances(j, seed * 64 + k), _fluxes(j)))
                for k, j in enumerate(jobs)]
    if c["profile"] == "spline" or _cost(c) > EXACT_MOST:
        return None
    F = _fluxes(c)
    if c["kind"] == "fresh":
        return _stats(_groups(c, _generated(seed, c["Nl"], c["ppl"]), *_instances(c, seed), F))
    loops = _ensemble(c["Nl"], c["ppl"], seed)
    if c["kind"] in ("eval", "device"):
        return _stats(_groups(c, loops, *_instances(c, seed), F))
    norm = 1.0 / (4.0 * math.pi) if c["fermion"] else -1.0 / (2.0 * math.pi)
    if c["kind"] == "tint":
        rho, T = _rho_T(c, seed)
        I = _integrals(c, loops, rho, T, _log_weights(T), F)
        bins = I.reshape(len(rho), len(F), c["nbins"], -1)
        nb, n = c["nbins"], I.shape[2]
        loo = (I.sum(2, keepdim=True) - bins.sum(3)) / (n - n // nb)
        err = torch.sqrt((nb - 1) / nb * ((loo - I.mean(2, keepdim=True)) ** 2).sum(2))
        return [(norm * I.mean(2)).cpu().numpy(), (abs(norm) * err).cpu().numpy(), None]
    T, w = _subst(c["panels"])
    if c["kind"] == "chain":
        return _integrals(c, loops, [_chain_rho(c, seed)], T, w, F)[0, 0].cpu().numpy()
    h, rho, wr = 1.0 / c["nrho"], [], []
    for k in range(1, 2 * c["nrho"] + 1):  # rho = (1 - t)/t, panels in t
        t = 0.5 * h * k
        rho.append((1 - t) / t)
        wr.append((4.0 if k % 2 else 2.0) * h / 6 / t ** 2)
    I = _integrals(c, loops, rho, T, w, F)[:, 0]
    gam = norm * sum(v * r * i for v, r, i in zip(wr, rho, I))
    n = len(gam)
    return [gam.mean().item(), (gam.std() / math.sqrt(n)).item(), None, gam.cpu().numpy()]


def _cost(c):
    """Node evaluations in 64 bits, a lattice or continued fraction weighted."""
    w = {"lattice": 15.0, "fixflux": 40.0, "periodic": 6.0}.get(c["profile"], 1.0)
    return float(c["Nl"]) * c["ppl"] * _ninst(c) * (c["nint"] + 1) * w
