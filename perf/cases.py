"""Timed cases of the cubature framework: what its users have it do, through
the public Python front end (``cubature.Context`` and the per-step and network
entry points), over the sizes that its tests, its benchmark and its own
workloads use.

Kinds of case (``kind``):

* ``single``  -- one ``integrate`` call per listed integral, the drop-in call of
  the reference's API: latency of one result.
* ``batch``   -- ``integrate_batch``: many independent integrals of one family
  in one call, breadth-first or with the reference's two phases.
* ``table7``  -- ``integrate_table7_batch``: integrands on device tables.
* ``lclt``    -- ``integrate_lclt``: the 3-D five-table integrand over a box.
* ``steps``   -- one hand-driven breadth-first iteration on the caller's own
  tensors: ``rule_eval``, ``reduce``, ``split``.
* ``network`` -- the control-variate network by itself: gradients of a
  minibatch (forward and backward), a short training, inference.
* ``cv``      -- ``cv_integrate_batch``: train on the integrand, integrate the
  residual and the network.
"""
from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = Path(__file__).resolve().parents[1] / "old-gpuintegration_b200"
if str(_PKG) not in sys.path:
    sys.path.insert(0, str(_PKG))

import cubature as cub  # noqa: E402
from cubature import tables as cub_tables  # noqa: E402

EPSABS = 1e-12
LCLT_LO, LCLT_HI = (5.0, 0.12, 1.0), (60.0, 0.28, 5.0)


def listed():
    return [
        # One small integral, the smallest call there is: a 5-D Gaussian peak
        # at a loose tolerance.  Launch and host latency decide it.
        {"name": "gaussian_5d", "kind": "single", "items": "gaussian:5:4.5:5.5", "epsrel": 1e-3},
        # The headline pair: an 8-D oscillatory and an 8-D corner peak
        # integral, one call each, at epsrel 1e-6 (1 and about 10 iterations).
        {"name": "oscillatory_cornerpeak_8d", "kind": "single",
         "items": "oscillatory:8:1.0:1.2,corner_peak:8:0.45:0.55", "epsrel": 1e-6},
        # One hard integral under the reference's default policy: the first
        # phase fills up and the leftover boxes go through the second phase.
        {"name": "productpeak_5d_two_phase", "kind": "single", "items": "product_peak:5:15:25",
         "epsrel": 1e-6},
        # A parameter scan: some hundred easy integrals in one call, their
        # lists short enough for the persistent kernel throughout.
        {"name": "gaussian_4d_scan", "kind": "batch", "family": "gaussian", "ndim": 4,
         "count": 300, "amin": 1.0, "amax": 6.0, "epsrel": 1e-5, "policy": "reference"},
        # Integrals of uneven difficulty, breadth-first (the 6-D product-peak
        # batch of the benchmark, a sixteenth of it).
        {"name": "productpeak_6d_breadth", "kind": "batch", "family": "product_peak", "ndim": 6,
         "count": 256, "amin": 1.0, "amax": 50.0, "epsrel": 1e-5, "policy": "breadth"},
        # The same integrals under the reference's two-phase policy.
        {"name": "productpeak_6d_two_phase", "kind": "batch", "family": "product_peak", "ndim": 6,
         "count": 256, "amin": 1.0, "amax": 50.0, "epsrel": 1e-5, "policy": "reference"},
        # A smooth family whose value needs a transcendental of a sum over
        # the axes, in the largest dimension; an odd count.
        {"name": "cornerpeak_8d_breadth", "kind": "batch", "family": "corner_peak", "ndim": 8,
         "count": 37, "amin": 0.5, "amax": 2.0, "epsrel": 1e-6, "policy": "breadth"},
        # A model integrand built from interpolation tables (512-knot spline,
        # 128 x 128 grid), a few parameter sets per call.
        {"name": "table7", "kind": "table7", "count": 4, "epsrel": 1e-5},
        # The reference's own physics integrand over a box, one call.
        {"name": "lclt_3d", "kind": "lclt", "epsrel": 1e-6},
        # A user's own loop on its own tensors: rule, sums and split of a
        # million 6-D regions (not a multiple of any tile).
        {"name": "steps_6d_1m", "kind": "steps", "family": "gaussian", "ndim": 6,
         "regions": 1000003, "layout": 0},
        # The network alone: gradients, one epoch of training, inference.
        {"name": "network_16x8192", "kind": "network", "count": 16, "samples": 8192,
         "batch": 1024, "epochs": 1, "points": 20000},
        # The learned control variate end to end on 7-D product peaks.
        {"name": "cv_productpeak_7d", "kind": "cv", "count": 2, "amax": 8.0, "samples": 8192,
         "batch": 1024, "epochs": 30, "epsrel": 1e-4},
    ]


def _log_uniform(rng, a, b):
    return math.exp(rng.uniform(math.log(a), math.log(b)))


def _round(v):
    return float(f"{v:.3g}")


def draw(rng):
    kind = rng.choice(["single", "single", "single", "batch", "batch", "batch", "table7", "lclt",
                       "steps", "steps", "network", "cv"])
    eps = _round(_log_uniform(rng, 1e-6, 1e-3))
    if kind == "single":
        fam, nmin, nmax, a0, a1, emin = rng.choice([
            ("gaussian", 2, 6, 1.0, 5.0, 1e-5), ("oscillatory", 2, 8, 0.5, 2.0, 1e-6),
            ("corner_peak", 2, 8, 0.2, 1.0, 1e-6), ("product_peak", 2, 5, 2.0, 20.0, 1e-6),
            ("continuous", 2, 4, 1.0, 4.0, 1e-5), ("discontinuous", 2, 3, 0.2, 1.0, 1e-4)])
        n = rng.randint(nmin, nmax)
        return {"kind": kind, "items": f"{fam}:{n}:{a0}:{_round(rng.uniform(a0, a1) + 0.1)}",
                "epsrel": max(eps, emin)}
    if kind == "batch":
        fam = rng.choice(["product_peak", "product_peak", "gaussian", "corner_peak"])
        n = rng.randint(3, 6 if fam == "product_peak" else 5)
        amax = {"product_peak": _log_uniform(rng, 5, 50), "gaussian": _log_uniform(rng, 2, 8),
                "corner_peak": rng.uniform(0.6, 2.0)}[fam]
        return {"kind": kind, "family": fam, "ndim": n,
                "count": int(_log_uniform(rng, 16, 256 if n == 6 else 700)),
                "amin": 0.5 if fam == "corner_peak" else 1.0, "amax": _round(amax),
                "epsrel": max(eps, 1e-5), "policy": rng.choice(["breadth", "reference"])}
    if kind == "table7":
        return {"kind": kind, "count": rng.randint(1, 8),
                "epsrel": _round(_log_uniform(rng, 1e-5, 1e-3))}
    if kind == "lclt":
        return {"kind": kind, "epsrel": max(eps, 1e-6)}
    if kind == "steps":
        n = rng.randint(2, 8)
        return {"kind": kind,
                "family": rng.choice(["gaussian", "oscillatory", "corner_peak", "product_peak",
                                      "continuous"]),
                "ndim": n, "regions": int(_log_uniform(rng, 100, 1.2e6 if n < 7 else 4e5)),
                "layout": rng.randint(0, 1)}
    if kind == "network":
        batch = 128 * rng.choice([1, 2, 4, 8])
        return {"kind": kind, "count": rng.randint(1, 24), "samples": batch * rng.randint(1, 8),
                "batch": batch, "epochs": rng.randint(1, 2),
                "points": int(_log_uniform(rng, 100, 20000))}
    return {"kind": kind, "count": rng.randint(1, 2), "amax": _round(rng.uniform(2.0, 8.0)),
            "samples": 1024 * rng.randint(4, 8), "batch": 1024, "epochs": rng.randint(10, 30),
            "epsrel": _round(_log_uniform(rng, 1e-4, 1e-3))}


# ---- inputs ---------------------------------------------------------------

_CTX = []


def _ctx():
    """The program's one context, kept for its lifetime."""
    if not _CTX:
        _CTX.append(cub.Context(0))
    return _CTX[0]


def _family_params(rng, family, n, a0, a1):
    """Parameters of one integral: difficulty log-uniform in [a0, a1]."""
    a = np.exp(rng.uniform(math.log(a0), math.log(a1), n))
    if family == "oscillatory":
        u = np.full(n, rng.uniform(0.25, 0.35))
    elif family == "corner_peak":
        u = np.zeros(n)
    elif family == "product_peak":
        u = rng.uniform(0.1, 0.9, n)
    elif family == "discontinuous":
        u = rng.uniform(0.4, 0.8, n)
    else:
        u = rng.uniform(0.3, 0.7, n)
    return tuple(float(v) for v in a), tuple(float(v) for v in u)


def _items(case, seed):
    """(family, ndim, a, u) of each integral of a single, batch or cv case."""
    rng = np.random.default_rng([int(seed), 1])
    if case["kind"] == "single":
        out = []
        for it in case["items"].split(","):
            fam, n, a0, a1 = it.split(":")
            out.append((fam, int(n), *_family_params(rng, fam, int(n), float(a0), float(a1))))
        return out
    if case["kind"] == "cv":
        fam, n, a0, a1 = "product_peak", 7, 1.0, case["amax"]
    else:
        fam, n, a0, a1 = case["family"], case["ndim"], case["amin"], case["amax"]
    return [(fam, n, *_family_params(rng, fam, n, a0, a1)) for _ in range(case["count"])]


def _step_boxes(case, seed):
    """A region list as refinement leaves it: dyadic boxes of the unit cube,
    up to six halvings per axis, most of the list at the deeper levels."""
    n, m = case["ndim"], case["regions"]
    rng = np.random.default_rng([int(seed), 2])
    level = rng.binomial(6, 0.5, (n, m))
    length = np.ldexp(1.0, -level)
    lo = np.floor(rng.random((n, m)) / length) * length
    return lo, length


def _step_item(case, seed):
    fam = case["family"]
    a0, a1 = {"gaussian": (1, 6), "oscillatory": (0.5, 2), "corner_peak": (0.2, 1),
              "product_peak": (1, 20), "continuous": (1, 4)}[fam]
    return _family_params(np.random.default_rng([int(seed), 3]), fam, case["ndim"], a0, a1)


def _network_data(case, seed):
    """Samples of 7-D product peaks, weights of a start (He-uniform) and query points."""
    rng = np.random.default_rng([int(seed), 4])
    e, s = case["count"], case["samples"]
    x = rng.random((e, s, 7))
    a = np.exp(rng.uniform(0, math.log(5), (e, 1, 7)))
    u = rng.uniform(0.2, 0.8, (e, 1, 7))
    y = np.prod(1.0 / (a ** -2 + (x - u) ** 2), axis=2)
    p = np.zeros((e, cub.MLP_PARAMS), dtype=np.float32)
    w0 = np.zeros((e, 128, 16))
    w0[:, :, :7] = rng.uniform(-1, 1, (e, 128, 7)) / math.sqrt(7)
    p[:, :2048] = w0.reshape(e, -1)
    for k, m in ((2176, 16384), (18688, 16384), (35200, 128)):
        p[:, k:k + m] = rng.uniform(-1, 1, (e, m)) / math.sqrt(128)
    return x, y, p, rng.random((e, case["points"], 7))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "single":
        return {"case": case, "ctx": _ctx(),
                "f": [cub.Integrand(fam, n, a, u) for fam, n, a, u in _items(case, seed)]}
    if kind in ("batch", "cv"):
        st = {"case": case, "ctx": _ctx(),
              "params": [cub.make_params(n, a, u) for _, n, a, u in _items(case, seed)]}
        if kind == "batch":
            st["opts"] = cub.options(policy=cub.POLICY_BREADTH if case["policy"] == "breadth"
                                     else cub.POLICY_REFERENCE)
        return st
    if kind == "table7":
        return {"case": case, "ctx": _ctx(),
                "tables": cub_tables.Table7(cub_tables.table7_data(seed), 0),
                "offsets": list(cub_tables.table7_offsets(case["count"], seed + 1)),
                "opts": cub.options(policy=cub.POLICY_BREADTH)}
    if kind == "lclt":
        return {"case": case, "ctx": _ctx(),
                "tables": cub_tables.LcLtTables(cub_tables.lclt_data(seed), 0)}
    if kind == "steps":
        lo, length = _step_boxes(case, seed)
        a, u = _step_item(case, seed)
        # the program refines half of its list, by a rule of its own
        refine = np.zeros(case["regions"], dtype=np.int32)
        refine[np.random.default_rng([int(seed), 5]).permutation(case["regions"])[::2]] = 1
        return {"case": case, "f": cub.Integrand(case["family"], case["ndim"], a, u),
                "refine": torch.from_numpy(refine).cuda(), "lo": torch.from_numpy(lo).cuda(), "len": torch.from_numpy(length).cuda()}
    x, y, p, q = _network_data(case, seed)
    return {"case": case, "params": p, "x": torch.from_numpy(x).cuda(),
            "y": torch.from_numpy(y).cuda(), "q": torch.from_numpy(q).cuda()}


# ---- one pass -------------------------------------------------------------

def _results(res):
    return {"value": np.array([r.integral for r in res]),
            "error": np.array([r.error for r in res]),
            "nregions": np.array([r.nregions for r in res], dtype=np.int64),
            "neval": np.array([r.neval for r in res], dtype=np.int64),
            "status": np.array([r.status for r in res], dtype=np.int64)}


STEP_EPSREL = 1e-4


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "single":
        return _results([state["ctx"].integrate(f, case["epsrel"], EPSABS) for f in state["f"]])
    if kind == "batch":
        return _results(state["ctx"].integrate_batch(case["family"], case["ndim"],
                                                     state["params"], case["epsrel"], EPSABS,
                                                     state["opts"]))
    if kind == "cv":
        res, _ = state["ctx"].cv_integrate_batch(
            "product_peak", state["params"], case["epsrel"], EPSABS, samples=case["samples"],
            batch=case["batch"], epochs=case["epochs"])
        return _results(res)
    if kind == "table7":
        return _results(state["ctx"].integrate_table7_batch(
            state["tables"], state["offsets"], case["epsrel"], EPSABS, state["opts"]))
    if kind == "lclt":
        return _results([state["ctx"].integrate_lclt(state["tables"], LCLT_LO, LCLT_HI,
                                                     case["epsrel"], EPSABS)])
    if kind == "steps":
        lo, length = state["lo"], state["len"]
        avg, err, axis, active = cub.rule_eval(state["f"], lo, length, STEP_EPSREL, EPSABS)
        sums = cub.reduce(avg, err, active)
        clo, clen = cub.split(lo, length, state["refine"], axis, layout=case["layout"])
        return {"avg": avg, "err": err, "axis": axis, "active": active, "sums": sums,
                "child_lo": clo, "child_len": clen}
    # the network: a program creates it, gives it data, looks at a gradient,
    # trains it and evaluates it
    net = cub.Mlp(case["count"], case["samples"], case["batch"])
    net.set_params(state["params"])
    net.set_data(state["x"], state["y"])
    loss, grads = net.grad(0)
    last = net.train(case["epochs"], 1e-3)
    out = {"loss": loss, "grads": grads, "last_loss": last, "params": net.params(),
           "g": net.eval(state["q"])}
    net.close()
    return out


# ---- the work a pass cannot do without ------------------------------------

# FP64 operations of one integrand value (FMA = 2, a transcendental = 1) and
# of one rule node around it: coordinates 2n, five weighted sums 10, Jacobian 1.
_F = {"gaussian": lambda n: 4 * n + 1, "oscillatory": lambda n: 2 * n + 2,
      "corner_peak": lambda n: 2 * n + 6, "product_peak": lambda n: 6 * n,
      "continuous": lambda n: 4 * n + 1, "discontinuous": lambda n: 2 * n + 1,
      "table7": lambda n: 28, "lclt": lambda n: 120}


def _region_flops(family, n):
    return cub.npoints(n) * (2 * n + 11 + _F[family](n)) + 5 * n + 89


def _regions(family, n, a1, epsrel, policy="reference"):
    """Typical regions of one integral (the count depends on its parameters)."""
    grid = (2 if n >= 5 else 4) ** n
    tight = (1e-3 / epsrel)
    if family == "oscillatory":
        return grid * 1.5
    if family == "corner_peak":
        return grid * (1 + 0.6 * a1 * tight ** 0.4)
    if family == "product_peak":
        return grid * (1 + 0.02 * a1 * n * tight ** 0.8)
    if family == "gaussian":
        return grid * (1 + 2 * a1 * tight ** 0.3)
    return grid * (10 + 10 * tight ** 0.5)


def work(case):
    kind = case["kind"]
    if kind == "single":
        flops = 0.0
        items = case["items"].split(",")
        for it in items:
            fam, n, _, a1 = it.split(":")
            flops += _regions(fam, int(n), float(a1), case["epsrel"]) * _region_flops(fam, int(n))
        return {"bytes": len(items) * (32 * 8 + 56), "flops": flops}
    if kind == "batch":
        fam, n = case["family"], case["ndim"]
        flops = (case["count"] * _regions(fam, n, case["amax"], case["epsrel"], case["policy"]) *
                 _region_flops(fam, n))
        return {"bytes": case["count"] * (32 * 8 + 56), "flops": flops}
    if kind == "table7":
        regions = 128 * (1 + 60 * (1e-3 / case["epsrel"]) ** 1.2)
        return {"bytes": (3 * 512 + 128 * 128 + 256) * 8 + case["count"] * 64,
                "flops": case["count"] * regions * _region_flops("table7", 7)}
    if kind == "lclt":
        regions = 64 * (1 + 5 * (1e-3 / case["epsrel"]) ** 0.5)
        return {"bytes": 5 * 22 * 5 * 8 + 56, "flops": regions * _region_flops("lclt", 3)}
    if kind == "steps":
        n, m = case["ndim"], case["regions"]
        # boxes read by the rule and by the split, results written and read
        # once, half the list's children written
        return {"bytes": m * (2 * 16 * n + 2 * 24 + 16 * n),
                "flops": m * _region_flops(case["family"], n)}
    layers = 16 * 128 + 2 * 128 * 128 + 128
    if kind == "network":
        e = case["count"]
        rows = e * (case["batch"] + case["epochs"] * case["samples"])
        steps = 1 + case["epochs"] * (case["samples"] // case["batch"])
        return {"bytes": e * (case["samples"] * 8 * 8 + case["points"] * 8 * 8 +
                              2 * 4 * cub.MLP_PARAMS) + e * steps * 16 * cub.MLP_PARAMS,
                "flops": 6.0 * rows * layers + 2.0 * e * case["points"] * layers}
    rows = case["count"] * case["epochs"] * case["samples"]
    regions = 128 * (1 + 0.1 * case["amax"] ** 2 * (1e-3 / case["epsrel"]))
    return {"bytes": case["count"] * case["samples"] * 64,
            "flops": 6.0 * rows * layers +
            case["count"] * regions * cub.npoints(7) * (2.0 * layers + 60)}


# ---- 64-bit values --------------------------------------------------------

def _exact_integral(family, n, a, u):
    """Closed form of a family's integral over the unit cube."""
    if family == "gaussian":
        return math.prod(math.sqrt(math.pi) / (2 * a[i]) *
                         (math.erf(a[i] * (1 - u[i])) + math.erf(a[i] * u[i])) for i in range(n))
    if family == "oscillatory":
        z = complex(math.cos(2 * math.pi * u[0]), math.sin(2 * math.pi * u[0]))
        for i in range(n):
            z *= complex(math.sin(a[i]), 1 - math.cos(a[i])) / a[i]
        return z.real
    if family == "corner_peak":
        terms = []
        for m in range(1 << n):
            s = 1.0 + sum(a[i] for i in range(n) if m >> i & 1)
            terms.append((-1) ** bin(m).count("1") / s)
        return math.fsum(terms) / (math.factorial(n) * math.prod(a[:n]))
    if family == "product_peak":
        return math.prod(a[i] * (math.atan(a[i] * (1 - u[i])) + math.atan(a[i] * u[i]))
                         for i in range(n))
    if family == "continuous":
        return math.prod((2 - math.exp(-a[i] * u[i]) - math.exp(-a[i] * (1 - u[i]))) / a[i]
                         for i in range(n))
    top = [min(1.0, u[i]) if i < 2 else 1.0 for i in range(n)]
    return math.prod(math.expm1(a[i] * top[i]) / a[i] for i in range(n))


def _exact_table7(data, offset):
    """Integral of the 7-D table integrand: it factorises into the spline,
    the bilinear table and the kernel (its x3 axis in closed form, the others
    by Gauss-Legendre rules)."""
    sx, sy = data["spline_x"], data["spline_y"]
    k = len(sx)
    h = np.diff(sx)
    m = np.zeros((k, k))
    r = np.zeros(k)
    m[0, 0] = m[-1, -1] = 1.0
    i = np.arange(1, k - 1)
    m[i, i - 1], m[i, i], m[i, i + 1] = h[:-1], 2 * (h[:-1] + h[1:]), h[1:]
    r[1:-1] = 6 * (np.diff(sy)[1:] / h[1:] - np.diff(sy)[:-1] / h[:-1])
    y2 = np.linalg.solve(m, r)
    spline = float(np.sum(h * (sy[:-1] + sy[1:]) / 2 - h ** 3 * (y2[:-1] + y2[1:]) / 24))
    z = data["grid_z"]
    cell = np.outer(np.diff(data["grid_x"]), np.diff(data["grid_y"])) / 4
    grid = float(np.sum(cell * (z[:-1, :-1] + z[1:, :-1] + z[:-1, 1:] + z[1:, 1:])))
    x, w = np.polynomial.legendre.leggauss(60)
    x, w = (x + 1) / 2, w / 2
    x4 = ((x[:, None] + np.arange(8)) / 8).ravel()
    w4 = np.repeat(w / 8, 8)
    mu = offset + 2 * x4[:, None, None] + 0.1 * (x[:, None] + x)
    q = math.sqrt(2.0) * data["sigma"]
    erf = torch.special.erf
    inner = (erf(torch.from_numpy((4 - mu) / q)) - erf(torch.from_numpy(-mu / q))).numpy()
    inner *= math.sqrt(math.pi) * q / 8
    kern = float(np.einsum("i,j,k,ijk->", w4, w, w, inner))
    return spline * grid * kern


def _exact_lclt(data):
    """Gauss-Legendre over every table cell inside the box."""
    xs, ys, z = data["xs"], data["ys"], [torch.from_numpy(t) for t in data["z"]]
    x, w = np.polynomial.legendre.leggauss(24)
    x, w = torch.from_numpy((x + 1) / 2), torch.from_numpy(w / 2)
    cuts = lambda lo, hi, k: sorted({lo, hi, *[float(v) for v in k if lo < v < hi]})  # noqa: E731
    lc = torch.cat([LCLT_LO[2] + (LCLT_HI[2] - LCLT_LO[2]) * (x + p) / 24 for p in range(24)])
    wc = w.repeat(24) * (LCLT_HI[2] - LCLT_LO[2]) / 24
    bx, by = cuts(LCLT_LO[0], LCLT_HI[0], xs), cuts(LCLT_LO[1], LCLT_HI[1], ys)
    total = 0.0
    for x0, x1 in zip(bx, bx[1:]):
        i = int(np.searchsorted(xs, (x0 + x1) / 2)) - 1
        for y0, y1 in zip(by, by[1:]):
            j = int(np.searchsorted(ys, (y0 + y1) / 2)) - 1
            lt, zt = (x0 + (x1 - x0) * x)[:, None, None], (y0 + (y1 - y0) * x)[None, :, None]
            tx, ty = (lt - xs[i]) / (xs[i + 1] - xs[i]), (zt - ys[j]) / (ys[j + 1] - ys[j])
            tau, mu, sg, fm, fp = [
                (t[i, j] * (1 - tx) + t[i + 1, j] * tx) * (1 - ty) +
                (t[i, j + 1] * (1 - tx) + t[i + 1, j + 1] * tx) * ty for t in z]
            c = lc[None, None, :]
            et = torch.exp(tau * (2 * mu + tau * sg * sg - 2 * c) / 2)
            r, mts = math.sqrt(2.0) * sg, mu + tau * sg * sg
            erfc = torch.special.erfc
            v = ((1 - fm) * (1 - fp) * torch.exp(-((c - mu) / sg) ** 2 / 2) /
                 (math.sqrt(2 * math.pi) * sg) +
                 0.5 * ((1 - fm) * fp * tau + fm * fp / lt) * et * erfc((mts - c) / r) +
                 0.5 * fm / lt * (erfc((c - mu) / r) - erfc((c + lt - mu) / r)) -
                 0.5 * fm * fp / lt * torch.exp(-tau * lt) * et * erfc((mts - c - lt) / r))
            total += float(torch.einsum("i,j,k,ijk->", w, w, wc, v)) * (x1 - x0) * (y1 - y0)
    return total


def _exact_steps(case, seed):
    """The regions' values: the basic rule of degree 9 from its own points,
    one generator set at a time."""
    n = case["ndim"]
    lo, length = (torch.from_numpy(v) for v in _step_boxes(case, seed))
    a, u = _step_item(case, seed)
    fam = case["family"]
    gen = (.47795365790226950619, .20302858736911986780, .44762735462617812882, .125,
           .34303789878087814570)
    t = lambda d, c: (lo[d] + (0.5 + c) * length[d])  # noqa: E731

    def term(d, x):
        if fam == "gaussian":
            return (a[d] * (x - u[d])) ** 2
        if fam in ("oscillatory", "corner_peak"):
            return a[d] * x
        if fam == "product_peak":
            return torch.log(a[d] ** -2 + (x - u[d]) ** 2)
        return a[d] * (x - u[d]).abs()

    def value(s):
        if fam == "oscillatory":
            return torch.cos(2 * math.pi * u[0] + s)
        if fam == "corner_peak":
            return (1 + s) ** -(n + 1)
        return torch.exp(-s)

    cen = [term(d, t(d, 0.0)) for d in range(n)]
    tot = sum(cen)
    pm = [[[term(d, t(d, sg * g)) - cen[d] for sg in (1, -1)] for g in gen] for d in range(n)]
    sets = [value(tot)]
    for g in range(4):
        sets.append(sum(value(tot + v) for d in range(n) for v in pm[d][g]))
    sets.append(sum(value(tot + v + w) for d in range(n) for e in range(d + 1, n)
                    for v in pm[d][0] for w in pm[e][0]))
    sets.append(sum(value(tot + v + w) for d in range(n) for e in range(n) if e != d
                    for v in pm[d][0] for w in pm[e][1]))
    if n >= 3:
        sets.append(sum(value(tot + v + w + x) for d in range(n) for e in range(d + 1, n)
                        for f in range(e + 1, n) for v in pm[d][0] for w in pm[e][0]
                        for x in pm[f][0]))
    else:
        sets.append(torch.zeros_like(tot))
    sets.append(sum(value(tot + sum(pm[d][4][m >> d & 1] for d in range(n)))
                    for m in range(1 << n)))
    wt = (n * (n * (n * (-.0023611709677855117884) + .11415390023857325268) -
               .63833920076702389094) + .74849988504685208004,
          n * (n * .0035417564516782676826 - .072609367395893679605) + .10557491625218991012,
          n * -.04508628929435784076 + .21415883524352793401, .057693384490973483573, 0.0,
          .015532417276607053264 - n * .0035417564516782676826, .02254314464717892038,
          .0017708782258391338413, .25150011495314791996 / (1 << n))
    vol = torch.ones_like(tot)
    for d in range(n):
        vol = vol * length[d]
    return (sum(w * s for w, s in zip(wt, sets)) * vol).numpy()


def _network_forward(p, x):
    """The network in 64 bits from parameters p [e][...] at x [e][s][7]."""
    e = p.shape[0]
    w0, b0 = p[:, :2048].view(e, 128, 16)[:, :, :7], p[:, 2048:2176]
    w1, b1 = p[:, 2176:18560].view(e, 128, 128), p[:, 18560:18688]
    w2, b2 = p[:, 18688:35072].view(e, 128, 128), p[:, 35072:35200]
    w3, b3 = p[:, 35200:35328], p[:, 35328:35329]
    h = 2 * x - 1
    for w, b in ((w0, b0), (w1, b1), (w2, b2)):
        h = torch.nn.functional.silu(torch.bmm(h, w.transpose(1, 2)) + b[:, None, :])
    return torch.bmm(h, w3[:, :, None])[:, :, 0] + b3


def _exact_network(case, seed):
    x, y, p, _ = (torch.from_numpy(v).double() for v in _network_data(case, seed))
    scale = y.abs().amax(dim=1, keepdim=True)
    p.requires_grad_(True)
    d = (_network_forward(p, x[:, :case["batch"]]) - (y / scale)[:, :case["batch"]])
    loss = (d * d).mean(dim=1)
    loss.sum().backward()
    return {"loss": loss.detach().numpy(), "grads": p.grad.numpy(), "last_loss": None,
            "params": None, "g": None}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("single", "batch", "cv"):
        value = [_exact_integral(*it) for it in _items(case, seed)]
    elif kind == "table7":
        data = cub_tables.table7_data(seed)
        value = [_exact_table7(data, o)
                 for o in cub_tables.table7_offsets(case["count"], seed + 1)]
    elif kind == "lclt":
        value = [_exact_lclt(cub_tables.lclt_data(seed))]
    elif kind == "network":
        return _exact_network(case, seed)
    else:
        if case["regions"] * cub.npoints(case["ndim"]) > 1.5e9:
            return None  # over 20 seconds
        avg = _exact_steps(case, seed)
        return {"avg": avg, "err": None, "axis": None, "active": None, "sums": None,
                "child_lo": None, "child_len": None}
    return {"value": np.array(value), "error": None, "nregions": None, "neval": None,
            "status": None}
