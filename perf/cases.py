"""Performance cases: the work a user of this package has it do, through its
public entry points, over the range of sizes it is used at.

- interp_steps / InterpPlan, neighbour method 'all': ordinary, simple and
  external-drift kriging with the ordinary-kriging variance and IDW, in both
  precisions, from a handful of stations to thousands.
- interp_steps with the neighbour methods 'nrst' and 'pie'.
- the single-neighbourhood classes' computation on CUDA tensors
  (legacy.krige_points).
- leave-one-out cross-validation (steps.krige_loo).
- the variogram fitter (fitvgs.Empirical, fitvgs.fit_steps).

A case is a dict of plain values; sizes are those of the package's own bench
configurations and tests, with fewer steps or cells where a whole
configuration would take too long. Stations are uniform in a square of
8 km * sqrt(stations) (the density of those configurations) or clustered;
values are a smooth random field plus noise; variograms are the
configurations' (Exp, Sph with a nugget; Gau regularised by a micro-range
structure, the form under which its systems are not singular).
"""
import math

import numpy as np
import torch

# --------------------------------------------------------------- the cases

_INTERP = dict(path="interp", whole_call=False, methods="OK,IDW", variance=True,
               precision="fp64", models="Exp", missing=0.0, drifts=0, shared=False,
               clustered=False, f64_fields=False)


def _interp(name=None, **kw):
    c = dict(_INTERP, **kw)
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: a handful of gauges, three steps, a coarse grid,
        # numpy in and out (the package's smoke case)
        _interp("tiny_call_fp64", whole_call=True, stations=40, steps=3, nx=16, ny=12,
                f64_fields=True, missing=0.01),
        # the small configuration: a day of hourly steps of one region, every
        # gauge present, one variogram, in the default precision
        _interp("small_fp64", stations=150, steps=24, nx=200, ny=200, shared=True),
        # the same region with gaps in the series (every step its own system)
        # in mixed precision
        _interp("small_gaps_mixed", stations=150, steps=24, nx=200, ny=200, precision="mixed",
                missing=0.1, models="Sph"),
        # the batched configuration in the default precision: 1000 gauges with
        # gaps, ordinary kriging with its variance, simple kriging and IDW
        _interp("batched_fp64", stations=1000, steps=4, nx=250, ny=250, methods="OK,SK,IDW",
                models="mix", missing=0.25),
        # the batched configuration in mixed precision
        _interp("batched_mixed", stations=1000, steps=8, nx=500, ny=500, methods="OK,SK,IDW",
                models="mix", missing=0.25, precision="mixed"),
        # the large configuration: thousands of gauges, two drifts, a fine
        # grid, estimates only
        _interp("large_edk_mixed", stations=4000, steps=8, nx=1000, ny=1000, methods="EDK",
                variance=False, drifts=2, missing=0.275, precision="mixed"),
        # a long period of complete series: one system shared by every step
        _interp("edk_shared_fp64", stations=400, steps=200, nx=500, ny=500, methods="EDK",
                variance=False, drifts=1, shared=True, clustered=True, models="Sph"),
        # kriging and IDW from each cell's 16 nearest gauges
        dict(name="nearest16", path="nebs", neighbours="nrst", n_nebs=16, n_pies=1,
             stations=1000, steps=12, nx=250, ny=250, methods="OK,IDW", variance=True,
             models="mix", missing=0.25),
        # kriging from gauges spread over eight sectors around each cell, odd
        # grid sides
        dict(name="sectors12", path="nebs", neighbours="pie", n_nebs=12, n_pies=8,
             stations=300, steps=12, nx=151, ny=133, methods="OK", variance=True,
             models="Exp", missing=0.1),
        # one krige() of the single-neighbourhood ordinary kriging class, with
        # the weights of every point
        dict(name="single_ok", path="single", kind="OK", stations=400, points=250000,
             models="Exp"),
        # cross-validation of two months of daily variograms
        dict(name="loo_60_days", path="loo", stations=500, steps=60, models="mix",
             missing=0.25),
        # fitting the variograms of a month of days
        dict(name="fit_30_days", path="fit", stations=300, steps=30, missing=0.25),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sides(rng, cells):
    """An nx x ny grid of about that many cells, sides not alike."""
    nx = max(3, int(round(math.sqrt(cells) * rng.uniform(0.7, 1.4))))
    return nx, max(3, int(cells // nx))


def draw(rng):
    kind = rng.choices(["call", "fp64", "mixed", "edk", "shared", "nebs", "single", "loo", "fit"],
                       [2, 4, 4, 2, 2, 3, 1, 1, 1])[0]
    miss = rng.choice([0.0, 0.1, 0.25, 0.4])
    models = rng.choice(["Exp", "Sph", "mix"])
    if kind == "call":
        nx, ny = _sides(rng, _log(rng, 100, 20000))
        return _interp(whole_call=True, stations=_log(rng, 12, 200), steps=rng.randint(1, 24),
                       nx=nx, ny=ny, missing=miss, models=rng.choice(["Exp", "Sph"]),
                       precision=rng.choice(["fp64", "mixed"]), variance=rng.random() < 0.7,
                       methods=rng.choice(["OK", "OK,IDW", "OK,SK", "IDW"]))
    if kind in ("fp64", "mixed"):
        mixed = kind == "mixed"
        n = _log(rng, 30, 1000)
        steps = rng.randint(1, 8 if mixed else 6)
        most = (250000 * 8 if mixed else 62500 * 4) // steps
        nx, ny = _sides(rng, min(_log(rng, 2000, 250000), most))
        return _interp(stations=n, steps=steps, nx=nx, ny=ny, missing=miss, models=models,
                       precision=kind, variance=rng.random() < 0.75,
                       methods=rng.choice(["OK", "OK,IDW", "OK,SK,IDW", "SK"]))
    if kind == "edk":
        nx, ny = _sides(rng, _log(rng, 20000, 500000))
        return _interp(stations=_log(rng, 200, 3000), steps=rng.randint(1, 6), nx=nx, ny=ny,
                       methods="EDK", variance=False, drifts=rng.randint(1, 3), missing=miss,
                       models=rng.choice(["Exp", "Sph"]), precision="mixed")
    if kind == "shared":
        nx, ny = _sides(rng, _log(rng, 5000, 200000))
        drifts = rng.randint(0, 2)
        return _interp(stations=_log(rng, 50, 400), steps=_log(rng, 20, 200), nx=nx, ny=ny,
                       methods="EDK" if drifts else "OK", variance=not drifts, drifts=drifts,
                       shared=True, clustered=rng.random() < 0.5,
                       models=rng.choice(["Exp", "Sph"]))
    if kind == "nebs":
        nx, ny = _sides(rng, _log(rng, 1000, 60000))
        pie = rng.random() < 0.4
        return dict(path="nebs", neighbours="pie" if pie else "nrst",
                    n_nebs=rng.randint(8, 24), n_pies=rng.choice([4, 8]) if pie else 1,
                    stations=_log(rng, 100, 600 if pie else 1000), steps=rng.randint(2, 10),
                    nx=nx, ny=ny, methods=rng.choice(["OK", "OK,IDW"]), variance=True,
                    models=rng.choice(["Exp", "mix"]), missing=rng.choice([0.0, 0.1, 0.25]))
    if kind == "single":
        return dict(path="single", kind=rng.choice(["OK", "SK"]), stations=_log(rng, 30, 400),
                    points=_log(rng, 1000, 250000), models=rng.choice(["Exp", "Sph"]))
    if kind == "loo":
        return dict(path="loo", stations=_log(rng, 40, 600), steps=rng.randint(3, 60),
                    models=models, missing=miss)
    return dict(path="fit", stations=_log(rng, 60, 400), steps=rng.randint(3, 30), missing=miss)


# --------------------------------------------------------------- the inputs


def _field(rng, x, y, steps, scale):
    """[steps, points] smooth random fields (random cosines of wavelengths
    around ``scale``), unit variance, at the points."""
    k = 48
    w = rng.normal(size=(steps, k, 2)) * (2.0 / scale)
    ph = rng.uniform(0, 2 * math.pi, (steps, k, 1))
    out = np.empty((steps, x.size))
    for t in range(steps):
        a = w[t, :, :1] * x[None] + w[t, :, 1:] * y[None] + ph[t]
        out[t] = math.sqrt(2.0 / k) * np.cos(a).sum(0)
    return out


def _stations(rng, n, box, clustered):
    if not clustered:
        return rng.uniform(0, box, n), rng.uniform(0, box, n)
    px, py = rng.uniform(0, box, 20), rng.uniform(0, box, 20)
    k = rng.integers(0, 20, n)
    return px[k] + rng.normal(0, 0.01 * box, n), py[k] + rng.normal(0, 0.01 * box, n)


def _variograms(rng, steps, models, shared):
    out = []
    for t in range(steps):
        m = models if models != "mix" else ("Sph", "Exp", "Gau")[t % 3]
        sill, nug = rng.uniform(0.5, 2.0), rng.uniform(0.02, 0.2)
        if m == "Gau":
            out.append("%.8f Exp(1.0) + %.5f Gau(%.1f)" % (1e-5 * sill, sill,
                                                           rng.uniform(10e3, 30e3)))
        else:
            out.append("%.5f Nug(0.0) + %.5f %s(%.1f)" % (nug * sill, sill - nug * sill, m,
                                                          rng.uniform(15e3, 80e3)))
    return [out[0]] * steps if shared else out


def _inputs(case, seed):
    """Stations, values, grid, variograms and drifts, as numpy arrays."""
    rng = np.random.default_rng([seed, case["stations"]])
    n = case["stations"]
    steps = case.get("steps", 1)
    box = 8e3 * math.sqrt(n)
    sx, sy = _stations(rng, n, box, case.get("clustered", False))
    z = 3.0 + _field(rng, sx, sy, steps, 40e3) + 0.2 * rng.normal(size=(steps, n))
    z = np.maximum(z, 0.0)
    if case.get("missing", 0.0) > 0:
        gone = rng.uniform(size=z.shape) < case["missing"]
        gone[:, :8] = False
        z[gone] = np.nan
    vgs = _variograms(rng, steps, case.get("models", "Exp"), case.get("shared", False))
    w = dict(sx=sx, sy=sy, z=z, vgs=vgs, cx=None, cy=None, sd=None, cd=None)
    if "points" in case:
        w["cx"], w["cy"] = (rng.uniform(0, box, case["points"]) for _ in range(2))
    elif "nx" in case:
        xs = (np.arange(case["nx"]) + 0.5) * (box / case["nx"])
        ys = (np.arange(case["ny"])[::-1] + 0.5) * (box / case["ny"])
        gx, gy = np.meshgrid(xs, ys)
        w["cx"], w["cy"] = gx.ravel().copy(), gy.ravel().copy()
    k = case.get("drifts", 0)
    if k:
        # smooth terrain-like drifts, the same function at stations and cells
        px, py = np.concatenate([sx, w["cx"]]), np.concatenate([sy, w["cy"]])
        d = np.empty((k, px.size))
        for i in range(k):
            a, b, p = rng.uniform(1, 4), rng.uniform(1, 4), rng.uniform(0, 6.28)
            d[i] = 500.0 + 400.0 * np.sin(a * px / box * 3 + p) * np.cos(b * py / box * 3)
        w["sd"], w["cd"] = d[:, :n].T.copy(), d[:, n:].copy()
    return w


def _methods(case):
    return [("IDW", 2.0) if m == "IDW" else m for m in case["methods"].split(",")]


_MIN_VG = 1e-4


def _most_bins(case):
    """Bins of 50 pairs that complete series would fill."""
    n = case["stations"]
    return case["steps"] * ((n * (n - 1) // 2 + 49) // 50)


def prepare(case, seed):
    from spinterps_gb300 import fitvgs, legacy, steps
    w = _inputs(case, seed)
    p = case["path"]
    if p in ("interp", "nebs"):
        var = bool(case["variance"]) and "OK" in case["methods"].split(",")
        iargs = steps.interp_args_for(_methods(case), est_vars=var)
        kw = dict(est_vars=var, min_var_cut=0.0, min_vg_val=_MIN_VG)
        if p == "nebs":
            kw.update(neb_sel_mthd=case["neighbours"], n_nebs=case["n_nebs"],
                      n_pies=case["n_pies"])
        else:
            kw.update(precision=case["precision"], stn_drifts=w["sd"], cell_drifts=w["cd"],
                      intrp_dtype=np.float64 if case["f64_fields"] else np.float32)
        args = (w["sx"], w["sy"], w["z"], w["cx"], w["cy"], w["vgs"], iargs)
        if p == "nebs" or case["whole_call"]:
            return dict(call=steps.interp_steps, args=args, kw=kw)
        # a program that runs a job repeatedly keeps its plan
        return dict(plan=steps.InterpPlan(*args, **kw))
    if p == "single":
        dev = [torch.as_tensor(a, device="cuda") for a in
               (w["sx"], w["sy"], np.ascontiguousarray(w["z"][0]), w["cx"], w["cy"])]
        return dict(single=legacy.krige_points, kind=case["kind"], dev=dev, model=w["vgs"][0])
    if p == "loo":
        return dict(loo=steps.krige_loo, args=(w["sx"], w["sy"], w["z"], w["vgs"]),
                    kw=dict(min_vg_val=_MIN_VG), shape=w["z"].shape)
    return dict(fit=fitvgs, points=fitvgs.step_points(w["sx"], w["sy"], w["z"]),
                bins=_most_bins(case))


def run(state):
    if "plan" in state:
        state["plan"].execute()
        return dict(state["plan"].flds)
    if "call" in state:
        return dict(state["call"](*state["args"], **state["kw"])[0])
    if "single" in state:
        r = state["single"](state["kind"], *state["dev"], state["model"])
        return {k: v for k, v in r.items() if isinstance(v, torch.Tensor)}
    if "loo" in state:
        res, rmse = state["loo"](*state["args"], **state["kw"])
        table = np.full(state["shape"], np.nan)
        for row, r in zip(table, res):
            row[:r.size] = r
        return dict(residuals=table, rmse=rmse)
    fit = state["fit"]
    emp = fit.Empirical(None, None, None, points=state["points"]).run()
    _, det = fit.fit_steps(None, None, None, emp=emp, seed=1, return_details=True)
    steps = [d for k, d in sorted((k, d) for k, d in det.items() if not isinstance(k, str))]
    best = np.zeros((len(steps), 4))
    for row, d in zip(best, steps):
        row[:d["params"].size] = d["params"]
    pad = (0, state["bins"] - emp.bin_h.numel())
    return dict(objective=np.array([list(d["objective"].values()) for d in steps]),
                generations=np.array([list(d["generations"].values()) for d in steps]),
                best=best, bin_h=torch.nn.functional.pad(emp.bin_h, pad),
                bin_g=torch.nn.functional.pad(emp.bin_g, pad), n_bins=emp.n_bins)


# --------------------------------------------------------- work and exact


def work(case):
    p = case["path"]
    n = case["stations"] * (1.0 - case.get("missing", 0.0))
    T = case.get("steps", 1)
    if p in ("interp", "nebs"):
        C = case["nx"] * case["ny"]
        fields = case["methods"].split(",")
        nout = len(fields) + (1 if case["variance"] and "OK" in fields else 0)
        size = 8 if case.get("f64_fields") else 4
        by = nout * T * C * size + 16.0 * C * (1 + case.get("drifts", 0)) + 8.0 * T * n
        if p == "nebs":
            # the neighbour search's output, one system per neighbour list
            # (about four per station) and its use at the cells
            k = case["n_nebs"]
            fl = T * (4 * n * 2 / 3 * k ** 3 + C * (2.0 * k * k + 4 * k))
            return dict(bytes=by + 4.0 * T * C * k, flops=fl)
        S = 1 if case["shared"] else T
        fl = 0.0
        for f in fields:
            if f == "IDW":
                fl += 4.0 * n * T * C
                continue
            fl += S * n ** 3 / 3 + 2.0 * n * T * C
            if f == "OK" and case["variance"]:
                fl += S * (n ** 3 / 3 + n * n * C)
            fl += 2.0 * n * S * C * (1 + case["drifts"])
        return dict(bytes=by, flops=fl)
    if p == "single":
        m = n + 1
        return dict(bytes=8.0 * case["points"] * (2 * m + 4), flops=2 * m ** 3 / 3
                    + 2.0 * m * m * case["points"])
    if p == "loo":
        return dict(bytes=16.0 * T * n, flops=T * 2 * n ** 3 / 3)
    # the pairs of every step, and the search's model evaluations (about
    # 200 generations of 200 members over the bins for 5 model nests)
    return dict(bytes=24.0 * T * n * n / 2, flops=T * (n * n * 8 + 5 * 200 * 200 * 40 * 10.0))


def _parse(vg):
    out = []
    for c in vg.split("+"):
        s, m = c.split()
        name, r = m[:-1].split("(")
        out.append((name, float(s), max(1e-5, float(r))))
    return out


def _gamma(vg, h):
    g = torch.zeros_like(h)
    for name, s, r in _parse(vg):
        if name == "Nug":
            g += s
        elif name == "Exp":
            g += s * (1.0 - torch.exp(-3.0 * h / r))
        elif name == "Gau":
            g += s * (1.0 - torch.exp(-3.0 * (h / r) ** 2))
        else:
            t = torch.clamp(h / r, max=1.0)
            g += s * (1.5 * t - 0.5 * t ** 3)
    return g


def _sill(vg):
    return sum(c[1] for c in _parse(vg))


def _dist(ax, ay, bx, by):
    return torch.sqrt((ax[:, None] - bx[None]) ** 2 + (ay[:, None] - by[None]) ** 2)


def _cut(g):
    return torch.where(g <= _MIN_VG, torch.zeros_like(g), g)


def _exact_step(kind, vg, x, y, z, cx, cy, sd, cd, want_var):
    """(estimate, variance) of one step over all cells, the whole saddle
    system in float64."""
    n = x.numel()
    h = _dist(x, y, x, y)
    if kind == "SK":
        M = _cut(_sill(vg) - _gamma(vg, h))
        a = 0
    else:
        F = torch.ones((n, 1), dtype=x.dtype, device=x.device)
        if kind == "EDK":
            F = torch.cat([F, sd], 1)
        a = F.shape[1]
        M = torch.zeros((n + a, n + a), dtype=x.dtype, device=x.device)
        M[:n, :n] = _cut(_gamma(vg, h))
        M[:n, n:] = F
        M[n:, :n] = F.T
    rhs = torch.zeros((n + a, 2), dtype=x.dtype, device=x.device)
    rhs[:n, 0] = z
    rhs[:n, 1] = 1.0
    w = torch.linalg.solve(M, rhs)
    P = torch.linalg.inv(M) if want_var else None
    est = torch.empty_like(cx)
    var = torch.empty_like(cx) if want_var else None
    step = max(1, int(2e8 // (8 * (n + a))) * 4)
    for b in range(0, cx.numel(), step):
        e = min(cx.numel(), b + step)
        d = _dist(cx[b:e], cy[b:e], x, y)
        r = _cut(_sill(vg) - _gamma(vg, d)) if kind == "SK" else _cut(_gamma(vg, d))
        if a:
            f = torch.ones((e - b, a), dtype=x.dtype, device=x.device)
            if kind == "EDK":
                f[:, 1:] = cd[:, b:e].T
            r = torch.cat([r, f], 1)
        both = r @ w
        ok = (both[:, 1] - 1.0).abs() <= 1e-8 + 1e-5
        near = z[d.argmin(1)]
        est[b:e] = torch.where(ok, both[:, 0], near)
        if want_var:
            lam = r @ P
            v = (lam * r).sum(1) + lam[:, n]
            var[b:e] = torch.where(ok, v, torch.zeros_like(v))
    return est, var


def _neighbours(case, cx, cy, x, y):
    """[cells, k] neighbour indices by the method's rule."""
    out = []
    for b in range(0, cx.numel(), 8192):
        d = _dist(cx[b:b + 8192], cy[b:b + 8192], x, y)
        if case["neighbours"] == "nrst":
            out.append(d.topk(min(case["n_nebs"], x.numel()), 1, largest=False).indices)
            continue
        # sector of every station as seen from the cell, its rank by
        # distance within the sector, then the order (rank, distance)
        dx = x[None] - cx[b:b + 8192, None]
        dy = y[None] - cy[b:b + 8192, None]
        ang = torch.atan2(dy, dx)
        ang = torch.where(ang < 0, ang + 2 * math.pi, ang)
        sec = (ang * case["n_pies"] / (2 * math.pi)).long().clamp(max=case["n_pies"] - 1)
        order = d.argsort(1)
        sec_o = sec.gather(1, order)
        hot = torch.nn.functional.one_hot(sec_o, case["n_pies"]).to(torch.int32)
        rank = hot.cumsum(1).gather(2, sec_o[..., None])[..., 0]
        pos = rank.to(torch.int64) * x.numel() + torch.arange(x.numel(), device=x.device)
        out.append(order.gather(1, pos.argsort(1)[:, :case["n_nebs"]]))
    return torch.cat(out)


def _exact_nebs(case, w, t, kind, cx, cy, x, y, z):
    nb = _neighbours(case, cx, cy, x, y)
    est, var = torch.empty_like(cx), torch.empty_like(cx)
    k = nb.shape[1]
    for b in range(0, cx.numel(), 16384):
        e = min(cx.numel(), b + 16384)
        i = nb[b:e]
        X, Y, Z = x[i], y[i], z[i]
        d = torch.sqrt((X - cx[b:e, None]) ** 2 + (Y - cy[b:e, None]) ** 2)
        if kind == "IDW":
            wt = (d / d.amin(1, keepdim=True)) ** -2.0
            est[b:e] = (wt * Z).sum(1) / wt.sum(1)
            continue
        M = torch.ones((e - b, k + 1, k + 1), dtype=x.dtype, device=x.device)
        M[:, k, k] = 0.0
        h = torch.sqrt((X[:, :, None] - X[:, None]) ** 2 + (Y[:, :, None] - Y[:, None]) ** 2)
        M[:, :k, :k] = _cut(_gamma(w["vgs"][t], h))
        r = torch.ones((e - b, k + 1), dtype=x.dtype, device=x.device)
        r[:, :k] = _cut(_gamma(w["vgs"][t], d))
        lam = torch.linalg.solve(M, r[..., None])[..., 0]
        est[b:e] = (lam[:, :k] * Z).sum(1)
        var[b:e] = (lam * r).sum(1) + lam[:, k]
    return est, var


def exact(case, seed):
    w = _inputs(case, seed)
    p = case["path"]
    if p == "fit":
        return None  # a seeded random search: no value in closed form
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    t64 = lambda a: None if a is None else torch.as_tensor(a, dtype=torch.float64, device=dev)  # noqa: E731
    sx, sy, z, cx, cy, sd, cd = (t64(w[k]) for k in ("sx", "sy", "z", "cx", "cy", "sd", "cd"))
    if p == "single":
        return _exact_single(case, w["vgs"][0], sx, sy, z[0].contiguous(), cx, cy)
    if p == "loo":
        res = []
        for t in range(z.shape[0]):
            i = torch.isfinite(z[t])
            n = int(i.sum())
            M = torch.ones((n + 1, n + 1), dtype=torch.float64, device=dev)
            M[:n, :n] = _cut(_gamma(w["vgs"][t], _dist(sx[i], sy[i], sx[i], sy[i])))
            M[n, n] = 0.0
            P = torch.linalg.inv(M)
            res.append((P[:n, :n] @ z[t][i]) / P.diagonal()[:n])
        rmse = torch.stack([torch.sqrt((r * r).mean()) for r in res])
        table = torch.full_like(z, math.nan)
        for row, r in zip(table, res):
            row[:r.numel()] = r
        return dict(residuals=table, rmse=rmse)
    out = {}
    var = bool(case["variance"]) and "OK" in case["methods"].split(",")
    names = [("IDW_000", m) if m == "IDW" else (m, m) for m in case["methods"].split(",")]
    if p == "nebs":
        used = torch.unique(_neighbours(case, cx, cy, sx, sy))
        sx, sy, z = sx[used], sy[used], z[:, used]
    for label, m in names:
        est, vs = [], []
        for t in range(z.shape[0]):
            i = torch.isfinite(z[t])
            x, y, zt = sx[i], sy[i], z[t][i]
            if p == "nebs":
                e, v = _exact_nebs(case, w, t, m, cx, cy, x, y, zt)
            elif m == "IDW":
                e, v = torch.empty_like(cx), None
                for b in range(0, cx.numel(), 65536):
                    wt = _dist(cx[b:b + 65536], cy[b:b + 65536], x, y)
                    wt = (wt / wt.amin(1, keepdim=True)) ** -2.0
                    e[b:b + 65536] = (wt @ zt) / wt.sum(1)
            else:
                e, v = _exact_step(m, w["vgs"][t], x, y, zt, cx, cy, sd[i] if sd is not None
                                   else None, cd, var and m == "OK")
            est.append(e.clamp(min=0.0))
            vs.append(v)
        out[label] = torch.stack(est)
        if var and m == "OK":
            out["EST_VARS_OK"] = torch.stack(vs)
    return out


def _exact_single(case, vg, x, y, z, cx, cy):
    n, sk = x.numel(), case["kind"] == "SK"
    h = _dist(x, y, x, y)
    g = _gamma(vg, h)
    g.fill_diagonal_(0.0)
    a = 0 if sk else 1
    M = torch.zeros((n + a, n + a), dtype=x.dtype, device=x.device)
    M[:n, :n] = -g if sk else g
    if a:
        M[n, :n] = M[:n, n] = 1.0
    P = torch.linalg.inv(M)
    r = _gamma(vg, _dist(cx, cy, x, y))
    r = _sill(vg) - r if sk else torch.cat([r, torch.ones_like(cx)[:, None]], 1)
    lam = r @ P
    lk = lam[:, :n]
    out = dict(in_dists=h, lhs=M, lhs_inv=P, rhss=r, lambdas=lk, zk=lk @ z)
    if sk:
        out["est"] = (_sill(vg) - (lk * r).sum(1)).clamp(min=0.0)
    else:
        out["mus"] = lam[:, n:].T
        out["est"] = ((lk * r[:, :n]).sum(1) + lam[:, n]).clamp(min=0.0)
    return out
