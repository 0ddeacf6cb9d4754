"""The FP64 cell pass as sliced tensor-core products (csrc/spi_slices.cu) at
the sizes where it can go wrong: around a 16-station stage, a 64-row block, a
128-station drain, a 128-cell tile; several blocks of steps; every model with
a fixed-point form, nests, and models without one (which keep the FP64
kernels) in the same batch.

Against the oracle at the FP64 path's bar, 1e-9 of the field's largest
magnitude, and against the FP64 kernels (tensor_cores=False) at 1e-11: both
are FP64 evaluations of the same formulas from the same factor (condition up
to 1e5, so rounding of 1e-16 may grow to 1e-11).
"""
import numpy as np
import pytest

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oracle import port  # noqa: E402


def _run(n, T, C, methods, vgs, seed, drifts=0, min_vg=1e-4, oracle=True, precision="fp64"):
    from spinterps_gb300 import steps
    rng = np.random.default_rng(seed)
    box = 8e3 * np.sqrt(n)
    sx, sy = rng.uniform(0, box, n), rng.uniform(0, box, n)
    z = 3.0 + rng.normal(size=(T, n))
    cx, cy = rng.uniform(0, box, C), rng.uniform(0, box, C)
    cx[0], cy[0] = sx[1], sy[1]          # a cell on a station
    est_vars = "OK" in methods
    args = port.interp_args_for(methods, est_vars=est_vars)
    kw = dict(est_vars=est_vars, min_vg_val=min_vg, intrp_dtype=np.float64)
    if drifts:
        kw.update(stn_drifts=rng.uniform(0, 1, (n, drifts)),
                  cell_drifts=rng.uniform(0, 1, (drifts, C)))
    vgs = [vgs[t % len(vgs)] for t in range(T)]
    got, plain = (steps.interp_steps(sx, sy, z, cx, cy, vgs, args, precision=precision,
                                     tensor_cores=tc, **kw)[0] for tc in (True, False))
    bar = 1e-11 if precision == "fp64" else 1e-5
    for lab in plain:
        sc = np.nanmax(np.abs(plain[lab]))
        assert np.nanmax(np.abs(got[lab] - plain[lab])) <= bar * sc, (n, lab)
    if oracle:
        ref, _ = port.interp_steps(sx, sy, z, cx, cy, vgs, args, **kw)
        for lab in ref:
            sc = np.nanmax(np.abs(ref[lab]))
            assert np.nanmax(np.abs(got[lab] - ref[lab])) <= max(bar, 1e-9) * sc, (n, lab)


EXP = "0.05 Nug(0.0) + 0.95 Exp(20000)"


@pytest.mark.parametrize("n", [64, 65, 79, 80, 81, 127, 128, 129, 144, 145, 192, 193, 257])
def test_station_counts(n):
    _run(n, 3, 131, ["OK", "SK"], [EXP], 10 + n)


@pytest.mark.parametrize("C", [1, 127, 128, 129, 257])
def test_cell_counts(C):
    _run(70, 2, C + 1, ["OK"], [EXP], 30 + C)


@pytest.mark.parametrize("T,drifts", [(63, 0), (64, 0), (65, 0), (62, 1), (130, 3)])
def test_blocks_of_steps(T, drifts):
    _run(66, T, 40, ["EDK"] if drifts else ["OK"], [EXP], 50 + T, drifts)


@pytest.mark.parametrize("vg", ["0.9 Sph(60000)", "0.9 Lin(400000)", "0.00001 Exp(1.0) + 0.9 Gau(15000)",
                                "0.3 Sph(50000) + 0.1 Nug(0.0) + 0.6 Exp(90000)",
                                "0.00005 Nug(0.0) + 1.4 Sph(30000)"])
def test_models(vg):
    _run(100, 2, 150, ["OK", "SK"], [vg], 70, oracle="Lin" not in vg)


def test_models_without_a_sliced_form():
    """Hol and Pow beside Exp in one batch."""
    _run(90, 6, 140, ["OK"], [EXP, "0.9 Hol(9000) + 0.3 Exp(20000)", "0.0001 Pow(0.9)"], 80,
         oracle=False)


@pytest.mark.parametrize("min_vg", [0.0, 0.02, 0.3])
def test_cut(min_vg):
    _run(80, 2, 200, ["OK"], ["0.95 Exp(30000)"], 90, min_vg=min_vg, oracle=min_vg < 0.1)


def test_double_float_tier():
    """Mixed precision: ill-conditioned systems take the sliced variance."""
    _run(150, 3, 300, ["OK"], ["0.00001 Exp(1.0) + 0.9 Gau(25000)"], 95, precision="mixed")


@pytest.mark.parametrize("kind", ["OK", "SK", "EDK"])
@pytest.mark.parametrize("n,C", [(63, 600), (64, 513), (95, 640), (96, 700), (127, 515), (200, 900)])
def test_single_neighbourhood(kind, n, C, monkeypatch):
    """The classes' weights as sliced products and their matrix inverted step
    by step over the GPU, against the oracle's restatement of the classes:
    1e-9 of each array's largest value (condition up to 1e5)."""
    import torch
    from spinterps_gb300 import legacy
    monkeypatch.setattr(legacy, "SLICES_MIN_WORK", 0)
    rng = np.random.default_rng(n)
    xi, yi, zi = rng.uniform(0, 1e5, n), rng.uniform(0, 1e5, n), rng.gamma(1.2, 3.0, n)
    xk, yk = rng.uniform(0, 1e5, C), rng.uniform(0, 1e5, C)
    xk[0], yk[0] = xi[2], yi[2]
    si = rng.uniform(0, 2, (2, n)) if kind == "EDK" else None
    sk = rng.uniform(0, 2, (2, C)) if kind == "EDK" else None
    model = "0.1 Nug(0.0) + 0.9 Exp(30000)"
    d = lambda a: None if a is None else torch.as_tensor(a, device="cuda")  # noqa: E731
    got = legacy.krige_points(kind, d(xi), d(yi), d(zi), d(xk), d(yk), model, si=d(si), sk=d(sk))
    cls = {"OK": "OrdinaryKriging", "SK": "SimpleKriging", "EDK": "ExternalDriftKriging_MD"}[kind]
    ref = port.legacy_krige(cls, xi, yi, zi, xk, yk, model, si=si, sk=sk)
    for k in ("zk", "lambdas", "rhss", "in_dists"):
        a, b = got[k].cpu().numpy(), ref[k]
        assert np.abs(a - b).max() <= 1e-9 * np.abs(b).max(), k


@pytest.mark.parametrize("kind", ["OK", "SK", "EDK"])
@pytest.mark.parametrize("model", ["0.1 Nug(0.0) + 0.9 Exp(30000)", "2.5 Sph(60000)",
                                   "0.3 Nug(0.0) + 1.2 Gau(9000)", "1.0 Lin(50000)",
                                   "0.2 Nug(0.0) + 0.5 Exp(9000) + 0.7 Sph(50000)",
                                   "0.5 Exp(1e-5)", "0.7 Hol(20000)", "1.0 Pow(1.2)", "2.0 Nug(0.0)"])
def test_single_neighbourhood_right_hand_sides(kind, model, monkeypatch):
    """Fixed-point right-hand sides (512 points on) against the FP64 formulas
    (the same points 511 at a time), coinciding pairs included, also a
    distance of an ulp. Either evaluation rounds a structure at most about 8
    times at up to 1.5 times its sill: 16 * 2^-53 of the sills, twice."""
    import torch
    from spinterps_gb300 import legacy
    monkeypatch.setattr(legacy, "SLICES_MIN_WORK", 0)
    n, C = 97, 1500
    rng = np.random.default_rng(5)
    xi, yi, zi = 4e6 + rng.uniform(0, 1e5, n), 5e6 + rng.uniform(0, 1e5, n), rng.gamma(1.2, 3.0, n)
    xk, yk = 4e6 + rng.uniform(0, 1e5, C), 5e6 + rng.uniform(0, 1e5, C)
    xk[:3], yk[:3] = xi[2:5], yi[2:5]
    xk[1] = np.nextafter(xk[1], 0)
    si = rng.uniform(0, 2, (1, n)) if kind == "EDK" else None
    sk = rng.uniform(0, 2, (1, C)) if kind == "EDK" else None
    d = lambda a: None if a is None else torch.as_tensor(a, device="cuda")  # noqa: E731

    def rhss(sl):
        s = None if sk is None else np.ascontiguousarray(sk[:, sl])
        return legacy.krige_points(kind, d(xi), d(yi), d(zi), d(xk[sl]), d(yk[sl]), model, si=d(si),
                                   sk=d(s))["rhss"].cpu().numpy()

    got = rhss(slice(0, C))
    ref = np.concatenate([rhss(slice(a, a + 511)) for a in range(0, C, 511)])
    scale = np.abs(ref[:, :n]).max() if "Pow" in model else sum(
        c[1] for c in legacy.parse_model(model))
    assert np.abs(got[:, :n] - ref[:, :n]).max() <= 32 * 2.0 ** -53 * scale
    assert np.array_equal(got[:, n:], ref[:, n:])
    for i in (0, 2):     # the coinciding pairs
        assert got[i, 2 + i] == ref[i, 2 + i]
