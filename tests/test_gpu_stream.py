"""The streamed FP32-tier cell kernel (spi_krige_cells_stream, mixed
precision) at the sizes where it can go wrong: two cells to a lane and 64 to
a CTA, station chunks of 256 and the FP64 flush every 2048 stations; every
model with a pair form, with a nugget, nested and without a form; entries on
both sides of a min_vg_val cut.

Against the FP64 path. The pair entries are good to 2^-38 of the sill, the
dual weights to 2^-48, the sums to 2^-44: with a nugget of a twentieth of the
sill the weights' magnitudes sum to at most ~1e4 times the field's, so the
estimates agree to 1e4 * 2^-38 = 4e-8; the OK variance (three TF32 terms)
keeps the mixed path's own 1e-5.
"""
import numpy as np
import pytest

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

BAR, VAR_BAR = 4e-8, 1e-5
NUG = "0.05 Nug(0.0) + "


def _run(n, T, C, methods, vgs, seed, drifts=0, min_vg=1e-4):
    from spinterps_gb300 import steps
    rng = np.random.default_rng(seed)
    box = 8e3 * np.sqrt(n)
    sx, sy = rng.uniform(0, box, n), rng.uniform(0, box, n)
    z = 3.0 + rng.normal(size=(T, n))
    cx, cy = rng.uniform(0, box, C), rng.uniform(0, box, C)
    cx[0], cy[0] = sx[1], sy[1]          # a cell on a station
    est_vars = "OK" in methods
    args = steps.interp_args_for(methods, est_vars=est_vars)
    kw = dict(est_vars=est_vars, min_vg_val=min_vg, intrp_dtype=np.float64)
    if drifts:
        kw.update(stn_drifts=rng.uniform(0, 1, (n, drifts)),
                  cell_drifts=rng.uniform(0, 1, (drifts, C)))
    vgs = [vgs[t % len(vgs)] for t in range(T)]
    mixed, _, info = steps.interp_steps(sx, sy, z, cx, cy, vgs, args, precision="mixed",
                                        return_info=True, **kw)
    ref, _ = steps.interp_steps(sx, sy, z, cx, cy, vgs, args, **kw)
    for lab in ref:
        bar = VAR_BAR if lab.startswith("EST_VARS") else BAR
        sc = np.nanmax(np.abs(ref[lab]))
        assert np.array_equal(np.isnan(ref[lab]), np.isnan(mixed[lab]))
        assert np.nanmax(np.abs(mixed[lab] - ref[lab])) <= bar * sc, (lab, n, C)
    return info


@pytest.mark.parametrize("C", [1, 31, 32, 33, 63, 64, 65, 129])
def test_cell_counts(C):
    _run(150, 2, C, ["EDK", "SK"], [NUG + "0.95 Exp(20000)"], C, drifts=2)


@pytest.mark.parametrize("n", [65, 255, 256, 257, 520, 2047, 2049])
def test_station_counts(n):
    info = _run(n, 2, 200, ["EDK"], [NUG + "0.95 Exp(30000)"], n, drifts=1)
    assert info["fp32_tier_steps"]["EDK"]


@pytest.mark.parametrize("model", ["0.95 Exp(20000)", "0.95 Sph(60000)", "0.95 Lin(90000)",
                                   "0.95 Gau(9000)", "0.95 Exp(2e-3)", "0.5 Exp(9000) + 0.45 Sph(50000)",
                                   "0.95 Hol(1000)"])
@pytest.mark.parametrize("min_vg", [0.0, 1e-4, 0.3])
def test_models(model, min_vg):
    # six vectors: two passes over the stations
    _run(150, 6, 300, ["OK", "SK", "EDK"], [NUG + model], 7, drifts=1, min_vg=min_vg)
