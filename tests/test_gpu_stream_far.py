"""The streamed FP32-tier kernel (csrc/spi_cells_stream.cu) at cells and gauges
whose squared distances leave FP32's range, or that have no place: the FP64
kernels' values at the mixed path's 1e-5 of the field's largest magnitude. The
cells lie outside the probe, so that the tier is taken."""
import numpy as np
import pytest

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

N, C = 150, 6000
MODELS = ["0.95 Exp(20000)", "0.95 Gau(9000)", "0.95 Sph(60000)", "0.95 Lin(90000)",
          "0.5 Exp(9000) + 0.45 Sph(50000)"]


def _both(sx, cx, model, seed):
    from spinterps_gb300 import steps
    rng = np.random.default_rng(seed)
    sy, cy = rng.uniform(0, 1e5, sx.size), rng.uniform(0, 1e5, C)
    z = 3.0 + rng.normal(size=(2, sx.size))
    args = steps.interp_args_for(["OK", "SK", "EDK"])
    kw = dict(min_vg_val=1e-4, intrp_dtype=np.float64, stn_drifts=rng.uniform(0, 1, (sx.size, 1)),
              cell_drifts=rng.uniform(0, 1, (1, C)), return_info=True)
    vgs = ["0.05 Nug(0.0) + " + model] * 2
    got, _, info = steps.interp_steps(sx, sy, z, cx, cy, vgs, args, precision="mixed", **kw)
    want, _, _ = steps.interp_steps(sx, sy, z, cx, cy, vgs, args, tensor_cores=False, **kw)
    for lab, w in want.items():
        assert np.array_equal(np.isnan(got[lab]), np.isnan(w)), lab
        sc = np.nanmax(np.abs(w))
        assert np.nanmax(np.abs(got[lab] - w)) <= 1e-5 * sc, lab
    return info


@pytest.mark.parametrize("model", MODELS)
@pytest.mark.parametrize("far", [np.nan, 1e20, 9.969209968386869e36])
def test_cells(model, far):
    rng = np.random.default_rng(7)
    sx, cx = rng.uniform(0, 1e5, N), rng.uniform(0, 1e5, C)
    probe = np.unique(np.linspace(0, C - 1, 1024).round().astype(int))
    cx[np.setdiff1d(np.arange(11, 90), probe)[::3]] = far
    info = _both(sx, cx, model, 8)
    if np.isnan(far):   # (a far cell also coarsens the split coordinates)
        assert any(len(v) for v in info["fp32_tier_steps"].values())


@pytest.mark.parametrize("model", MODELS)
@pytest.mark.parametrize("far", [1e20, 9.969209968386869e36])
def test_a_gauge_in_use(model, far):
    rng = np.random.default_rng(9)
    sx, cx = rng.uniform(0, 1e5, 2 * N), rng.uniform(0, 1e5, C)
    sx[260] = far
    _both(sx, cx, model, 10)
