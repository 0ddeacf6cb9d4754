"""The refinement over FP32 factors (mixed precision, no variance) where the
matrix is singular: two gauges in one place leave the FP32 factor a pivot of
rounding, the refinement does not converge, and the FP64 factor of the
fallback is off the Cholesky path. Such systems take the exact inverse and its
pseudo-inverse check as without refinement (refine=False): the same fields at
the mixed path's 1e-5, and every step's route."""
import numpy as np
import pytest

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [6, 40, 130])
@pytest.mark.parametrize("drifts", [1, 2])
@pytest.mark.parametrize("model", ["0.1 Nug(0.0) + 0.9 Exp(20000)", "1.2 Nug(0.0) + 5.7 Sph(21000)",
                                   "0.3 Nug(0.0) + 1.6 Gau(9000)"])
def test_gauges_in_one_place(n, drifts, model):
    from spinterps_gb300 import steps
    back = 0
    for seed in range(4):
        rng = np.random.default_rng(seed)
        sx, sy = rng.uniform(0, 1e5, n), rng.uniform(0, 1e5, n)
        sx[1], sy[1] = sx[0], sy[0]
        sd = rng.uniform(0, 1, (n, drifts))
        z = 3.0 + rng.normal(size=(7, n))
        if n > 6:
            z[4:, 2] = np.nan
        cx, cy = rng.uniform(0, 1e5, 50), rng.uniform(0, 1e5, 50)
        kw = dict(min_vg_val=1e-4, intrp_dtype=np.float64, stn_drifts=sd, precision="mixed",
                  cell_drifts=rng.uniform(0, 1, (drifts, 50)), return_info=True)
        args = steps.interp_args_for(["EDK", "SK"])
        got, _, a = steps.interp_steps(sx, sy, z, cx, cy, [model] * 7, args, **kw)
        want, _, b = steps.interp_steps(sx, sy, z, cx, cy, [model] * 7, args, refine=False, **kw)
        for lab, w in want.items():
            assert np.abs(got[lab] - w).max() <= 1e-5 * np.abs(w).max(), (lab, seed)
            assert a["exact_inverse_steps"][lab] == b["exact_inverse_steps"][lab]
            assert a["pinv_steps"][lab] == b["pinv_steps"][lab]
            back += len(a["ir_fallback_steps"][lab])
    print("fallback steps", back)
