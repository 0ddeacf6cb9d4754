"""The FP64 inverse-square weights from integers (k_idw_sq, csrc/spi_idw.cu):
around its tiles and thread groups (16 and 32 cells, up to 32 steps at once),
gaps, a cell on a station present at some steps only, two stations at one
place, a cell a hair from a station, steps under the threshold, large offsets.

Against the oracle at 1e-12 of the field's largest value (sums of up to 1000
positive products, 2^-53 each and their roundings), NaN where it has NaN."""
import numpy as np
import pytest

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oracle import port  # noqa: E402


@pytest.mark.parametrize("n,T,C,off", [(2, 1, 5, 0.0), (31, 2, 33, 4e6), (64, 3, 31, 0.0),
                                       (150, 15, 32, -3e5), (400, 16, 40, 0.0),
                                       (401, 17, 16, 0.0), (700, 31, 17, 5.2e6),
                                       (1000, 33, 20, 0.0)])
def test_inverse_square(n, T, C, off):
    from spinterps_gb300 import steps
    rng = np.random.default_rng(n + T)
    sx, sy = off + rng.uniform(0, 9e4, n), rng.uniform(0, 6e4, n)
    z = 3.0 + rng.normal(size=(T, n))
    cx, cy = off + rng.uniform(0, 9e4, C), rng.uniform(0, 6e4, C)
    if n > 8:
        sx[5], sy[5] = sx[4], sy[4]
        z[rng.uniform(size=z.shape) < 0.2] = np.nan
        z[:, 4:6] = 1.0
        z[:, 0] = 2.0
        z[-1, 3] = np.nan
        cx[0], cy[0] = sx[3], sy[3]
        cx[1], cy[1] = sx[5], sy[5]
        cx[2], cy[2] = sx[7] + 1e-7, sy[7]
    if T > 1:
        z[0] = np.where(np.isfinite(z[0]), 0.1, np.nan)
    args = port.interp_args_for([("IDW", 2.0), ("IDW", 1.5)], est_vars=False)
    kw = dict(intrp_dtype=np.float64, min_var_thr=0.5 if T > 1 else 0.0)
    got, _ = steps.interp_steps(sx, sy, z, cx, cy, None, args, **kw)
    ref, _ = port.interp_steps(sx, sy, z, cx, cy, None, args, **kw)
    for lab in ref:
        assert np.array_equal(np.isnan(got[lab]), np.isnan(ref[lab])), lab
        sc = np.nanmax(np.abs(ref[lab]))
        assert np.nanmax(np.abs(got[lab] - ref[lab])) <= 1e-12 * sc, lab
