"""Every cell of every step is written, at the sizes around the tiles of the
sliced passes (csrc/spi_slices.cu: 16 stations, 64 rows, 128 cells) and of the
factorisation (csrc/spi_chol.cu, csrc/spi_duals.cu: 32 and 64 rows, cluster
sizes at 96 and 256). Fields start as NaN, which a nanmax over differences
would not see."""
import numpy as np
import pytest

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _finite(n, T, C, methods, precision="fp64", drifts=0, gaps=False, **kw):
    from spinterps_gb300 import steps
    rng = np.random.default_rng(n + 1000 * T + C)
    box = 8e3 * np.sqrt(n)
    sx, sy = rng.uniform(0, box, n), rng.uniform(0, box, n)
    z = 3.0 + rng.normal(size=(T, n))
    if gaps and n > 8:
        z[1::2, : max(1, n // 7)] = np.nan
    cx, cy = rng.uniform(0, box, C), rng.uniform(0, box, C)
    if drifts:
        kw.update(stn_drifts=rng.uniform(0, 1, (n, drifts)),
                  cell_drifts=rng.uniform(0, 1, (drifts, C)))
    var = "OK" in methods
    args = steps.interp_args_for(methods, est_vars=var)
    vgs = ["0.05 Nug(0.0) + 0.95 Exp(20000)"] * T
    got, _ = steps.interp_steps(sx, sy, z, cx, cy, vgs, args, est_vars=var, min_vg_val=1e-4,
                                precision=precision, **kw)
    for lab, f in got.items():
        assert f.shape == (T, C) and np.isfinite(f).all(), lab


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [2, 31, 32, 33, 63, 64, 65, 79, 80, 81, 96, 97, 127, 128, 129, 145,
                               192, 193, 255, 257, 320])
def test_station_counts(n, precision):
    _finite(n, 3, 131, ["OK", "SK", ("IDW", 2.0)], precision)
    _finite(n, 6, 23, ["OK", "SK"], precision, gaps=True)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("C", [1, 31, 33, 63, 65, 127, 128, 129, 255, 257, 19457])
def test_cell_counts(C, dtype):
    for precision in ("fp64", "mixed"):
        _finite(70, 2, C, ["OK", "SK", ("IDW", 2.0)], precision, intrp_dtype=dtype)


@pytest.mark.parametrize("T,drifts", [(1, 0), (62, 1), (63, 0), (64, 0), (65, 0), (127, 2),
                                      (130, 3)])
def test_blocks_of_steps(T, drifts):
    for precision in ("fp64", "mixed"):
        _finite(66, T, 40, ["EDK"] if drifts else ["OK"], precision, drifts)
        _finite(98, T, 40, ["EDK"] if drifts else ["OK", "SK"], precision, drifts, gaps=True)
