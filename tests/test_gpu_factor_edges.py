"""The factorisation, the inverse factor and the dual vectors spread over the
GPU (csrc/spi_chol.cu, csrc/spi_duals.cu) at the sizes where their tiling can
go wrong: around one panel of 32 rows, around the 64-row FP32 tiles, around
the cluster sizes' limits (96, 256), uneven systems in one batch, several
steps per system, more dual columns than vectors in a pass.

Against the oracle at the FP64 path's bar, 1e-9 of the field's largest
magnitude (Exp variograms: condition 1e2 to 1e5, rounding 1e-11 at most);
the refinement path (mixed precision, no variance) at the mixed bar, 1e-5.
"""
import numpy as np
import pytest

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oracle import port  # noqa: E402


def _case(n, T, seed, drifts=0, gaps=True):
    rng = np.random.default_rng(seed)
    box = 8e3 * np.sqrt(n)
    sx, sy = rng.uniform(0, box, n), rng.uniform(0, box, n)
    z = 3.0 + rng.normal(size=(T, n))
    if gaps and n > 8:
        z[1::2, : max(1, n // 7)] = np.nan   # every other step: a smaller system
    cx, cy = rng.uniform(0, box, 23), rng.uniform(0, box, 23)
    sd = rng.uniform(0, 1, (n, drifts)) if drifts else None
    cd = rng.uniform(0, 1, (drifts, 23)) if drifts else None
    return sx, sy, z, cx, cy, sd, cd


def _check(n, T, methods, est_vars, seed, drifts=0, precision="fp64", bar=1e-9):
    import spinterps_gb300 as spi
    sx, sy, z, cx, cy, sd, cd = _case(n, T, seed, drifts)
    args = port.interp_args_for(methods, est_vars=est_vars)
    kw = dict(est_vars=est_vars, min_vg_val=1e-4, intrp_dtype=np.float64, stn_drifts=sd,
              cell_drifts=cd)
    vgs = ["0.05 Nug(0.0) + 0.95 Exp(20000)"] * T
    got, _ = spi.interp_steps(sx, sy, z, cx, cy, vgs, args, precision=precision, **kw)
    ref, _ = port.interp_steps(sx, sy, z, cx, cy, vgs, args, **kw)
    for lab in ref:
        sc = np.nanmax(np.abs(ref[lab]))
        assert np.nanmax(np.abs(got[lab] - ref[lab])) <= bar * sc, (n, lab)


@pytest.mark.parametrize("n", [2, 31, 32, 33, 63, 64, 65, 96, 97, 129, 255, 257, 320])
def test_ok_variance_and_sk(n):
    _check(n, 6, ["OK", "SK"], True, 100 + n)


@pytest.mark.parametrize("n,drifts", [(33, 1), (64, 3), (98, 4), (130, 7), (257, 2)])
@pytest.mark.parametrize("precision,bar", [("fp64", 1e-9), ("mixed", 1e-5)])
def test_edk_without_variance(n, drifts, precision, bar):
    _check(n, 11, ["EDK"], False, 200 + n, drifts, precision, bar)


def test_loo_of_uneven_systems():
    """Every other step a smaller system, one batch: each step's residuals
    equal those of a batch of its own, bit for bit."""
    from spinterps_gb300 import steps
    sx, sy, z, *_ = _case(161, 4, 7)
    vgs = ["0.05 Nug(0.0) + 0.95 Exp(20000)"] * 4
    res, rmse = steps.krige_loo(sx, sy, z, vgs)
    for t in range(4):
        one, r = steps.krige_loo(sx, sy, z[t:t + 1], vgs[:1])
        assert np.array_equal(res[t], one[0]) and rmse[t] == r[0], t


@pytest.mark.parametrize("drifts", [4, 5, 7])
def test_many_drifts_in_the_streamed_kernel(drifts):
    """More dual columns than the streamed kernel contracts in a pass of its
    four vectors: the sum check needs them all (with the columns of the
    later passes missing, cells fell back to their nearest station, by what
    shared memory held)."""
    for seed in range(4):
        _check(90, 3, ["EDK"], False, 400 + seed, drifts, "mixed", 1e-5)
