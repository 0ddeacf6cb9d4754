"""Inverse-square weights from integers (k_idw_sq, csrc/spi_idw.cu) where one
grid does not hold all coordinates: gauges and cells far away or without a
place, a cluster around the origin of a wide domain.

Against the oracle at 1e-13 of each value: both sum 90 positive products,
rounded 2^-53 each and a few times per weight."""
import numpy as np
import pytest

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oracle import port  # noqa: E402

FAR = [1e12, 1e20, 9.969209968386869e36, 1e160, np.inf, np.nan]


def _job(n=90, T=3, C=70, seed=1):
    rng = np.random.default_rng(seed)
    z = 3.0 + rng.uniform(size=(T, n))
    z[:, 5:9] = np.nan
    return [rng.uniform(0, 9e4, n), rng.uniform(0, 6e4, n), z, rng.uniform(0, 9e4, C),
            rng.uniform(0, 6e4, C)]


def _both(job, ref=None):
    from spinterps_gb300 import steps
    args = port.interp_args_for([("IDW", 2.0)], est_vars=False)
    got, _ = steps.interp_steps(*job, None, args, intrp_dtype=np.float64)
    with np.errstate(all="ignore"):
        want, _ = port.interp_steps(*(ref or job), None, args, intrp_dtype=np.float64)
    (g,), (w,) = got.values(), want.values()
    return g, w


@pytest.mark.parametrize("far", FAR)
@pytest.mark.parametrize("axis", [0, 1])
def test_a_far_gauge_without_a_value(far, axis):
    job = _job()
    ref = list(job)
    job[axis] = np.append(job[axis], far)
    job[1 - axis] = np.append(job[1 - axis], 1e4)
    job[2] = np.column_stack([job[2], np.full(3, np.nan)])
    g, w = _both(job, ref)
    assert np.isfinite(w).all() and (np.abs(g - w) <= 1e-13 * np.abs(w)).all()


@pytest.mark.parametrize("far", FAR[:3])
@pytest.mark.parametrize("where", [0, 1, 3, 4])
def test_a_far_gauge_in_use_and_a_far_cell(far, where):
    job = _job()
    job[where][11] = far
    g, w = _both(job)
    assert np.isfinite(w).all() and (np.abs(g - w) <= 1e-13 * np.abs(w)).all()


@pytest.mark.parametrize("far", FAR[4:])
@pytest.mark.parametrize("axis", [3, 4])
def test_a_cell_without_a_place(far, axis):
    job = _job()
    ref = [a.copy() for a in job]
    job[axis][11] = far
    g, w = _both(job, ref)
    rest = np.arange(70) != 11
    assert np.isnan(g[:, 11]).all()
    assert (np.abs(g - w)[:, rest] <= 1e-13 * np.abs(w)[:, rest]).all()


def test_a_gauge_in_use_without_a_place():
    """NaN for every cell, as the weights' sum; infinitely far away counts
    nothing."""
    for far, nan in ((np.nan, True), (np.inf, False)):
        job = _job()
        ref = [np.delete(a, 11, -1) if k < 3 else a for k, a in enumerate(job)]
        job[0][11] = far
        g, w = _both(job, ref)
        assert np.isnan(g).all() if nan else (np.abs(g - w) <= 1e-13 * np.abs(w)).all()


@pytest.mark.parametrize("span", [1e-6, 1e-2, 1.0, 1e3])
def test_around_the_origin_of_a_wide_domain(span):
    """Half of the gauges and of the cells within `span` of the origin: their
    coordinates have places that a grid over 1e7 has not."""
    job = _job(seed=3)
    for a in (0, 1, 3, 4):
        job[a] *= 1e2
        job[a][::2] *= span / 9e6
    g, w = _both(job)
    assert (np.abs(g - w) <= 1e-13 * np.abs(w)).all()
