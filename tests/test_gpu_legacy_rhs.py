"""Right-hand sides of the single-neighbourhood classes in fixed point
(k_leg_rhs_fx, csrc/spi_legacy.cu): the points where that form must step aside
for the FP64 formulas, which the same points take 511 at a time."""
import numpy as np
import pytest

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture
def rhss(monkeypatch):
    import torch
    from spinterps_gb300 import legacy
    monkeypatch.setattr(legacy, "SLICES_MIN_WORK", 0)
    d = lambda a: torch.as_tensor(a, device="cuda")  # noqa: E731

    def both(kind, xi, yi, xk, yk, model):
        zi = np.arange(xi.size, dtype=np.float64)
        run = lambda s: legacy.krige_points(kind, d(xi), d(yi), d(zi), d(xk[s]), d(yk[s]),  # noqa: E731
                                            model)["rhss"].cpu().numpy()[:, :xi.size]
        return run(slice(None)), np.concatenate([run(slice(a, a + 511))
                                                 for a in range(0, xk.size, 511)])

    return both


def _points(seed, n=97, C=1200):
    rng = np.random.default_rng(seed)
    return (rng.uniform(0, 1e5, n), rng.uniform(0, 1e5, n), rng.uniform(0, 1e5, C),
            rng.uniform(0, 1e5, C))


@pytest.mark.parametrize("kind", ["OK", "SK"])
@pytest.mark.parametrize("far", [1e12, 1e20, 9.969209968386869e36, np.inf, np.nan])
def test_one_point_far_away(rhss, kind, far):
    """The other points' entries stay: both evaluations round a few times at
    the sill, 32 * 2^-53 as in the general test."""
    xi, yi, xk, yk = _points(1)
    xk[700] = far
    got, want = rhss(kind, xi, yi, xk, yk, "0.1 Nug(0.0) + 0.9 Exp(30000)")
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.nanmax(np.abs(got - want)) <= 32 * 2.0 ** -53


@pytest.mark.parametrize("model", ["0.7 Exp(20)", "0.7 Sph(100)", "0.7 Gau(50)", "0.7 Lin(90)"])
def test_ranges_short_of_the_domain(rhss, model):
    xi, yi, xk, yk = _points(2)
    rng = np.random.default_rng(3)
    xk[:97], yk[:97] = xi + rng.uniform(-20, 20, 97), yi + rng.uniform(-20, 20, 97)
    for kind in ("OK", "SK"):
        got, want = rhss(kind, xi, yi, xk, yk, model)
        assert np.abs(got - want).max() <= 8 * 2.0 ** -53 * 0.7, kind


@pytest.mark.parametrize("model", ["0.7 Sph(60000)", "1.3 Lin(50000)",
                                   "0.5 Sph(60000) + 0.2 Lin(30000)"])
def test_semivariances_beside_a_station(rhss, model):
    """Relative: the FP64 formulas of a spherical or linear lose a few
    roundings at any distance (16 * 2^-53 bounds both evaluations)."""
    xi, yi, xk, yk = _points(4)
    rng = np.random.default_rng(5)
    near = rng.integers(0, 97, 900)
    d = np.exp(rng.uniform(np.log(1e-4), np.log(3e3), 900))
    a = rng.uniform(0, 2 * np.pi, 900)
    xk[:900], yk[:900] = xi[near] + d * np.cos(a), yi[near] + d * np.sin(a)
    got, want = rhss("OK", xi, yi, xk, yk, model)
    assert (want > 0).all()
    assert (np.abs(got - want) / want).max() <= 16 * 2.0 ** -53
