"""The single-neighbourhood weights as sliced products (spi_slices.cu) where a
right-hand side's parts differ in size: semivariances of any unit beside the
unbiasedness condition's 1 and the drifts.

Against the same points 511 at a time, whose weights an FP64 kernel computes
from the same inverse. An FP64 sum of m products is off by at most m 2^-53 of
the products' magnitudes; the bar is both evaluations' bound, entry by entry."""
import numpy as np
import pytest

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,drift", [("OK", 1.0), ("SK", 1.0), ("EDK", 1e-8), ("EDK", 1e4),
                                        ("EDK", 1e9)])
@pytest.mark.parametrize("sill", [1e-9, 1.0, 1e9])
def test_weights_of_any_unit(kind, sill, drift, monkeypatch):
    import torch
    from spinterps_gb300 import legacy
    monkeypatch.setattr(legacy, "SLICES_MIN_WORK", 0)
    rng = np.random.default_rng(11)
    n, C = 90, 1022
    xi, yi, zi = rng.uniform(0, 1e5, n), rng.uniform(0, 1e5, n), rng.gamma(1.2, 3.0, n)
    xk, yk = rng.uniform(0, 1e5, C), rng.uniform(0, 1e5, C)
    si, sk = drift * rng.uniform(1, 2, (2, n)), drift * rng.uniform(1, 2, (2, C))
    d = lambda a: torch.as_tensor(np.ascontiguousarray(a), device="cuda")  # noqa: E731
    model = "%.17g Nug(0.0) + %.17g Exp(30000)" % (0.1 * sill, 0.9 * sill)

    def run(s):
        kw = dict(si=d(si), sk=d(sk[:, s])) if kind == "EDK" else {}
        return legacy.krige_points(kind, d(xi), d(yi), d(zi), d(xk[s]), d(yk[s]), model, **kw)

    got = run(slice(None))
    parts = [run(slice(a, a + 511)) for a in (0, 511)]
    P = got["lhs_inv"]
    for p in parts:
        assert torch.equal(P, p["lhs_inv"])
    rhs = torch.cat([p["rhss"] for p in parts])
    bar = 2 * P.shape[0] * 2.0 ** -53 * (rhs.abs() @ P.abs().T)
    # (the right-hand sides themselves differ by their roundings)
    bar += (got["rhss"] - rhs).abs() @ P.abs().T
    err = (got["lambdas"] - torch.cat([p["lambdas"] for p in parts])).abs()
    assert (err <= bar[:, :n]).all()
    if kind != "SK":
        err = (got["mus"] - torch.cat([p["mus"] for p in parts], 1)).abs().T
        assert (err <= bar[:, n:]).all()
