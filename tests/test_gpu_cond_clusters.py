"""The condition estimate of many small systems at once (k_trinv_cond, a
cluster of eight CTAs per system, csrc/spi_chol.cu): just above one block of
32 rows most of a cluster's warps own no row, so their sums arrive in CTA 0's
shared memory at once.

n L_00^2 |Linv|_F^2 against numpy's from the same covariances, at 1e-9: the
inverse factor's rounding is n 2^-53 times its condition (1e4 at most here)."""
import numpy as np
import pytest

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [32, 33, 40, 65])
def test_condition_of_many_small_systems(n):
    from spinterps_gb300 import steps
    T = 600
    rng = np.random.default_rng(n)
    sx, sy = rng.uniform(0, 3e5, n + 3), rng.uniform(0, 3e5, n + 3)
    z = rng.normal(size=(T, n + 3))
    for t in range(T):                      # every step a system of its own
        z[t, rng.choice(n + 3, 3, replace=False)] = np.nan
    vgs = ["0.30000 Nug(0.0) + %.6f Exp(20000)" % (0.5 + 1e-3 * t) for t in range(T)]
    args = steps.interp_args_for(["OK"], est_vars=True)
    plan = steps.InterpPlan(sx, sy, z, sx[:1] + 10.0, sy[:1], vgs, args, est_vars=True)
    plan.execute()
    cond = plan.collect_info()["cond"]["OK"]
    assert len(cond) == T
    for t in range(T):
        on = np.isfinite(z[t])
        d = np.hypot(sx[on][:, None] - sx[on], sy[on][:, None] - sy[on])
        s = 0.5 + 1e-3 * t
        # (a nugget counts at distance 0 too: it leaves the covariance form)
        L = np.linalg.cholesky(s * np.exp(-3 * d / 2e4))
        want = n * L[0, 0] ** 2 * (np.linalg.inv(L) ** 2).sum()
        assert abs(cond[t] - want) <= 1e-9 * want, t
