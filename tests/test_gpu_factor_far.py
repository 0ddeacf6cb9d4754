"""The system matrices (k_build_sys, csrc/spi_factor.cu) with a gauge so far away
that distances to it overflow: its correlations are 0, as at any distance past
the ranges, and the other gauges' residuals stay."""
import numpy as np
import pytest

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model", ["0.95 Exp(20000)", "0.95 Sph(60000)", "0.95 Gau(9000)",
                                   "0.95 Lin(60000)", "0.5 Exp(9000) + 0.45 Sph(50000)"])
@pytest.mark.parametrize("far", [1e100, 1e148, 1e152, 1e160, 1e300])
def test_leave_one_out(model, far):
    from spinterps_gb300 import steps
    rng = np.random.default_rng(5)
    sx, sy = rng.uniform(0, 1e5, 50), rng.uniform(0, 1e5, 50)
    z = 3.0 + rng.normal(size=(1, 50))
    vg = ["0.05 Nug(0.0) + " + model]
    sx[7] = 1e12
    (want,), _ = steps.krige_loo(sx, sy, z, vg, min_vg_val=1e-4)
    sx[7] = far
    (got,), _ = steps.krige_loo(sx, sy, z, vg, min_vg_val=1e-4)
    assert np.array_equal(got, want)
