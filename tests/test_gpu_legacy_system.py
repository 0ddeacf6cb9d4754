"""spi_legacy_system (csrc/spi_legacy.cu) writes its n x n distances and
nothing past them, whichever way it inverts the m x m matrix: m = n + 1 +
drifts, so a few stations with many drifts make a large matrix with little
room in the distances."""
import ctypes

import numpy as np
import pytest

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,drifts", [(7, 87), (7, 88), (7, 90), (7, 91), (7, 95), (14, 90),
                                      (100, 1)])
def test_distances_and_nothing_past_them(n, drifts):
    import torch
    from spinterps_gb300 import _native as nat, legacy
    rng = np.random.default_rng(n + drifts)
    f64 = dict(dtype=torch.float64, device="cuda")
    x, y = (torch.as_tensor(rng.uniform(0, 1e5, n), device="cuda") for _ in range(2))
    si = torch.as_tensor(rng.uniform(0, 1, (drifts, n)), device="cuda")
    m = n + 1 + drifts
    room = torch.full((n * n + 64,), -7.0, **f64)
    lhs, inv = torch.empty((m, m), **f64), torch.empty((m, m), **f64)
    status, cond = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.zeros(1, **f64)
    vg = legacy._vg_struct(legacy.parse_model("1.0 Exp(30000)"))
    nat.call("spi_legacy_system", nat.KIND["EDK"], x.data_ptr(), y.data_ptr(), n, si.data_ptr(),
             drifts, ctypes.byref(vg), room.data_ptr(), lhs.data_ptr(), inv.data_ptr(),
             status.data_ptr(), cond.data_ptr(), None)
    torch.cuda.synchronize()
    got = room.cpu().numpy()
    assert (got[n * n:] == -7.0).all()
    xc, yc = x.cpu().numpy(), y.cpu().numpy()
    d = np.sqrt((xc[:, None] - xc) ** 2 + (yc[:, None] - yc) ** 2)
    assert np.abs(got[:n * n].reshape(n, n) - d).max() <= 1e-9
    if drifts < n:   # regular
        assert int(status.item()) == 0
        e = (lhs @ inv - torch.eye(m, **f64)).abs().max().item()
        assert e <= m * 2.0 ** -53 * cond.item()   # |A| |A^-1| in Frobenius norms



@pytest.mark.parametrize("n", [95, 96, 120, 348, 349, 400, 559, 560, 607, 801])
def test_inverse_around_the_grids_sizes(n):
    """The elimination's grid changes with the rows (csrc/spi_legacy.cu,
    leg_gj_ctas): |A P - 1| within the bound of an inverse's rounding,
    m 2^-53 |A| |P| in Frobenius norms."""
    import torch
    from spinterps_gb300 import _native as nat, legacy
    rng = np.random.default_rng(n)
    f64 = dict(dtype=torch.float64, device="cuda")
    x, y = (torch.as_tensor(rng.uniform(0, 1e5, n), device="cuda") for _ in range(2))
    m = n + 1
    dists = torch.empty((n, n), **f64)
    lhs, inv = torch.empty((m, m), **f64), torch.empty((m, m), **f64)
    status, cond = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.zeros(1, **f64)
    vg = legacy._vg_struct(legacy.parse_model("0.1 Nug(0.0) + 0.9 Exp(30000)"))
    nat.call("spi_legacy_system", nat.KIND["OK"], x.data_ptr(), y.data_ptr(), n, None, 0,
             ctypes.byref(vg), dists.data_ptr(), lhs.data_ptr(), inv.data_ptr(),
             status.data_ptr(), cond.data_ptr(), None)
    assert int(status.item()) == 0
    e = (lhs @ inv - torch.eye(m, **f64)).abs().max().item()
    assert e <= m * 2.0 ** -53 * cond.item()
