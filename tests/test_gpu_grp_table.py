"""spi_local_groups with and without the table of all stations' pairs
(k_grp_table; taken where the groups hold more entries than it and the
scratch has room): the same entries in the same order of operations, so the
same fields to the last bit, at the sizes around the 32 lanes of
k_grp_factor's element loop and in chunks of steps."""
import ctypes

import numpy as np
import pytest

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind_name,k", [("OK", 2), ("OK", 5), ("SK", 16), ("OK", 16),
                                         ("EDK", 14), ("SK", 31), ("SK", 32), ("OK", 32),
                                         ("EDK", 60)])
def test_table_and_direct_entries_agree(kind_name, k):
    import torch
    from spinterps_gb300 import _native as nat
    from spinterps_gb300.nebs import LOCAL_KIND, SpInterpNeighborGrouping, device_groups
    from spinterps_gb300.steps import (_Domain, _out_struct, _ptr, _stream, _vg_tensor, parse_vg)
    rng = np.random.default_rng(k)
    N, C, T = 70, 400, 3
    sx, sy, cx, cy = (rng.uniform(0, 1e5, s) for s in (N, N, C, C))
    nd = 2 if kind_name == "EDK" else 0
    sd, cd = rng.uniform(0, 1, (N, nd)), rng.uniform(0, 1, (nd, C))
    dom = _Domain(torch.device("cuda"), sx, sy, cx, cy, sd if nd else None, cd if nd else None,
                  1e-4, 0)
    nb = SpInterpNeighborGrouping("nrst", k, 1, cx, cy).neb_idxs_device(sx, sy)
    g, cg, order = device_groups(nb)
    G, kind = g.shape[0], LOCAL_KIND[kind_name]
    assert N * N <= G * k * k or k < 6   # (short lists: always direct)
    z = torch.as_tensor(3 + rng.normal(size=(T, N)), device="cuda")
    vg = _vg_tensor([parse_vg(v) for v in ("0.1 Nug(0.0) + 0.9 Exp(30000)", "1.0 Sph(60000)",
                                           "0.2 Nug(0.0) + 0.8 Gau(20000)")],
                    torch.device("cuda")).view(T, -1)
    nug = torch.zeros(T, dtype=torch.int32, device="cuda")
    steps = torch.arange(T, dtype=torch.int32, device="cuda")
    size = nat.lib().spi_local_groups_scratch_bytes
    per = size(kind, k, nd, G, 2) - size(kind, k, nd, G, 1)
    one = size(kind, k, nd, G, 1)
    res = []
    # one step without room for the table; all steps with it; two at a time
    for nbytes in (one, one + 2 * per + 3 * N * N * 8, one + per + 2 * N * N * 8):
        scratch = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
        est = torch.full((T, C), float("nan"), dtype=torch.float64, device="cuda")
        var = torch.full((T, C), float("nan"), dtype=torch.float64, device="cuda")
        pr = torch.zeros(T, dtype=torch.int32, device="cuda")
        out = _out_struct(est, var if kind_name == "OK" else None, None, None)
        nat.call("spi_local_groups", ctypes.byref(dom.st), kind, k, _ptr(g), G, _ptr(cg),
                 _ptr(order), T, _ptr(steps), _ptr(steps), _ptr(z), N, _ptr(vg), _ptr(nug), -1e9,
                 int(kind_name == "OK"), ctypes.byref(out), _ptr(scratch), nbytes, _ptr(pr),
                 _stream())
        res.append((est.cpu().numpy(), var.cpu().numpy(), pr.cpu().numpy()))
    assert np.isfinite(res[0][0]).all()
    for r in res[1:]:
        for a, b in zip(res[0], r):
            assert np.array_equal(a, b, equal_nan=True)
