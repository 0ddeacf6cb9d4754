"""Neighbour selection where its FP32 decisions end: ties, directions along
the axes and the pies' edges, destinations on stations, empty pies, list
lengths around the register lists' sizes (8, 16, 32, 64), station counts
around a tile (1024), coordinates far from the origin, scales beyond FP32's
range. Lists must equal the rule in FP64 with equal distances ordered by
index, station for station.
"""
import numpy as np
import pytest

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _nrst(cx, cy, sx, sy, k):
    d = ((cx[:, None] - sx) ** 2 + (cy[:, None] - sy) ** 2) ** 0.5
    return np.sort(np.argsort(d, axis=1, kind="stable")[:, :k], axis=1)


def _pie(cx, cy, sx, sy, k, n_pies):
    out = np.empty((cx.size, k), dtype=np.int64)
    for i in range(cx.size):
        xd, yd = sx - cx[i], sy - cy[i]
        d = (xd ** 2 + yd ** 2) ** 0.5
        with np.errstate(all="ignore"):
            a = np.arctan(yd / xd)
        a = np.where((xd < 0) & (yd != 0), np.pi + a, np.where((xd > 0) & (yd < 0), 2 * np.pi + a, a))
        a = np.where(xd == 0, 0.0, a)
        pie = np.clip((a * n_pies / (2 * np.pi)).astype(np.int64), 0, n_pies - 1)
        order = np.lexsort((np.arange(d.size), d))
        rank = np.empty(d.size, dtype=np.int64)
        for p in range(n_pies):
            m = order[pie[order] == p]
            rank[m] = np.arange(m.size)
        out[i] = np.sort(np.lexsort((np.arange(d.size), d, rank))[:k])
    return out


def _check(mth, k, n_pies, sx, sy, cx, cy):
    from spinterps_gb300.nebs import SpInterpNeighborGrouping
    got = SpInterpNeighborGrouping(mth, k, n_pies, cx, cy).neb_idxs(sx, sy)
    ref = _nrst(cx, cy, sx, sy, k) if mth == "nrst" else _pie(cx, cy, sx, sy, k, n_pies)
    assert np.array_equal(got, ref), (mth, k, n_pies, np.where((got != ref).any(1))[0][:5])


@pytest.mark.parametrize("k", [1, 7, 8, 9, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("n", [64, 1023, 1024, 1025, 2500])
def test_nrst_sizes(k, n):
    rng = np.random.default_rng(k * n)
    sx, sy = 4e6 + rng.uniform(0, 2e5, n), 5.5e6 + rng.uniform(0, 2e5, n)
    cx, cy = 4e6 + rng.uniform(-1e4, 2.1e5, 259), 5.5e6 + rng.uniform(-1e4, 2.1e5, 259)
    cx[:20], cy[:20] = sx[:20], sy[:20]
    _check("nrst", k, 1, sx, sy, cx, cy)


@pytest.mark.parametrize("mth,k,n_pies", [("nrst", 16, 1), ("nrst", 5, 1), ("pie", 12, 8),
                                          ("pie", 9, 3), ("pie", 16, 16), ("pie", 20, 5)])
@pytest.mark.parametrize("scale", [1.0, 1e3, 2.0 ** -66, 2.0 ** 73])
def test_lattice_ties(mth, k, n_pies, scale):
    # stations and destinations on the nodes and centres of one lattice:
    # ties, axis directions and diagonals everywhere (quarters are exact)
    g = np.arange(14, dtype=np.float64)
    sx, sy = [a.ravel() * scale for a in np.meshgrid(g, g)]
    h = np.arange(0, 13.5, 0.5)
    cx, cy = [a.ravel() * scale for a in np.meshgrid(h, h)]
    _check(mth, k, n_pies, sx, sy, cx, cy)


@pytest.mark.parametrize("k,n_pies", [(1, 1), (4, 4), (12, 8), (16, 5), (16, 16), (24, 7), (64, 8)])
@pytest.mark.parametrize("n", [64, 300, 1025])
def test_pie_sizes(k, n_pies, n):
    # destinations outside the stations' box: pies without stations
    rng = np.random.default_rng(k * n + n_pies)
    sx, sy = rng.uniform(0, 2e5, n), rng.uniform(0, 2e5, n)
    cx, cy = rng.uniform(-1e5, 3e5, 150), rng.uniform(-1e5, 3e5, 150)
    cx[:20], cy[:20] = sx[:20], sy[:20]
    cx[20:30], cy[30:40] = sx[20:30], sy[30:40]
    _check("pie", k, n_pies, sx, sy, cx, cy)


@pytest.mark.parametrize("C,k,lists", [(1, 1, 1), (2, 16, 1), (255, 3, 40), (256, 64, 256),
                                       (4097, 12, 1), (60000, 16, 9000)])
def test_groups_of_equal_lists(C, k, lists):
    import torch
    from spinterps_gb300.nebs import device_groups
    rng = np.random.default_rng(C + k)
    pool = np.sort(rng.integers(-1, 50, size=(lists, k)), axis=1).astype(np.int32)
    nb = pool[rng.integers(0, lists, C)]
    g, c, o = (t.cpu().numpy() for t in device_groups(torch.as_tensor(nb, device="cuda")))
    uniq, first, inv = np.unique(nb, axis=0, return_index=True, return_inverse=True)
    rank = np.empty(first.size, dtype=np.int64)      # groups in order of first cells
    rank[np.argsort(first)] = np.arange(first.size)
    assert np.array_equal(g, uniq[np.argsort(first)])
    assert np.array_equal(c, rank[inv.ravel()])
    assert np.array_equal(o, np.argsort(c, kind="stable"))
    assert g.dtype == c.dtype == o.dtype == np.int32
