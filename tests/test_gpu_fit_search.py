"""The differential-evolution search (spi_vg_de) against a NumPy replica of
its draws, trials and selection, at the edges of its bin tiles (2048 bins),
with one and two structures (one CTA and a cluster), and with distances that
leave the range of the fast quotient.

Tolerance: a member's FP32 energy is E = sum(d^2), d = g - m, where g and m
are good to a few ulp of FP32: |dd| <= 1e-6 max(g) for a member that is near
the data. So E is off by at most 2 sqrt(nb E) dd + nb dd^2, and a choice
between two members closer than that moves the result by as much again.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

M64 = (1 << 64) - 1


def _mix(z):
    z = (z + 0x9e3779b97f4a7c15) & M64
    z = ((z ^ (z >> 30)) * 0xbf58476d1ce4e5b9) & M64
    z = ((z ^ (z >> 27)) * 0x94d049bb133111eb) & M64
    return z ^ (z >> 31)


def _urand(seed, a, b, c):
    inner = _mix(((b * 0xcbf29ce484222325) & M64) ^ c)
    h = _mix(seed ^ _mix(((a * 0x100000001b3) & M64) ^ inner))
    return (h >> 11) / 9007199254740992.0


def _model(name, h, r, s):
    h, r, s = np.float64(h), np.float64(np.float32(r)), np.float64(np.float32(s))
    with np.errstate(all="ignore"):
        t = h / r
        if name == "Nug":
            return np.full_like(h, s)
        if name == "Sph":
            return np.where(h > r, s, s * (1.5 * t - 0.5 * t ** 3))
        if name == "Exp":
            return s * (1 - np.exp(-3 * t))
        if name == "Lin":
            return np.where(h > r, s, s * t)
        if name == "Gau":
            return s * (1 - np.exp(-3 * t * t))
        if name == "Pow":
            return s * h ** r
        return np.where(h > 0, s * (1 - np.sin(np.pi * t) / (np.pi * t)), 0.0)


def _search(names, fixed, h, g, var2, seed, gens):
    D = 2 * len(names)
    NP = 50 * D * D
    lo, sc = np.zeros(4), np.zeros(4)
    for k, nm in enumerate(names):
        rl, rh, sl, sh = h[0], 1e9, 1e-5, var2
        if nm == "Pow":
            rl, rh = 1e-5, 2.0
        elif fixed and k == 0:
            rl = rh = h[0]
            sl = sh = g[0]
        lo[2 * k:2 * k + 2] = rl, sl
        sc[2 * k:2 * k + 2] = rh - rl, sh - sl
    h32, g32 = np.float32(h), np.float32(g)

    def energy(u):
        x = lo + u * sc
        m = sum(_model(nm, h32, x[2 * k], x[2 * k + 1]) for k, nm in enumerate(names))
        return ((g32 - m) ** 2).sum()

    pop = np.zeros((NP, 4))
    for j in range(D):
        perm = list(range(NP))
        for i in range(NP - 1, 0, -1):
            k = int(_urand(seed, 0, j, i) * (i + 1))
            perm[i], perm[k] = perm[k], perm[i]
        for i in range(NP):
            pop[perm[i], j] = (i + _urand(seed, 1, j, i)) / NP
    E = np.array([energy(u) for u in pop])
    for gen in range(1, gens + 1):
        best = int(np.argmin(E))
        F = 0.5 + 0.5 * _urand(seed, 2, gen, 0)
        tri = pop.copy()
        for i in range(NP):
            r1 = next(r for r in (int(_urand(seed, 3, gen, i * 64 + c) * NP) for c in range(32))
                      if r != i)
            r2 = next(r for r in (int(_urand(seed, 7, gen, i * 64 + c) * NP) for c in range(32))
                      if r not in (i, r1))
            jr = int(_urand(seed, 4, gen, i) * D)
            for j in range(D):
                if _urand(seed, 5, gen, i * 4 + j) < 0.7 or j == jr:
                    v = pop[best, j] + F * (pop[r1, j] - pop[r2, j])
                    tri[i, j] = v if 0 <= v <= 1 else _urand(seed, 6, gen, i * 4 + j)
        Et = np.array([energy(u) for u in tri])
        ok = Et <= E
        E[ok], pop[ok] = Et[ok], tri[ok]
    x = lo + pop[int(np.argmin(E))] * sc
    m = sum(_model(nm, h, x[2 * k], x[2 * k + 1]) for k, nm in enumerate(names))
    return ((g - m) ** 2).sum()


@pytest.mark.parametrize("names,fixed", [(("Sph",), 0), (("Hol",), 0), (("Nug", "Exp"), 1),
                                         (("Nug", "Gau"), 0), (("Sph", "Lin"), 0),
                                         (("Nug", "Pow"), 1)])
@pytest.mark.parametrize("nb,tiny", [(1, 0), (7, 1), (2047, 0), (2048, 1), (2049, 0), (4097, 1)])
def test_search_matches_replica(names, fixed, nb, tiny):
    from spinterps_gb300 import _native as nat
    from spinterps_gb300.fitvgs import CODES, DeProblem
    rng = np.random.default_rng(nb + len(names))
    gens = 2
    probs, want, hs, gs, off = [], [], [], [], [0, 3]
    for step in range(2):
        h = np.sort(rng.uniform(1e6, 8e8, nb))
        if tiny:
            h[0] = 1e-15          # below the fast quotient's range
        g = 3.0 * (1 - np.exp(-h / 1e8)) + rng.uniform(0.3, 0.9, nb)
        if names[-1] == "Pow":
            g *= 1e6
        p = DeProblem()
        p.step, p.n_comp, p.fixed_first = step, len(names), fixed
        for c, nm in enumerate(names):
            p.code[c] = CODES[nm]
        p.var2, p.seed = 8.0, 1234567 + 99 * step
        probs.append(p)
        want.append(_search(names, fixed, h, g, p.var2, p.seed, gens))
        hs.append(h)
        gs.append(g)
    bins = lambda a: torch.from_numpy(np.concatenate([a[0], np.zeros(3), a[1]])).cuda()  # noqa
    bh, bg = bins(hs), bins(gs)
    off = torch.tensor([0, nb + 3], dtype=torch.int64, device="cuda")
    nbt = torch.tensor([nb, nb], dtype=torch.int32, device="cuda")
    raw = torch.frombuffer(bytearray(bytes((DeProblem * 2)(*probs))), dtype=torch.uint8).cuda()
    bx = torch.zeros((2, 4), dtype=torch.float64, device="cuda")
    bf = torch.zeros(2, dtype=torch.float64, device="cuda")
    ng = torch.zeros(2, dtype=torch.int32, device="cuda")
    nat.call("spi_vg_de", 2, raw.data_ptr(), off.data_ptr(), nbt.data_ptr(), bh.data_ptr(),
             bg.data_ptr(), gens, 0.0, bx.data_ptr(), bf.data_ptr(), ng.data_ptr(),
             torch.cuda.current_stream().cuda_stream)
    # an exact fit (a single bin) may end before the last generation
    assert all(1 <= k <= gens for k in ng.tolist())
    for k, got in enumerate(bf.tolist()):
        dd = 1e-6 * np.max(gs[k])
        tol = 2 * (2 * np.sqrt(nb * want[k]) * dd + nb * dd * dd)
        assert abs(got - want[k]) <= tol, (k, got, want[k], tol)
