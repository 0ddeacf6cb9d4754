"""The fixed-point covariance entries (csrc/spi_fx.cuh) on the CPU: the same
functions compiled for the host, against decimal arithmetic of 50 digits.

An entry's unit is 2^-62 of the structures' sills. Its error bound, in units of
2^-54: the grid's 2^-61 of the extent on each coordinate (3 sqrt(2) e^4 e^-1 of
it for the shortest range used here: 0.7), the distance's and its root's 2^-59
relative (3 e^-1 of that: 0.04), the products' 2 units of 2^-61 relative, the
exponential's 2^-60, each structure's weight rounding (2^-62): 2 hold with
room.
"""
import random
import shutil
import subprocess
from decimal import Decimal, getcontext
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CODES = {"Nug": 1, "Sph": 2, "Exp": 3, "Lin": 4, "Gau": 5}
MAIN = r'''
#include <cstdio>
#include "spi_fx.cuh"
using namespace spi;
int main() {
  uint64_t tab[256];
  for (int j = 0; j < 256; ++j) tab[j] = fx_exp2_entry(j);
  int n, q, sk;
  double mv, ox, oy;
  while (scanf("%d %d %d %la %la %la", &n, &q, &sk, &mv, &ox, &oy) == 6) {
    spi_vg_t vg = {};
    vg.n_comp = n;
    for (int c = 0; c < n; ++c) scanf("%d %la %la", &vg.code[c], &vg.sill[c], &vg.range[c]);
    double x[4];
    for (int i = 0; i < 4; ++i) scanf("%la", &x[i]);
    FxVg f;
    fx_init(f, vg, sk, mv, q);
    const int64_t v = fx_entry(f, fx_coord(x[0], ox, q), fx_coord(x[1], oy, q),
                               fx_coord(x[2], ox, q), fx_coord(x[3], oy, q), tab);
    printf("%d %lld %lld %lld\n", f.ok, (long long)v, (long long)f.cut, (long long)f.over);
  }
}
'''


@pytest.fixture(scope="module")
def fx(tmp_path_factory):
    cxx = shutil.which("g++")
    cuda = Path("/usr/local/cuda/include")
    if not cxx or not (cuda / "cuda_runtime.h").exists():
        pytest.skip("no host compiler or CUDA headers")
    d = tmp_path_factory.mktemp("fx")
    (d / "main.cpp").write_text(MAIN)
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", str(ROOT / "include"),
                    "-I", str(ROOT / "spinterps_gb300" / "csrc"), "-I", str(cuda),
                    str(d / "main.cpp"), "-o", str(d / "fx")], check=True)

    def run(cases):
        txt = []
        for c in cases:
            head = [len(c["vg"]), c["q"], c["sk"], c["mv"].hex(), c["o"][0].hex(), c["o"][1].hex()]
            for name, s, r in c["vg"]:
                head += [CODES[name], float(s).hex(), float(r).hex()]
            txt.append(" ".join(map(str, head + [v.hex() for v in c["x"]])))
        r = subprocess.run([str(d / "fx")], input="\n".join(txt), capture_output=True, text=True,
                           check=True)
        return [tuple(map(int, line.split())) for line in r.stdout.splitlines()]

    return run


def _exact(vg, x):
    """sum s rho in decimals, and the unit's sum of the structures' s (in
    doubles, as the device forms it)."""
    dx, dy = Decimal(x[0]) - Decimal(x[2]), Decimal(x[1]) - Decimal(x[3])
    h = (dx * dx + dy * dy).sqrt()
    c, tot = Decimal(0), 0.0
    for name, s, r in vg:
        if name == "Nug":
            continue
        tot += s
        s, r = Decimal(s), Decimal(r)
        t = h / r
        if name == "Exp":
            rho = (-3 * t).exp()
        elif name == "Gau":
            rho = (-3 * t * t).exp()
        elif name == "Sph":
            rho = 1 - t * (3 - t * t) / 2 if t < 1 else Decimal(0)
        else:
            rho = 1 - t if t < 1 else Decimal(0)
        c += s * rho
    return c, Decimal(tot)


def _cases(rng, names, count):
    import math
    out = []
    for _ in range(count):
        box = math.exp(rng.uniform(0, 14))
        off = rng.choice([0.0, 1e6 * rng.random(), -3e5 * rng.random()])
        vg = [(nm, 0.01 + 3 * rng.random(), box * math.exp(rng.uniform(-4, 1))) for nm in names]
        near = rng.choice([1.0, 0.05, 1e-4])
        cx, cy = off + box * rng.random(), off + box * rng.random()
        clip = lambda v: min(max(v, off), off + box)  # noqa: E731
        sx = clip(cx + near * box * (rng.random() - 0.5))
        sy = clip(cy + near * box * (rng.random() - 0.5))
        if rng.random() < 0.02:
            sx, sy = cx, cy
        q = 60 - math.frexp(box)[1]
        out.append(dict(vg=vg, q=q, sk=0, mv=0.0, o=(off, off), x=(cx, cy, sx, sy)))
    return out


@pytest.mark.parametrize("names", [("Exp",), ("Gau",), ("Sph",), ("Lin",), ("Nug", "Exp"),
                                   ("Exp", "Gau"), ("Sph", "Lin", "Exp", "Gau")])
def test_entries_against_decimals(fx, names):
    getcontext().prec = 50
    cases = _cases(random.Random("/".join(names)), names, 400)
    unit = Decimal(2) ** -54
    for c, (ok, v, cut, over) in zip(cases, fx(cases)):
        assert ok == 1 and cut == -1
        want, tot = _exact(c["vg"], c["x"])
        assert abs(v * unit / 256 - want / tot) <= 2 * unit, c


def test_min_vg_cut(fx):
    """The boundary of the min_vg_val zeroing and what lies past it, for the
    kinds; a cut that no entry reaches, or that every entry passes."""
    base = dict(q=40, o=(0.0, 0.0), x=(1e3, 2e3, 1.5e3, 2.5e3))
    exp = [("Exp", 0.9, 2e4)]
    one = 1 << 62
    got = fx([dict(base, vg=exp, sk=0, mv=1e-4), dict(base, vg=exp, sk=1, mv=1e-4),
              dict(base, vg=[("Nug", 0.1, 0.0), *exp], sk=0, mv=1e-4),
              dict(base, vg=[("Nug", 5e-5, 0.0), *exp], sk=0, mv=1e-4),
              dict(base, vg=exp, sk=0, mv=2.0), dict(base, vg=exp, sk=1, mv=2.0)])
    assert [g[0] for g in got] == [1, 1, 1, 1, 0, 0]
    assert abs(got[0][2] - round(one * (0.9 - 1e-4) / 0.9)) <= 1 << 14 and got[0][3] == one
    assert abs(got[1][2] - round(one * 1e-4 / 0.9)) <= 1 << 14 and got[1][3] == 0
    assert got[2][2] == -1  # the nugget alone exceeds the cut
    assert abs(got[3][3] - round(one * 0.90005 / 0.9)) <= 1 << 14
