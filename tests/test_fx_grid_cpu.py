"""When the fixed-point entries (csrc/spi_fx.cuh) may stand in for FP64 ones:
fx_grid and fx_resolves compiled for the host, against decimals of 50 digits.
Where fx_resolves says yes, the entries' rms error over pairs within a range is
no larger than that of the FP64 formula on the same pairs; a far coordinate or
a short range makes it say no, unless the grid holds the coordinates exactly."""
import math
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
  double b[4], x[4];
  int n, rule;  // rule: the points count as not exact
  while (scanf("%d %la %la %la %la %d", &rule, &b[0], &b[1], &b[2], &b[3], &n) == 6) {
    spi_vg_t vg = {};
    vg.n_comp = n;
    for (int c = 0; c < n; ++c) scanf("%d %la %la", &vg.code[c], &vg.sill[c], &vg.range[c]);
    for (int i = 0; i < 4; ++i) scanf("%la", &x[i]);
    FxGrid g;
    int place = 4096;
    for (int i = 0; i < 4; ++i) place = place < fx_place(x[i]) ? place : fx_place(x[i]);
    const int ok = fx_grid(b[0], b[1], b[2], b[3], rule ? -4096 : place, g) && fx_resolves(vg, g);
    FxVg f;
    fx_init(f, vg, 0, 0.0, g.q);
    const int64_t v = ok ? fx_entry(f, fx_coord(x[0], g.ox, g.q), fx_coord(x[1], g.oy, g.q),
                                    fx_coord(x[2], g.ox, g.q), fx_coord(x[3], g.oy, g.q), tab)
                         : 0;
    printf("%d %lld\n", ok, (long long)v);
  }
}
'''


@pytest.fixture(scope="module")
def fx(tmp_path_factory):
    cxx = shutil.which("g++")
    cuda = Path("/usr/local/cuda/include")
    if not cxx or not (cuda / "cuda_runtime.h").exists():
        pytest.skip("no host compiler or CUDA headers")
    d = tmp_path_factory.mktemp("fxgrid")
    (d / "main.cpp").write_text(MAIN)
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", str(ROOT / "include"),
                    "-I", str(ROOT / "spinterps_gb300" / "csrc"), "-I", str(cuda),
                    str(d / "main.cpp"), "-o", str(d / "fx")], check=True)

    def run(cases, rule=1):
        txt = []
        for box, vg, x in cases:
            head = [rule] + [float(v).hex() for v in box] + [len(vg)]
            for name, s, r in vg:
                head += [CODES[name], float(s).hex(), float(r).hex()]
            txt.append(" ".join(map(str, head + [float(v).hex() for v in x])))
        r = subprocess.run([str(d / "fx")], input="\n".join(txt), capture_output=True, text=True,
                           check=True)
        return [tuple(map(int, line.split())) for line in r.stdout.splitlines()]

    return run


def _rho(name, t, exp=math.exp):
    """The correlation at t = h / range; exp by the type of t."""
    if name == "Exp":
        return exp(-3 * t)
    if name == "Gau":
        return exp(-3 * t * t)
    if t >= 1:
        return 0 * t
    return 1 - t * (3 - t * t) / 2 if name == "Sph" else 1 - t


@pytest.mark.parametrize("name", ["Exp", "Gau", "Sph", "Lin"])
@pytest.mark.parametrize("at", ["corner", "anywhere", "exact"])
def test_no_larger_error_than_fp64(fx, name, at):
    getcontext().prec = 50
    rng = random.Random(name + at)
    cases = []
    for _ in range(3000):
        side = math.exp(rng.uniform(0, 30))
        r = side / math.exp(rng.uniform(1, 6 if at != "exact" else 16))
        span = 2 * r if at == "corner" else side
        lim = lambda v: min(max(v, 0.0), side)  # noqa: E731
        cx, cy = span * rng.random(), span * rng.random()
        x = (cx, cy, lim(cx + 2 * r * (rng.random() - 0.5)), lim(cy + 2 * r * (rng.random() - 0.5)))
        if at == "exact":   # coordinates of 53 bits of the side
            side, u = 2.0 ** math.frexp(side)[1], 2.0 ** (math.frexp(side)[1] - 53)
            x = tuple(round(v / u) * u for v in x)
        cases.append(((0.0, side, 0.0, side), [(name, 0.01 + rng.random(), r)], x))
    e_fx, e_64, n = Decimal(0), Decimal(0), 0
    for (_, vg, x), (ok, v) in zip(cases, fx(cases, int(at != "exact"))):
        if not ok:
            continue
        (_, s, r), n = vg[0], n + 1
        dx, dy = Decimal(x[0]) - Decimal(x[2]), Decimal(x[1]) - Decimal(x[3])
        want = _rho(name, (dx * dx + dy * dy).sqrt() / Decimal(r), Decimal.exp)
        h = math.sqrt((x[0] - x[2]) ** 2 + (x[1] - x[3]) ** 2)
        got = s - s * (1.0 - _rho(name, h / r))
        e_fx += (Decimal(v) / 2 ** 62 - want) ** 2
        e_64 += (Decimal(got) / Decimal(s) - want) ** 2
    assert n > 1000 if at != "exact" else n == len(cases)
    assert e_fx <= e_64


def test_what_is_refused(fx):
    inf, nan = math.inf, math.nan
    x = (10.0, 20.0, 30.0, 40.0)
    exp = [("Exp", 0.9, 2e4)]

    def ok(box, vg):
        return fx([(box, vg, x)])[0][0]

    # a network of 250 km, ranges of it down to a fortieth
    assert ok((0, 2.5e5, 0, 1e5), exp)
    assert ok((4e6, 4.25e6, -1e5, 1e5), [("Nug", 0.1, 0.0), ("Exp", 0.9, 6.3e3)])
    # a structure of little sill counts little
    assert ok((0, 2.5e5, 0, 1e5), [("Exp", 1e-5, 1.0), ("Gau", 0.9, 1e4)])
    assert not ok((0, 2.5e5, 0, 1e5), [("Exp", 0.5, 1.0), ("Gau", 0.9, 1e4)])
    # short ranges, far points, points without a place
    assert not ok((0, 2.5e5, 0, 1e5), [("Exp", 0.9, 500.0)])
    for far in (1e7, 1e12, 1e20, 9.969209968386869e36, 1e300, inf, nan):
        assert not ok((0, far, 0, 1e5), exp), far
        assert not ok((0, 1e5, -far, 1e5), exp), far
    # coordinates that the grid holds exactly: any range
    assert fx([((0, 2.5e5, 0, 1e5), [("Exp", 0.9, 1.0)], x)], rule=0)[0][0]
    assert not fx([((0, 2.5e5, 0, 1e5), [("Exp", 0.9, 1.0)], (1e-9, *x[1:]))], rule=0)[0][0]
    # all points in one place
    assert ok((5.0, 5.0, 7.0, 7.0), exp)
