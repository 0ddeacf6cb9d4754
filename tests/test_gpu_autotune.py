"""The cell-tile autotuner (InterpPlan.autotune) runs the passes that execute()
runs: the fields afterwards are those of before, bit for bit, without another
execute()."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [40, 150])
def test_autotune_leaves_the_fields(precision, n, monkeypatch):
    from spinterps_gb300 import steps
    monkeypatch.setattr(steps, "_TILE_CACHE", {})
    rng = np.random.default_rng(n)
    sx, sy = rng.uniform(0, 1e5, n), rng.uniform(0, 1e5, n)
    cx, cy = rng.uniform(0, 1e5, 3000), rng.uniform(0, 1e5, 3000)
    z = 3.0 + rng.normal(size=(4, n))
    z[1, :5] = np.nan
    # a regular system, and one on the exact-inverse path (two gauges in one
    # place), which keeps the FP64 kernel
    sx[9], sy[9] = sx[8], sy[8]
    z[2:, 9] = np.nan
    args = steps.interp_args_for(["OK", "SK"], est_vars=True)
    plan = steps.InterpPlan(sx, sy, z, cx, cy, ["0.1 Nug(0.0) + 0.9 Exp(30000)"] * 4, args,
                            est_vars=True, min_vg_val=1e-4, precision=precision,
                            intrp_dtype=np.float64)
    plan.execute()
    base = {k: v.clone() for k, v in plan.fields(numpy=False).items()}
    tiles = plan.autotune()
    if precision == "fp64":
        assert tiles and set(tiles.values()) <= {16, 32, 64}
    for k, v in plan.fields(numpy=False).items():
        assert torch.equal(v, base[k]), k
