"""A wave's tensors stay within the caller's budget, the scratch of the sliced
passes included (the next wave's plan is built while one runs: two budgets)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_waves_keep_the_budget():
    from spinterps_gb300 import steps, waves
    rng = np.random.default_rng(3)
    n, T, C = 1500, 72, 2000
    sx, sy = rng.uniform(0, 3e5, n), rng.uniform(0, 3e5, n)
    cx, cy = rng.uniform(0, 3e5, C), rng.uniform(0, 3e5, C)
    z = rng.normal(size=(T, n))
    z[np.arange(T), np.arange(T)] = np.nan
    args = steps.interp_args_for(["OK"], est_vars=True)
    vgs = ["0.1 Nug(0.0) + 0.9 Exp(30000)"] * T
    budget = 900 << 20
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    base = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    seen = []
    waves.interp_steps_waves(sx, sy, z, cx, cy, vgs, args, budget=budget, est_vars=True,
                             sink=lambda a, f: seen.append(a))
    assert len(seen) > 1
    # (coordinates, data and descriptors: a few MB)
    assert torch.cuda.max_memory_allocated() - base <= 2 * budget + (32 << 20)
