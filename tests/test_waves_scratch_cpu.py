"""The wave planner counts the scratch of the sliced passes, which a plan
allocates once: a wave's steps and scratch together keep the budget."""
import numpy as np
import pytest

from spinterps_gb300 import steps, waves


@pytest.mark.parametrize("n,T,kinds,var,drifts", [(4000, 30, ["EDK"], False, 2),
                                                  (2000, 20, ["OK"], True, 0),
                                                  (300, 50, ["OK", "SK", "EDK"], True, 1)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_waves_with_their_scratch_keep_the_budget(n, T, kinds, var, drifts, precision):
    rng = np.random.default_rng(n)
    data = rng.normal(size=(T, n))
    data[rng.uniform(size=data.shape) < 0.2] = np.nan
    args = [(k, None, k) for k in kinds]
    C, mixed = 10000, precision == "mixed"
    n_av = np.isfinite(data).sum(1)
    per = [waves.step_bytes(int(k), C, len(args), 4, kinds, var, mixed) for k in n_av]
    one = waves.scratch_bytes(n, 1, kinds, var, mixed, drifts)
    assert one > 0
    kw = dict(est_vars=var, precision=precision, n_drift=drifts)
    for budget in (one // 2, one + max(per), 2 * one + 4 * max(per), 10 ** 13):
        ws = waves.plan_waves(data, C, args, budget=budget, **kw)
        assert ws[0][0] == 0 and ws[-1][1] == T
        assert all(a < b for a, b in ws)
        assert all(ws[i][1] == ws[i + 1][0] for i in range(len(ws) - 1))
        for a, b in ws:
            # what a plan of these steps allocates: each its own system, or
            # all of them one
            most = int(n_av[a:b].max())
            for n_sys, n_steps in ((b - a, 1), (1, b - a)):
                scratch = max(steps.slices_scratch_bytes(
                    most, n_sys, n_steps, drifts if k == "EDK" else 0, var and k == "OK", mixed)
                    for k in kinds)
                assert b - a == 1 or sum(per[a:b]) + scratch <= budget
    assert len(waves.plan_waves(data, C, args, budget=10 ** 13, **kw)) == 1
    # without tensor cores there is none
    few = waves.plan_waves(data, C, args, budget=one // 2 + 2 * max(per), tensor_cores=False, **kw)
    assert any(b - a > 1 for a, b in few)
