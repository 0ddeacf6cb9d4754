"""The neighbour methods hold one scratch for all of a call's step groups, within
nebs.GRP_SCRATCH_BYTES (waves.nebs_fixed_bytes counts it once), and the fields
do not depend on it."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_one_scratch_for_all_step_groups(monkeypatch):
    from spinterps_gb300 import nebs, steps, waves
    rng = np.random.default_rng(2)
    n, T, C, k = 300, 20, 20000, 16
    sx, sy = rng.uniform(0, 1e5, n), rng.uniform(0, 1e5, n)
    cx, cy = rng.uniform(0, 1e5, C), rng.uniform(0, 1e5, C)
    z = rng.normal(size=(T, n))
    z[np.arange(T), np.arange(T)] = np.nan        # every step a group of its own
    args = steps.interp_args_for(["OK"], est_vars=True)
    vgs = ["0.1 Nug(0.0) + 0.9 Exp(30000)"] * T

    def run(nbytes):
        monkeypatch.setattr(nebs, "GRP_SCRATCH_BYTES", nbytes)
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        torch.cuda.reset_peak_memory_stats()
        base = torch.cuda.memory_allocated()
        f, _ = steps.interp_steps(sx, sy, z, cx, cy, vgs, args, est_vars=True, min_vg_val=1e-4,
                                  neb_sel_mthd="nrst", n_nebs=k)
        return f, torch.cuda.max_memory_allocated() - base

    want, _ = run(2 << 30)
    for nbytes in (64 << 20, 1):
        got, peak = run(nbytes)
        for lab in want:
            assert np.array_equal(got[lab], want[lab]), lab
        if nbytes > 1:
            fields = T * C * 4 * len(args)
            # the step groups' lists and groupings are kept to the end
            lists = T * (C * 4 * (3 * k + 4))
            assert peak <= fields + lists + waves.nebs_fixed_bytes(C, k) + (16 << 20)
