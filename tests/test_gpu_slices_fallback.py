"""Where the sliced tensor-core passes (csrc/spi_slices.cu) hand systems back
to the FP64 kernels, against those kernels alone (tensor_cores=False)."""
import numpy as np
import pytest

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

EXP = "0.05 Nug(0.0) + 0.95 Exp(20000)"


def _job(n, T, C, seed=0):
    rng = np.random.default_rng(seed)
    box = 8e3 * np.sqrt(n)
    sx, sy = rng.uniform(0, box, n), rng.uniform(0, box, n)
    return sx, sy, 3.0 + rng.normal(size=(T, n)), rng.uniform(0, box, C), rng.uniform(0, box, C)


def _plan(job, methods, vg, tensor_cores=True, **kw):
    from spinterps_gb300 import steps
    sx, sy, z, cx, cy = job
    kw.setdefault("est_vars", "OK" in methods)
    args = steps.interp_args_for(methods, est_vars=kw["est_vars"])
    kw = dict(dict(min_vg_val=1e-4, intrp_dtype=np.float64), **kw)
    return steps.InterpPlan(sx, sy, z, cx, cy, [vg] * len(z), args, tensor_cores=tensor_cores, **kw)


@pytest.mark.parametrize("precision,vg", [("fp64", EXP),
                                          ("mixed", "0.00001 Exp(1.0) + 0.9 Gau(25000)")])
def test_after_a_wait_that_ran_out(precision, vg):
    """With the error flag up (as a timed-out wait leaves it) every system is
    computed by the FP64 (double-float) kernels: the same bits as without
    tensor cores in FP64, the mixed tier's 1e-5 else (its own tensor-core
    variance stays on)."""
    job = _job(150, 3, 300)
    p = _plan(job, ["OK", "SK"], vg, precision=precision)
    p.slices_err.fill_(1)
    p.execute()
    got, plain = p.fields(), _plan(job, ["OK", "SK"], vg, False, precision=precision)
    plain.execute()
    want = plain.fields()
    for lab in want:
        g, w = (x[lab].cpu().numpy() if hasattr(x[lab], "cpu") else x[lab] for x in (got, want))
        if precision == "fp64":
            assert np.array_equal(g, w), lab
        else:
            assert np.isfinite(g).all()
            assert np.abs(g - w).max() <= 1e-5 * np.abs(w).max(), lab
    with pytest.raises(RuntimeError, match="timed out"):
        p.collect_info()


@pytest.mark.parametrize("drifts", [1, 2])
@pytest.mark.parametrize("T", [62, 63, 127])
def test_scratch_of_ok_beside_edk(T, drifts):
    """OK with its variance and EDK in one plan, one shared system: the OK
    batch's scratch holds its own rows (1 + T: a whole number of blocks of 64
    at 63 and 127), not the drifts'."""
    job = _job(70, T, 130)
    rng = np.random.default_rng(T)
    kw = dict(stn_drifts=rng.uniform(0, 1, (70, drifts)), cell_drifts=rng.uniform(0, 1, (drifts, 130)))
    a, b = (_plan(job, ["OK", "EDK"], EXP, tc, **kw) for tc in (True, False))
    a.execute()
    b.execute()
    for lab, w in b.fields().items():
        g = a.fields()[lab]
        assert np.isfinite(g).all() and np.abs(g - w).max() <= 1e-11 * np.abs(w).max(), lab


def _near(got, want, bar=1e-11):
    for lab, w in want.items():
        g = got[lab]
        assert np.array_equal(np.isnan(g), np.isnan(w)), lab
        if np.isfinite(w).any():
            assert np.nanmax(np.abs(g - w)) <= bar * np.nanmax(np.abs(w)), lab


FAR = [1e12, 1e20, 9.969209968386869e36, np.inf, np.nan]


@pytest.mark.parametrize("far", FAR)
@pytest.mark.parametrize("axis", [0, 1])
def test_a_far_gauge_without_a_value(far, axis):
    """Its coordinates (a fill value, say) are nobody's business."""
    job = list(_job(90, 3, 200))
    want = _plan(job, ["OK", "SK"], EXP, False)
    want.execute()
    job[axis] = np.append(job[axis], far)
    job[1 - axis] = np.append(job[1 - axis], 1e5)
    job[2] = np.column_stack([job[2], np.full(3, np.nan)])
    p = _plan(job, ["OK", "SK"], EXP)
    p.execute()
    _near(p.fields(), want.fields())


@pytest.mark.parametrize("far", FAR[:3])
@pytest.mark.parametrize("vg", [EXP, "0.9 Sph(60000)", "0.1 Nug(0.0) + 0.9 Gau(9000)"])
def test_a_far_gauge_in_use_and_a_far_cell(far, vg):
    for where in (0, 3):
        job = list(_job(90, 3, 200))
        job[where][7] = far
        a, b = (_plan(job, ["OK", "SK"], vg, tc) for tc in (True, False))
        a.execute()
        b.execute()
        _near(a.fields(), b.fields())


@pytest.mark.parametrize("far", FAR[3:])
@pytest.mark.parametrize("axis", [3, 4])
def test_a_cell_without_a_place(far, axis):
    """A domain ten times as long in x as in y, a cell at NaN or infinity: the
    other cells keep their values."""
    job = list(_job(90, 3, 200))
    job[1], job[4] = job[1] / 10, job[4] / 10
    want = _plan(job, ["OK", "SK"], EXP, False)
    want.execute()
    job[axis][11] = far
    p = _plan(job, ["OK", "SK"], EXP)
    p.execute()
    rest = np.arange(200) != 11
    _near({k: v[:, rest] for k, v in p.fields().items()},
          {k: v[:, rest] for k, v in want.fields().items()})


@pytest.mark.parametrize("off", [0.0, 4e5])
def test_a_range_short_of_the_domain(off):
    """Exp(12) in a domain of 76 km: stations a few metres apart; also with
    offsets, whose coordinates the grid holds exactly."""
    job = [a if k == 2 else a + off for k, a in enumerate(_job(90, 2, 200))]
    for a, b in ((0, 3), (1, 4)):
        job[b][:80] = job[a][:80] + np.random.default_rng(a).uniform(-9, 9, 80)
    a, b = (_plan(job, ["OK", "SK"], "0.9 Exp(12)", tc) for tc in (True, False))
    a.execute()
    b.execute()
    _near(a.fields(), b.fields(), 1e-14)
