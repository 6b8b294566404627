"""The column form of the FP64 z sweeps (column_kernel: even N1, more than 384 rows,
24576 lines or more) through its public calls (needs a B200): its results against
the oracle at the edges of its shapes, against the marching form on one grid, its use
of the spectrum, and the report of a copy that does not arrive."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# 25600 lines of 400 rows: thermal, dU, dV and dW all take the column form
CFG = dict(n1m=128, n2m=200, n3m=400, property_set=0, Pr=0.71, Ra=1e6, dtStart=1e-4, fixed_dt=1, seed=3, gamma2=1.2)
FIELDS = ("T", "U", "V", "W", "P", "dPhat")


@pytest.fixture(scope="module")
def tcs():
    import pascal_tcs_b200 as P
    P.load()
    return P


def test_a_copy_that_does_not_arrive_in_time_is_not_a_blow_up(tcs):
    # waits that run out at their first poll (the kernel still waits for its copies
    # before it leaves): every call that reads the scalars reports a CUDA error, and
    # after tcs_restore the case runs on as if nothing had happened
    ref = tcs.Solver(**CFG)
    ref.step(3)
    g = tcs.Solver(**CFG)
    g.step(1)
    g.snapshot()
    g.set_copy_polls(0)

    def failed(call):
        with pytest.raises(tcs.TcsError) as ei:
            call()
        assert ei.value.code == 2 and "did not arrive" in str(ei.value), str(ei.value)

    failed(lambda: g.step(2))
    assert g.scalars()["blowup"] == 2          # the step it happened in
    failed(lambda: g.step(1))
    g.restore()
    g.thermal_solver()
    failed(g.post_div)
    failed(g.post_cfl)
    g.restore()
    ens = tcs.Ensemble([g], batched=True)
    failed(lambda: ens.step(1))
    ens.close()
    g.set_copy_polls(1 << 22)
    g.restore()
    assert g.step(2) == 2
    for n in FIELDS:
        np.testing.assert_array_equal(g.get(n), ref.get(n), err_msg=n)


def test_no_steps_leave_a_pending_right_hand_side_alone(tcs):
    # the column form keeps its coefficients in the spectrum: after tcs_pressure_RHS it
    # must not run before the Poisson solve has taken the right-hand side, and a call for
    # no steps changes nothing about that
    a, b = tcs.Solver(**CFG), tcs.Solver(**CFG)
    ens = tcs.Ensemble([b])
    for s in (a, b):
        s.step(1)
        s.thermal_solver()
        s.momentum_coeffi()
        s.momentum_solvedU()
        s.momentum_solvedV()
        s.momentum_solvedW()
        s.momentum_blockLdV()
        s.momentum_blockLdU()
        s.momentum_pseudoupdateUVW()
        s.pressure_RHS()
        if s is b:
            s.step(0)
            ens.step(0)
            s.momentum_solvedU()
        s.pressure_Poisson_FFT2()
    np.testing.assert_array_equal(b.get("dP"), a.get("dP"))
    ens.close()


def _takes_the_column_form(g, sweep):
    # with waits that run out at once, a sweep in the column form reports a late copy
    g.set_copy_polls(0)
    sweep()
    try:
        g.post_cfl()
        late = False
    except Exception as e:
        assert e.code == 2
        late = True
    g.set_copy_polls(1 << 22)
    g.restore()
    return late


@pytest.mark.parametrize("n,column", [
    ((150, 180, 405), True),      # block width 32, a part-filled last block; segments of 203 and 202 rows
    ((180, 144, 405), True),      # block width 64, a part-filled last block
    ((64, 396, 486), True),       # full blocks; two segments of 243 rows
    ((135, 190, 400), False),     # odd N1: rows of i are not 16-byte aligned
    ((128, 200, 384), False),     # 384 rows: the marching form
])
def test_column_form_matches_oracle(tcs, oracle_mod, n, column):
    # the diffusion number of the z rows is above 0.1: a segment's coupling to its
    # neighbour lives for tens of rows, which the second march repairs
    cfg = dict(n1m=n[0], n2m=n[1], n3m=n[2], property_set=1, Pr=7.0, Ra=1e4, DeltaT=10.0, dtStart=1e-3 if n[1] < 300 else 2e-4,
               fixed_dt=1, seed=11, noise_amp=0.05, gamma2=1.2)
    g = tcs.Solver(**cfg)
    dz = g.metric("dx3")[1]
    assert 0.5 * (7.0 / 1e4) ** 0.5 * cfg["dtStart"] / dz**2 > 0.1
    g.momentum_coeffi()
    g.snapshot()
    for sweep in (g.thermal_solver, g.momentum_solvedU, g.momentum_solvedV, g.momentum_solvedW):
        assert _takes_the_column_form(g, sweep) == column, sweep.__name__
    o = oracle_mod.Oracle(**{k: v for k, v in g.config.items() if k not in ("device", "precision")})
    g.step(2)
    o.step(2)
    for f in ("T", "U", "V", "W", "P"):
        a, b = g.get(f), o.get(f)
        err = np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)
        print(f, f"{err:.2e}")
        assert np.all(np.isfinite(a)) and err <= 1e-10, (f, err)
    g.close()


def test_column_form_agrees_with_the_marching_form(tcs):
    # a pending right-hand side keeps the spectrum, so the same sweep then takes the
    # marching form: the same rows eliminated in another order
    g = tcs.Solver(**CFG)
    g.step(2)
    g.momentum_coeffi()
    g.snapshot()
    for sweep, field in ((g.momentum_solvedU, "dU"), (g.momentum_solvedV, "dV"), (g.momentum_solvedW, "dW"), (g.thermal_solver, "T")):
        assert _takes_the_column_form(g, sweep)
        sweep()
        a = g.get(field)
        g.restore()
        g.pressure_RHS()
        assert not _takes_the_column_form(g, sweep)
        sweep()
        b = g.get(field)
        g.restore()
        g.pressure_Poisson_FFT2()
        assert np.linalg.norm(a - b) <= 1e-12 * np.linalg.norm(b), field
