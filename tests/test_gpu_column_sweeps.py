"""The column form of the FP64 z sweeps (column_kernel: even N1, more than 384 rows,
24576 lines or more) through its public calls (needs a B200)."""
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
