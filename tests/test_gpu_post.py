"""The step's diagnostics and wall rows on both sides of the FP32 form's choice between
one launch and two (2^22 cells), against sums over the downloaded fields (needs a
B200).  The sums are FP64 in both forms and compensated, so they agree with numpy's
pairwise sums to a few rounding errors of the largest term: 1e-12."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(20, 7, 18), (128, 255, 128), (128, 256, 128), (250, 131, 162)]


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", SHAPES)
def test_diagnostics_and_wall_rows(n, precision):
    import pascal_tcs_b200 as P

    g = P.Solver(n1m=n[0], n2m=n[1], n3m=n[2], property_set=0, Pr=0.71, Ra=1e6, dtStart=1e-4, fixed_dt=1, seed=2, gamma2=1.3,
                 noise_amp=0.05, precision=precision)
    rng = np.random.default_rng(1)
    for f in "UVW":
        a = np.zeros(g.shape)
        a[1:-1, 2:-1, 1:-1] = 1e-3 * rng.standard_normal((n[2], n[1] - 1, n[0]))
        g.set(f, a)
    g.step(1)
    T, U, V, W = (g.get(f) for f in ("T", "U", "V", "W"))
    d = [g.metric(f"dx{a}") for a in (1, 2, 3)]
    dm2 = g.metric("dmx2")
    c = (slice(1, -1),) * 3
    r1, r2, r3 = (1.0 / x[1:-1] for x in d)
    x, y, z = (U[c], U[1:-1, 1:-1, 2:]), (V[c], V[1:-1, 2:, 1:-1]), (W[c], W[2:, 1:-1, 1:-1])
    div = (x[1] - x[0]) * r1 + (y[1] - y[0]) * r2[:, None] + (z[1] - z[0]) * r3[:, None, None]
    cfl = abs(x[1] + x[0]) / 2 * r1 + abs(y[1] + y[0]) / 2 * r2[:, None] + abs(z[1] + z[0]) / 2 * r3[:, None, None]
    ke = 0.5 * np.sum((x[0] ** 2 + y[0] ** 2 + z[0] ** 2) * d[0][1:-1] * d[1][1:-1, None] * d[2][1:-1, None, None]) / (
        d[0][1:-1].sum() * d[1][1:-1].sum() * d[2][1:-1].sum())
    sc = g.scalars()
    assert sc["step"] == 1 and sc["blowup"] == 0
    assert abs(sc["KE"] - ke) <= 1e-12 * ke
    assert abs(sc["CFL"] - 1e-4 * cfl.max()) <= 1e-12 * sc["CFL"]
    # a difference of terms of |u| / dx; U, V, W come down as FP64 (in the mixed form the sum of their two words)
    assert abs(sc["maxDivU"] - div.max()) <= 1e-14 * 8 * cfl.max()
    for key, want in (("Nu_bot", -(T[1:-1, 1, 1:-1] - 0.5) / dm2[1]), ("Nu_top", -(-0.5 - T[1:-1, n[1], 1:-1]) / dm2[n[1] + 1])):
        assert abs(sc[key] - want.mean()) <= 1e-12 * abs(want).max(), key
    # the wall rows, dP with its ghost columns, P with its periodic images: rounded once to the field's type
    tol = 1e-15 if precision == 0 else 1.2e-7
    for f, cols in (("dP", slice(None)), ("P", slice(None))):
        a = g.get(f)
        for wall, p, q, e in ((0, 1, 2, (dm2[1], dm2[2])), (n[1] + 1, n[1], n[1] - 1, (dm2[n[1] + 1], dm2[n[1]]))):
            s = (e[0] + e[1]) ** 2
            want = s / (s - e[0] ** 2) * a[1:-1, p, 1:-1] - e[0] ** 2 / (s - e[0] ** 2) * a[1:-1, q, 1:-1]
            np.testing.assert_allclose(a[1:-1, wall, 1:-1], want, rtol=0, atol=4 * tol * abs(a).max())
            np.testing.assert_array_equal(a[:, wall, 0], a[:, wall, -2])
            np.testing.assert_array_equal(a[0, wall, :], a[-2, wall, :])
    g.close()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_fields_that_are_not_finite_are_reported(value, precision):
    # the pressure solve spreads them over every cell, and a maximum of NaN divergences
    # is none of them: the step reports a blow-up by the kinetic energy
    import pascal_tcs_b200 as P

    for n in ((16, 12, 10), (128, 256, 128)):
        g = P.Solver(n1m=n[0], n2m=n[1], n3m=n[2], property_set=1, Pr=7.0, Ra=1e6, dtStart=5e-4, fixed_dt=1, precision=precision)
        g.step(1)
        T = g.get("T")
        T[5, 5, 5] = value
        g.set("T", T)
        with pytest.raises(P.TcsError) as ei:
            g.step(2)
        assert ei.value.code == 4
        assert g.scalars()["blowup"] == 2 and g.scalars()["step"] == 1
        g.close()
