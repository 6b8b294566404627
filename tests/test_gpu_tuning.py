"""The autotuner (tcs_autotune) and the launch-shape knobs it sets (needs a B200):
tuning leaves the case's state as it was, every knob setting gives the same
results to rounding, and a tuned shape is served from the cache."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CFG = dict(n1m=48, n2m=32, n3m=40, property_set=1, Pr=7.0, Ra=1e6, dtStart=5e-4, seed=7)


@pytest.fixture(scope="module")
def tcs():
    import pascal_tcs_b200 as P
    P.load()
    return P


def test_autotune_keeps_state_and_caches(tcs, tmp_path):
    cache = str(tmp_path / "tune.txt")
    g = tcs.Solver(**CFG)
    g.step(2)
    before = {n: g.get(n) for n in ("T", "U", "V", "W", "P", "dPhat", "dP0")}
    step0 = g.scalars()["step"]
    knobs, hit = g.autotune(trial_steps=2, cache_path=cache)
    assert not hit
    assert set(knobs) == set(tcs.tcs.TUNING)
    assert g.scalars()["step"] == step0
    for n, v in before.items():
        np.testing.assert_array_equal(g.get(n), v, err_msg=n)
    h = tcs.Solver(**CFG)
    knobs2, hit2 = h.autotune(cache_path=cache)
    assert hit2 and knobs2 == knobs
    with open(cache) as f:
        assert len(f.read().split()) == 4 + len(knobs)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("knob,value", [("lanes", 2), ("lanes", 4), ("lanes", 8), ("lanes", 16), ("fft_lines_x", 1),
                                        ("fft_lines_z", 8), ("ifft_lines_x", 8)])
def test_every_knob_setting_gives_the_same_step(tcs, knob, value, precision):
    # another split of the lines or of the transforms: another order of rounding in FP64
    # (1e-12), and so another FP32 rounding of some stored words in the mixed form (its
    # 1e-5 bar; V, the smallest component, sits 2.3e-6 apart after 3 steps)
    cfg = dict(CFG, precision=precision)
    a, b = tcs.Solver(**cfg), tcs.Solver(**cfg)
    b.set_tuning(knob, value)
    assert b.tuning()[knob] == value
    a.step(3); b.step(3)
    for n in ("T", "U", "V", "W", "P"):
        x, y = a.get(n), b.get(n)
        assert np.linalg.norm(x - y) <= (1e-12 if precision == 0 else 1e-5) * np.linalg.norm(x), n


@pytest.mark.parametrize("lanes", [2, 8])
def test_segment_bounds_on_long_lines(tcs, lanes):
    # 512 rows along y and z, 540 along x: more rows per segment, fewer lines per block
    cfg = dict(n1m=540, n2m=512, n3m=8, property_set=1, Pr=7.0, Ra=1e6, dtStart=5e-5, fixed_dt=1, seed=4)
    for c in (cfg, dict(cfg, n1m=8, n3m=512)):
        a, b = tcs.Solver(**c), tcs.Solver(**c)
        b.set_tuning("lanes", lanes)
        a.step(2); b.step(2)
        for n in ("T", "U", "V", "W", "P"):
            x, y = a.get(n), b.get(n)
            assert np.linalg.norm(x - y) <= 1e-12 * np.linalg.norm(x), n
        a.close(); b.close()


INERT = {"tl_strided": 64, "tl_contig": 64, "tl_modal": 64, "long_lines": 4, "y_solver": 4, "mixed_rows": 8, "z_staging": 2}


def test_knobs_without_effect_are_checked_and_kept(tcs):
    # they chose between line solvers that one solver has replaced: a value in range is
    # returned as set, anything else is refused
    g = tcs.Solver(n1m=36, n2m=24, n3m=64)
    for knob, most in INERT.items():
        v = 1
        while v <= most:
            g.set_tuning(knob, v)
            assert g.tuning()[knob] == v
            v *= 2
        for bad in (0, 3, 2 * most):
            with pytest.raises(tcs.TcsError) as ei:
                g.set_tuning(knob, bad)
            assert ei.value.code == 1, (knob, bad)
        assert g.tuning()[knob] == most
    # z_staging 2 stays refused in the FP32 form, for N3 no multiple of 64 and for an odd N1
    for bad in (dict(n1m=36, n2m=24, n3m=64, precision=1), dict(n1m=36, n2m=24, n3m=96), dict(n1m=45, n2m=24, n3m=64)):
        g = tcs.Solver(**bad)
        with pytest.raises(tcs.TcsError) as ei:
            g.set_tuning("z_staging", 2)
        assert ei.value.code == 1
        g.close()
