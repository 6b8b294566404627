"""The marching solvers of the line sweeps at the edges of their shapes (needs a
B200): few rows, lines of segments of unequal length, part-filled blocks, more than
32 segments along each axis and in the modal solves, against the oracle.  The
diffusion number of the z rows is above 0.1 in the long cases, so a segment's
coupling to its neighbour lives for tens of rows.  (The column form of long FP64 z
lines: test_gpu_column_sweeps.py.)

Bars: FP64 the parity bar of the other oracle tests (1e-10); FP32-mixed storage
keeps 6e-8 of each field per step, U, T and P within 1e-5 over two steps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [
    (4, 4, 4),        # one segment pair of 2 rows, 16-line blocks part-filled
    (5, 4, 6),        # segments of 3 rows along z, of 2 along y, of 1 and 2 in V's y sweep
    (12, 10, 25),     # of 3 and 4 rows along z, of 2 and 3 along y
    (20, 7, 25),      # segments of 3 and 4 rows
    (24, 20, 24),     # 8 segments of 3 rows along x and z, of 2 and 3 along y
    (18, 9, 384),     # 32 segments of 12 rows
    (36, 6, 400),     # 32 segments of 12 and 13 rows, three blocks of 16 lines
    (150, 5, 405),    # segments of 12 and 13 rows, a part-filled last block
    (45, 6, 400),     # odd N1: rows of i are not 16-byte aligned
    (45, 5, 640),     # z: 64 segments, reduced systems through shared memory
    (20, 643, 8),     # y: 64 segments of unequal length
    (540, 6, 8),      # x: 64 segments (from 531 cells on), several warps staging one line
    (2160, 5, 6),     # x: 128 segments
    (4096, 4, 4),     # x: 256 segments, one line per block
    (16, 900, 6),     # modal solves (two right-hand sides): 64 segments (from 837 rows on)
    (8, 4096, 4),     # y and modal: the longest lines
    (8, 6, 4096),     # z: the longest lines
]


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", SHAPES)
def test_strided_sweeps_match_oracle(n, precision):
    import pascal_tcs_b200 as P
    from oracle import oracle as O

    # (643 stretched rows at Ra = 1e4 and dt = 2e-3 are no test: the y rows of T lose
    # their dominance there, max |T| is 8e4 after two steps, and two restatements in
    # 64 bits differ by 3e-10; likewise 2160 cells along x (max |T| 1e6), 4096 along z,
    # and 4096 rows along y at Ra = 1e6 and dt = 1e-4 (2e4))
    ra, dt = (1e4, 2e-3) if n[1] < 100 and max(n) < 1000 else ((1e6, 1e-4) if n[1] < 1000 else (1e8, 1e-5))
    cfg = dict(n1m=n[0], n2m=n[1], n3m=n[2], property_set=0, Pr=0.71, Ra=ra, dtStart=dt, fixed_dt=1, seed=11,
               noise_amp=0.05, gamma2=1.2)
    g = P.Solver(precision=precision, **cfg)
    o = O.Oracle(**{k: v for k, v in g.config.items() if k not in ("device", "precision")})
    g.step(2)
    o.step(2)
    for f in ("T", "U", "V", "W", "P") if precision == 0 else ("T", "U", "P"):
        a, b = g.get(f), o.get(f)
        err = np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)
        assert np.all(np.isfinite(a)) and err <= (1e-10 if precision == 0 else 1e-5), (f, err)
    g.close()


@pytest.mark.parametrize("cyclic", [False, True])
@pytest.mark.parametrize("n_sys,n_row", [(1, 2), (63, 3), (64, 4), (65, 7), (200, 8), (129, 9), (70, 14), (130, 15), (66, 61)])
def test_tdma_many_bits_at_the_edges_of_its_prefetch(n_sys, n_row, cyclic):
    # rows around multiples of the rows loaded ahead, systems around a block: the bits of the strict evaluation
    import pascal_tcs_b200 as P
    from oracle import oracle as O

    rng = np.random.default_rng(100 * n_sys + n_row)
    A, C, D = (rng.uniform(-0.4, 0.4, (n_row, n_sys)) for _ in range(3))
    B = 1.0 + rng.uniform(0.0, 1.0, (n_row, n_sys))
    ref = O.tdma_many(A, B, C, D, cyclic=cyclic)
    Ag, Bg, Cg, Dg = A.copy(), B.copy(), C.copy(), D.copy()
    plan = P.TdmaPlan(n_sys)
    (plan.many_solve_cycle if cyclic else plan.many_solve)(Ag, Bg, Cg, Dg, n_sys, n_row)
    np.testing.assert_array_equal(Dg, ref)
