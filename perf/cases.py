"""The work that a user of pascal_tcs_b200 has it do, as cases that can be timed and compared.

A case is one call pattern of the public Python binding: whole time steps
(Solver.step), the driver sequence of the reference (Solver.driver_step), an
ensemble of cases (Ensemble.step) or the PaScaL_TDMA many-systems solve
(TdmaPlan).  The time steps start from a checkpoint kept on the device
(Solver.snapshot), and a pass returns to it first (Solver.restore), as the
benchmark does with the water cases: their states blow up within about ten
steps in the reference's own algorithm.

exact() restates the time step of the reference (main.f90:129-223) for one
rank in 64-bit torch, in the reference's own form of every expression.
"""
import math
import os

import numpy as np
import torch

import pascal_tcs_b200 as P

TUNE_CACHE = os.path.join(os.path.dirname(os.path.abspath(P.__file__)), "tune_cache.txt")

WATER = {"property_set": 1, "Pr": 7.0, "DeltaT": 10.0}
GLYCEROL = {"property_set": 2, "Pr": 7.0, "DeltaT": 10.0}
CONSTANT = {"property_set": 0, "Pr": 0.71, "DeltaT": 10.0}


def _step(name, n, ra, dt, props, **kw):
    c = {"kind": "step", "n1m": n[0], "n2m": n[1], "n3m": n[2], "Ra": ra, "dtStart": dt, "gamma2": 1.5,
         "fixed_dt": 1, "top_wall_mode": 0, "precision": 0, "steps": 2, "tuned": False}
    c.update(props)
    c.update(kw)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest grid of the tests: one step, bound by its launches (a control loop that looks at every step)
        _step("step_32", (32, 32, 32), 1e5, 1e-3, CONSTANT, steps=1),
        # the benchmark's 64^3 constant-property case
        _step("step_64", (64, 64, 64), 1e5, 1e-3, CONSTANT, steps=4),
        # the reference's own driver loop, one call per routine, CFL-adaptive dt, odd sizes
        _step("driver_96", (96, 77, 90), 1e6, 5e-4, CONSTANT, kind="driver", steps=1, fixed_dt=0, top_wall_mode=1),
        # sizes with every FFT radix and lines that are no power of two, on the default launch shapes
        _step("step_ragged", (180, 151, 250), 1e7, 2e-4, GLYCEROL, top_wall_mode=1),
        # the 256^3 water case the headline metric is quoted on, with the committed launch shapes, and its FP32-mixed
        # twin on the default ones
        _step("step_256", (256, 256, 256), 1e8, 2e-4, WATER, tuned=True),
        _step("step_256_mixed", (256, 256, 256), 1e8, 2e-4, WATER, precision=1),
        # the default benchmark workload: the largest grid
        _step("step_512", (512, 512, 512), 1e9, 5e-5, WATER, gamma2=2.0, tuned=True),
        # a large FP32-mixed run on a grid of its own shape, not in the tuning cache
        _step("step_mixed_wide", (400, 200, 384), 1e8, 1e-4, WATER, precision=1),
        # a parameter study: small cases of uneven sizes, both forms, advanced together
        {"name": "ensemble_8", "kind": "ensemble", "count": 8, "steps": 2},
        # PaScaL_TDMA as the ADI and Poisson stages of another code call it: many systems, one plane or one volume
        {"name": "tdma_plane", "kind": "tdma", "n_sys": 4096, "n_row": 64, "cyclic": False},
        {"name": "tdma_cycle", "kind": "tdma", "n_sys": 30000, "n_row": 333, "cyclic": True},
        {"name": "tdma_volume", "kind": "tdma", "n_sys": 65536, "n_row": 256, "cyclic": False},
    ]


def _smooth(rng, lo, hi):
    """A size that factors into 2, 3 and 5 (the FFT axes), log-uniform."""
    sizes = [n for n in range(lo, hi + 1) if _is_smooth(n)]
    want = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(sizes, key=lambda n: abs(n - want))


def _is_smooth(n):
    for p in (2, 3, 5):
        while n % p == 0:
            n //= p
    return n == 1


def draw(rng):
    kind = rng.choice(["step", "step", "step", "driver", "tdma"])
    if kind == "tdma":
        rows = int(math.exp(rng.uniform(math.log(8), math.log(700))))
        most = min(200000, 40_000_000 // rows)
        return {"kind": "tdma", "n_sys": int(math.exp(rng.uniform(math.log(64), math.log(most)))), "n_row": rows,
                "cyclic": rng.random() < 0.5}
    while True:
        n = (_smooth(rng, 20, 512), int(math.exp(rng.uniform(math.log(20), math.log(400)))), _smooth(rng, 20, 512))
        if n[0] * n[1] * n[2] <= 40_000_000:
            break
    props = rng.choice([WATER, GLYCEROL, CONSTANT])
    fine = max(n[0] / 2.0, n[1] / 1.0, n[2] / 2.0)
    return _step(None, n, 10.0 ** rng.uniform(5.0, 8.0), 0.05 / fine, props, kind=kind,
                 steps=1 if kind == "driver" else rng.choice([1, 2]), gamma2=rng.choice([1.2, 1.5, 2.0]),
                 # a dt that follows the CFL number jumps after the first step: constant properties stand that
                 fixed_dt=rng.choice([1, 0]) if props is CONSTANT else 1, top_wall_mode=rng.choice([0, 1]),
                 precision=rng.choice([0, 0, 1]))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
CONFIG = ("n1m", "n2m", "n3m", "Ra", "Pr", "DeltaT", "dtStart", "gamma2", "property_set", "fixed_dt",
          "top_wall_mode", "precision")
STATE = ("T", "U", "V", "W", "P", "dPhat", "dP0")
FIELDS = ("T", "U", "V", "W", "P", "dPhat")


def _config(case):
    return {k: case[k] for k in CONFIG}


def _members(case):
    """The cases of the ensemble: sizes, Rayleigh numbers and forms of a parameter study."""
    sizes = ((64, 96, 64), (128, 64, 96), (96, 128, 80), (64, 64, 160), (128, 96, 128), (80, 100, 64), (160, 64, 64), (96, 96, 96))
    out = []
    for i in range(case["count"]):
        water = i % 2 == 0
        out.append(_step(None, sizes[i % len(sizes)], 10.0 ** (5.0 + 0.25 * i), 2e-4, WATER if water else CONSTANT,
                         precision=1 if i % 4 == 3 else 0, steps=case["steps"]))
    return out


def _modes(gen, count, dev):
    kx = torch.randint(1, 5, (count,), generator=gen).double()
    kz = torch.randint(0, 5, (count,), generator=gen).double()
    ph = 2.0 * math.pi * torch.rand(count, generator=gen, dtype=torch.float64)
    am = torch.randn(count, generator=gen, dtype=torch.float64) / count
    return [tuple(float(v) for v in q) for q in zip(kx, kz, ph, am)]


def _fill_periodic(a):
    a[:, :, 0] = a[:, :, -2]
    a[:, :, -1] = a[:, :, 1]
    a[0] = a[-2]
    a[-1] = a[1]


def _fields(case, seed, dev):
    """A checkpoint in 64 bits, padded (k, j, i): convection rolls (divergence-free on the staggered grid, free-fall
    velocities of about 0.2), the conduction profile with plumes and noise, a smooth pressure and its correction history.
    With variable properties a twentieth of that: such runs are young, for the reference's own algorithm ends them early."""
    size = 1.0 if case["property_set"] == 0 else 0.05
    m = _mesh(case, dev)
    gen = torch.Generator().manual_seed(int(seed))
    N1, N2, N3 = case["n1m"], case["n2m"], case["n3m"]
    lx, lz = 2.0, 2.0
    x, y, z = m["x1"], m["x2"], m["x3"]
    xc, yc, zc = (torch.cat([0.5 * (q[1:] + q[:-1]), q[-1:]]) for q in (x, y, z))

    def plane(zz, xx, modes, s=0.0):
        out = torch.zeros(zz.numel(), 1, xx.numel(), dtype=torch.float64, device=dev)
        for kx, kz, ph, am in modes:
            out += am * torch.cos(2.0 * math.pi * (kx * xx / lx)[None, None, :] + 2.0 * math.pi * (kz * zz / lz)[:, None, None] + ph + s)
        return out

    shape = torch.sin(math.pi * y.clamp(0.0, 1.0)) ** 2          # 0 on both walls: no flow through them
    shape[0] = 0.0
    shape[-1] = 0.0
    psi3 = 0.1 * size * plane(zc, x, _modes(gen, 4, dev)) * shape[None, :, None]   # on the edges along z
    psi1 = 0.1 * size * plane(z, xc, _modes(gen, 4, dev)) * shape[None, :, None]   # on the edges along x
    U, V, W = (torch.zeros(N3 + 2, N2 + 2, N1 + 2, dtype=torch.float64, device=dev) for _ in range(3))
    i1, i2, i3 = slice(1, N1 + 1), slice(1, N2 + 1), slice(1, N3 + 1)
    n1, n2, n3 = slice(2, N1 + 2), slice(2, N2 + 2), slice(2, N3 + 2)
    d1, d2, d3 = m["dx1"][i1][None, None, :], m["dx2"][i2][None, :, None], m["dx3"][i3][:, None, None]
    U[i3, i2, i1] = (psi3[i3, n2, i1] - psi3[i3, i2, i1]) / d2
    V[i3, i2, i1] = -(psi3[i3, i2, n1] - psi3[i3, i2, i1]) / d1 + (psi1[n3, i2, i1] - psi1[i3, i2, i1]) / d3
    W[i3, i2, i1] = -(psi1[i3, n2, i1] - psi1[i3, i2, i1]) / d2
    V[:, 1] = 0.0
    for a in (U, V, W):
        # the edges' images of the last face make the rolls periodic
        _fill_periodic(a)
    bump = torch.sin(math.pi * yc)[None, :, None]
    noise = torch.rand(N3 + 2, N2 + 2, N1 + 2, generator=torch.Generator(device=dev).manual_seed(int(seed) + 1), dtype=torch.float64, device=dev)
    T = 0.5 - yc[None, :, None] + 0.05 * size * bump * plane(zc, xc, _modes(gen, 6, dev)) + 0.01 * (2.0 * noise - 1.0)
    T[:, 0] = 0.5
    T[:, -1] = -0.5 if case["top_wall_mode"] else 0.0
    _fill_periodic(T)
    cosy = torch.cos(math.pi * yc)[None, :, None]
    Pr = (0.002 * size * cosy * plane(zc, xc, _modes(gen, 4, dev))).contiguous()
    ph, p0 = (1e-5 * size * cosy * plane(zc, xc, _modes(gen, 4, dev)) for _ in range(2))
    for a in (ph, p0):                                                       # no values outside the walls, as the projection leaves them
        a[:, 0] = 0.0
        a[:, -1] = 0.0
    for a in (Pr, ph, p0):
        _fill_periodic(a)
    out = dict(zip(STATE, (T, U, V, W, Pr, ph, p0)))
    if case["precision"]:                                                    # a checkpoint of the FP32-mixed form holds FP32 values
        out = {k: v.float().double() for k, v in out.items()}
    return out


class _Device:
    """A device buffer of the solver, for torch; the tensor made of it keeps the solver."""

    def __init__(self, s, name):
        self.solver = s
        kind = "<f4" if s.precision == P.PREC_FP32_MIXED else "<f8"
        self.__cuda_array_interface__ = {"shape": s.shape, "typestr": kind, "data": (s.device_ptr(name), False), "version": 3}


def _view(s, name):
    return torch.as_tensor(_Device(s, name), device="cuda")


def _solver(case, seed):
    s = P.Solver(**_config(case))
    if case["tuned"]:
        s.autotune(cache_path=TUNE_CACHE)
    for name, a in _fields(case, seed, "cuda").items():
        _view(s, name).copy_(a)
    torch.cuda.synchronize()
    s.snapshot()
    return s


def prepare(case, seed):
    if case["kind"] == "tdma":
        given = _systems(case, seed, "cuda")
        return {"case": case, "plan": P.TdmaPlan(case["n_sys"]), "given": given, "work": [torch.empty_like(t) for t in given]}
    if case["kind"] == "ensemble":
        solvers = [_solver(m, 100 * seed + i) for i, m in enumerate(_members(case))]
        e = P.Ensemble(solvers)
        e.step(8)                       # an ensemble measures its two forms over its first eight steps
        for s in solvers:
            s.restore()
            s.synchronize()
        return {"case": case, "ensemble": e, "solvers": solvers}
    s = _solver(case, seed)
    if case["kind"] == "step":
        s.step(case["steps"])           # a run's graphs exist by the time that it restarts from a checkpoint
        s.restore()
        s.synchronize()
    return {"case": case, "solver": s}


def _run_tdma(state, case):
    for w, g in zip(state["work"], state["given"]):     # the solve overwrites its rows
        w.copy_(g)
    A, B, C, D = state["work"]
    torch.cuda.current_stream().synchronize()           # the plan solves on a stream of its own
    solve = state["plan"].many_solve_cycle if case["cyclic"] else state["plan"].many_solve
    solve(A, B, C, D, case["n_sys"], case["n_row"])
    return D


def run(state):
    case = state["case"]
    if case["kind"] == "tdma":
        return _run_tdma(state, case)
    if case["kind"] == "ensemble":
        for s in state["solvers"]:
            s.restore()
        state["ensemble"].step(case["steps"])
        return [{n: _view(s, n) for n in FIELDS} for s in state["solvers"]]
    s = state["solver"]
    s.restore()
    if case["kind"] == "driver":
        for _ in range(case["steps"]):
            s.driver_step()
    else:
        s.step(case["steps"])
    return {n: _view(s, n) for n in FIELDS}


def _systems(case, seed, dev):
    """Diagonally dominant rows of the strength that an implicit diffusion or wave-number solve has."""
    gen = torch.Generator(device=dev).manual_seed(int(seed))
    n, m = case["n_row"], case["n_sys"]
    r = [torch.rand(n, m, generator=gen, dtype=torch.float64, device=dev) for _ in range(4)]
    A, C = -0.2 - 0.8 * r[0], -0.2 - 0.8 * r[1]
    B = 0.05 + r[2] - A - C
    return A, B, C, 2.0 * r[3] - 1.0


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
# Arrays read and written by the routines of a step, each an entry point with outputs that a user can read after it:
# thermal_solver 5 (T U V W, T), solvedU 6 (U V W P T, dU), solvedV 6, solvedW 7, blockLdV 4, blockLdU 5, the pseudo-update
# with the pressure right-hand side 11, the Poisson solve 2, the projection 13, the diagnostics 3.
STEP_ARRAYS = 62
# the velocity's low words of the FP32-mixed form: right-hand side 6, projection 6, diagnostics 3
LOW_ARRAYS = 15
# operators of the nine stencils and their twelve tridiagonal solves
STEP_FLOPS = 2000


def _step_work(case):
    cells = case["n1m"] * case["n2m"] * case["n3m"]
    arrays = STEP_ARRAYS + (LOW_ARRAYS if case["precision"] else 0)
    fft = 4 * 2.5 * (math.log2(case["n1m"]) + math.log2(case["n3m"]))
    return case["steps"] * cells * arrays * (4 if case["precision"] else 8), case["steps"] * cells * (STEP_FLOPS + fft)


def work(case):
    if case["kind"] == "tdma":
        n = case["n_sys"] * case["n_row"]
        return {"bytes": n * 8 * 5, "flops": n * 20}
    parts = [_step_work(m) for m in _members(case)] if case["kind"] == "ensemble" else [_step_work(case)]
    return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}


def tolerance(case):
    if case["kind"] == "tdma":
        return "exact"                  # the interface promises the bits of the reference's IEEE arithmetic
    mixed = case["kind"] == "ensemble" or case["precision"]
    # four times the largest distance from exact() over the listed and 26 drawn cases: dPhat, the smallest output
    return {"rel": 1.2e-5, "max": 7e-5} if mixed else {"rel": 2e-10, "max": 1e-9}


# ---------------------------------------------------------------------------
# the time step in 64 bits
# ---------------------------------------------------------------------------
def _mesh(case, dev):
    """mpi_subdomain_mesh on one rank (module_mpi_subdomain.f90:153-299): x1..x3, dx1..dx3, dmx1..dmx3."""
    m = {}
    for d, n, uniform, gamma, length in ((1, case["n1m"], True, 0.0, 2.0),
                                         (2, case["n2m"], False, case["gamma2"], 1.0), (3, case["n3m"], True, 0.0, 2.0)):
        q = np.arange(n + 2, dtype=np.float64) - 1.0
        x = q * length / n if uniform else length * 0.5 * (1.0 + np.tanh(0.5 * gamma * (2.0 * q / n - 1.0)) / np.tanh(gamma * 0.5))
        if d == 2:
            x[0] = x[1]
        dx, dmx = np.zeros(n + 2), np.zeros(n + 2)
        dx[1:n + 1] = x[2:n + 2] - x[1:n + 1]
        if d != 2:
            dx[0], dx[n + 1] = dx[n], dx[1]
        dmx[1:n + 1] = 0.5 * (dx[0:n] + dx[1:n + 1])
        if d != 2:
            dmx[0], dmx[n + 1] = dmx[n], dmx[1]
        else:
            dmx[n + 1] = 0.5 * (dx[n] + dx[n + 1])
        for name, v in (("x", x), ("dx", dx), ("dmx", dmx)):
            m["%s%d" % (name, d)] = torch.tensor(v, dtype=torch.float64, device=dev)
    return m


# density, heat capacity, conductivity and viscosity polynomials (module_global.f90:113-132)
_PROPERTIES = {
    0: ((1.0,), (1.0,), (1.0,), (1.0,)),
    1: ((0.9922e+3, -3.736e-4, -3.98e-6), (4.1690e+3, 0.084e-4, 4.60e-6), (float(np.float32(0.6297)), 21.99e-4, -17.8e-6),
        (0.6690e-6, -175.9e-4, 295.8e-6, -460.e-8)),
    2: ((1.2477e+3, -4.789e-4, -0.3795e-6), (2.5108e+3, 22.511e-4), (2.9351e-3, 3.863e-4),
        (238.71e-6, -702.83e-4, 2393.1e-6, -6923.0e-8, 33131.3e-10, -71517.5e-12)),
}


def _poly(c, t):
    """c[0] (1 + c[1] t + c[2] t^2 + ...)."""
    s = torch.zeros_like(t)
    for q in reversed(c[1:]):
        s = (s + q) * t
    return c[0] * (1.0 + s)


def _dpoly(c, t):
    s = torch.zeros_like(t)
    for k in range(len(c) - 1, 0, -1):
        s = s * t + k * c[k]
    return c[0] * s


def _thomas(a, b, c, d, dim):
    """Tridiagonal systems along dim; a of the first and c of the last row are not used."""
    a, b, c, d = (torch.broadcast_to(t, d.shape).movedim(dim, 0) for t in (a, b, c, d))
    n = d.shape[0]
    cp, x = torch.empty_like(d), torch.empty_like(d)
    den = b[0]
    cp[0], x[0] = c[0] / den, d[0] / den
    for r in range(1, n):
        den = b[r] - a[r] * cp[r - 1]
        cp[r] = c[r] / den
        x[r] = (d[r] - a[r] * x[r - 1]) / den
    for r in range(n - 2, -1, -1):
        x[r] -= cp[r] * x[r + 1]
    return x.movedim(0, dim)


def _cyclic(a, b, c, d, dim):
    """Cyclic systems: the last unknown is bordered out of the other rows."""
    a, b, c, d = (torch.broadcast_to(t, d.shape).movedim(dim, 0) for t in (a, b, c, d))
    n = d.shape[0]
    cp, x, e = torch.empty_like(d), torch.empty_like(d), torch.empty_like(d)
    cp[0], x[0], e[0] = c[0] / b[0], d[0] / b[0], a[0] / b[0]
    for r in range(1, n - 1):
        den = b[r] - a[r] * cp[r - 1]
        cp[r] = c[r] / den
        x[r] = (d[r] - a[r] * x[r - 1]) / den
        e[r] = -a[r] * e[r - 1] / den
    e[n - 2] += cp[n - 2]
    for r in range(n - 3, -1, -1):
        x[r] -= cp[r] * x[r + 1]
        e[r] -= cp[r] * e[r + 1]
    # rows 0..n-2 are x - e last; the last row closes the system
    last = (d[n - 1] - a[n - 1] * x[n - 2] - c[n - 1] * x[0]) / (b[n - 1] - a[n - 1] * e[n - 2] - c[n - 1] * e[0])
    x[n - 1] = last
    x[:n - 1] -= e[:n - 1] * last
    return x.movedim(0, dim)


class _Exact:
    """One case's time step, every expression as the reference has it (citations: its source files)."""

    def __init__(self, case, fields):
        self.N = (case["n1m"], case["n2m"], case["n3m"])
        dev = fields["T"].device
        self.m = _mesh(case, dev)
        self.f = dict(fields)
        self.prop = _PROPERTIES[case["property_set"]]
        self.dT, self.dt, self.fixed = case["DeltaT"], case["dtStart"], case["fixed_dt"]
        self.Cmu, self.Ct = math.sqrt(case["Pr"] / case["Ra"]), 1.0 / math.sqrt(case["Ra"] * case["Pr"])
        self.dt_max = 100.0 * min(2.0 / self.N[0], 1.0 / self.N[1], 2.0 / self.N[2])
        self.Tbt, self.Tup = 0.5, -0.5
        a = self.prop[0] + (0.0,) * 3
        self.a12pera11 = 0.0 if a[2] < 1e-14 else a[2] / a[1]

    # metric values of the cells of a block, shaped for (k, j, i); s shifts, j0 is the first j
    def mx(self, name, s=0, j0=1):
        v, d = self.m[name], int(name[-1])
        n = self.N[d - 1]
        lo = j0 if d == 2 else 1
        return v[lo + s:n + 1 + s].reshape([-1 if q == 3 - d else 1 for q in range(3)])

    def at(self, A, dk=0, dj=0, di=0, j0=1):
        N1, N2, N3 = self.N
        return A[1 + dk:N3 + 1 + dk, j0 + dj:N2 + 1 + dj, 1 + di:N1 + 1 + di]

    def tab(self, A, dj=0, dk=0, j0=1):
        """A (k, j) table's values, constant along i."""
        return A[1 + dk:self.N[2] + 1 + dk, j0 + dj:self.N[1] + 1 + dj, None]

    def padded(self, inner, j0=1):
        N1, N2, N3 = self.N
        A = torch.zeros(N3 + 2, N2 + 2, N1 + 2, dtype=torch.float64, device=inner.device)
        A[1:N3 + 1, j0:N2 + 1, 1:N1 + 1] = inner
        _fill_periodic(A)
        return A

    def masks(self, j0=1):
        """0 on the lowest and on the highest row of the block (the rows next to the walls), else 1."""
        n = self.N[1] + 1 - j0
        lo = torch.ones(1, n, 1, dtype=torch.float64, device=self.f["T"].device)
        hi = lo.clone()
        lo[0, 0, 0] = 0.0
        hi[0, -1, 0] = 0.0
        return lo, hi

    def thermal(self):
        """mpi_thermal_coeffi and mpi_thermal_solver (module_solve_thermal.f90:129-154, 236-524)."""
        f, mx, at, dt = self.f, self.mx, self.at, self.dt
        T, U, V, W = f["T"], f["U"], f["V"], f["W"]
        a, b, c, _ = self.prop
        t = self.dT * T
        K, dK = _poly(c, t) / c[0], _dpoly(c, t) / c[0]
        ra, rb = _poly(a, t) / a[0], _poly(b, t) / b[0]
        irc = 1.0 / (ra * rb)
        dirc = -(_dpoly(a, t) / a[0] * rb + ra * _dpoly(b, t) / b[0]) * irc * irc
        jem, jep = self.masks()
        d1, d1m, d1p, e1, e1p = mx("dx1"), mx("dx1", -1), mx("dx1", 1), mx("dmx1"), mx("dmx1", 1)
        d2, d2m, d2p, e2, e2p = mx("dx2"), mx("dx2", -1), mx("dx2", 1), mx("dmx2"), mx("dmx2", 1)
        d3, d3m, d3p, e3, e3p = mx("dx3"), mx("dx3", -1), mx("dx3", 1), mx("dmx3"), mx("dmx3", 1)
        h, Tc = 0.5 * self.Ct * at(irc), at(T)
        dh = 0.5 * self.Ct * at(dirc)

        def faces(A, dim, lo, hi):
            """Face values of A at the lower and upper face along dim."""
            dd, dm, dp, em, ep = ((d1, d1m, d1p, e1, e1p), (d2, d2m, d2p, e2, e2p), (d3, d3m, d3p, e3, e3p))[dim]
            mid = at(A)
            return 0.5 / em * (dd * lo + dm * mid), 0.5 / ep * (dp * mid + dd * hi)

        def sh(A, dim, s):
            return at(A, **{("di", "dj", "dk")[dim]: s})

        kp, dkp, ee, de = [], [], [], []
        for dim, (em, ep) in enumerate(((e1, e1p), (e2, e2p), (e3, e3p))):
            kp.append(faces(K, dim, sh(K, dim, -1), sh(K, dim, 1)))
            dkp.append(faces(dK, dim, sh(dK, dim, -1), sh(dK, dim, 1)))
            ee.append(faces(T, dim, sh(T, dim, -1), sh(T, dim, 1)))
            de.append(((Tc - sh(T, dim, -1)) / em, (sh(T, dim, 1) - Tc) / ep))
        u = ((at(U), at(U, di=1)), (at(V), at(V, dj=1)), (at(W), at(W, dk=1)))
        dd = (d1, d2, d3)
        rhs = torch.zeros_like(Tc)
        dv = torch.zeros_like(Tc)
        rows = []
        for dim, (dm, dp, em, ep) in enumerate(((d1m, d1p, e1, e1p), (d2m, d2p, e2, e2p), (d3m, d3p, e3, e3p))):
            (k0, k1), (q0, q1), (g0, g1), (t0, t1), (u0, u1) = kp[dim], dkp[dim], de[dim], ee[dim], u[dim]
            lo, hi = (jem, jep) if dim == 1 else (1.0, 1.0)
            rhs = rhs - 0.25 * (u0 * g0 + u1 * g1) + h * (k1 * g1 - k0 * g0 - t1 * q1 * g1 + t0 * q0 * g0) / dd[dim]
            dv = dv + (k1 * g1 - k0 * g0) / dd[dim]
            ac = h / dd[dim] * (k1 / ep + k0 / em - dp * 0.5 / ep * q1 * g1 * hi + dm * 0.5 / em * q0 * g0 * lo) + (0.25 * u0 / em - 0.25 * u1 / ep)
            ap = (-h / dd[dim] * (k1 / ep + dd[dim] * 0.5 / ep * q1 * g1) + 0.25 * u1 / ep) * hi
            am = (-h / dd[dim] * (k0 / em - dd[dim] * 0.5 / em * q0 * g0) - 0.25 * u0 / em) * lo
            rows.append((am, ac, ap))
        (k0, k1), (q0, q1), (g0, g1), (u0, u1) = kp[1], dkp[1], de[1], u[1]
        up = -0.25 * u1 / e2p * self.Tup + h / d2 * k1 / e2p * self.Tup + h / d2 * q1 * g1 * self.Tup
        dn = 0.25 * u0 / e2 * self.Tbt + h / d2 * k0 / e2 * self.Tbt - h / d2 * q0 * g0 * self.Tbt
        rhs = rhs + (1.0 - jem) * dn + (1.0 - jep) * up
        for dim, (am, ac, ap) in enumerate(rows):
            rhs = rhs - (ap * sh(T, dim, 1) + ac * Tc + am * sh(T, dim, -1))
        am, ac, ap = rows[2]
        r = _cyclic(am * dt, 1.0 + ac * dt - 0.5 * dh * dv * dt, ap * dt, rhs * dt, 0)
        # stages 2 and 3 read the neighbours with the indices that the stage before left: N-1 and N+1
        N1, N2, N3 = self.N

        def stale(dim):
            n = (N1, N2, N3)[dim]
            cut = {1: (lambda q: (slice(1, N3 + 1), slice(q, q + 1), slice(1, N1 + 1))), 2: (lambda q: (slice(q, q + 1), slice(1, N2 + 1), slice(1, N1 + 1)))}[dim]
            d, e = self.m["dx%d" % (dim + 1)], self.m["dmx%d" % (dim + 1)]
            dd, em = (d2, e2) if dim == 1 else (d3, e3)
            Km, Kp, Tm, Tp = K[cut(n - 1)], K[cut(n + 1)], T[cut(n - 1)], T[cut(n + 1)]
            km = 0.5 / em * (dd * Km + d[n - 1] * at(K))
            kq = 0.5 / e[n + 1] * (d[n + 1] * at(K) + dd * Kp)
            return (kq * (Tp - Tc) / e[n + 1] - km * (Tc - Tm) / em) / dd

        x = (kp[0][1] * de[0][1] - kp[0][0] * de[0][0]) / d1
        yv = (kp[1][1] * de[1][1] - kp[1][0] * de[1][0]) / d2
        zs = stale(2)
        am, ac, ap = rows[0]
        r = _cyclic(am * dt, 1.0 + (ac - 0.5 * h * (x + stale(1) + zs)) * dt, ap * dt, r, 2)
        am, ac, ap = rows[1]
        r = _thomas(am * dt, 1.0 + (ac - 0.5 * h * (x + yv + zs)) * dt, ap * dt, r, 1)
        new = self.padded(Tc + r)
        new[:, 0], new[:, -1] = T[:, 0], T[:, -1]
        f["T"] = new

    def tables(self):
        """mpi_momentum_coeffi (module_solve_momentum.f90:145-173): rows of T(n1sub, j, k)."""
        a, _, _, d = self.prop
        t = self.dT * self.f["T"][:, :, -1]
        ra = _poly(a, t)
        self.Mu, self.iR = ra * _poly(d, t) / (a[0] * d[0]), a[0] / ra

    def momentum(self):
        """solvedU, solvedV, solvedW, blockLdV, blockLdU (module_solve_momentum.f90:225-1460).  The wall velocities are 0."""
        f, mx, at, dt, Mu, iR = self.f, self.mx, self.at, self.dt, self.Mu, self.iR
        T, U, V, W, Pp = f["T"], f["U"], f["V"], f["W"], f["P"]
        N1, N2, N3 = self.N
        d1, d1m, d1p, e1, e1p = mx("dx1"), mx("dx1", -1), mx("dx1", 1), mx("dmx1"), mx("dmx1", 1)
        d3, d3m, d3p, e3, e3p = mx("dx3"), mx("dx3", -1), mx("dx3", 1), mx("dmx3"), mx("dmx3", 1)
        d2, d2m, d2p, e2, e2p = mx("dx2"), mx("dx2", -1), mx("dx2", 1), mx("dmx2"), mx("dmx2", 1)
        tab = self.tab
        lo, hi = self.masks()

        # ---- dU
        Uc = at(U)
        u1, u2 = 0.5 * (at(U, di=-1) + Uc), 0.5 * (at(U, di=1) + Uc)
        v3 = 0.5 * (d1m * at(V) + d1 * at(V, di=-1)) / e1
        v4 = 0.5 * (d1m * at(V, dj=1) + d1 * at(V, dj=1, di=-1)) / e1
        w5 = 0.5 * (d1m * at(W) + d1 * at(W, di=-1)) / e1
        w6 = 0.5 * (d1m * at(W, dk=1) + d1 * at(W, dk=1, di=-1)) / e1
        g1, g2 = (Uc - at(U, di=-1)) / d1m, (at(U, di=1) - Uc) / d1
        g3, g4 = (Uc - at(U, dj=-1)) / e2, (at(U, dj=1) - Uc) / e2p
        g5, g6 = (Uc - at(U, dk=-1)) / e3, (at(U, dk=1) - Uc) / e3p
        vx3, vx4 = (at(V) - at(V, di=-1)) / e1, (at(V, dj=1) - at(V, dj=1, di=-1)) / e1
        wx5, wx6 = (at(W) - at(W, di=-1)) / e1, (at(W, dk=1) - at(W, dk=1, di=-1)) / e1
        mc = tab(Mu)
        m3, m4 = 0.5 * (d2m * mc + d2 * tab(Mu, -1)) / e2, 0.5 * (d2p * mc + d2 * tab(Mu, 1)) / e2p
        m5, m6 = 0.5 * (d3m * mc + d3 * tab(Mu, 0, -1)) / e3, 0.5 * (d3p * mc + d3 * tab(Mu, 0, 1)) / e3p
        ir = tab(iR)
        ih = 0.5 * self.Cmu * ir
        A1 = (-2 * ih / e1 * mc / d1m + 0.25 * (-u1 / d1m + 0.5 * g1), 2 * ih / e1 * mc * (1 / d1 + 1 / d1m) + 0.25 * (0.5 * g2 + 0.5 * g1 - u2 / d1 + u1 / d1m),
              -2 * ih / e1 * mc / d1 + 0.25 * (u2 / d1 + 0.5 * g2))
        A2 = ((-ih / d2 * m3 / e2 - 0.25 * v3 / e2) * lo, ih / d2 * (m4 / e2p + m3 / e2) + 0.25 * (-v4 / e2p + v3 / e2), (-ih / d2 * m4 / e2p + 0.25 * v4 / e2p) * hi)
        A3 = (-ih / d3 * m5 / e3 - 0.25 * w5 / e3, ih / d3 * (m6 / e3p + m5 / e3) + 0.25 * (-w6 / e3p + w5 / e3), -ih / d3 * m6 / e3p + 0.25 * w6 / e3p)
        rhs = 2 * ih * mc * (g2 - g1) / e1 + ih * ((m4 * g4 - m3 * g3) / d2 + (m6 * g6 - m5 * g5) / d3)
        # the x diffusion and the cross derivatives of the full stress tensor
        rhs = rhs + ih * ((m4 * vx4 - m3 * vx3) / d2 + (m6 * wx6 - m5 * wx5) / d3)
        Tf = 0.5 * (d1m * at(T) + d1 * at(T, di=-1)) / e1
        rhs = rhs - ir * (at(Pp) - at(Pp, di=-1)) / e1 + (Tf + self.a12pera11 * Tf * Tf * self.dT) * ir
        rhs = rhs - (A1[2] * at(U, di=1) + A1[1] * Uc + A1[0] * at(U, di=-1)) - (A2[2] * at(U, dj=1) + A2[1] * Uc + A2[0] * at(U, dj=-1)) \
            - (A3[2] * at(U, dk=1) + A3[1] * Uc + A3[0] * at(U, dk=-1))
        rhs = rhs - (0.25 * (v4 * hi * g4 + v3 * lo * g3) - ih / d2 * (m4 * vx4 * hi - m3 * vx3 * lo)) \
            - (0.25 * (w6 * g6 + w5 * g5) - ih / d3 * (m6 * wx6 - m5 * wx5))
        r = self._sweeps(A1, A2, A3, rhs)
        dU = self.padded(r)
        ihu, mu_u = ih, (m3, m4, m5, m6, g3, g4, g5, g6)

        # ---- dV: rows j = 2 .. N2
        j0 = 2
        at2 = lambda A, **s: at(A, j0=2, **s)  # noqa: E731
        d2, d2m, d2p, e2 = mx("dx2", 0, 2), mx("dx2", -1, 2), mx("dx2", 1, 2), mx("dmx2", 0, 2)
        t2 = lambda A, dj=0, dk=0: tab(A, dj, dk, 2)  # noqa: E731
        lo, hi = self.masks(2)

        def ymean(A, **s):
            s1 = dict(s)
            s1["dj"] = s.get("dj", 0) - 1
            return (d2m * at2(A, **s) + d2 * at2(A, **s1)) / e2 * 0.5

        def ygrad(A, **s):
            s1 = dict(s)
            s1["dj"] = s.get("dj", 0) - 1
            return (at2(A, **s) - at2(A, **s1)) / e2

        Vc = at2(V)
        v3, v4 = 0.5 * (at2(V, dj=-1) + Vc), 0.5 * (Vc + at2(V, dj=1))
        u1, u2, w5, w6 = ymean(U), ymean(U, di=1), ymean(W), ymean(W, dk=1)
        p1, p2 = ymean(dU), ymean(dU, di=1)
        g1, g2 = (Vc - at2(V, di=-1)) / e1, (at2(V, di=1) - Vc) / e1p
        g3, g4 = (Vc - at2(V, dj=-1)) / d2m, (at2(V, dj=1) - Vc) / d2
        g5, g6 = (Vc - at2(V, dk=-1)) / e3, (at2(V, dk=1) - Vc) / e3p
        mxy = 0.5 * (d2m * t2(Mu) + d2 * t2(Mu, -1)) / e2
        m1 = 0.5 * (d1m + d1) / e1 * mxy
        m2 = 0.5 * (d1p + d1) / e1p * mxy
        ma, mb = 0.5 * (d2m * t2(Mu, 0, -1) + d2 * t2(Mu, -1, -1)) / e2, 0.5 * (d2m * t2(Mu, 0, 1) + d2 * t2(Mu, -1, 1)) / e2
        m5, m6 = 0.5 * (d3m * mxy + d3 * ma) / e3, 0.5 * (d3p * mxy + d3 * mb) / e3p
        ir = 0.5 * (d2m * t2(iR) + d2 * t2(iR, -1)) / e2
        ih = 0.5 * self.Cmu * ir
        # the upper coefficient carries the mask of the row below, the lower one that of the row above (:864-889)
        A2 = ((-2 * ih / e2 * t2(Mu, -1) / d2m + 0.25 * (-v3 / d2m + 0.5 * g3)) * hi,
              2 * ih / e2 * (t2(Mu) / d2 + t2(Mu, -1) / d2m) + 0.25 * (0.5 * g4 + 0.5 * g3 - v4 / d2 + v3 / d2m),
              (-2 * ih / e2 * t2(Mu) / d2 + 0.25 * (v4 / d2 + 0.5 * g4)) * lo)
        A1 = (-ih / d1 * m1 / e1 - 0.25 * u1 / e1, ih / d1 * (m2 / e1p + m1 / e1) + 0.25 * (-u2 / e1p + u1 / e1), -ih / d1 * m2 / e1p + 0.25 * u2 / e1p)
        A3 = (-ih / d3 * m5 / e3 - 0.25 * w5 / e3, ih / d3 * (m6 / e3p + m5 / e3) + 0.25 * (-w6 / e3p + w5 / e3), -ih / d3 * m6 / e3p + 0.25 * w6 / e3p)
        uy1, uy2, wy5, wy6 = ygrad(U), ygrad(U, di=1), ygrad(W), ygrad(W, dk=1)
        rhs = ih * ((m2 * g2 - m1 * g1) / d1 + 2 * (t2(Mu) * g4 - t2(Mu, -1) * g3) / e2 + (m6 * g6 - m5 * g5) / d3)
        rhs = rhs + ih * ((m2 * uy2 - m1 * uy1) / d1 + (m6 * wy6 - m5 * wy5) / d3)
        rhs = rhs - ir * (at2(Pp) - at2(Pp, dj=-1)) / e2
        rhs = rhs - (A1[2] * at2(V, di=1) + A1[1] * Vc + A1[0] * at2(V, di=-1)) - (A2[2] * at2(V, dj=1) + A2[1] * Vc + A2[0] * at2(V, dj=-1)) \
            - (A3[2] * at2(V, dk=1) + A3[1] * Vc + A3[0] * at2(V, dk=-1))
        rhs = rhs - (0.25 * (u2 * g2 + u1 * g1) - ih / d1 * (m2 * uy2 - m1 * uy1)) - (0.25 * (w6 * g6 + w5 * g5) - ih / d3 * (m6 * wy6 - m5 * wy5))
        rhs = rhs - (0.25 * (p2 * g2 + p1 * g1) - ih / d1 * (m2 * ygrad(dU, di=1) - m1 * ygrad(dU)))
        # stage 2 keeps the mu1, mu2 of the last cell of stage 1
        s1, s2 = (torch.broadcast_to(q, rhs.shape)[-1, -1, -1] for q in (m1, m2))
        A1s = (-ih / d1 * s1 / e1 - 0.25 * u1 / e1, ih / d1 * (s2 / e1p + s1 / e1) + 0.25 * (-u2 / e1p + u1 / e1), -ih / d1 * s2 / e1p + 0.25 * u2 / e1p)
        dV = self.padded(self._sweeps(A1s, A2, A3, rhs), 2)
        bv = (v3, v4, g5, g6, m5, m6, ih, ymean, ygrad)

        # ---- dW
        d2, d2m, d2p, e2, e2p = mx("dx2"), mx("dx2", -1), mx("dx2", 1), mx("dmx2"), mx("dmx2", 1)
        lo, hi = self.masks()

        def zmean(A, **s):
            s1 = dict(s)
            s1["dk"] = s.get("dk", 0) - 1
            return (d3m * at(A, **s) + d3 * at(A, **s1)) / e3 * 0.5

        def zgrad(A, **s):
            s1 = dict(s)
            s1["dk"] = s.get("dk", 0) - 1
            return (at(A, **s) - at(A, **s1)) / e3

        Wc = at(W)
        w5, w6 = 0.5 * (Wc + at(W, dk=-1)), 0.5 * (Wc + at(W, dk=1))
        u1, u2, v3, v4 = zmean(U), zmean(U, di=1), zmean(V), zmean(V, dj=1)
        p1, p2, p3, p4 = zmean(dU), zmean(dU, di=1), zmean(dV) * lo, zmean(dV, dj=1) * hi
        g1, g2 = (Wc - at(W, di=-1)) / e1, (at(W, di=1) - Wc) / e1p
        g3, g4 = (Wc - at(W, dj=-1)) / e2, (at(W, dj=1) - Wc) / e2p
        g5, g6 = (Wc - at(W, dk=-1)) / d3m, (at(W, dk=1) - Wc) / d3
        mxz = 0.5 * (d3m * tab(Mu) + d3 * tab(Mu, 0, -1)) / e3
        m1, m2 = 0.5 * (d1m + d1) / e1 * mxz, 0.5 * (d1p + d1) / e1p * mxz
        ma, mb = 0.5 * (d3m * tab(Mu, -1) + d3 * tab(Mu, -1, -1)) / e3, 0.5 * (d3m * tab(Mu, 1) + d3 * tab(Mu, 1, -1)) / e3
        m3, m4 = 0.5 * (d2m * mxz + d2 * ma) / e2, 0.5 * (d2p * mxz + d2 * mb) / e2p
        ir = 0.5 * (d3m * tab(iR) + d3 * tab(iR, 0, -1)) / e3
        ih = 0.5 * self.Cmu * ir
        uz1, uz2, vz3, vz4 = zgrad(U), zgrad(U, di=1), zgrad(V), zgrad(V, dj=1)
        q1, q2, q3, q4 = zgrad(dU), zgrad(dU, di=1), zgrad(dV), zgrad(dV, dj=1)

        def a1(n1, n2):
            return (-ih / d1 * n1 / e1 - 0.25 * u1 / e1, ih / d1 * (n2 / e1p + n1 / e1) + 0.25 * (-u2 / e1p + u1 / e1), -ih / d1 * n2 / e1p + 0.25 * u2 / e1p)

        def a2(n3, n4, v3, v4, ih):
            return ((-ih / d2 * n3 / e2 - 0.25 * v3 / e2) * lo, ih / d2 * (n4 / e2p + n3 / e2) + 0.25 * (-v4 / e2p + v3 / e2), (-ih / d2 * n4 / e2p + 0.25 * v4 / e2p) * hi)

        A1, A2 = a1(m1, m2), a2(m3, m4, v3, v4, ih)
        k0, k1 = tab(Mu, 0, -1), tab(Mu)
        A3 = (-2 * ih / e3 * k0 / d3m + 0.25 * (-w5 / d3m + 0.5 * g5), 2 * ih / e3 * (k1 / d3 + k0 / d3m) + 0.25 * (-w6 / d3 + w5 / d3m + 0.5 * g6 + 0.5 * g5),
              -2 * ih / e3 * k1 / d3 + 0.25 * (w6 / d3 + 0.5 * g6))
        rhs = ih * ((m2 * g2 - m1 * g1) / d1 + (m4 * g4 - m3 * g3) / d2 + 2 * (k1 * g6 - k0 * g5) / e3)
        rhs = rhs + ih * ((m2 * uz2 - m1 * uz1) / d1 + (m4 * vz4 - m3 * vz3) / d2)
        rhs = rhs - ir * (at(Pp) - at(Pp, dk=-1)) / e3
        rhs = rhs - (A1[2] * at(W, di=1) + A1[1] * Wc + A1[0] * at(W, di=-1)) - (A2[2] * at(W, dj=1) + A2[1] * Wc + A2[0] * at(W, dj=-1)) \
            - (A3[2] * at(W, dk=1) + A3[1] * Wc + A3[0] * at(W, dk=-1))
        rhs = rhs - (0.25 * (u2 * g2 + u1 * g1) - ih / d1 * (m2 * uz2 - m1 * uz1)) - (0.25 * (v3 * lo * g3 + v4 * hi * g4) - ih / d2 * (m4 * vz4 * hi - m3 * vz3 * lo))
        rhs = rhs - (0.25 * (p2 * g2 + p1 * g1) - ih / d1 * (m2 * q2 - m1 * q1)) - (0.25 * (p3 * lo * g3 + p4 * hi * g4) - ih / d2 * (m4 * q4 * hi - m3 * q3 * lo))
        s1, s2, s3, s4 = (torch.broadcast_to(q, rhs.shape)[-1, -1, -1] for q in (m1, m2, m3, m4))
        # stage 3: mu3, mu4 of the last cell of stage 1 and km = N3 - 1 throughout
        dk, jn = self.m["dx3"][N3 - 1], slice(1, N2 + 1)
        below = lambda A, dj=0: A[N3 - 1:N3, 1 + dj:N2 + 1 + dj, 1:N1 + 1]  # noqa: E731
        z3, z4 = (dk * at(V) + d3 * below(V)) / e3 * 0.5, (dk * at(V, dj=1) + d3 * below(V, 1)) / e3 * 0.5
        ihs = 0.5 * self.Cmu * 0.5 * (dk * tab(iR) + d3 * iR[N3 - 1:N3, jn, None]) / e3
        dW = self.padded(self._sweeps(a1(s1, s2), a2(s3, s4, z3, z4, ihs), A3, rhs))

        # ---- blockLdV, blockLdU
        v3, v4, g5, g6, m5, m6, ih, ymean, ygrad = bv
        d2, d2m, d2p, e2 = mx("dx2", 0, 2), mx("dx2", -1, 2), mx("dx2", 1, 2), mx("dmx2", 0, 2)
        new = at2(dV) - dt * (0.25 * (ymean(dW) * g5 + ymean(dW, dk=1) * g6) - ih / d3 * (m6 * ygrad(dW, dk=1) - m5 * ygrad(dW)))
        dV = self.padded(new, 2)
        m3, m4, m5, m6, g3, g4, g5, g6 = mu_u
        d2 = mx("dx2")
        lo, hi = self.masks()
        mean = lambda A, **s: (d1 * at(A, di=-1, **s) + d1m * at(A, **s)) / e1 * 0.5  # noqa: E731
        grad = lambda A, **s: (at(A, **s) - at(A, di=-1, **s)) / e1  # noqa: E731
        new = at(dU) - dt * (0.25 * (mean(dV, dj=1) * hi * g4 + mean(dV) * lo * g3) - ihu / d2 * (m4 * grad(dV, dj=1) * hi - m3 * grad(dV) * lo)) \
            - dt * (0.25 * (mean(dW, dk=1) * g6 + mean(dW) * g5) - ihu / d3 * (m6 * grad(dW, dk=1) - m5 * grad(dW)))
        # the pseudo-update (:178-208); the lower wall row of V stays
        dV[:, 1] = 0.0
        for name, inc in (("U", new), ("V", at(dV)), ("W", at(dW))):
            a = self.padded(at(f[name]) + inc)
            a[:, 0], a[:, -1] = 0.0, 0.0
            f[name] = a

    def _sweeps(self, A1, A2, A3, rhs):
        dt = self.dt
        r = _cyclic(A3[0] * dt, 1.0 + A3[1] * dt, A3[2] * dt, rhs * dt, 0)
        r = _cyclic(A1[0] * dt, 1.0 + A1[1] * dt, A1[2] * dt, r, 2)
        return _thomas(A2[0] * dt, 1.0 + A2[1] * dt, A2[2] * dt, r, 1)

    def pressure(self):
        """mpi_pressure_RHS, Poisson_FFT2 and Projection (module_solve_pressure.f90:140-231, 489-744, 756-874)."""
        f, mx, at, tab, dt, iR = self.f, self.mx, self.at, self.tab, self.dt, self.iR
        N1, N2, N3 = self.N
        U, V, W, ph = f["U"], f["V"], f["W"], f["dPhat"]
        d1, d1m, d1p, e1, e1p = mx("dx1"), mx("dx1", -1), mx("dx1", 1), mx("dmx1"), mx("dmx1", 1)
        d2, d2m, d2p, e2, e2p = mx("dx2"), mx("dx2", -1), mx("dx2", 1), mx("dmx2"), mx("dmx2", 1)
        d3, d3m, d3p, e3, e3p = mx("dx3"), mx("dx3", -1), mx("dx3", 1), mx("dmx3"), mx("dmx3", 1)
        lo, hi = self.masks()
        div = (at(U, di=1) - at(U)) / d1 + (hi * at(V, dj=1) - lo * at(V)) / d2 + (at(W, dk=1) - at(W)) / d3
        c = at(ph)
        ir = tab(iR)
        i3, i4 = 0.5 / e2 * (d2m * ir + d2 * tab(iR, -1)), 0.5 / e2p * (d2p * ir + d2 * tab(iR, 1))
        i5, i6 = 0.5 / e3 * (d3m * ir + d3 * tab(iR, 0, -1)), 0.5 / e3p * (d3p * ir + d3 * tab(iR, 0, 1))
        extra = ((1 - ir) * (at(ph, di=1) - c) / e1p - (1 - ir) * (c - at(ph, di=-1)) / e1) / d1 \
            + ((1 - i4) * (at(ph, dj=1) - c) / e2p - (1 - i3) * (c - at(ph, dj=-1)) / e2) / d2 \
            + ((1 - i6) * (at(ph, dk=1) - c) / e3p - (1 - i5) * (c - at(ph, dk=-1)) / e3) / d3
        S = torch.fft.fft(torch.fft.rfft(div / dt + extra, dim=2), dim=0)
        # modified wave numbers and the modal systems (:93-129, 597-652)
        dev = S.device
        h = N1 // 2 + 1
        q1, q3 = torch.arange(h, dtype=torch.float64, device=dev), torch.arange(N3, dtype=torch.float64, device=dev)
        q3 = torch.where(q3 <= N3 // 2, q3, N3 - q3)
        dd1, dd3 = 2.0 / N1, 2.0 / N3
        kx = 2.0 * (1.0 - torch.cos(2.0 * math.pi * q1 * dd1 / 2.0)) / dd1 ** 2
        kz = 2.0 * (1.0 - torch.cos(2.0 * math.pi * q3 * dd3 / 2.0)) / dd3 ** 2
        am, ap = 1.0 / d2 / e2 * lo, 1.0 / d2 / e2p * hi
        b = torch.broadcast_to(-am - ap - kx[None, None, :] - kz[:, None, None], S.shape).clone()
        am, ap = (torch.broadcast_to(t, S.shape).clone() for t in (am, ap))
        b[0, 0, 0], ap[0, 0, 0] = 1.0, 0.0
        re = S.real.clone()
        re[0, 0, 0] = 0.0
        re, im = _thomas(am, b, ap, re, 1), _thomas(am, b, ap, S.imag.clone(), 1)
        im[0, :, 0] = 0.0
        im[N3 // 2, :, 0] = 0.0
        x = torch.fft.ifft(torch.complex(re, im), dim=0)
        x = torch.fft.irfft(x, n=N1, dim=2)
        x = x - re[0, :, 0].sum() / (N1 * N2 * N3)
        dP = self.padded(x)
        e = self.m["dmx2"]

        def wall(A):
            s1, s2 = (e[1] + e[2]) ** 2, (e[N2 + 1] + e[N2]) ** 2
            A[:, 0] = s1 / (s1 - e[1] ** 2) * A[:, 1] - e[1] ** 2 / (s1 - e[1] ** 2) * A[:, 2]
            A[:, -1] = s2 / (s2 - e[N2 + 1] ** 2) * A[:, N2] - e[N2 + 1] ** 2 / (s2 - e[N2 + 1] ** 2) * A[:, N2 - 1]

        wall(dP)
        # the projection sweeps upwards and changes dPhat as it goes, so the lower neighbours (not across the
        # periodic boundary, nor row 1 from row 2) are the new ones
        p0 = 0.5 * (c + at(f["dP0"]))
        new = self.padded(2.0 * at(dP) - p0)
        Xi, Xj, Xk = at(ph, di=-1).clone(), at(ph, dj=-1).clone(), at(ph, dk=-1).clone()
        Xi[:, :, 1:] = at(new, di=-1)[:, :, 1:]
        Xj[:, 2:] = at(new, dj=-1)[:, 2:]
        Xk[1:] = at(new, dk=-1)[1:]
        un = at(U) - dt * ((at(dP) - at(dP, di=-1)) / e1 + (ir - 1) * (c - Xi) / e1)
        j3 = 0.5 / e2 * (d2 * tab(iR, -1) + d2m * ir)
        vn = at(V) - lo * dt * ((at(dP) - at(dP, dj=-1)) / e2 + (j3 - 1) * (c - Xj) / e2)
        k3 = 0.5 / e3 * (d3 * tab(iR, 0, -1) + d3m * ir)
        wn = at(W) - dt * ((at(dP) - at(dP, dk=-1)) / e3 + (k3 - 1) * (c - Xk) / e3)
        for name, v in (("U", un), ("V", vn), ("W", wn)):
            f[name] = self.padded(v)
        p = self.padded(at(f["P"]) + at(dP))
        wall(p)
        f["P"], f["dPhat"], f["dP0"] = p, new, self.padded(p0)

    def time_step(self):
        """mpi_Post_CFL (module_post.f90:168-230)."""
        if self.fixed:
            return
        f, at, mx = self.f, self.at, self.mx
        q = abs(at(f["U"], di=1) + at(f["U"])) / 2 / mx("dx1") + abs(at(f["V"], dj=1) + at(f["V"])) / 2 / mx("dx2") \
            + abs(at(f["W"], dk=1) + at(f["W"])) / 2 / mx("dx3")
        self.dt = min(1.0 / float(q.max()), self.dt_max)

    def step(self, n):
        for _ in range(n):
            self.thermal()
            self.tables()
            self.momentum()
            self.pressure()
            self.time_step()
        return {k: self.f[k] for k in FIELDS}


def exact(case, seed, device="cuda"):
    if case["kind"] == "tdma":
        A, B, C, D = _systems(case, seed, device)
        return (_cyclic if case["cyclic"] else _thomas)(A, B, C, D, 0)
    if case["kind"] == "ensemble":
        return [_Exact(m, _fields(m, 100 * seed + i, device)).step(m["steps"]) for i, m in enumerate(_members(case))]
    return _Exact(case, _fields(case, seed, device)).step(case["steps"])
