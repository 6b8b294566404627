// tcs_device.cuh -- device-side building blocks shared by every kernel of the
// PaScaL_TCS time step on one B200 (sm_100a).
//
// Layout: every 3-D field is one padded array (0:N1+1, 0:N2+1, 0:N3+1) with i
// fastest, exactly the reference's Fortran arrays (0:n1sub, 0:n2sub, 0:n3sub)
// on one rank, so host<->device copies are plain memcpys.
//
// Two numerical forms share the code through the field type R:
//   R = double  FP64 plain, the reference's arithmetic;
//   R = float   FP32-mixed: fields stored in FP32, stencils and ADI rows built
//               in FP32; eliminations, FFTs, modal pressure solves, the
//               divergence of the pressure right-hand side, the projection and
//               all reductions in FP64 arithmetic.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <type_traits>

namespace tcs {

// ---------------------------------------------------------------------------
// Metric tables of one direction (length n+2, index 0..n+1), as computed by
// mpi_subdomain_mesh (module_mpi_subdomain.f90:153-299), plus reciprocals.
// ---------------------------------------------------------------------------
template <class R>
struct MetricT {
    const R *dx, *dmx;       // dx_sub, dmx_sub
    const R *rdx, *rdmx;     // 1/dx, 1/dmx (0 where dx or dmx is 0)
};

// Physical constants of module_global (module_global.f90:107-141) and the
// property polynomial coefficients (water/glycerol/constant).  Every member
// is of type R, so the host converts the FP64 set member by member.
template <class R>
struct PhysT {
    R Cmu, Cmt, Ct, Cmp, DeltaT, a12pera11;
    R a10, a11, a12, a13, a14, a15;
    R b10, b11, b12, b13, b14, b15;
    R c10, c11, c12, c13, c14, c15;
    R d10, d11, d12, d13, d14, d15;
    R KPP0, Rho0, Cp0, Mu0;
    R Tup, Tbt, Uup, Ubt, Vup, Vbt, Wup, Wbt;
    R MaxCFL, dtMax;
    R L1, L2, L3;
    R cK;                       // c10 / KPP0
    R cRC;                      // Rho0 * Cp0 / (a10 * b10)
    R k2, k3, k4, k5;           // 2 c12, 3 c13, 4 c14, 5 c15 (dKPP in Horner form)
    R n0, n1, n2, n3, n4, n5;   // d(invRhoCp)/dT numerator collected in powers of DeltaT*T
};
using Phys = PhysT<double>;

template <class R>
inline PhysT<R> phys_cast(const Phys &p)
{
    static_assert(sizeof(Phys) % sizeof(double) == 0, "Phys holds doubles only");
    PhysT<R> q;
    const double *src = reinterpret_cast<const double *>(&p);
    R *dst = reinterpret_cast<R *>(&q);
    for (size_t i = 0; i < sizeof(Phys) / sizeof(double); i++) dst[i] = (R)src[i];
    return q;
}

// Device scalar block (one per case, FP64 in both forms).  dt is read by
// every kernel so the step needs no host synchronisation and can be replayed
// as a CUDA graph.
enum : int {
    S_DT = 0, S_TIME, S_CFL, S_MAXDIV, S_NUBOT, S_NUTOP, S_KE, S_BLOWUP, S_AVER,
    S_STEP, S_FIXED_DT, S_NSCAL
};
// Device doubles past the public scalars: S_OOB, in a build with
// -DTCS_BOUNDS_CHECK, the number of out-of-range indices the kernels met
// (each one recorded here and its access redirected to a valid cell instead of
// made; the stand-in for a memory checker; 0 in the normal build); S_TIMEOUT,
// the number of blocks whose bounded wait on an asynchronous copy ran out (a
// kernel that records one also sets S_BLOWUP, so that the rest of the step is
// skipped, and the host reports TCS_ERR_CUDA, not a blow-up); S_CTR,
// the count of diagnostics blocks done (an unsigned in the double's place); S_ROWS,
// in the bounds-check build, the number of rows the line sweeps have checked.
enum : int { S_TIMEOUT = S_NSCAL, S_OOB, S_CTR, S_ROWS, S_NALLOC };   // S_TIMEOUT next to the public ones: one copy restores them

#if defined(TCS_BOUNDS_CHECK) && defined(__CUDA_ARCH__)
#define TCS_OOB(scal, bad, fix)                          \
    do {                                                 \
        if (bad) { atomicAdd((scal) + S_OOB, 1.0); fix; } \
    } while (0)
// one row of a line sweep, reached by stepping an offset or a pointer
#define TCS_ROW(scal, bad, fix)                          \
    do {                                                 \
        atomicAdd((scal) + S_ROWS, 1.0);                 \
        TCS_OOB(scal, bad, fix);                         \
    } while (0)
#else
#define TCS_OOB(scal, bad, fix) do { } while (0)
#define TCS_ROW(scal, bad, fix) do { } while (0)
#endif

template <class R>
struct GridT {
    int N1, N2, N3;             // interior cells
    int P1, P2;                 // padded strides: P1 = N1+2, P2 = N2+2
    long long NP;               // padded element count
    MetricT<R> m1, m2, m3;      // metrics in the field type
    MetricT<double> d1, d2, d3; // FP64 metrics (the FP64 parts of the mixed form)
    PhysT<R> ph;                // constants in the field type
    Phys phd;                   // FP64 constants
    double *scal;               // device scalars (S_*)
    int kdeg2;                  // KPP has no terms above t^2 (c13 = c14 = c15 = 0: water, glycerol, constant)
};
using Grid = GridT<double>;

// complex type of a precision
template <class R> struct CplxOf;
template <> struct CplxOf<double> { using T = double2; };
template <> struct CplxOf<float> { using T = float2; };
template <class R> using cplx_t = typename CplxOf<R>::T;

template <class R>
__host__ __device__ __forceinline__ cplx_t<R> mkc(R x, R y)
{
    cplx_t<R> c;
    c.x = x; c.y = y;
    return c;
}

// Division by a loop-invariant divisor d (1 <= d < 2^31) of x < 2^31 by a
// multiply-high and a shift: m = ceil(2^(32+s) / d) - 2^32 with 2^s >= d
// (Granlund and Montgomery, "Division by invariant integers using
// multiplication", PLDI 1994).
struct FastDiv {
    unsigned d, m, s;
    __device__ __forceinline__ unsigned div(unsigned x) const
    {
        return (unsigned)(((unsigned long long)__umulhi(x, m) + x) >> s);
    }
};
inline FastDiv make_fastdiv(unsigned d)
{
    FastDiv f;
    f.d = d; f.s = 0;
    while ((1ull << f.s) < d) f.s++;
    f.m = (unsigned)((((1ull << (32 + f.s)) + d - 1) / d) - (1ull << 32));
    return f;
}

template <class R>
__host__ __device__ __forceinline__ long long ix(const GridT<R> &g, int i, int j, int k)
{
    TCS_OOB(g.scal, (unsigned)i > (unsigned)(g.N1 + 1) || (unsigned)j > (unsigned)(g.N2 + 1) || (unsigned)k > (unsigned)(g.N3 + 1),
            (i = 1, j = 1, k = 1));
    return (long long)i + (long long)g.P1 * ((long long)j + (long long)g.P2 * (long long)k);
}

// 2-D (j,k) tables: Mu and invRho are constant along i (module_solve_momentum.f90:156-171
// assigns whole rows Mu(:,j,k) inside the i loop, leaving f(T(n1sub,j,k))).
template <class R>
__host__ __device__ __forceinline__ int ix2(const GridT<R> &g, int j, int k)
{
    TCS_OOB(g.scal, (unsigned)j > (unsigned)(g.N2 + 1) || (unsigned)k > (unsigned)(g.N3 + 1), (j = 1, k = 1));
    return j + g.P2 * k;
}

// Read-only loads through the non-coherent cache.
template <class V>
__device__ __forceinline__ V ld(const V *p) { return __ldg(p); }

// Store one interior value and its periodic images: the on-device form of
// mpi_subdomain_ghostcell_update (module_mpi_subdomain.f90:758-791) on one
// rank -- x faces, then z faces including the x-ghost columns.
template <class R, class V>
__device__ __forceinline__ void store_periodic(const GridT<R> &g, V *a, int i, int j, int k, V v)
{
    a[ix(g, i, j, k)] = v;
    const int ig = (i == 1) ? g.N1 + 1 : ((i == g.N1) ? 0 : -1);
    const int kg = (k == 1) ? g.N3 + 1 : ((k == g.N3) ? 0 : -1);
    if (ig >= 0) a[ix(g, ig, j, k)] = v;
    if (kg >= 0) {
        a[ix(g, i, j, kg)] = v;
        if (ig >= 0) a[ix(g, ig, j, kg)] = v;
    }
}

// ---------------------------------------------------------------------------
// Temperature-dependent properties: mpi_thermal_coeffi
// (module_solve_thermal.f90:129-154), evaluated at the point where the
// stencil needs them instead of being stored.
// ---------------------------------------------------------------------------
// Horner forms of KPP = c10 (1 + c11 t + ... + c15 t^5) / KPP0 and its
// derivative.  With d2 (c13 = c14 = c15 = 0) the zero leading terms are
// skipped; in Horner form they only add exact zeros, so the values are the same.
template <class R>
__device__ __forceinline__ void kpp_eval(const PhysT<R> &p, bool d2, R T, R &kpp, R &dkpp)
{
    const R t = p.DeltaT * T;
    if (d2) {
        kpp = p.cK * (R(1) + t * (p.c11 + t * p.c12));
        dkpp = p.cK * (p.c11 + t * p.k2);
    } else {
        kpp = p.cK * (R(1) + t * (p.c11 + t * (p.c12 + t * (p.c13 + t * (p.c14 + t * p.c15)))));
        dkpp = p.cK * (p.c11 + t * (p.k2 + t * (p.k3 + t * (p.k4 + t * p.k5))));
    }
}

template <class R>
__device__ __forceinline__ R kpp_only(const PhysT<R> &p, bool d2, R T)
{
    const R t = p.DeltaT * T;
    if (d2) return p.cK * (R(1) + t * (p.c11 + t * p.c12));
    return p.cK * (R(1) + t * (p.c11 + t * (p.c12 + t * (p.c13 + t * (p.c14 + t * p.c15)))));
}

// invRhoCp = Rho0 Cp0 / (a10 (1 + A)) / (b10 (1 + B)) and its T-derivative
// share one reciprocal of q1 q2 = (1 + A)(1 + B): every property set of
// module_global.f90 has a14 = a15 = b14 = b15 = 0, so 1 + A is the q1 of
// module_solve_thermal.f90:149.  The derivative's numerator (:144-148) is
// collected into a polynomial in t = DeltaT*T with coefficients n0..n5.
template <class R>
__device__ __forceinline__ R qrcp(R b);
template <>
__device__ __forceinline__ double qrcp<double>(double b);

template <class R>
__device__ __forceinline__ void rhocp_eval(const PhysT<R> &p, R T, R &irc, R &dirc)
{
    const R t = p.DeltaT * T;
    const R q1 = R(1) + t * (p.a11 + t * (p.a12 + t * p.a13));
    const R q2 = R(1) + t * (p.b11 + t * (p.b12 + t * p.b13));
    const R rq = qrcp(q1 * q2);
    irc = p.cRC * rq;
    dirc = -(p.n0 + t * (p.n1 + t * (p.n2 + t * (p.n3 + t * (p.n4 + t * p.n5))))) * (rq * rq);
}

// Reciprocals of the line solver.  FP64: the hardware's approximate
// reciprocal refined by two Newton-Raphson steps y <- y + y (1 - b y), the
// classical iteration (P. Markstein, "Computation of elementary functions on
// the IBM RISC System/6000 processor", IBM J. Res. Develop. 34(1), 1990):
// each step squares the relative error, so the result is within about one ulp
// of the correctly rounded 1/b for |b| from 2^-1022 to 2^1022 (tcs_check_reciprocal
// measures it against the correctly rounded quotient).  For a zero, subnormal or
// infinite b it gives NaN where a division gives infinity or 0: a sweep's row with an
// infinite diagonal has an infinite off-diagonal entry too (the diagonal is 1 minus
// their sum, or sums the same terms), so its elimination is NaN with either.  A test
// for these b costs 2 to 3% of a step (256^3 FP64 2.2%, 400 x 200 x 384 mixed 2.6%).  It takes a handful of
// instructions where the correctly rounded quotient takes a few tens.  FP32:
// the approximate FP32 reciprocal refined by one Newton-Raphson step.
template <class R>
__device__ __forceinline__ R qrcp(R b) { return R(1) / b; }
template <>
__device__ __forceinline__ float qrcp<float>(float b)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(b));
    return fmaf(y, fmaf(-b, y, 1.0f), y);
}
template <>
__device__ __forceinline__ double qrcp<double>(double b)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    double e = fma(-b, y, 1.0);
    y = fma(y, e, y);
    e = fma(-b, y, 1.0);
    return fma(y, e, y);
}

} // namespace tcs
