// tcs_fields.cuh -- the device-resident state of one case and the small
// helpers the stage kernels share.
#pragma once

#include "tcs_device.cuh"

namespace tcs {

template <class R>
struct FieldsT {
    // persistent fields (padded, i fastest)
    R *T, *U, *V, *W, *P, *dPhat, *dP0;
    // second buffers of the fields that a kernel rewrites while other threads
    // still read the old values (T in the thermal y sweep, U/V/W in the fused
    // pseudo-update, dPhat/dP0 in the projection)
    R *Tn, *Un, *Vn, *Wn, *dPhatn, *dP0n;
    // FP32 form only: low words of the velocity (U = U + Ulo to FP64 accuracy)
    // and of its second buffers.  The stencils read the FP32 high word; the
    // pressure right-hand side, the projection and the diagnostics read both,
    // so the storage rounding of the velocity never reaches the divergence.
    R *Ulo, *Vlo, *Wlo, *Unlo, *Vnlo, *Wnlo;
    // per-step increments and pressure correction
    R *dU, *dV, *dW, *dP;
    // interior stage scratch (padded layout)
    R *scr;
    // the pressure right-hand side of the split form (FP64, padded layout): the
    // FP64 form's scr, the FP32 form's FP64 staging array; null where the split
    // form does not run
    double *prhs;
    // 2-D (j,k) property tables: Mu of mpi_momentum_coeffi in the field type, invRho
    // in FP64 in both forms (the sweeps read both from the face tables below).  invRho differs from 1 by about 1e-3 for water, and
    // the pressure right-hand side and the projection use 1 - invRho: from an
    // FP32 table those terms carried 6e-5 relative error, which left P 2-3e-5
    // off the FP64 form after 5-8 steps of the 256^3 and 512^3 water cases
    // (3-8e-6 with the FP64 table).
    R *Mu2;
    double *iR2d;
    // the same properties with their face averages, four words per (j,k) entry
    // (momentum_coeffi): Mu, Mu_y, Mu_z, Mu_yz and invRho, invRho_y, invRho_z, 0
    R *MuT, *iRT;
    double *iRTd;            // the invRho words in FP64 (the same array in the FP64 form)
    // Poisson spectral work array: (h1p, N2, N3) complex, kx fastest
    cplx_t<R> *S;
    // modified wavenumbers and y coefficients of the modal solves (FP64 in both forms)
    const double *dxk2, *dzk, *fam, *fap;
    // FFT twiddles exp(-2 pi i e / n) for n = N1 and n = N3 (FFT arithmetic is FP64 in both forms)
    const double2 *tw1, *tw3;
    // reduction scratch
    double *part;
    double *hist;            // per-step diagnostics history (7 doubles per step)
    int hist_cap;
};

// Skip all work once the divergence check has flagged a blow-up, so the
// fields stay at the state of the step that blew up (main.f90:208-212).
template <class R>
__device__ __forceinline__ bool blown(const GridT<R> &g) { return g.scal[S_BLOWUP] != 0.0; }

// The FP32 form keeps low words of the velocity.
template <class R> struct HasLo { static constexpr bool on = std::is_same<R, float>::value; };

// Two adjacent words of a table (16-byte aligned in FP64, 8-byte in FP32).
__device__ __forceinline__ double2 ld2(const double *p) { return __ldg(reinterpret_cast<const double2 *>(p)); }
__device__ __forceinline__ float2 ld2(const float *p) { return __ldg(reinterpret_cast<const float2 *>(p)); }

// The line sweeps step offsets and pointers from row to row.  In the bounds-check
// build every row is looked at as it is reached (elsewhere nothing happens).
// The cell at offset c of a padded field is interior: its stencil stays inside the
// padding.
template <class R>
__device__ __forceinline__ void row_cell(const GridT<R> &g, long long &c)
{
    TCS_ROW(g.scal, c < 0 || c >= g.NP || (unsigned)(c % g.P1 - 1) >= (unsigned)g.N1 || (unsigned)(c / g.P1 % g.P2 - 1) >= (unsigned)g.N2 ||
            (unsigned)(c / g.P1 / g.P2 - 1) >= (unsigned)g.N3, c = ix(g, 1, 1, 1));
}
// ... and word t4 of the face tables starts the entry of that cell's (j, k).
template <class R>
__device__ __forceinline__ void row_cell(const GridT<R> &g, long long &c, int &t4)
{
    row_cell(g, c);
    TCS_OOB(g.scal, t4 != 4 * (int)(c / g.P1), t4 = 4 * (int)(c / g.P1));
}
// p points at an interior cell of the padded field a.
template <class R, class V>
__device__ __forceinline__ void row_ptr(const GridT<R> &g, V *a, V *&p)
{
#if defined(TCS_BOUNDS_CHECK) && defined(__CUDA_ARCH__)
    long long c = p - a;
    row_cell(g, c);
    p = a + c;
#endif
}

// Weights of the wall extrapolations (Pbc_a and Pbc_b of the lower and upper wall).
struct WallRows { double ab, bb, at, bt; };

// dP wall extrapolation (module_solve_pressure.f90:719-736) on every (i,k)
// including ghost columns, which is what the extrapolation followed by
// ghost(dP) produces.
template <class R>
__device__ __forceinline__ void dp_wall_cell(const GridT<R> &g, R *dP, int i, int k, const WallRows &w)
{
    dP[ix(g, i, 0, k)] = R(w.ab * (double)dP[ix(g, i, 1, k)] - w.bb * (double)dP[ix(g, i, 2, k)]);
    dP[ix(g, i, g.N2 + 1, k)] = R(w.at * (double)dP[ix(g, i, g.N2, k)] - w.bt * (double)dP[ix(g, i, g.N2 - 1, k)]);
}
// P(i,0,k) = Pbc_a P(i,1,k) - Pbc_b P(i,2,k) and the top-wall counterpart
// (:853-869), then ghost(P).
template <class R>
__device__ __forceinline__ void p_wall_cell(const GridT<R> &g, R *P, int i, int k, const WallRows &w)
{
    store_periodic(g, P, i, 0, k, R(w.ab * (double)P[ix(g, i, 1, k)] - w.bb * (double)P[ix(g, i, 2, k)]));
    store_periodic(g, P, i, g.N2 + 1, k, R(w.at * (double)P[ix(g, i, g.N2, k)] - w.bt * (double)P[ix(g, i, g.N2 - 1, k)]));
}

// v = hi + lo in FP64, and its split back into an FP32 pair.
__device__ __forceinline__ double join(float hi, float lo) { return (double)hi + (double)lo; }
__device__ __forceinline__ void split(double v, float &hi, float &lo)
{
    hi = (float)v;
    lo = (float)(v - (double)hi);
}

} // namespace tcs
