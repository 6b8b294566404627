// tcs_march.cuh -- the strided line sweeps (lines along z or y, i fastest in
// memory): a marching, segmented tridiagonal solver.
//
// A block owns TI consecutive i (one line each) and cuts every line into NS
// segments; thread (line l, segment s) marches along its segment row by row.
// It keeps what the next row's stencil shares with this one in registers (the
// problem's March object: the values and fluxes of the face between two rows are
// loaded and computed once), eliminates the row as soon as it is built, and
// parks the eliminated row in shared memory:
//
//     x_r + c_r x_{r+1} + e_r X_{s-1} = d_r
//
// where X_{s-1} is the last unknown of the segment before it.  The last rows of
// the segments form a (cyclic) tridiagonal system in the X_s, closed by the
// first unknown of each segment as a combination of X_{s-1} and X_s (sd, se, p,
// accumulated on the way down); it is solved by parallel cyclic reduction
// across the lanes, one line per group of NS lanes.  Each thread then
// substitutes back through its rows and emits them.  It is the partitioned
// solve of pascal_tdma.f90:487-578 with one partition per thread.
//
// Elimination, rows and solution are FP64 in both numerical forms; the
// FP32-mixed form builds its rows in FP32 and rounds the solution once.
//
// What it bought (ms, from sweeps that built every row apart and solved in a
// separate phase): dw_z at 256^3 0.51 -> 0.36, FP32-mixed 0.44 -> 0.30; at 180 x
// 151 x 250 0.23 -> 0.17; at 512^3 (column form) 5.94 -> 3.07; du_y at 256^3
// FP32-mixed 0.26 -> 0.17.  What bounds it now: load latency at the 16 warps per
// SM that 128 registers allow (long-scoreboard stalls 4 to 5 per issue, issue
// slots 40% busy, FP64 pipe 25 to 33%, DRAM 20 to 32%).
#pragma once

#include "tcs_fields.cuh"
#include "tcs_tma.cuh"

namespace tcs {

struct MarchPlan {
    int n;        // rows per line
    int lgNS;     // log2 of the segments per line
    int lgTI;     // log2 of the lines per block
    int m0, rem;  // segment s has m0 + (s < rem) rows
    int cyclic;
};

__host__ __device__ __forceinline__ size_t march_words(int n, int NS, int TI, int nrhs)
{
    // eliminated rows c, e, d[nrhs] of every line, then the reduced systems (padded lines)
    return (size_t)n * TI * (2 + nrhs) + (size_t)(4 + 2 * nrhs) * NS * (TI + 1);
}

// The reduced systems of a block: words e, c, se, p, d[NR], sd[NR] of the last
// row of segment s of line L at q NS TP + s TP + L of red, NS a power of two, NS
// lines = the block's threads.  Parallel cyclic reduction, one row per thread:
// across the lanes of a group of NS (row t mod NS of line t / NS in thread t),
// or, for more than 32 segments, through shared memory (row t / lines of line
// t mod lines).  Leaves X in words 0 .. NR-1.  Ends with a barrier; the caller
// has put one before it.
template <int NR>
__device__ void march_reduce_wide(double *red, int lgNS, int TP, bool cyc)
{
    const int NS = 1 << lgNS, RS = NS * TP, TI = TP - 1;
    const int g = threadIdx.x / TI, L = threadIdx.x - g * TI;
    double *const own = red + g * TP + L;
    const double *const nxt = red + ((g + 1) & (NS - 1)) * TP + L;
    const double cp = (cyc || g < NS - 1) ? own[RS] : 0.0;
    double al = own[0], be = 1.0, ga = 0.0, de[NR];
#pragma unroll
    for (int q = 0; q < NR; q++) de[q] = own[(4 + q) * RS];
    if (cyc || g < NS - 1) {
        be = 1.0 - cp * nxt[2 * RS];
        ga = cp * nxt[3 * RS];
#pragma unroll
        for (int q = 0; q < NR; q++) de[q] -= cp * nxt[(4 + NR + q) * RS];
    }
    for (int h = 1; h < NS; h <<= 1) {
        __syncthreads();                           // the words of the step before have been read
        own[0] = al; own[RS] = qrcp(be); own[2 * RS] = ga;
#pragma unroll
        for (int q = 0; q < NR; q++) own[(3 + q) * RS] = de[q];
        __syncthreads();
        const bool lok = cyc || g >= h, hok = cyc || g + h < NS;
        const double *const lo = red + ((g - h) & (NS - 1)) * TP + L, *const hi = red + ((g + h) & (NS - 1)) * TP + L;
        const double k1 = lok ? al * lo[RS] : 0.0, k2 = hok ? ga * hi[RS] : 0.0;
#pragma unroll
        for (int q = 0; q < NR; q++) {
            if (lok) de[q] = fma(-k1, lo[(3 + q) * RS], de[q]);
            if (hok) de[q] = fma(-k2, hi[(3 + q) * RS], de[q]);
        }
        if (lok) be = fma(-k1, lo[2 * RS], be);
        if (hok) be = fma(-k2, hi[0], be);
        al = lok ? -k1 * lo[0] : 0.0;
        ga = hok ? -k2 * hi[2 * RS] : 0.0;
    }
    const double den = qrcp(al + be + ga);
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NR; q++) own[q * RS] = de[q] * den;
    __syncthreads();
}

template <int NR>
__device__ __forceinline__ void march_reduce(double *red, int lgNS, int TP, bool cyc)
{
    if (lgNS > 5) {
        march_reduce_wide<NR>(red, lgNS, TP, cyc);
        return;
    }
    const int NS = 1 << lgNS, RS = NS * TP;
    const int g = threadIdx.x & (NS - 1), L = threadIdx.x >> lgNS;
    const int gn = (g + 1) & (NS - 1);
    const double *const own = red + g * TP + L, *const nxt = red + gn * TP + L;
    const double cp = own[RS];
    double al = own[0], be = 1.0 - cp * nxt[2 * RS], ga = cp * nxt[3 * RS], de[NR];
#pragma unroll
    for (int q = 0; q < NR; q++) de[q] = own[(4 + q) * RS] - cp * nxt[(4 + NR + q) * RS];
    if (!cyc && g == NS - 1) {
        be = 1.0; ga = 0.0;
#pragma unroll
        for (int q = 0; q < NR; q++) de[q] = own[(4 + q) * RS];
    }
    for (int h = 1; h < NS; h <<= 1) {
        const int lo = (g - h) & (NS - 1), hi = (g + h) & (NS - 1);
        const bool lok = cyc || g >= h, hok = cyc || g + h < NS;
        const double rb = qrcp(be);
        const double alm = __shfl_sync(0xffffffffu, al, lo, NS), gam = __shfl_sync(0xffffffffu, ga, lo, NS);
        const double alp = __shfl_sync(0xffffffffu, al, hi, NS), gap = __shfl_sync(0xffffffffu, ga, hi, NS);
        const double rbm = __shfl_sync(0xffffffffu, rb, lo, NS), rbp = __shfl_sync(0xffffffffu, rb, hi, NS);
        const double k1 = lok ? al * rbm : 0.0, k2 = hok ? ga * rbp : 0.0;
#pragma unroll
        for (int q = 0; q < NR; q++) {
            const double dm = __shfl_sync(0xffffffffu, de[q], lo, NS), dq = __shfl_sync(0xffffffffu, de[q], hi, NS);
            if (lok) de[q] = fma(-k1, dm, de[q]);
            if (hok) de[q] = fma(-k2, dq, de[q]);
        }
        if (lok) be = fma(-k1, gam, be);
        if (hok) be = fma(-k2, alp, be);
        al = lok ? -k1 * alm : 0.0;
        ga = hok ? -k2 * gap : 0.0;
    }
    const double den = qrcp(al + be + ga);
    __syncthreads();                               // every lane has read its rows: X takes the place of the first words
#pragma unroll
    for (int q = 0; q < NR; q++) red[q * RS + g * TP + L] = de[q] * den;
    __syncthreads();
}

// Problems that want the sum of line 0's solution in the first block row
// (Out::total, set_total).
template <class P, class = void>
struct HasTotal { static constexpr bool on = false; };
template <class P>
struct HasTotal<P, std::void_t<decltype(P::TOTAL)>> { static constexpr bool on = true; };

// Stores of a line's rows from the last to the first: into the sweep scratch, ...
template <class R>
struct ScratchOut {
    R *p;
    long long step;
    __device__ __forceinline__ ScratchOut(const GridT<R> &g, R *a, int i, int j, int k, long long st) : p(a + ix(g, i, j, k)), step(st) {}
    __device__ __forceinline__ void put(const GridT<R> &g, R *a, R v)
    {
        row_ptr(g, a, p);
        *p = v;
        p -= step;
    }
};
// ... or into a field with its periodic images, along y (see store_periodic).
template <class R>
struct PeriodicOut {
    R *p;
    long long gi, gk, step;      // offsets of the x and z images, 0: none
    __device__ __forceinline__ PeriodicOut(const GridT<R> &g, R *a, int i, int j, int k)
        : p(a + ix(g, i, j, k)), gi(i == 1 ? g.N1 : (i == g.N1 ? -g.N1 : 0)),
          gk((long long)g.P1 * g.P2 * (k == 1 ? g.N3 : (k == g.N3 ? -g.N3 : 0))), step(g.P1) {}
    __device__ __forceinline__ void put(const GridT<R> &g, R *a, R v)
    {
        row_ptr(g, a, p);
        *p = v;
        if (gi) p[gi] = v;
        if (gk) {
            p[gk] = v;
            if (gi) p[gi + gk] = v;
        }
        p -= step;
    }
};

// The problem supplies
//   static constexpr int NRHS, AHEAD (rows whose inputs are loaded ahead), ROWS, LGTI (most rows per segment, most lines per block), TPS
//   static constexpr bool LONG64 (long lines in 64 segments, march_plan)
//   skip(), lines() (count of lines along i of the block row)
//   struct March { March(const Prob &, int line, int by, int r0);               // line: clamped to a valid one
//                  struct In;  void load(const Prob &, int r, In &);             // the inputs of row r, rows in order from r0
//                  void row(const Prob &, int r, const In &, double &a, double &b, double &c, double d[NRHS]); }
//   struct Out { Out(const Prob &, int line, int by, int r);  void put(const Prob &, const double x[NRHS]); }   // row r, then r - 1, ...
template <class Prob>
__device__ __forceinline__ void march_block(const Prob &prob, const MarchPlan &mp, int bx, int by)
{
    constexpr int NR = Prob::NRHS, W = 2 + NR;
    extern __shared__ __align__(16) double msm[];
    const bool skip = prob.skip();   // tested before the stores: its load does not delay the others
    const int TI = 1 << mp.lgTI, NS = 1 << mp.lgNS, TP = TI + 1;
    const int l = threadIdx.x & (TI - 1), s = threadIdx.x >> mp.lgTI;
    const int line = (bx << mp.lgTI) + l, nl = prob.lines();
    const int m = mp.m0 + (s < mp.rem ? 1 : 0), r0 = s * mp.m0 + min(s, mp.rem);
    double *const row0 = msm + (size_t)r0 * W * TI + l;
    double *const red = msm + (size_t)mp.n * W * TI;   // e, c, d[NR], se, p, sd[NR] of the last rows: word q of (s, l) at q NS TP + s TP + l
    const int RS = NS * TP;
    TCS_OOB(prob.g.scal, blockDim.x != NS * TI || mp.m0 < 1 || NS * mp.m0 + mp.rem != mp.n, return);   // the same for the whole block
    {
        typename Prob::March st(prob, min(line, nl - 1), by, r0);
        double cp = 0.0, e = -1.0, p = 1.0, se = 0.0, dp[NR], sd[NR];
#pragma unroll
        for (int q = 0; q < NR; q++) { dp[q] = 0.0; sd[q] = 0.0; }
        double *w = row0;
        auto eliminate = [&](int r, const typename Prob::March::In &in) {
            double a, b, c, d[NR];
            st.row(prob, r, in, a, b, c, d);
            const double rr = qrcp(fma(-a, cp, b));
            e = -(a * rr) * e;
#pragma unroll
            for (int q = 0; q < NR; q++) dp[q] = fma(-a, dp[q], d[q]) * rr;
            cp = c * rr;
            if (!mp.cyclic) {                          // no unknown before the first row, none after the last
                if (r == 0) e = 0.0;
                if (r == mp.n - 1) cp = 0.0;
            }
        };
        auto park = [&]() {
            TCS_OOB(prob.g.scal, w < msm || w + (W - 1) * TI >= msm + (size_t)mp.n * W * TI, w = row0);
            w[0] = cp; w[TI] = e;
#pragma unroll
            for (int q = 0; q < NR; q++) { w[(2 + q) * TI] = dp[q]; sd[q] = fma(p, dp[q], sd[q]); }
            se = fma(p, e, se);
            p = -p * cp;
            w += W * TI;
        };
        // AHEAD rows of inputs are on their way while a row is worked on (0: it waits for its own)
        constexpr int D = Prob::AHEAD, NB = D + 1;
        const int last = r0 + m - 1;
        typename Prob::March::In in[NB];
#pragma unroll
        for (int q = 0; q < (D ? D : 1); q++)
            if (r0 + q <= last) st.load(prob, r0 + q, in[q]);
        if constexpr (D == 0) {
            int r = r0;
            while (r < last) {
                eliminate(r, in[0]);
                park();
                st.load(prob, ++r, in[0]);
            }
            eliminate(last, in[0]);
        } else {
            for (int r = r0; r <= last; r += NB) {
#pragma unroll
                for (int q = 0; q < NB; q++) {
                    if (r + q > last) break;
                    if (r + q + D <= last) st.load(prob, r + q + D, in[(q + D) % NB]);
                    eliminate(r + q, in[q]);
                    if (r + q < last) park();
                }
            }
        }
        double *const o = red + s * TP + l;
        o[0] = e; o[RS] = cp; o[2 * RS] = se; o[3 * RS] = p;
#pragma unroll
        for (int q = 0; q < NR; q++) { o[(4 + q) * RS] = dp[q]; o[(4 + NR + q) * RS] = sd[q]; }
    }
    __syncthreads();
    march_reduce<NR>(red, mp.lgNS, TP, mp.cyclic != 0);
    if (line < nl && !skip) {
        double x[NR], xp[NR];
        const int sp = (s - 1) & (NS - 1);
#pragma unroll
        for (int q = 0; q < NR; q++) { x[q] = red[q * RS + s * TP + l]; xp[q] = red[q * RS + sp * TP + l]; }
        typename Prob::Out out(prob, line, by, r0 + m - 1);
        out.put(prob, x);
        const double *w = row0 + (m - 2) * W * TI;
        int left = m - 1;
        constexpr int B = 4;                           // parked rows read ahead of the substitution
        for (; left >= B; left -= B, w -= B * W * TI) {
            TCS_OOB(prob.g.scal, w - (B - 1) * W * TI < msm || w + (W - 1) * TI >= msm + (size_t)mp.n * W * TI, break);
            double c[B], y[B][NR];
#pragma unroll
            for (int t = 0; t < B; t++) {
                c[t] = w[-t * W * TI];
                const double e = w[-t * W * TI + TI];
#pragma unroll
                for (int q = 0; q < NR; q++) y[t][q] = fma(-e, xp[q], w[-t * W * TI + (2 + q) * TI]);
            }
#pragma unroll
            for (int t = 0; t < B; t++) {
#pragma unroll
                for (int q = 0; q < NR; q++) x[q] = fma(-c[t], x[q], y[t][q]);
                out.put(prob, x);
            }
        }
        for (; left > 0; left--, w -= W * TI) {
            TCS_OOB(prob.g.scal, w < msm || w + (W - 1) * TI >= msm + (size_t)mp.n * W * TI, break);
            const double c = w[0], e = w[TI];
#pragma unroll
            for (int q = 0; q < NR; q++) x[q] = fma(-c, x[q], fma(-e, xp[q], w[(2 + q) * TI]));
            out.put(prob, x);
        }
        if constexpr (HasTotal<Prob>::on)
            if (bx == 0 && by == 0 && l == 0) msm[r0 * W * TI] = out.total;   // over a row that this thread has used
    }
    if constexpr (HasTotal<Prob>::on) {
        // the total of line 0 of the first block row, segment by segment
        if (bx == 0 && by == 0 && !skip) {
            __syncthreads();
            if (threadIdx.x == 0) {
                double t = 0.0;
                for (int q = 0; q < NS; q++) t += msm[(q * mp.m0 + min(q, mp.rem)) * W * TI];
                prob.set_total(t);
            }
        }
    }
}

// NT: the most threads per block; Prob::TPS threads per SM.
template <class Prob, int NT>
__global__ void __launch_bounds__(NT, Prob::TPS / NT) march_kernel(const __grid_constant__ Prob prob, MarchPlan mp)
{
    march_block(prob, mp, blockIdx.x, blockIdx.y);
}

// ---------------------------------------------------------------------------
// The x sweeps (lines contiguous in memory): the same march over lines held in
// shared memory.  A block stages the inputs of TI lines (consecutive j at one k)
// word plane by word plane, a warp per line with consecutive i in consecutive
// lanes; thread (line l, segment s) marches over its rows there, parks d, c and e
// in the places of the words it has used (planes 0, 1, 2), and the solution
// leaves plane 0 as it came, a warp per line.  The line stride is odd, so the
// TI lines of a warp's march sit on distinct banks.  Two blocks per SM: one
// stages while the other marches.  Against the lane-per-partition solver that was
// here before (du_x, ps per cell, before and now): FP64 256 cells along x 19.6 and
// 15.7, 400 14.2 and 13.1, 512 12.7 and 12.2, but slower from 540 on, where fewer lines
// fit a block (540 13.6 and 14.9, 1024 16.7 and 19.4, 4096 37.2 and 51.2); FP32-mixed
// faster at every length (256 23.8 and 14.3, 540 18.5 and 13.2, 4096 91.7 and 45.6).
// It moves 3 or 4 arrays at 2.5 to 2.7 TB/s: latency at 16 warps per SM bounds it.
// The problem supplies
//   static constexpr int WORDS;                                             // planes staged: 0 the right-hand side, 1.. the stencil
//   struct Stage { Stage(const Prob &, int line, int by);  void put(const Prob &, int r, double *w, int PL); }   // row r of the line, words PL apart
//   struct March { March(const Prob &, int line, int by, int r0, int m, int n, const double *w, int PL);  // reads across segment edges
//                  void row(const Prob &, int r, bool last, const double *w, int PL, double &a, double &b, double &c, double &d); }
//   lines(), out(line, by)                                                   // the row of the sweep scratch (i = 1)
// ---------------------------------------------------------------------------
__host__ __device__ __forceinline__ int xmarch_stride(int n) { return n | 1; }
__host__ __device__ __forceinline__ size_t xmarch_words(int n, int NS, int TI, int words)
{
    return (size_t)words * TI * xmarch_stride(n) + (size_t)6 * NS * (TI + 1);
}

template <class Prob>
__global__ void __launch_bounds__(256, 2) xmarch_kernel(const __grid_constant__ Prob prob, MarchPlan mp)
{
    using R = typename Prob::Real;
    extern __shared__ __align__(16) double xsm[];
    const bool skip = prob.skip();
    const int n = mp.n, TI = 1 << mp.lgTI, NS = 1 << mp.lgNS, TP = TI + 1, LS = xmarch_stride(n), PL = TI * LS;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5, by = blockIdx.y;
    const int line0 = blockIdx.x << mp.lgTI, nl = prob.lines();
    double *const red = xsm + (size_t)Prob::WORDS * PL;
    const int RS = NS * TP;
    // a warp per line, or, with fewer lines than warps, nw / TI warps side by side on one
    const int share = nw > TI ? nw >> mp.lgTI : 1;
    auto stage = [&](int l, int first, int step) {
        const typename Prob::Stage st(prob, min(line0 + l, nl - 1), by);
        double *const w = xsm + l * LS;
#pragma unroll Prob::UNROLL
        for (int r = first; r < n; r += step) {
            TCS_ROW(prob.g.scal, r < 0 || l < 0 || l >= TI, break);
            st.put(prob, r, w + r, PL);
        }
    };
    if (share == 1)
        for (int l = warp; l < TI; l += nw) stage(l, lane, 32);
    else
        stage(warp / share, lane + 32 * (warp % share), 32 * share);
    __syncthreads();
    const int l = threadIdx.x & (TI - 1), s = threadIdx.x >> mp.lgTI;
    const int m = mp.m0 + (s < mp.rem ? 1 : 0), r0 = s * mp.m0 + min(s, mp.rem);
    double *const w = xsm + l * LS;
    TCS_OOB(prob.g.scal, blockDim.x != NS * TI || mp.m0 < 1 || NS * mp.m0 + mp.rem != n, return);   // the same for the whole block
    {
        typename Prob::March st(prob, min(line0 + l, nl - 1), by, r0, m, n, w, PL);
        __syncthreads();                               // the words across segment edges have been read
        double cp = 0.0, e = -1.0, p = 1.0, se = 0.0, dp = 0.0, sd = 0.0;
        const int last = r0 + m - 1;
        for (int r = r0; r <= last; r++) {
            double a, b, c, d;
            st.row(prob, r, r == last, w, PL, a, b, c, d);
            const double rr = qrcp(fma(-a, cp, b));
            e = -(a * rr) * e;
            dp = fma(-a, dp, d) * rr;
            cp = c * rr;
            TCS_OOB(prob.g.scal, r < 0 || r >= n, break);
            if (r < last) {
                w[r] = dp; w[PL + r] = cp; w[2 * PL + r] = e;
                sd = fma(p, dp, sd);
                se = fma(p, e, se);
                p = -p * cp;
            }
        }
        double *const o = red + s * TP + l;
        o[0] = e; o[RS] = cp; o[2 * RS] = se; o[3 * RS] = p; o[4 * RS] = dp; o[5 * RS] = sd;
    }
    __syncthreads();
    march_reduce<1>(red, mp.lgNS, TP, true);
    {
        double x = red[s * TP + l];
        const double xp = red[((s - 1) & (NS - 1)) * TP + l];
        int r = r0 + m - 1;
        w[r] = x;
        for (r--; r - 3 >= r0; r -= 4) {
            TCS_OOB(prob.g.scal, r >= n || r - 3 < 0, break);
            double c[4], y[4];
#pragma unroll
            for (int t = 0; t < 4; t++) { c[t] = w[PL + r - t]; y[t] = fma(-w[2 * PL + r - t], xp, w[r - t]); }
#pragma unroll
            for (int t = 0; t < 4; t++) { x = fma(-c[t], x, y[t]); w[r - t] = x; }
        }
        for (; r >= r0; r--) {
            x = fma(-w[PL + r], x, fma(-w[2 * PL + r], xp, w[r]));
            w[r] = x;
        }
    }
    __syncthreads();
    if (skip) return;
    for (int q = warp / share; q < TI && line0 + q < nl; q += nw / share) {
        R *const o = prob.out(line0 + q, by);
        const double *const v = xsm + q * LS;
        for (int r = lane + 32 * (warp % share); r < n; r += 32 * share) {
            TCS_ROW(prob.g.scal, r < 0 || r >= prob.g.N1, break);
            o[r] = R(v[r]);
        }
    }
}

// ---------------------------------------------------------------------------
// The column form (FP64, z lines): a block of w consecutive i marches up NS
// segments of the lines together (w NS threads).  The rows of i that a plane needs
// (the problem's stream: its arrays at j-1, j, j+1) come one bulk copy each into a
// ring of COL_SLOTS planes, up to two (COL_SLOTS - 2) ahead of the one being worked
// on, so no load latency is left on the march; c and d of the eliminated rows go to global scratch
// (consecutive i: coalesced) and the second march substitutes back.  The
// segment's coupling e_r to the unknown before it is not stored: it dies out
// within a few rows of a diagonally dominant line, so the rows up to the last
// one with |e_r| above COL_TINY are built once more (their coefficients alone)
// and d_r -= e_r X is applied to them.
// ---------------------------------------------------------------------------
constexpr int COL_SLOTS = 4;
constexpr double COL_TINY = 7.8886090522101181e-31;   // 2^-100
constexpr int COL_WAIT = 1 << 22;                     // polls of a bounded wait (a block's first: Shapes::copy_polls)

// FP64 problems that name their stream (Prob::NROW): the cyclic z sweeps.
template <class P, class = void>
struct Streams { static constexpr bool on = false; };
template <class P>
struct Streams<P, std::void_t<decltype(P::NROW)>> { static constexpr bool on = std::is_same<typename P::Real, double>::value; };

// Words of one segment's plane: NROW rows of w + 2, then the table words of rows
// j-1, j, j+1 (Mu) and j (iR).
template <class Prob>
__host__ __device__ constexpr int col_slot_words(int w) { return Prob::NROW * (w + 2) + 16; }
template <class Prob>
__host__ __device__ constexpr size_t col_smem(int w, int NS) { return ((size_t)COL_SLOTS * NS * col_slot_words<Prob>(w) + COL_SLOTS) * sizeof(double); }

template <class Prob>
__global__ void __launch_bounds__(128, 4) column_kernel(const __grid_constant__ Prob prob, int n, int w, int lgNS, double *cscr, int cpitch, int polls)
{
    using March = typename Prob::March;
    extern __shared__ __align__(16) double csm[];
    const GridT<double> &g = prob.g;
    const int NS = 1 << lgNS, s = threadIdx.x / w, l = threadIdx.x - s * w, by = blockIdx.y, x0 = w * blockIdx.x;
    const int SW = col_slot_words<Prob>(w) * NS;                     // words of a ring slot
    uint64_t *const bar = reinterpret_cast<uint64_t *>(csm + COL_SLOTS * SW);
    double *const mine = csm + s * col_slot_words<Prob>(w);
    const int nl = prob.lines(), line = x0 + l, sline = min(line, nl - 1);
    const int i = 1 + sline, j = Prob::J0 + by;
    const int m0 = n >> lgNS, rem = n & (NS - 1), m = m0 + (s < rem), r0 = s * m0 + min(s, rem), mmax = m0 + (rem > 0);
    const long long sk = (long long)g.P1 * g.P2;
    const uint32_t rowb = (uint32_t)min(w + 2, g.P1 - x0) * 8u;
    TCS_OOB(g.scal, blockDim.x != NS * w || m0 < 1 || n != g.N3 || cpitch < g.N1 || cpitch > 2 * (g.N1 / 2 + 1), return);   // the same for the whole block
    if (threadIdx.x == 0) {
        for (int q = 0; q < COL_SLOTS; q++) mbar_init(&bar[q], NS);
        mbar_init_fence();
    }
    if (__syncthreads_or(prob.skip())) return;                       // as one block: another block's failed wait may set the flag now
    // one thread of each segment: plane k of the segment's row r (k = r0 + r + 1) into
    // slot (r + 1) mod COL_SLOTS (r = -1: what the first row needs of the plane below)
    auto issue = [&](int r) {
        const int sl = (r + 1) % COL_SLOTS, k = r0 + r + 1;
        if (r >= m) {                                                // a shorter segment has no such row
            mbar_arrive_expect_tx(&bar[sl], 0);
            return;
        }
        double *const dst = mine + sl * SW;
        mbar_arrive_expect_tx(&bar[sl], Prob::NROW * rowb + (Prob::TABLES ? 128u : 0u));
#pragma unroll
        for (int q = 0; q < Prob::NROW; q++) {
            int jq = j + Prob::row_dj(q), kq = k + Prob::row_dk(q);
            TCS_OOB(g.scal, (unsigned)jq > (unsigned)g.N2 + 1u || (unsigned)kq > (unsigned)g.N3 + 1u || (x0 & 1) || x0 < 0 || x0 + (int)(rowb / 8) > g.P1 ||
                    (int)(rowb / 8) > w + 2, jq = kq = 1);
            bulk_load(dst + q * (w + 2), prob.row_src(q) + (x0 + (long long)g.P1 * (jq + (long long)g.P2 * kq)), rowb, &bar[sl]);
        }
        if (Prob::TABLES) {
            double *const t = dst + Prob::NROW * (w + 2);
            int jt = j, kt = k + 1;
            TCS_OOB(g.scal, jt < 1 || jt > g.N2 || kt < 0 || kt > g.N3 + 1, jt = kt = 1);
            bulk_load(t, prob.f.MuT + 4 * (jt - 1 + g.P2 * kt), 96, &bar[sl]);
            bulk_load(t + 12, prob.f.iRT + 4 * (jt + g.P2 * kt), 32, &bar[sl]);
        }
    };
    if (l == 0)
        for (int r = -1; r < COL_SLOTS - 1 && r < mmax; r++) issue(r);
    const long long ck = (long long)cpitch * g.N2;
    double *const sc = cscr + (i - 1) + (long long)cpitch * (j - 1) + r0 * ck;
    double *const sd_ = prob.f.scr + ix(g, i, j, 1 + r0);
    double cp = 0.0, dp = 0.0, e = -1.0, p = 1.0, se = 0.0, sd = 0.0;
    int K = -1;
    {
        March st(prob, sline, by, r0);
        double a, b, c, d;
        int r = 0;
        bool ok = true, got = mbar_wait(&bar[0], 0, polls);   // (one bound for every wait, kept through the march, spilled: dw_z at 512^3 2.98 -> 3.20 ms)
        for (; r < mmax; r++) {
            got = mbar_wait(&bar[(r + 1) % COL_SLOTS], ((r + 1) / COL_SLOTS) & 1, COL_WAIT) && got;
            if (got && r < m) {
                typename March::In in;
                st.fill(prob, r0 + r, in, mine + ((r + 1) % COL_SLOTS) * SW, mine + (r % COL_SLOTS) * SW, w, sline - x0);
                st.row(prob, r0 + r, in, a, b, c, &d);
                const double rr = qrcp(fma(-a, cp, b));
                e = -(a * rr) * e;
                dp = fma(-a, dp, d) * rr;
                cp = c * rr;
                if (r < m - 1) {
                    bool in = line < nl;
                    TCS_ROW(g.scal, r0 + r >= n || i > g.N1 || j > g.N2, in = false);
                    if (in) {
                        sc[r * ck] = cp;
                        sd_[r * sk] = dp;
                    }
                    sd = fma(p, dp, sd);
                    se = fma(p, e, se);
                    p = -p * cp;
                    if (!(fabs(e) <= COL_TINY)) K = r;
                }
            }
            if (__syncthreads_or(!got)) { ok = false; break; }     // every thread is done with the slot below
            if (l == 0 && r + COL_SLOTS - 1 < mmax) {
                fence_proxy_async();
                issue(r + COL_SLOTS - 1);
            }
        }
        if (!ok) {
            // a copy did not arrive in time: record it, stop the step, and wait
            // (bounded) for this block's copies still in flight before leaving: the
            // planes of rows r - 1 (the first row may not have got it) to r + COL_SLOTS - 2
            if (threadIdx.x == 0) {
                atomicAdd(g.scal + S_TIMEOUT, 1.0);
                g.scal[S_BLOWUP] = g.scal[S_STEP] + 1.0;
                for (int q = r; q < r + COL_SLOTS && q <= mmax; q++) mbar_wait(&bar[q % COL_SLOTS], (q / COL_SLOTS) & 1, COL_WAIT);
            }
            __syncthreads();
            return;
        }
    }
    // the ring is idle now: it holds the reduced systems
    const int TP = w + 1, RS = NS * TP;
    double *const o = csm + s * TP + l;
    o[0] = e; o[RS] = cp; o[2 * RS] = se; o[3 * RS] = p; o[4 * RS] = dp; o[5 * RS] = sd;
    __syncthreads();
    march_reduce<1>(csm, lgNS, TP, true);
    const double X = o[0], Xp = csm[((s - 1) & (NS - 1)) * TP + l];
    K = __reduce_max_sync(0xffffffffu, K);
    {
        March st(prob, sline, by, r0);
        double c2 = 0.0, e2 = -1.0, a, b, c, d;
        for (int r = 0; r <= K; r++) {
            typename March::In in;
            st.load(prob, r0 + r, in);
            st.row(prob, r0 + r, in, a, b, c, &d);
            const double rr = qrcp(fma(-a, c2, b));
            e2 = -(a * rr) * e2;
            c2 = c * rr;
            TCS_OOB(g.scal, r >= m - 1, break);
            if (line < nl) sd_[r * sk] = fma(-e2, Xp, sd_[r * sk]);
        }
    }
    if (line >= nl) return;
    double x = X;
    TCS_ROW(g.scal, r0 + m > n || i > g.N1 || j > g.N2, return);
    sd_[(m - 1) * sk] = x;
    int r = m - 2;
    for (; r >= 7; r -= 8) {
        double cc[8], dd[8];
#pragma unroll
        for (int q = 0; q < 8; q++) { cc[q] = sc[(r - q) * ck]; dd[q] = sd_[(r - q) * sk]; }
#pragma unroll
        for (int q = 0; q < 8; q++) {
            x = fma(-cc[q], x, dd[q]);
            sd_[(r - q) * sk] = x;
        }
    }
    for (; r >= 0; r--) {
        x = fma(-sc[r * ck], x, sd_[r * sk]);
        sd_[r * sk] = x;
    }
}

} // namespace tcs
