// tcs_kernels.h -- host-side view of one case (Ctx), kernel identifiers and
// the launch helpers shared by the stage files.
#pragma once

#include "tcs_march.cuh"

#include <cuda_runtime.h>
#include <stdint.h>
#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

namespace tcs {

// The probed kernels, in launch order.  A step launches neither K_PSEUDO (part of the
// right-hand side) nor K_DP_WALL and K_P_WALL (part of K_POST); K_FINAL is launched where
// the diagnostics end in a launch of their own.  K_MEAN (part of K_MODAL) and K_TDMA_API
// have no launch; their ids are kept.
enum KernelId : int {
    K_THERMAL_Z = 0, K_THERMAL_X, K_THERMAL_Y, K_MOM_COEFFI,
    K_DU_Z, K_DU_X, K_DU_Y, K_DV_Z, K_DV_X, K_DV_Y, K_DW_Z, K_DW_X, K_DW_Y,
    K_BLOCKLDV, K_BLOCKLDU, K_PSEUDO, K_PRHS_FFTX, K_FFTZ_FWD, K_MODAL, K_MEAN,
    K_FFTZ_INV, K_IFFTX, K_DP_WALL, K_PROJECT, K_P_WALL, K_POST, K_FINAL, K_TDMA_API,
    K_COUNT
};

const char *kernel_name(int kid);

struct FFTPlan {
    int n, npass;
    int radix[24];
    FastDiv dnb[24], dns[24];   // per pass: n / radix and the span Ns
    FastDiv dn, dh;             // n and n/2 + 1
};

// A block's z-FFT lines in shared memory: element (line l, row q) of NL lines at
// (q + q/8) NL + l -- lines fastest, so that the threads of a warp, which take
// consecutive lines and then consecutive butterflies, touch consecutive
// words; the pad row after every 8 rows spreads the strided writes of a pass
// with span 1 over the banks.
__host__ __device__ __forceinline__ int frow(int q) { return q + (q >> 3); }
__host__ __device__ __forceinline__ size_t fft_buf_elems(int NL, int n) { return (size_t)NL * (size_t)frow(n); }

// The form of a z transform of NL lines per block: 1 the one-radix form (every
// pass of radix 4 or 8, one butterfly per thread: NL n / radix <= 1024 threads,
// one buffer), 2 the general form (256 threads, two buffers), 0 neither fits
// the 227 KB a block may take.
inline size_t fftz_smem(const FFTPlan &fp, int NL, int form) { return (size_t)form * fft_buf_elems(NL, fp.n) * 16; }
inline int fftz_form(const FFTPlan &fp, int NL)
{
    bool uni = fp.npass >= 1 && (fp.radix[0] == 8 || fp.radix[0] == 4);
    for (int p = 1; p < fp.npass; p++) uni = uni && fp.radix[p] == fp.radix[0];
    if (uni && (long long)NL * (fp.n / fp.radix[0]) <= 1024 && fftz_smem(fp, NL, 1) <= 227 * 1024) return 1;
    return fftz_smem(fp, NL, 2) <= 227 * 1024 ? 2 : 0;
}

// The form of the inverse x transform of NL lines per block: 1 the one-radix
// form (fpu of one radix 4 or 8, packed lines x N1 / radix <= 512 threads, one
// line-major buffer), 2 the general form (256 threads, two buffers, the
// radix-4 plan), 0 neither fits.
inline size_t ifftx_smem(const FFTPlan &fpu, int NL, int form)
{
    const size_t nfl = (size_t)((NL + 1) / 2);
    return form == 1 ? nfl * (size_t)frow(fpu.n) * 16 : nfl * (size_t)fpu.n * 2 * 16;
}
inline int ifftx_form(const FFTPlan &fpu, int NL)
{
    bool uni = fpu.npass >= 1 && (fpu.radix[0] == 8 || fpu.radix[0] == 4);
    for (int p = 1; p < fpu.npass; p++) uni = uni && fpu.radix[p] == fpu.radix[0];
    if (uni && (long long)((NL + 1) / 2) * (fpu.n / fpu.radix[0]) <= 512 && ifftx_smem(fpu, NL, 1) <= 227 * 1024) return 1;
    return ifftx_smem(fpu, NL, 2) <= 227 * 1024 ? 2 : 0;
}

struct ProbeState;   // CUDA-event probes (tcs_capi.cu)

// Launch shapes shared by both forms.
struct Shapes {
    int fft_lines_x, fft_lines_z;
    int ifft_lines_x;                            // lines per block of the inverse x transform
    int lanes;                                   // at most this many partitions (lanes) per line
    int tl_strided, tl_contig, tl_modal, long_lines, y_solver, mixed_rows, z_staging;   // knobs without effect: kept and returned
    int copy_polls;                              // polls of a block's first wait for its copies in the column form
    bool spec_live;                              // the spectrum holds a right-hand side that no Poisson solve has taken yet
    FFTPlan fp1, fp3;
    FFTPlan fp1u;                                // N1 with radices up to 8 (the inverse x transform's one-radix form)
    int h1p;
    double wall_ab, wall_bb, wall_at, wall_bt;   // Pbc_a, Pbc_b of the two walls
    ProbeState *probe;
};

template <class R>
struct Ctx : Shapes {
    GridT<R> g;
    FieldsT<R> f;
};

bool make_fft_plan(int n, FFTPlan &fp, int maxr);   // radices 2, 3, 4, 5 and (maxr >= 8) 8
void probe_begin(const Shapes &cx, int kid, cudaStream_t s);
void probe_end(const Shapes &cx, int kid, cudaStream_t s);
int record_launch_error(const char *what);
int set_error(int code, const std::string &msg);

// Opt a kernel in to smem bytes of dynamic shared memory on the current
// device.  The attribute belongs to the function on each device, so the
// largest size set so far is kept per device (cache: one entry per ordinal).
inline void smem_opt_in(const void *fn, size_t smem, size_t *cache)
{
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    if (smem > cache[dev]) {
        cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        cache[dev] = smem;
    }
}

// The shape of a marching sweep (march_block) of `lines` lines in all: TI lines
// and NS segments of every line per block.  Rows per segment, m = n / NS: at
// most P::ROWS, and at least 4, because every segment loads its first plane
// twice; with few lines, short segments fill the SMs.  Up to 8192 threads in all a
// sweep is one chain of loads per segment, so segments of 2 rows are taken there
// (x sweeps alike; not where 4 rows are on their way at once, P::AHEAD).  With 4 the
// FP64 step at 12 x 10 x 12 took 143 us against 131 before the sweeps marched, with 2
// 118; 24^3 141, 141 and 118.  Up to 65536 threads a 32^3 or 48^3 step would gain 8% too,
// but 48 such cases side by side, which fill the SMs, lose 15% by the planes loaded
// twice (2.65 -> 3.07 ms), and a case has one plan, alone or not.  P::ROWS is 12 for the z
// sweeps: the parked rows (24 B each, 512 threads per SM) then leave L1 room for
// the stencil's x neighbours and tables (measured in FP64, ps per cell of dw_z:
// m = 16 at 256^3 36, m = 8 22; m = 12 at 192^3 23, m = 6 28).  The y sweeps read
// little through L1 and run best with 16 rows in two blocks per SM (256^3, ps per
// cell of du_y: m = 16 12.0, m = 8 14.2; FP32-mixed 9.7 and 13.0).  Lines too long
// for 16 of them to fit keep 512 threads and take more rows.
template <class P>
inline MarchPlan march_plan(int n, bool cyclic, int lanes, long long lines)
{
    MarchPlan mp;
    mp.n = n; mp.cyclic = cyclic ? 1 : 0;
    mp.lgNS = 1;
    const int cap = lanes < 32 ? lanes : 256;
    auto more = [&](int rows) { return (2 << mp.lgNS) <= cap && (n >> (mp.lgNS + 1)) >= rows; };
    while (more(4) && mp.lgNS < 5 && (n > (P::ROWS << mp.lgNS) || (lines << mp.lgNS) < 131072)) mp.lgNS++;
    if (P::AHEAD < 4)
        while (more(2) && mp.lgNS < 5 && (lines << (mp.lgNS + 1)) <= 8192) mp.lgNS++;
    mp.lgTI = P::LGTI;
    // FP64 z lines (P::LONG64) of more than 416 rows in too few lines for the column
    // form: 64 segments of 8 lines (64 x 64 x 512, ps per cell of dw_z: 33 against 45)
    if (P::LONG64 && mp.lgNS == 5 && n > 416 && cap >= 64) {
        mp.lgNS = 6;
        mp.lgTI = 3;
    }
    auto words = [&]() { return march_words(n, 1 << mp.lgNS, 1 << mp.lgTI, P::NRHS) * sizeof(double); };
    while (mp.lgTI > 0 && words() > 227 * 1024) {
        mp.lgTI--;
        if (more(4) && mp.lgNS + mp.lgTI < 9) mp.lgNS++;
    }
    while (words() > 227 * 1024 || mp.lgTI + mp.lgNS < 5) {   // fits, in whole warps
        if (words() > 227 * 1024) mp.lgTI--;
        else mp.lgNS++;
    }
    mp.m0 = n >> mp.lgNS; mp.rem = n & ((1 << mp.lgNS) - 1);
    return mp;
}

template <int NT, class P>
inline void launch_march_nt(const Shapes &cx, const P &prob, const MarchPlan &mp, int nlines, int gy, cudaStream_t s, int kid)
{
    const int TI = 1 << mp.lgTI;
    const size_t smem = march_words(mp.n, 1 << mp.lgNS, TI, P::NRHS) * sizeof(double);
    static size_t conf[64] = {};
    smem_opt_in((const void *)march_kernel<P, NT>, smem, conf);
    probe_begin(cx, kid, s);
    march_kernel<P, NT><<<dim3((nlines + TI - 1) / TI, gy), TI << mp.lgNS, smem, s>>>(prob, mp);
    probe_end(cx, kid, s);
    record_launch_error(kernel_name(kid));
}

// The column form of a z sweep (column_kernel), in two segments per line: 24576
// or more FP64 lines (a thread for each segment then half fills the SMs; with
// 6240 lines of 400 rows the step took 1.2 times march_kernel's) of more than 384
// rows, with rows of i that start on 16 bytes, while the spectrum is idle.  Measured
// at 512^3 (ms, thermal_z, du_z, dv_z, dw_z): 3.17, 2.54, 2.81, 3.02 against 4.64,
// 3.80, 4.85, 5.06 for march_kernel, whose parked rows then fill the shared
// memory; at 384 rows the two are level, and below it march_kernel leads.
template <class P>
inline bool launch_column(const Shapes &cx, const P &prob, int n, int nlines, int gy, cudaStream_t s, int kid)
{
    constexpr int lgNS = 1;
    if (cx.spec_live || n <= 384 || (prob.g.P1 & 1) || (long long)nlines * gy < 24576) return false;
    int w = 0, best = 1 << 30;
    for (int c = 32; c <= (128 >> lgNS); c += 32) {       // the widest of the block widths that waste least
        const int waste = (nlines + c - 1) / c * c;
        if (waste <= best) { best = waste; w = c; }
    }
    const size_t smem = col_smem<P>(w, 1 << lgNS);
    static size_t conf[64] = {};
    smem_opt_in((const void *)column_kernel<P>, smem, conf);
    probe_begin(cx, kid, s);
    column_kernel<P><<<dim3((nlines + w - 1) / w, gy), w << lgNS, smem, s>>>(prob, n, w, lgNS, reinterpret_cast<double *>(prob.f.S), 2 * cx.h1p,
                                                                              cx.copy_polls);
    probe_end(cx, kid, s);
    record_launch_error(kernel_name(kid));
    return true;
}

// A strided line sweep: nlines x gy lines of n rows.
template <class P>
inline void launch_march(const Shapes &cx, const P &prob, int n, bool cyclic, int nlines, int gy, cudaStream_t s, int kid)
{
    if constexpr (Streams<P>::on)
        if (launch_column(cx, prob, n, nlines, gy, s, kid)) return;
    const MarchPlan mp = march_plan<P>(n, cyclic, cx.lanes, (long long)nlines * gy);
    if (mp.lgTI + mp.lgNS > 8) launch_march_nt<512>(cx, prob, mp, nlines, gy, s, kid);
    else launch_march_nt<256>(cx, prob, mp, nlines, gy, s, kid);
}

// The shape of an x sweep: as many lines as two blocks per SM hold, segments for
// 256 threads, of at least 4 rows (2 on small grids, as above).
template <class P>
inline MarchPlan xmarch_plan(int n, int lanes, long long lines)
{
    MarchPlan mp;
    mp.n = n; mp.cyclic = 1;
    const int cap = lanes < 32 ? lanes : 256;
    for (mp.lgTI = 4;; mp.lgTI--) {
        mp.lgNS = 1;
        while (mp.lgNS + mp.lgTI < 8 && (2 << mp.lgNS) <= cap && (n >> (mp.lgNS + 1)) >= ((lines << (mp.lgNS + 1)) <= 8192 ? 2 : 4)) mp.lgNS++;
        while (mp.lgNS + mp.lgTI < 5) mp.lgNS++;          // whole warps
        if (mp.lgTI == 0 || xmarch_words(n, 1 << mp.lgNS, 1 << mp.lgTI, P::WORDS) * sizeof(double) <= 113 * 1024) break;
    }
    mp.m0 = n >> mp.lgNS; mp.rem = n & ((1 << mp.lgNS) - 1);
    return mp;
}

template <class P>
inline void launch_xmarch(const Shapes &cx, const P &prob, int n, int nlines, int gy, cudaStream_t s, int kid)
{
    const MarchPlan mp = xmarch_plan<P>(n, cx.lanes, (long long)nlines * gy);
    const int TI = 1 << mp.lgTI;
    const size_t smem = xmarch_words(n, 1 << mp.lgNS, TI, P::WORDS) * sizeof(double);
    static size_t conf[64] = {};
    smem_opt_in((const void *)xmarch_kernel<P>, smem, conf);
    probe_begin(cx, kid, s);
    xmarch_kernel<P><<<dim3((nlines + TI - 1) / TI, gy), TI << mp.lgNS, smem, s>>>(prob, mp);
    probe_end(cx, kid, s);
    record_launch_error(kernel_name(kid));
}

// ---------------------------------------------------------------------------
// Ensemble launches: the streams a stage's launches run on side by side (forked
// from and joined back to the stage's stream).
// ---------------------------------------------------------------------------
struct MultiArena {
    std::vector<cudaStream_t> aux;
    std::vector<cudaEvent_t> join;       // one per aux stream
    cudaEvent_t fork = nullptr;
};

// A marching sweep for a group of cases: one launch per case, side by side on
// the aux streams.  (A persistent multi-case form of march_block was a second
// compilation of the same source, whose multiply-adds the compiler fused
// differently: the ensemble's results left its members' by one bit.)
template <class R, class Launch>
inline void march_stage(const std::vector<Ctx<R> *> &cs, MultiArena &A, cudaStream_t s, Launch launch)
{
    if (cs.empty()) return;
    const size_t side = std::min(A.aux.size(), cs.size());
    if (side) cudaEventRecord(A.fork, s);
    for (size_t i = 0; i < side; i++) cudaStreamWaitEvent(A.aux[i], A.fork, 0);
    for (size_t i = 0; i < cs.size(); i++) launch(*cs[i], side ? A.aux[i % side] : s);
    for (size_t i = 0; i < side; i++) {
        cudaEventRecord(A.join[i], A.aux[i]);
        cudaStreamWaitEvent(s, A.join[i], 0);
    }
}

// Stage launchers (one per reference routine or fused group), instantiated
// for R = double and R = float.
template <class R> void launch_thermal(const Ctx<R> &cx, cudaStream_t s);
template <class R> void launch_momentum_coeffi(const Ctx<R> &cx, cudaStream_t s);
template <class R> void launch_solve_du(const Ctx<R> &cx, cudaStream_t s);
template <class R> void launch_solve_dv(const Ctx<R> &cx, cudaStream_t s);
template <class R> void launch_solve_dw(const Ctx<R> &cx, cudaStream_t s);
template <class R> void launch_blockld_v(const Ctx<R> &cx, cudaStream_t s);
template <class R> void launch_blockld_u(const Ctx<R> &cx, cudaStream_t s);
template <class R> void launch_pseudo_update(const Ctx<R> &cx, cudaStream_t s);   // standalone (Un = U + dU, ...)
template <class R> void launch_pseudo_prhs_fftx(const Ctx<R> &cx, cudaStream_t s, bool with_pseudo);
// walls: write the wall rows of dP (of P) too; a step leaves both to launch_post
template <class R> void launch_poisson_rest(const Ctx<R> &cx, cudaStream_t s, bool walls);
template <class R> void launch_modal(const Ctx<R> &cx, cudaStream_t s);
template <class R> void launch_poisson_fwd(const Ctx<R> &cx, cudaStream_t s);   // z FFTs (forward)
template <class R> void launch_poisson_back(const Ctx<R> &cx, cudaStream_t s, bool walls);  // z and x inverse FFTs, dP walls
template <class R> void launch_projection(const Ctx<R> &cx, cudaStream_t s, bool walls);
template <class R> void launch_post(const Ctx<R> &cx, cudaStream_t s, int record_hist, bool walls);
template <class R> void launch_ghost(const Ctx<R> &cx, R *a, cudaStream_t s);
// the line stages of a step for a group of same-precision cases
template <class R> void launch_thermal_multi(const std::vector<Ctx<R> *> &cs, MultiArena &A, cudaStream_t s);
template <class R> void launch_momentum_multi(const std::vector<Ctx<R> *> &cs, MultiArena &A, cudaStream_t s);
template <class R> void launch_modal_multi(const std::vector<Ctx<R> *> &cs, MultiArena &A, cudaStream_t s);
template <class R> void launch_convert(const R *src, double *dst, long long n, cudaStream_t s);   // field -> FP64 staging
template <class R> void launch_convert_in(const double *src, R *dst, long long n, cudaStream_t s); // FP64 staging -> field
void launch_join(const float *hi, const float *lo, double *dst, long long n, cudaStream_t s);       // FP32 pair -> FP64 staging
template <class R> void launch_pack(const Ctx<R> &cx, const R *src, const R *lo, double *dst, int k0, int nk, cudaStream_t s);
template <class R> void launch_unpack(const Ctx<R> &cx, const double *src, R *dst, R *dst2, R *lo, int k0, int nk, cudaStream_t s);
template <class R> void launch_plane(const Ctx<R> &cx, const R *src, const R *lo, double *dst, int axis, int index, cudaStream_t s);
void launch_split(const double *src, float *hi, float *lo, long long n, cudaStream_t s);          // FP64 staging -> FP32 pair

} // namespace tcs
