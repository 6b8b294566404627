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

// Every kernel the time step launches, in launch order.
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
    int tl_strided, tl_contig, tl_modal;
    int fft_lines_x, fft_lines_z;
    int ifft_lines_x;                            // lines per block of the inverse x transform
    int lanes;                                   // at most this many partitions (lanes) per line
    int long_lines, y_solver;                    // accepted and kept; one solver runs the strided lines
    int mixed_rows;                              // likewise
    int z_staging;                               // likewise
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

LinePlan make_line_plan(int n, bool cyclic, int TL, int pmax = 32);
bool make_fft_plan(int n, FFTPlan &fp, int maxr);   // radices 2, 3, 4, 5 and (maxr >= 8) 8
void probe_begin(const Shapes &cx, int kid, cudaStream_t s);
void probe_end(const Shapes &cx, int kid, cudaStream_t s);
int record_launch_error(const char *what);
int set_error(int code, const std::string &msg);

// Dynamic shared memory of a line-solver launch.
template <class Prob>
inline size_t line_smem(const LinePlan &lp)
{
    return (size_t)line_words<Prob>() * lp.TL * lp.LS * sizeof(typename Prob::Real) + (size_t)lp.n * sizeof(int);
}

// The plan of a line problem: make_line_plan's partitions, and for the
// non-cyclic strided problems (the modal solves) a
// line stride LS chosen for the build and the emission, where one warp
// touches TL lines x 32/TL rows: LS = banks/TL (mod banks), banks = 32
// four-byte words (FP32 rows) or 16 eight-byte words per half-warp (FP64
// rows), puts those accesses on distinct banks.  The solve (one line per
// warp) only uses the odd partition stride PS.  Measured at 256^3: the y
// sweeps 2-5% and the modal solves 3-4% faster in both forms.
template <class Prob>
inline LinePlan plan_for(int n, bool cyclic, int tl, int pmax)
{
    LinePlan lp = make_line_plan(n, cyclic, tl, pmax);
    if (!Prob::CONTIG && !cyclic && tl > 1) {
        const int banks = sizeof(typename Prob::Real) == 4 ? 32 : 16;
        const int want = tl < banks ? banks / tl : 1;
        const int ls = lp.P * lp.PS;
        lp.LS = ls + ((want - ls) % banks + banks) % banks;
    }
    return lp;
}

// Lines per block: the requested count, halved until MINB blocks fit in the
// SM's shared memory (228 KiB, 1 KB reserved per block); extra: static shared
// memory the kernel adds per block.
template <class Prob>
inline int fit_tl(int n, bool cyclic, int want, int pmax, size_t extra = 0)
{
    const size_t budget = (size_t)228 * 1024 / Prob::MINB - 1024 - extra;
    int tl = want;
    while (tl > 1 && line_smem<Prob>(plan_for<Prob>(n, cyclic, tl, pmax)) > budget) tl /= 2;
    return tl;
}

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

template <class Prob>
inline void launch_lines(const Prob &p, const LinePlan &lp, dim3 grid, cudaStream_t s, int kid, const Shapes &cx)
{
    const size_t smem = line_smem<Prob>(lp);
    static size_t configured[64] = {};
    smem_opt_in((const void *)line_solve_kernel<Prob>, smem, configured);
    probe_begin(cx, kid, s);
    line_solve_kernel<Prob><<<grid, Prob::NT, smem, s>>>(p, lp);
    probe_end(cx, kid, s);
    record_launch_error(kernel_name(kid));
}

// The shape of a marching sweep (march_block) of `lines` lines in all: TI lines
// and NS segments of every line per block.  Rows per segment, m = n / NS: at
// most P::ROWS, and at least 4, because every segment loads its first plane
// twice; with few lines, short segments fill the SMs.  P::ROWS is 12 for the z
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
    auto more = [&]() { return (2 << mp.lgNS) <= cap && (n >> (mp.lgNS + 1)) >= 4; };
    while (more() && mp.lgNS < 5 && (n > (P::ROWS << mp.lgNS) || (lines << mp.lgNS) < 131072)) mp.lgNS++;
    mp.lgTI = 4;
    auto words = [&]() { return march_words(n, 1 << mp.lgNS, 1 << mp.lgTI, P::NRHS) * sizeof(double); };
    while (mp.lgTI > 0 && words() > 227 * 1024) {
        mp.lgTI--;
        if (more() && mp.lgNS + mp.lgTI < 9) mp.lgNS++;
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

// The column form of a z sweep (column_kernel), in two segments per line: FP64
// lines of more than 384 rows, with rows of i that start on 16 bytes.  Measured
// at 512^3 (ms, thermal_z, du_z, dv_z, dw_z): 3.17, 2.54, 2.81, 3.02 against 4.64,
// 3.80, 4.85, 5.06 for march_kernel, whose parked rows then fill the shared
// memory; at 384 rows the two are level, and below it march_kernel leads.
template <class P>
inline bool launch_column(const Shapes &cx, const P &prob, int n, int nlines, int gy, cudaStream_t s, int kid)
{
    constexpr int lgNS = 1;
    if (n <= 384 || (prob.g.P1 & 1)) return false;
    int w = 0, best = 1 << 30;
    for (int c = 32; c <= (128 >> lgNS); c += 32) {       // the widest of the block widths that waste least
        const int waste = (nlines + c - 1) / c * c;
        if (waste <= best) { best = waste; w = c; }
    }
    const size_t smem = col_smem<P>(w, 1 << lgNS);
    static size_t conf[64] = {};
    smem_opt_in((const void *)column_kernel<P>, smem, conf);
    probe_begin(cx, kid, s);
    column_kernel<P><<<dim3((nlines + w - 1) / w, gy), w << lgNS, smem, s>>>(prob, n, w, lgNS, reinterpret_cast<double *>(prob.f.S), 2 * cx.h1p);
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
// 256 threads.
template <class P>
inline MarchPlan xmarch_plan(int n, int lanes)
{
    MarchPlan mp;
    mp.n = n; mp.cyclic = 1;
    const int cap = lanes < 32 ? lanes : 256;
    for (mp.lgTI = 4;; mp.lgTI--) {
        mp.lgNS = 1;
        while (mp.lgNS + mp.lgTI < 8 && (2 << mp.lgNS) <= cap && (n >> (mp.lgNS + 1)) >= 4) mp.lgNS++;
        while (mp.lgNS + mp.lgTI < 5) mp.lgNS++;          // whole warps
        if (mp.lgTI == 0 || xmarch_words(n, 1 << mp.lgNS, 1 << mp.lgTI, P::WORDS) * sizeof(double) <= 113 * 1024) break;
    }
    mp.m0 = n >> mp.lgNS; mp.rem = n & ((1 << mp.lgNS) - 1);
    return mp;
}

template <class P>
inline void launch_xmarch(const Shapes &cx, const P &prob, int n, int nlines, int gy, cudaStream_t s, int kid)
{
    const MarchPlan mp = xmarch_plan<P>(n, cx.lanes);
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
// Ensemble launches: one line stage of many cases as line_solve_multi
// launches of up to MultiParams::K cases each.  An ensemble builds each
// step's launches twice in the same order: in planning mode every launch
// reserves its item counter in the arena, then (after one upload of the
// arena) in launch mode each launch takes its counter's device address.
// The launches of one stage run concurrently on the aux streams (forked from
// and joined back to the stage's stream).
// ---------------------------------------------------------------------------
struct MultiArena {
    std::vector<unsigned char> host;
    unsigned char *dev = nullptr;
    size_t cursor = 0;
    bool planning = true;
    std::vector<cudaStream_t> aux;       // streams for a stage's second and later launches
    std::vector<cudaEvent_t> join;       // one per aux stream
    cudaEvent_t fork = nullptr;
    int *counter()
    {
        const size_t off = (cursor + 15) & ~(size_t)15;
        cursor = off + 16;
        if (planning) {
            host.resize(cursor, 0);
            return nullptr;
        }
        return (int *)(dev + off);
    }
};

// One case's share of a multi-case line stage: the line length, cyclicity,
// requested lines per block, and the block grid (lines / TL rounded up, gy).
struct StageShape {
    int n;
    bool cyclic;
    int want, lines, gy;
};

template <class Prob>
inline void launch_lines_multi(MultiParams<Prob> &mp, int ncase, cudaStream_t s, const char *what)
{
    size_t smem = 0;
    for (int c = 0; c < ncase; c++) smem = std::max(smem, line_smem<Prob>(mp.lp[c]));
    static size_t conf[64] = {};
    smem_opt_in((const void *)line_solve_multi<Prob>, smem, conf);
    int dev = 0, sms = 148, occ = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, line_solve_multi<Prob>, Prob::NT, smem);
    const int grid = (int)std::min<long long>(mp.nitems, (long long)std::max(occ, 1) * sms);
    line_solve_multi<Prob><<<grid, Prob::NT, smem, s>>>(mp);
    record_launch_error(what);
}

// A line stage for a group of same-precision cases: per case the same plan
// and block grid as its one-case launch; the cases with the longest blocks
// first (so the blocks that pull the last items finish close together),
// MultiParams::K cases per launch.
template <class P, class R, class Shape, class Make>
inline void multi_stage(const std::vector<Ctx<R> *> &cs, MultiArena &A, cudaStream_t s, const char *what, Shape shape,
                        Make make)
{
    struct Entry { P prob; LinePlan lp; int gx, gy; long long cost; };
    std::vector<Entry> es;
    for (const Ctx<R> *xp : cs) {
        const Ctx<R> &x = *xp;
        const StageShape sh = shape(x);
        const LinePlan lp = plan_for<P>(sh.n, sh.cyclic, fit_tl<P>(sh.n, sh.cyclic, sh.want, x.lanes, 64), x.lanes);
        es.push_back({make(x, lp.TL), lp, (sh.lines + lp.TL - 1) / lp.TL, sh.gy, (long long)sh.n * lp.TL});
    }
    std::stable_sort(es.begin(), es.end(), [](const Entry &a, const Entry &b) { return a.cost > b.cost; });
    constexpr int K = MultiParams<P>::K;
    const int nl = (int)((es.size() + K - 1) / K);
    const bool fan = !A.planning && nl > 1 && (int)A.aux.size() >= nl - 1;
    if (fan) cudaEventRecord(A.fork, s);
    for (int l = 0; l < nl; l++) {
        const size_t c0 = (size_t)l * K;
        const int nc = (int)std::min<size_t>(K, es.size() - c0);
        int *ctr = A.counter();
        if (A.planning) continue;
        MultiParams<P> mp;
        mp.start[0] = 0;
        for (int c = 0; c < nc; c++) {
            const Entry &e = es[c0 + c];
            mp.p[c] = e.prob;
            mp.lp[c] = e.lp;
            mp.gx[c] = e.gx;
            mp.start[c + 1] = mp.start[c] + e.gx * e.gy;
        }
        mp.nitems = mp.start[nc];
        mp.ctr = ctr;
        cudaStream_t ls = s;
        if (fan && l > 0) {
            ls = A.aux[l - 1];
            cudaStreamWaitEvent(ls, A.fork, 0);
        }
        launch_lines_multi(mp, nc, ls, what);
        if (fan && l > 0) {
            cudaEventRecord(A.join[l - 1], ls);
            cudaStreamWaitEvent(s, A.join[l - 1], 0);
        }
    }
}

// A marching sweep for a group of cases: one launch per case, side by side on
// the aux streams.  (A persistent multi-case form of march_block was a second
// compilation of the same source, whose multiply-adds the compiler fused
// differently: the ensemble's results left its members' by one bit.)
template <class R, class Launch>
inline void march_stage(const std::vector<Ctx<R> *> &cs, MultiArena &A, cudaStream_t s, Launch launch)
{
    if (A.planning || cs.empty()) return;
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
template <class R> void launch_poisson_rest(const Ctx<R> &cx, cudaStream_t s);
template <class R> void launch_modal(const Ctx<R> &cx, cudaStream_t s);
template <class R> void launch_poisson_fwd(const Ctx<R> &cx, cudaStream_t s);   // z FFTs (forward)
template <class R> void launch_poisson_back(const Ctx<R> &cx, cudaStream_t s);  // mean, z and x inverse FFTs, dP walls
template <class R> void launch_projection(const Ctx<R> &cx, cudaStream_t s);
template <class R> void launch_post(const Ctx<R> &cx, cudaStream_t s, int record_hist);
template <class R> void launch_ghost(const Ctx<R> &cx, R *a, cudaStream_t s);
// the line stages of a step for a group of same-precision cases, one launch per stage
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
