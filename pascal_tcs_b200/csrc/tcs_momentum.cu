// tcs_momentum.cu -- momentum increments: mpi_momentum_coeffi, solvedU/V/W,
// blockLdV/U and the standalone pseudo-update (module_solve_momentum.f90).
//
// Each solved* routine is three fused kernels (z, x, y sweeps, tcs_march.cuh); the y sweep writes the increment with its periodic ghosts, which
// is the ghost update the driver performs right after (main.f90:151-169).
//
// Mu and invRho are the 2-D (j,k) tables of mpi_momentum_coeffi: the
// reference assigns whole rows Mu(:,j,k) inside its i loop (:156-171), so every
// value along i equals the one computed from T(n1sub,j,k).
#include "tcs_kernels.h"

namespace tcs {

#define MU(jj, kk) ld(f.Mu2 + ix2(g, (jj), (kk)))

// ---------------------------------------------------------------------------
// mpi_momentum_coeffi (:145-173) -> (j,k) tables from T(n1sub, j, k).
// ---------------------------------------------------------------------------
// Evaluated in FP64 in both forms; invRho stays FP64 (FieldsT::iR2d, iRTd) for the
// pressure right-hand side and the projection.
template <class R>
__global__ void momentum_coeffi_kernel(GridT<R> g, FieldsT<R> f)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x, k = blockIdx.y;
    if (j > g.N2 + 1 || blown(g)) return;
    const Phys &p = g.phd;
    auto props = [&](int jj, int kk, double &mu, double &ir) {
        const double t1 = p.DeltaT * (double)f.T[ix(g, g.N1 + 1, jj, kk)];
        const double t2 = t1 * t1, t3 = t2 * t1, t4 = t3 * t1, t5 = t4 * t1;
        const double ra = (p.a10 + p.a10 * (p.a11 * t1 + p.a12 * t2 + p.a13 * t3 + p.a14 * t4 + p.a15 * t5));
        ir = p.Rho0 / ra;
        mu = ra * (p.d10 + p.d10 * (p.d11 * t1 + p.d12 * t2 + p.d13 * t3 + p.d14 * t4 + p.d15 * t5)) / p.Mu0;
    };
    double mu, ir;
    props(j, k, mu, ir);
    const int c = ix2(g, j, k);
    f.Mu2[c] = (R)mu;
    f.iR2d[c] = ir;
    // the averages at the faces between row j-1 and j (y), plane k-1 and k (z)
    // and at the edge between them (yz), which the sweeps read instead of
    // forming them again at every i: Mu, Mu_y, Mu_z, Mu_yz and iR, iR_y, iR_z
    double mj, rj, mk, rk, mjk, rjk;
    props(max(j - 1, 0), k, mj, rj);
    props(j, max(k - 1, 0), mk, rk);
    props(max(j - 1, 0), max(k - 1, 0), mjk, rjk);
    const double y0 = j ? 0.5 * g.d2.dx[j - 1] * g.d2.rdmx[j] : 0.0, y1 = j ? 0.5 * g.d2.dx[j] * g.d2.rdmx[j] : 0.0;
    const double z0 = k ? 0.5 * g.d3.dx[k - 1] * g.d3.rdmx[k] : 0.0, z1 = k ? 0.5 * g.d3.dx[k] * g.d3.rdmx[k] : 0.0;
    R *const mt = f.MuT + 4 * c, *const rt = f.iRT + 4 * c;
    mt[0] = (R)mu;
    mt[1] = (R)(y0 * mu + y1 * mj);
    mt[2] = (R)(z0 * mu + z1 * mk);
    mt[3] = (R)(z0 * (y0 * mu + y1 * mj) + z1 * (y0 * mk + y1 * mjk));
    const double ry = y0 * ir + y1 * rj, rz = z0 * ir + z1 * rk;
    rt[0] = (R)ir; rt[1] = (R)ry; rt[2] = (R)rz; rt[3] = R(0);
    if constexpr (HasLo<R>::on) {
        double *const rd = f.iRTd + 4 * c;
        rd[0] = ir; rd[1] = ry; rd[2] = rz; rd[3] = 0.0;
    }
}

template <class R>
void launch_momentum_coeffi(const Ctx<R> &cx, cudaStream_t s)
{
    const GridT<R> &g = cx.g;
    probe_begin(cx, K_MOM_COEFFI, s);
    momentum_coeffi_kernel<<<dim3((g.N2 + 2 + 127) / 128, g.N3 + 2), 128, 0, s>>>(g, cx.f);
    probe_end(cx, K_MOM_COEFFI, s);
    record_launch_error("momentum_coeffi");
}

// ---------------------------------------------------------------------------
// solvedU (:225-563)
// ---------------------------------------------------------------------------
template <class R>
struct DUZ {
    using Real = R;
    static constexpr int NRHS = 1;
    static constexpr int AHEAD = std::is_same<R, float>::value ? 1 : 0, TPS = 512, ROWS = 12, LGTI = 4;   // FP64 inputs of two rows do not fit the registers
    static constexpr bool LONG64 = std::is_same<R, double>::value;
    GridT<R> g; FieldsT<R> f;
    __device__ bool skip() const { return blown(g); }
    __device__ int lines() const { return g.N1; }
    // the rows of i that a plane needs in the column form
    static constexpr int NROW = 8, J0 = 1;
    static constexpr bool TABLES = true;
    __device__ static constexpr int row_dj(int q) { constexpr int v[] = {0, -1, 1, 0, 1, 0, 0, 0}; return v[q]; }
    __device__ static constexpr int row_dk(int q) { constexpr int v[] = {1, 0, 0, 0, 0, 1, 0, 0}; return v[q]; }
    __device__ __forceinline__ const R *row_src(int q) const
    {
        switch (q) {
        case 0: return f.U;
        case 1: return f.U;
        case 2: return f.U;
        case 3: return f.V;
        case 4: return f.V;
        case 5: return f.W;
        case 6: return f.P;
        default: return f.T;
        }
    }
    // Averages over a face weigh the two cells by w and 1 - w (dmx is the mean
    // of the two dx on every mesh), and Mu and invRho are constant along i.
    // The reduced right-hand side: the explicit operator minus the implicit
    // ones applied to U.  Per direction the coefficient terms of the two
    // cancel in exact arithmetic; on the wall-adjacent planes (j = 1, N2), where
    // the jC_BC masks and the wall terms break that, the difference is added.
    struct March {
        R cu, rdx1, rdx1m, rdmx1, rdx2, rdmx2, rdmx2p, dt;   // fixed along the line; cu: weight of cell i at x face i (cell i-1: 1 - cu)
        R Uc, F, G, ma, wa;                                  // the face below the row
        long long c;
        int t4, j;
        __device__ __forceinline__ March(const DUZ &q, int line, int by, int r0)
        {
            const GridT<R> &g = q.g;
            const FieldsT<R> &f = q.f;
            const int i = 1 + line, im = i - 1, k = r0 + 1;
            j = 1 + by;
            rdmx1 = ld(g.m1.rdmx + i); rdx1 = ld(g.m1.rdx + i); rdx1m = ld(g.m1.rdx + im);
            cu = R(0.5) * ld(g.m1.dx + im) * rdmx1;
            rdx2 = ld(g.m2.rdx + j); rdmx2 = ld(g.m2.rdmx + j); rdmx2p = ld(g.m2.rdmx + j + 1);
            dt = R(g.scal[S_DT]);
            c = ix(g, i, j, k);
            t4 = 4 * ix2(g, j, k);
            Uc = ld(f.U + c);
            face(ld(f.U + c - (long long)g.P1 * g.P2), Uc, ld(f.W + c), ld(f.W + c - 1), ld(f.MuT + t4 + 2), ld(g.m3.rdmx + k));
        }
        // the z face between planes k-1 and k: stress, convection and matrix terms
        __device__ __forceinline__ void face(R Um, R Up, R W0, R Wxm, R mu, R rdmx3)
        {
            const R dw = W0 - Wxm, w = Wxm + cu * dw, du = (Up - Um) * rdmx3;
            F = mu * (du + dw * rdmx1);
            G = w * du;
            ma = mu * rdmx3;
            wa = R(0.25) * w * rdmx3;
        }
        struct In { R Uxm, Uxp, Uym, Uyp, Uzp, Vc, Vxm, Vyp, Vxmyp, Wzp, Wxmzp, Pc, Pxm, T0, Txm, muy4, muz6, iR, rdx3, rdmx3; cplx_t<R> mt; };
        __device__ __forceinline__ void load(const DUZ &q, int r, In &n)
        {
            row_cell(q.g, c, t4);
            const GridT<R> &g = q.g;
            const FieldsT<R> &f = q.f;
            const long long sj = g.P1, sk = (long long)g.P1 * g.P2;
            n.Uxm = ld(f.U + c - 1); n.Uxp = ld(f.U + c + 1); n.Uym = ld(f.U + c - sj); n.Uyp = ld(f.U + c + sj); n.Uzp = ld(f.U + c + sk);
            n.Vc = ld(f.V + c); n.Vxm = ld(f.V + c - 1); n.Vyp = ld(f.V + c + sj); n.Vxmyp = ld(f.V + c - 1 + sj);
            n.Wzp = ld(f.W + c + sk); n.Wxmzp = ld(f.W + c - 1 + sk);
            n.Pc = ld(f.P + c); n.Pxm = ld(f.P + c - 1); n.T0 = ld(f.T + c); n.Txm = ld(f.T + c - 1);
            n.mt = ld2(f.MuT + t4);                        // Mu, Mu at the lower y face
            n.muy4 = ld(f.MuT + t4 + 5); n.muz6 = ld(f.MuT + t4 + 4 * g.P2 + 2); n.iR = ld(f.iRT + t4);
            n.rdx3 = ld(g.m3.rdx + r + 1); n.rdmx3 = ld(g.m3.rdmx + r + 2);
            c += sk;
            t4 += 4 * g.P2;
        }
        // the same values from the ring: slot a holds plane k's rows, b the plane below's
        __device__ __forceinline__ void fill(const DUZ &q, int r, In &n, const double *a, const double *b, int w, int l)
        {
            const GridT<R> &g = q.g;
            const int s = w + 2;
            a += l + 1; b += l + 1;
            const double *const ta = a - (l + 1) + NROW * s, *const tb = b - (l + 1) + NROW * s;   // table words of planes k + 1 and k
            n.Uxm = b[-1]; n.Uxp = b[1]; n.Uzp = a[0]; n.Uym = a[s]; n.Uyp = a[2 * s];
            n.Vc = a[3 * s]; n.Vxm = a[3 * s - 1]; n.Vyp = a[4 * s]; n.Vxmyp = a[4 * s - 1];
            n.Wzp = a[5 * s]; n.Wxmzp = a[5 * s - 1];
            n.Pc = a[6 * s]; n.Pxm = a[6 * s - 1]; n.T0 = a[7 * s]; n.Txm = a[7 * s - 1];
            n.mt.x = tb[4]; n.mt.y = tb[5]; n.muy4 = tb[9]; n.muz6 = ta[6]; n.iR = tb[12];
            n.rdx3 = ld(g.m3.rdx + r + 1); n.rdmx3 = ld(g.m3.rdmx + r + 2);
        }
        __device__ __forceinline__ void row(const DUZ &q, int r, const In &n, double &a, double &b, double &cc, double *d)
        {
            const GridT<R> &g = q.g;
            const PhysT<R> &p = g.ph;
            const R Uxm = n.Uxm, Uxp = n.Uxp, Uym = n.Uym, Uyp = n.Uyp, Uzp = n.Uzp, Vc = n.Vc, Vxm = n.Vxm, Vyp = n.Vyp, Vxmyp = n.Vxmyp;
            const R Wzp = n.Wzp, Wxmzp = n.Wxmzp, Pc = n.Pc, Pxm = n.Pxm, T0 = n.T0, Txm = n.Txm, muy4 = n.muy4, muz6 = n.muz6, iR = n.iR;
            const cplx_t<R> mt = n.mt;
            const R rdx3 = n.rdx3;
            const R ih = R(0.5) * p.Cmu * iR;
            const R u1 = R(0.5) * (Uxm + Uc), u2 = R(0.5) * (Uxp + Uc);
            const R dx1 = (Uc - Uxm) * rdx1m, dx2 = (Uxp - Uc) * rdx1;
            const R dv3 = Vc - Vxm, dv4 = Vyp - Vxmyp;
            const R v3 = Vxm + cu * dv3, v4 = Vxmyp + cu * dv4;
            const R dy3 = (Uc - Uym) * rdmx2, dy4 = (Uyp - Uc) * rdmx2p;
            const R vx3 = dv3 * rdmx1, vx4 = dv4 * rdmx1;
            const R mu3 = mt.y, mu4 = muy4;
            const R F5 = F, G5 = G, ma5 = ma, wa5 = wa, U0 = Uc;
            Uc = Uzp;
            face(U0, Uzp, Wzp, Wxmzp, muz6, n.rdmx3);
            const R vs = R(2) * mt.x * ((dx2 - dx1) * rdmx1) + (F - F5) * rdx3 + (mu4 * (dy4 + vx4) - mu3 * (dy3 + vx3)) * rdx2;
            R rhs = R(2) * ih * vs - R(0.5) * ((u1 * dx1 + u2 * dx2) + (G5 + G) + (v3 * dy3 + v4 * dy4));
            const R Tc = Txm + cu * (T0 - Txm);
            rhs = rhs + iR * (p.Cmt * (Tc + p.a12pera11 * (Tc * Tc) * p.DeltaT) - p.Cmp * ((Pc - Pxm) * rdmx1));
            if (j == 1) {
                const R am = -(ih * rdx2 * mu3 + R(0.25) * v3) * rdmx2;
                rhs = rhs + am * (Uym - p.Ubt) + R(0.25) * dy3 * (v3 - p.Vbt) + ih * rdx2 * mu3 * vx3;
            }
            if (j == g.N2) {
                const R ap = (R(0.25) * v4 - ih * rdx2 * mu4) * rdmx2p;
                rhs = rhs + ap * (Uyp - p.Uup) + R(0.25) * dy4 * (v4 - p.Vup) - ih * rdx2 * mu4 * vx4;
            }
            const R h3 = ih * rdx3;
            const R am = -(h3 * ma5 + wa5) * dt, ap = (wa - h3 * ma) * dt;
            a = am; cc = ap; b = 1.0 - ((double)am + (double)ap);
            d[0] = rhs * dt;
        }
    };
    struct Out : ScratchOut<R> {
        __device__ __forceinline__ Out(const DUZ &q, int line, int by, int r) : ScratchOut<R>(q.g, q.f.scr, 1 + line, 1 + by, r + 1, (long long)q.g.P1 * q.g.P2) {}
        __device__ __forceinline__ void put(const DUZ &q, const double *x) { ScratchOut<R>::put(q.g, q.f.scr, R(x[0])); }
    };
};

template <class R>
struct DUX {
    using Real = R;
    static constexpr int WORDS = 3, UNROLL = 4;
    GridT<R> g; FieldsT<R> f;
    __device__ bool skip() const { return blown(g); }
    __device__ int lines() const { return g.N2; }
    __device__ R *out(int line, int by) const { return f.scr + ix(g, 1, 1 + line, 1 + by); }
    struct Stage {
        long long c;
        __device__ __forceinline__ Stage(const DUX &q, int line, int by) : c(ix(q.g, 1, 1 + line, 1 + by)) {}
        __device__ __forceinline__ void put(const DUX &q, int r, double *w, int PL) const
        {
            TCS_OOB(q.g.scal, r < 0 || r >= q.g.N1, return);
            w[0] = (double)q.f.scr[c + r];
            w[PL] = (double)ld(q.f.U + c + r);
        }
    };
    struct March {
        R mu, h, dt, Uc, Un, A, B, C;                   // Un: U beyond the segment; A, B, C: the cell below the row
        __device__ __forceinline__ March(const DUX &q, int line, int by, int r0, int m, int n, const double *w, int PL)
        {
            const int t4 = 4 * ix2(q.g, 1 + line, 1 + by);
            mu = ld(q.f.MuT + t4);
            h = q.g.ph.Cmu * ld(q.f.iRT + t4);
            dt = R(q.g.scal[S_DT]);
            Uc = R(w[PL + r0]);
            Un = R(w[PL + (r0 + m < n ? r0 + m : 0)]);
            cell(R(w[PL + (r0 ? r0 - 1 : n - 1)]), Uc, ld(q.g.m1.rdx + r0));
        }
        __device__ __forceinline__ void cell(R Um, R Up, R rdx1)
        {
            A = mu * rdx1;
            B = R(0.125) * (Um + Up) * rdx1;
            C = R(0.125) * (Up - Um) * rdx1;
        }
        __device__ __forceinline__ void row(const DUX &q, int r, bool last, const double *w, int PL, double &a, double &b, double &c, double &d)
        {
            const R rdx1 = ld(q.g.m1.rdx + r + 1), hd = h * ld(q.g.m1.rdmx + r + 1);
            const R Up = last ? Un : R(w[PL + r + 1]);
            const R A1 = A, B1 = B, C1 = C, U0 = Uc;
            Uc = Up;
            cell(U0, Up, rdx1);
            const R am = (C1 - B1 - hd * A1) * dt, ap = (B + C - hd * A) * dt;
            a = am; c = ap; b = (1.0 - ((double)am + (double)ap)) + (double)(R(2) * (C1 + C) * dt);
            d = w[r];
        }
    };
};

// The rows along x of V and W: face velocities U averaged to the line (word 1)
// and one pair of viscosities, the mu1 and mu2 left by the last cell of stage 1.
template <class R>
struct FaceRows {
    R mu1, mu2, h, dt, un, w1, rdm;                     // un: the face velocity beyond the segment; w1, rdm: the face below the row
    __device__ __forceinline__ void begin(const GridT<R> &g, R ih, int r0, int m, int n, const double *w, int PL)
    {
        h = ih;
        dt = R(g.scal[S_DT]);
        un = R(w[PL + (r0 + m < n ? r0 + m : 0)]);
        rdm = ld(g.m1.rdmx + r0 + 1);
        w1 = R(0.25) * R(w[PL + r0]) * rdm;
    }
    __device__ __forceinline__ void rows(const GridT<R> &g, int r, bool last, const double *w, int PL, double &a, double &b, double &c, double &d)
    {
        const R rdp = ld(g.m1.rdmx + r + 2), hd = h * ld(g.m1.rdx + r + 1);
        const R w2 = R(0.25) * (last ? un : R(w[PL + r + 1])) * rdp;
        const R am = -(hd * (mu1 * rdm) + w1) * dt, ap = (w2 - hd * (mu2 * rdp)) * dt;
        a = am; c = ap; b = 1.0 - ((double)am + (double)ap);
        d = w[r];
        w1 = w2; rdm = rdp;
    }
};

template <class R>
struct DUY {
    using Real = R;
    static constexpr int NRHS = 1;
    static constexpr int AHEAD = 2, TPS = 512, ROWS = 16, LGTI = 4;
    static constexpr bool LONG64 = false;
    GridT<R> g; FieldsT<R> f;
    __device__ bool skip() const { return blown(g); }
    __device__ int lines() const { return g.N1; }
    struct March {
        R cu, dt, m, w;                                 // m, w: stress and convection terms of the face below the row
        long long c;
        int t4;
        __device__ __forceinline__ March(const DUY &q, int line, int by, int r0)
        {
            const GridT<R> &g = q.g;
            const int i = 1 + line, j = r0 + 1, k = 1 + by;
            cu = R(0.5) * ld(g.m1.dx + i - 1) * ld(g.m1.rdmx + i);
            dt = R(g.scal[S_DT]);
            c = ix(g, i, j, k);
            t4 = 4 * ix2(g, j, k);
            face(ld(q.f.V + c), ld(q.f.V + c - 1), ld(q.f.MuT + t4 + 1), ld(g.m2.rdmx + j));
        }
        __device__ __forceinline__ void face(R V, R Vxm, R mu, R rdmx2)
        {
            m = mu * rdmx2;
            w = R(0.25) * (Vxm + cu * (V - Vxm)) * rdmx2;
        }
        struct In { R V, Vxm, mu, iR, rdx2, rdmx2, d; };
        __device__ __forceinline__ void load(const DUY &q, int r, In &n)
        {
            row_cell(q.g, c, t4);
            const long long sj = q.g.P1;
            n.V = ld(q.f.V + c + sj); n.Vxm = ld(q.f.V + c + sj - 1);
            n.mu = ld(q.f.MuT + t4 + 5); n.iR = ld(q.f.iRT + t4);
            n.rdx2 = ld(q.g.m2.rdx + r + 1); n.rdmx2 = ld(q.g.m2.rdmx + r + 2);
            n.d = q.f.scr[c];
            c += sj;
            t4 += 4;
        }
        __device__ __forceinline__ void row(const DUY &q, int r, const In &n, double &a, double &b, double &cc, double *d)
        {
            const R m3 = m, w3 = w, h = R(0.5) * q.g.ph.Cmu * n.iR * n.rdx2;
            face(n.V, n.Vxm, n.mu, n.rdmx2);
            const R am = -(h * m3 + w3) * dt, ap = (w - h * m) * dt;
            a = r == 0 ? R(0) : am; cc = r == q.g.N2 - 1 ? R(0) : ap; b = 1.0 - ((double)am + (double)ap);
            d[0] = n.d;
        }
    };
    struct Out : PeriodicOut<R> {
        __device__ __forceinline__ Out(const DUY &q, int line, int by, int r) : PeriodicOut<R>(q.g, q.f.dU, 1 + line, r + 1, 1 + by) {}
        __device__ __forceinline__ void put(const DUY &q, const double *x) { PeriodicOut<R>::put(q.g, q.f.dU, R(x[0])); }
    };
};

// ---------------------------------------------------------------------------
// solvedV (:569-924): rows j = j_indexS(=2)..N2.  Stage 2 uses mu1, mu2 left
// by the last stage-1 iteration (i=N1, j=N2, k=N3); the y stage scales the
// upper coefficient by jvp = jS_BC(j-1) and the lower one by jvm = jS_BC(j+1).
// ---------------------------------------------------------------------------
template <class R>
struct DVZ {
    using Real = R;
    static constexpr int NRHS = 1;
    static constexpr int AHEAD = std::is_same<R, float>::value ? 1 : 0, TPS = 512, ROWS = 12, LGTI = 4;   // FP64 inputs of two rows do not fit the registers
    static constexpr bool LONG64 = std::is_same<R, double>::value;
    GridT<R> g; FieldsT<R> f;
    __device__ bool skip() const { return blown(g); }
    __device__ int lines() const { return g.N1; }
    // the rows of i that a plane needs in the column form
    static constexpr int NROW = 11, J0 = 2;
    static constexpr bool TABLES = true;
    __device__ static constexpr int row_dj(int q) { constexpr int v[] = {0, -1, 1, 0, -1, 0, -1, 0, -1, 0, -1}; return v[q]; }
    __device__ static constexpr int row_dk(int q) { constexpr int v[] = {1, 0, 0, 0, 0, 0, 0, 1, 1, 0, 0}; return v[q]; }
    __device__ __forceinline__ const R *row_src(int q) const
    {
        switch (q) {
        case 0: return f.V;
        case 1: return f.V;
        case 2: return f.V;
        case 3: return f.U;
        case 4: return f.U;
        case 5: return f.dU;
        case 6: return f.dU;
        case 7: return f.W;
        case 8: return f.W;
        case 9: return f.P;
        default: return f.P;
        }
    }
    // The reduced right-hand side (see DUZ), with solvedU's increment beside U in
    // every term (U + dU/2); on the planes next to the walls (j = 2, N2) the
    // reference masks the upper coefficient by jS_BC(j-1) and the lower one by
    // jS_BC(j+1).
    struct March {
        R cy, rdx1, rdmx1, rdmx1p, rdx2, rdx2m, rdmx2, dt;     // cy: weight of row j at y face j (row j-1: 1 - cy)
        R Vc, F, G, ma, wa;
        long long c;
        int t4, j;
        __device__ __forceinline__ March(const DVZ &q, int line, int by, int r0)
        {
            const GridT<R> &g = q.g;
            const FieldsT<R> &f = q.f;
            const int i = 1 + line, k = r0 + 1;
            j = 2 + by;
            rdx1 = ld(g.m1.rdx + i); rdmx1 = ld(g.m1.rdmx + i); rdmx1p = ld(g.m1.rdmx + i + 1);
            rdx2 = ld(g.m2.rdx + j); rdx2m = ld(g.m2.rdx + j - 1); rdmx2 = ld(g.m2.rdmx + j);
            cy = R(0.5) * ld(g.m2.dx + j - 1) * rdmx2;
            dt = R(g.scal[S_DT]);
            c = ix(g, i, j, k);
            t4 = 4 * ix2(g, j, k);
            Vc = ld(f.V + c);
            face(ld(f.V + c - (long long)g.P1 * g.P2), Vc, ld(f.W + c), ld(f.W + c - g.P1), ld(f.MuT + t4 + 3), ld(g.m3.rdmx + k));
        }
        __device__ __forceinline__ void face(R Vm, R Vp, R W0, R Wym, R mu, R rdmx3)
        {
            const R dw = W0 - Wym, w = Wym + cy * dw, dv = (Vp - Vm) * rdmx3;
            F = mu * (dv + dw * rdmx2);
            G = w * dv;
            ma = mu * rdmx3;
            wa = R(0.25) * w * rdmx3;
        }
        struct In { R Vxm, Vxp, Vym, Vyp, Vzp, U0, Uym, Uxp, Uxpym, D0, Dym, Dxp, Dxpym, Wzp, Wzpym, Pc, Pym, Mm, muz6, iR, rdx3, rdmx3; cplx_t<R> mt; };
        __device__ __forceinline__ void load(const DVZ &q, int r, In &n)
        {
            row_cell(q.g, c, t4);
            const GridT<R> &g = q.g;
            const FieldsT<R> &f = q.f;
            const long long sj = g.P1, sk = (long long)g.P1 * g.P2;
            n.Vxm = ld(f.V + c - 1); n.Vxp = ld(f.V + c + 1); n.Vym = ld(f.V + c - sj); n.Vyp = ld(f.V + c + sj); n.Vzp = ld(f.V + c + sk);
            n.U0 = ld(f.U + c); n.Uym = ld(f.U + c - sj); n.Uxp = ld(f.U + c + 1); n.Uxpym = ld(f.U + c + 1 - sj);
            n.D0 = ld(f.dU + c); n.Dym = ld(f.dU + c - sj); n.Dxp = ld(f.dU + c + 1); n.Dxpym = ld(f.dU + c + 1 - sj);
            n.Wzp = ld(f.W + c + sk); n.Wzpym = ld(f.W + c + sk - sj);
            n.Pc = ld(f.P + c); n.Pym = ld(f.P + c - sj);
            n.mt = ld2(f.MuT + t4);
            n.Mm = ld(f.MuT + t4 - 4); n.muz6 = ld(f.MuT + t4 + 4 * g.P2 + 3); n.iR = ld(f.iRT + t4 + 1);
            n.rdx3 = ld(g.m3.rdx + r + 1); n.rdmx3 = ld(g.m3.rdmx + r + 2);
            c += sk;
            t4 += 4 * g.P2;
        }
        // the same values from the ring: slot a holds plane k's rows, b the plane below's
        __device__ __forceinline__ void fill(const DVZ &q, int r, In &n, const double *a, const double *b, int w, int l)
        {
            const GridT<R> &g = q.g;
            const int s = w + 2;
            a += l + 1; b += l + 1;
            const double *const ta = a - (l + 1) + NROW * s, *const tb = b - (l + 1) + NROW * s;   // table words of planes k + 1 and k
            n.Vxm = b[-1]; n.Vxp = b[1]; n.Vzp = a[0]; n.Vym = a[s]; n.Vyp = a[2 * s];
            n.U0 = a[3 * s]; n.Uxp = a[3 * s + 1]; n.Uym = a[4 * s]; n.Uxpym = a[4 * s + 1];
            n.D0 = a[5 * s]; n.Dxp = a[5 * s + 1]; n.Dym = a[6 * s]; n.Dxpym = a[6 * s + 1];
            n.Wzp = a[7 * s]; n.Wzpym = a[8 * s];
            n.Pc = a[9 * s]; n.Pym = a[10 * s];
            n.mt.x = tb[4]; n.mt.y = tb[5]; n.Mm = tb[0]; n.muz6 = ta[7]; n.iR = tb[13];
            n.rdx3 = ld(g.m3.rdx + r + 1); n.rdmx3 = ld(g.m3.rdmx + r + 2);
        }
        __device__ __forceinline__ void row(const DVZ &q, int r, const In &n, double &a, double &b, double &cc, double *d)
        {
            const GridT<R> &g = q.g;
            const PhysT<R> &p = g.ph;
            const R Vxm = n.Vxm, Vxp = n.Vxp, Vym = n.Vym, Vyp = n.Vyp, Vzp = n.Vzp, U0 = n.U0, Uym = n.Uym, Uxp = n.Uxp, Uxpym = n.Uxpym;
            const R D0 = n.D0, Dym = n.Dym, Dxp = n.Dxp, Dxpym = n.Dxpym, Wzp = n.Wzp, Wzpym = n.Wzpym, Pc = n.Pc, Pym = n.Pym;
            const R Mm = n.Mm, muz6 = n.muz6, iR = n.iR;
            const cplx_t<R> mt = n.mt;
            const R rdx3 = n.rdx3;
            const R ih = R(0.5) * p.Cmu * iR;
            const R dx1 = (Vc - Vxm) * rdmx1, dx2 = (Vxp - Vc) * rdmx1p;
            const R v3 = R(0.5) * (Vym + Vc), v4 = R(0.5) * (Vc + Vyp);
            const R dy3 = (Vc - Vym) * rdx2m, dy4 = (Vyp - Vc) * rdx2;
            // differences of U and dU apart: U is the larger by orders of magnitude
            const R ds1 = (U0 - Uym) + R(0.5) * (D0 - Dym), ds2 = (Uxp - Uxpym) + R(0.5) * (Dxp - Dxpym);
            const R s1 = (Uym + R(0.5) * Dym) + cy * ds1, s2 = (Uxpym + R(0.5) * Dxpym) + cy * ds2;
            const R F5 = F, G5 = G, ma5 = ma, wa5 = wa, V0 = Vc;
            Vc = Vzp;
            face(V0, Vzp, Wzp, Wzpym, muz6, n.rdmx3);
            const R vs = mt.y * (((dx2 - dx1) + (ds2 - ds1) * rdmx2) * rdx1) + (F - F5) * rdx3 + R(2) * (mt.x * dy4 - Mm * dy3) * rdmx2;
            R rhs = R(2) * ih * vs - R(0.5) * ((s1 * dx1 + s2 * dx2) + (G5 + G) + (v3 * dy3 + v4 * dy4));
            rhs = rhs - p.Cmp * iR * (Pc - Pym) * rdmx2;
            if (j == 2) {
                const R ap = -R(2) * ih * rdmx2 * mt.x * rdx2 + R(0.25) * (v4 * rdx2 + R(0.5) * dy4);
                rhs = rhs + ap * (Vyp - p.Vup);
            }
            if (j == g.N2) {
                const R am = -R(2) * ih * rdmx2 * Mm * rdx2m + R(0.25) * (R(0.5) * dy3 - v3 * rdx2m);
                rhs = rhs + am * (Vym - p.Vbt);
            }
            const R h3 = ih * rdx3;
            const R am = -(h3 * ma5 + wa5) * dt, ap = (wa - h3 * ma) * dt;
            a = am; cc = ap; b = 1.0 - ((double)am + (double)ap);
            d[0] = rhs * dt;
        }
    };
    struct Out : ScratchOut<R> {
        __device__ __forceinline__ Out(const DVZ &q, int line, int by, int r) : ScratchOut<R>(q.g, q.f.scr, 1 + line, 2 + by, r + 1, (long long)q.g.P1 * q.g.P2) {}
        __device__ __forceinline__ void put(const DVZ &q, const double *x) { ScratchOut<R>::put(q.g, q.f.scr, R(x[0])); }
    };
};

// mu1, mu2 of solvedV's last stage-1 iteration (i = N1, j = N2, k = N3).
template <class R>
__device__ __forceinline__ void dv_stale_mu12(const GridT<R> &g, const FieldsT<R> &f, R &mu1, R &mu2)
{
    const int i = g.N1, j = g.N2, k = g.N3, im = i - 1, ip = i + 1, jm = j - 1;
    const R *dx1 = g.m1.dx, *dx2 = g.m2.dx, *rdmx1 = g.m1.rdmx, *rdmx2 = g.m2.rdmx;
    const R mxy = R(0.5) * (dx2[jm] * MU(j, k) + dx2[j] * MU(jm, k)) * rdmx2[j];
    mu1 = R(0.5) * (dx1[im] * mxy + dx1[i] * mxy) * rdmx1[i];
    mu2 = R(0.5) * (dx1[ip] * mxy + dx1[i] * mxy) * rdmx1[ip];
}

template <class R>
struct DVX {
    using Real = R;
    static constexpr int WORDS = 3, UNROLL = 4;
    GridT<R> g; FieldsT<R> f;
    __device__ bool skip() const { return blown(g); }
    __device__ int lines() const { return g.N2 - 1; }
    __device__ R *out(int line, int by) const { return f.scr + ix(g, 1, 2 + line, 1 + by); }
    struct Stage {
        long long c;
        R cy;
        __device__ __forceinline__ Stage(const DVX &q, int line, int by)
            : c(ix(q.g, 1, 2 + line, 1 + by)), cy(R(0.5) * ld(q.g.m2.dx + 1 + line) * ld(q.g.m2.rdmx + 2 + line)) {}
        __device__ __forceinline__ void put(const DVX &q, int r, double *w, int PL) const
        {
            TCS_OOB(q.g.scal, r < 0 || r >= q.g.N1, return);
            w[0] = (double)q.f.scr[c + r];
            const R U0 = ld(q.f.U + c + r), Um = ld(q.f.U + c + r - q.g.P1);
            w[PL] = (double)(Um + cy * (U0 - Um));
        }
    };
    struct March : FaceRows<R> {
        __device__ __forceinline__ March(const DVX &q, int line, int by, int r0, int m, int n, const double *w, int PL)
        {
            dv_stale_mu12(q.g, q.f, this->mu1, this->mu2);
            this->begin(q.g, R(0.5) * q.g.ph.Cmu * ld(q.f.iRT + 4 * ix2(q.g, 2 + line, 1 + by) + 1), r0, m, n, w, PL);
        }
        __device__ __forceinline__ void row(const DVX &q, int r, bool last, const double *w, int PL, double &a, double &b, double &c, double &d)
        {
            this->rows(q.g, r, last, w, PL, a, b, c, d);
        }
    };
};

template <class R>
struct DVY {
    using Real = R;
    static constexpr int NRHS = 1;
    static constexpr int AHEAD = 2, TPS = 512, ROWS = 16, LGTI = 4;
    static constexpr bool LONG64 = false;
    GridT<R> g; FieldsT<R> f;
    __device__ bool skip() const { return blown(g); }
    __device__ int lines() const { return g.N1; }
    struct March {
        R dt, Vc, A, B, C;                              // the cell below the row
        long long c;
        int t4;
        __device__ __forceinline__ March(const DVY &q, int line, int by, int r0)
        {
            const GridT<R> &g = q.g;
            const int i = 1 + line, j = r0 + 2, k = 1 + by;
            dt = R(g.scal[S_DT]);
            c = ix(g, i, j, k);
            t4 = 4 * ix2(g, j, k);
            Vc = ld(q.f.V + c);
            cell(ld(q.f.V + c - g.P1), Vc, ld(q.f.MuT + t4 - 4), ld(g.m2.rdx + j - 1));
        }
        __device__ __forceinline__ void cell(R Vm, R Vp, R mu, R rdx2)
        {
            A = mu * rdx2;
            B = R(0.125) * (Vm + Vp) * rdx2;
            C = R(0.125) * (Vp - Vm) * rdx2;
        }
        struct In { R V, mu, iR, rdx2, rdmx2, d; };
        __device__ __forceinline__ void load(const DVY &q, int r, In &n)
        {
            row_cell(q.g, c, t4);
            const long long sj = q.g.P1;
            n.V = ld(q.f.V + c + sj);
            n.mu = ld(q.f.MuT + t4); n.iR = ld(q.f.iRT + t4 + 1);
            n.rdx2 = ld(q.g.m2.rdx + r + 2); n.rdmx2 = ld(q.g.m2.rdmx + r + 2);
            n.d = q.f.scr[c];
            c += sj;
            t4 += 4;
        }
        __device__ __forceinline__ void row(const DVY &q, int r, const In &n, double &a, double &b, double &cc, double *d)
        {
            const R A3 = A, B3 = B, C3 = C, h = q.g.ph.Cmu * n.iR * n.rdmx2, V0 = Vc;
            Vc = n.V;
            cell(V0, n.V, n.mu, n.rdx2);
            const R am = (C3 - B3 - h * A3) * dt, ap = (B + C - h * A) * dt;
            // the upper coefficient carries the mask of the row below, the lower one that of the row above (:864-889)
            a = r == q.g.N2 - 2 ? R(0) : am; cc = r == 0 ? R(0) : ap;
            b = (1.0 - ((double)am + (double)ap)) + (double)(R(2) * (C3 + C) * dt);
            d[0] = n.d;
        }
    };
    struct Out : PeriodicOut<R> {
        __device__ __forceinline__ Out(const DVY &q, int line, int by, int r) : PeriodicOut<R>(q.g, q.f.dV, 1 + line, r + 2, 1 + by) {}
        __device__ __forceinline__ void put(const DVY &q, const double *x) { PeriodicOut<R>::put(q.g, q.f.dV, R(x[0])); }
    };
};

// ---------------------------------------------------------------------------
// solvedW (:930-1272).  Stage 2 uses stale mu1, mu2 and stage 3 stale mu3,
// mu4 (last stage-1 iteration) and a stale km = N3-1 (last stage-2 iteration).
// ---------------------------------------------------------------------------
template <class R>
struct DWZ {
    using Real = R;
    static constexpr int NRHS = 1;
    static constexpr int AHEAD = std::is_same<R, float>::value ? 1 : 0, TPS = 512, ROWS = 12, LGTI = 4;   // FP64 inputs of two rows do not fit the registers
    static constexpr bool LONG64 = std::is_same<R, double>::value;
    GridT<R> g; FieldsT<R> f;
    __device__ bool skip() const { return blown(g); }
    __device__ int lines() const { return g.N1; }
    // the rows of i that a plane needs in the column form
    static constexpr int NROW = 10, J0 = 1;
    static constexpr bool TABLES = true;
    __device__ static constexpr int row_dj(int q) { constexpr int v[] = {0, -1, 1, 0, 0, 0, 1, 0, 1, 0}; return v[q]; }
    __device__ static constexpr int row_dk(int q) { constexpr int v[] = {1, 0, 0, 0, 0, 0, 0, 0, 0, 0}; return v[q]; }
    __device__ __forceinline__ const R *row_src(int q) const
    {
        switch (q) {
        case 0: return f.W;
        case 1: return f.W;
        case 2: return f.W;
        case 3: return f.U;
        case 4: return f.dU;
        case 5: return f.V;
        case 6: return f.V;
        case 7: return f.dV;
        case 8: return f.dV;
        default: return f.P;
        }
    }
    // The reduced right-hand side (see DUZ), with the increments of solvedU and
    // solvedV beside U and V.
    struct March {
        R rdx1, rdmx1, rdmx1p, rdx2, rdmx2, rdmx2p, dt;
        R U0, Uxp, D0, Dxp, V0, Vyp, E0, Eyp, P0;       // the plane below: U, dU at i, i+1; V, dV at j, j+1; P
        R Wc, G, H, A, B, C, dx3;                       // the cell below (between W rows k-1 and k)
        long long c;
        int t4, j;
        __device__ __forceinline__ March(const DWZ &q, int line, int by, int r0)
        {
            const GridT<R> &g = q.g;
            const FieldsT<R> &f = q.f;
            const int i = 1 + line, k = r0 + 1;
            const long long sj = g.P1, sk = (long long)g.P1 * g.P2;
            j = 1 + by;
            rdx1 = ld(g.m1.rdx + i); rdmx1 = ld(g.m1.rdmx + i); rdmx1p = ld(g.m1.rdmx + i + 1);
            rdx2 = ld(g.m2.rdx + j); rdmx2 = ld(g.m2.rdmx + j); rdmx2p = ld(g.m2.rdmx + j + 1);
            dt = R(g.scal[S_DT]);
            c = ix(g, i, j, k);
            t4 = 4 * ix2(g, j, k);
            const long long cm = c - sk;
            U0 = ld(f.U + cm); Uxp = ld(f.U + cm + 1); D0 = ld(f.dU + cm); Dxp = ld(f.dU + cm + 1);
            V0 = ld(f.V + cm); Vyp = ld(f.V + cm + sj); E0 = ld(f.dV + cm); Eyp = ld(f.dV + cm + sj);
            P0 = ld(f.P + cm);
            Wc = ld(f.W + c);
            cell(ld(f.W + cm), Wc, ld(f.MuT + t4 - 4 * g.P2), ld(g.m3.dx + k - 1), ld(g.m3.rdx + k - 1));
        }
        // the cell between W rows k and k + 1
        __device__ __forceinline__ void cell(R Wm, R Wp, R mu, R dz, R rdx3)
        {
            dx3 = dz;
            const R w = R(0.5) * (Wm + Wp), dw = (Wp - Wm) * rdx3;
            G = w * dw;
            H = mu * dw;
            A = mu * rdx3;
            B = R(0.25) * w * rdx3;
            C = R(0.125) * dw;
        }
        struct In { R Wxm, Wxp, Wym, Wyp, Wzp, U, Ux, D, Dx, V, Vy, E, Ey, P, Mc, muyz4, iR, dx3, rdx3, rdmx3; cplx_t<R> mt; };
        __device__ __forceinline__ void load(const DWZ &q, int r, In &n)
        {
            row_cell(q.g, c, t4);
            const GridT<R> &g = q.g;
            const FieldsT<R> &f = q.f;
            const long long sj = g.P1, sk = (long long)g.P1 * g.P2;
            n.Wxm = ld(f.W + c - 1); n.Wxp = ld(f.W + c + 1); n.Wym = ld(f.W + c - sj); n.Wyp = ld(f.W + c + sj); n.Wzp = ld(f.W + c + sk);
            n.U = ld(f.U + c); n.Ux = ld(f.U + c + 1); n.D = ld(f.dU + c); n.Dx = ld(f.dU + c + 1);
            n.V = ld(f.V + c); n.Vy = ld(f.V + c + sj); n.E = ld(f.dV + c); n.Ey = ld(f.dV + c + sj);
            n.P = ld(f.P + c);
            n.Mc = ld(f.MuT + t4);
            n.mt = ld2(f.MuT + t4 + 2);                    // Mu at the lower z face, at the lower yz edge
            n.muyz4 = ld(f.MuT + t4 + 7); n.iR = ld(f.iRT + t4 + 2);
            n.dx3 = ld(g.m3.dx + r + 1); n.rdx3 = ld(g.m3.rdx + r + 1); n.rdmx3 = ld(g.m3.rdmx + r + 1);
            c += sk;
            t4 += 4 * g.P2;
        }
        // the same values from the ring: slot a holds plane k's rows, b the plane below's
        __device__ __forceinline__ void fill(const DWZ &q, int r, In &n, const double *a, const double *b, int w, int l)
        {
            const GridT<R> &g = q.g;
            const int s = w + 2;
            a += l + 1; b += l + 1;
            const double *const tb = b - (l + 1) + NROW * s;   // table words of plane k
            n.Wxm = b[-1]; n.Wxp = b[1]; n.Wzp = a[0]; n.Wym = a[s]; n.Wyp = a[2 * s];
            n.U = a[3 * s]; n.Ux = a[3 * s + 1]; n.D = a[4 * s]; n.Dx = a[4 * s + 1];
            n.V = a[5 * s]; n.Vy = a[6 * s]; n.E = a[7 * s]; n.Ey = a[8 * s];
            n.P = a[9 * s];
            n.Mc = tb[4]; n.mt.x = tb[6]; n.mt.y = tb[7]; n.muyz4 = tb[11]; n.iR = tb[14];
            n.dx3 = ld(g.m3.dx + r + 1); n.rdx3 = ld(g.m3.rdx + r + 1); n.rdmx3 = ld(g.m3.rdmx + r + 1);
        }
        __device__ __forceinline__ void row(const DWZ &q, int r, const In &n, double &a, double &b, double &cc, double *d)
        {
            const GridT<R> &g = q.g;
            const PhysT<R> &p = g.ph;
            const R Wxm = n.Wxm, Wxp = n.Wxp, Wym = n.Wym, Wyp = n.Wyp, Wzp = n.Wzp, nU = n.U, nUx = n.Ux, nD = n.D, nDx = n.Dx;
            const R nV = n.V, nVy = n.Vy, nE = n.E, nEy = n.Ey, nP = n.P, Mc = n.Mc, muyz4 = n.muyz4, iR = n.iR;
            const cplx_t<R> mt = n.mt;
            const R rdmx3 = n.rdmx3;
            const R dx3m = dx3, G5 = G, H5 = H, A5 = A, B5 = B, C5 = C, W0 = Wc;
            Wc = Wzp;
            cell(W0, Wzp, Mc, n.dx3, n.rdx3);
            const R cz = R(0.5) * dx3m * rdmx3;                            // weight of plane k at z face k (plane k-1: 1 - cz)
            const R ih = R(0.5) * p.Cmu * iR;
            const R dx1 = (W0 - Wxm) * rdmx1, dx2 = (Wxp - W0) * rdmx1p;
            const R dy3 = (W0 - Wym) * rdmx2, dy4 = (Wyp - W0) * rdmx2p;
            const R ds1 = (nU - U0) + R(0.5) * (nD - D0), ds2 = (nUx - Uxp) + R(0.5) * (nDx - Dxp);
            const R dv3 = nV - V0, dv4 = nVy - Vyp, de3 = nE - E0, de4 = nEy - Eyp;
            const R dt3 = dv3 + R(0.5) * de3, dt4 = dv4 + R(0.5) * de4;
            const R s1 = (U0 + R(0.5) * D0) + cz * ds1, s2 = (Uxp + R(0.5) * Dxp) + cz * ds2;
            const R t3 = (V0 + R(0.5) * E0) + cz * dt3, t4_ = (Vyp + R(0.5) * Eyp) + cz * dt4;
            const R mu3 = mt.y, mu4 = muyz4;
            const R vs = mt.x * (((dx2 - dx1) + (ds2 - ds1) * rdmx3) * rdx1) + (mu4 * (dy4 + dt4 * rdmx3) - mu3 * (dy3 + dt3 * rdmx3)) * rdx2 + R(2) * (H - H5) * rdmx3;
            R rhs = R(2) * ih * vs - R(0.5) * ((s1 * dx1 + s2 * dx2) + (t3 * dy3 + t4_ * dy4) + (G5 + G));
            rhs = rhs - p.Cmp * iR * (nP - P0) * rdmx3;
            if (j == 1) {
                const R v3 = V0 + cz * dv3, am = -(ih * rdx2 * mu3 + R(0.25) * v3) * rdmx2;
                rhs = rhs + am * Wym + (R(0.5) * t3 - R(0.25) * v3) * dy3 + ih * rdx2 * mu3 * ((dv3 + de3) * rdmx3);
                rhs = rhs + R(0.25) * v3 * rdmx2 * p.Wbt - R(0.25) * dy3 * p.Vbt + ih * rdx2 * mu3 * rdmx2p * p.Wbt;
            }
            if (j == g.N2) {
                const R v4 = Vyp + cz * dv4, ap = (R(0.25) * v4 - ih * rdx2 * mu4) * rdmx2p;
                rhs = rhs + ap * Wyp + (R(0.5) * t4_ - R(0.25) * v4) * dy4 - ih * rdx2 * mu4 * ((dv4 + de4) * rdmx3);
                rhs = rhs - R(0.25) * v4 * rdmx2p * p.Wup - R(0.25) * dy4 * p.Vup + ih * rdx2 * mu4 * rdmx2 * p.Wup;
            }
            const R h3 = R(2) * ih * rdmx3;
            const R am = (C5 - B5 - h3 * A5) * dt, ap = (B + C - h3 * A) * dt;
            a = am; cc = ap; b = (1.0 - ((double)am + (double)ap)) + (double)(R(2) * (C5 + C) * dt);
            d[0] = rhs * dt;
            U0 = nU; Uxp = nUx; D0 = nD; Dxp = nDx; V0 = nV; Vyp = nVy; E0 = nE; Eyp = nEy; P0 = nP;
        }
    };
    struct Out : ScratchOut<R> {
        __device__ __forceinline__ Out(const DWZ &q, int line, int by, int r) : ScratchOut<R>(q.g, q.f.scr, 1 + line, 1 + by, r + 1, (long long)q.g.P1 * q.g.P2) {}
        __device__ __forceinline__ void put(const DWZ &q, const double *x) { ScratchOut<R>::put(q.g, q.f.scr, R(x[0])); }
    };
};

// mu1..mu4 of solvedW's last stage-1 iteration (i = N1, j = N2, k = N3).
template <class R>
__device__ __forceinline__ void dw_stale_mu(const GridT<R> &g, const FieldsT<R> &f, R &mu1, R &mu2, R &mu3, R &mu4)
{
    const int i = g.N1, j = g.N2, k = g.N3, im = i - 1, ip = i + 1, jm = j - 1, jp = j + 1, km = k - 1;
    const R *dx1 = g.m1.dx, *dx2 = g.m2.dx, *dx3 = g.m3.dx;
    const R *rdmx1 = g.m1.rdmx, *rdmx2 = g.m2.rdmx, *rdmx3 = g.m3.rdmx;
    const R mxz = R(0.5) * (dx3[km] * MU(j, k) + dx3[k] * MU(j, km)) * rdmx3[k];
    mu1 = R(0.5) * (dx1[im] * mxz + dx1[i] * mxz) * rdmx1[i];
    mu2 = R(0.5) * (dx1[ip] * mxz + dx1[i] * mxz) * rdmx1[ip];
    const R mua = R(0.5) * (dx3[km] * MU(jm, k) + dx3[k] * MU(jm, km)) * rdmx3[k];
    const R mub = R(0.5) * (dx3[km] * MU(jp, k) + dx3[k] * MU(jp, km)) * rdmx3[k];
    mu3 = R(0.5) * (dx2[jm] * mxz + dx2[j] * mua) * rdmx2[j];
    mu4 = R(0.5) * (dx2[jp] * mxz + dx2[j] * mub) * rdmx2[jp];
}

template <class R>
struct DWX {
    using Real = R;
    static constexpr int WORDS = 3, UNROLL = 4;
    GridT<R> g; FieldsT<R> f;
    __device__ bool skip() const { return blown(g); }
    __device__ int lines() const { return g.N2; }
    __device__ R *out(int line, int by) const { return f.scr + ix(g, 1, 1 + line, 1 + by); }
    struct Stage {
        long long c, sk;
        R cz;
        __device__ __forceinline__ Stage(const DWX &q, int line, int by)
            : c(ix(q.g, 1, 1 + line, 1 + by)), sk((long long)q.g.P1 * q.g.P2), cz(R(0.5) * ld(q.g.m3.dx + by) * ld(q.g.m3.rdmx + 1 + by)) {}
        __device__ __forceinline__ void put(const DWX &q, int r, double *w, int PL) const
        {
            TCS_OOB(q.g.scal, r < 0 || r >= q.g.N1, return);
            w[0] = (double)q.f.scr[c + r];
            const R U0 = ld(q.f.U + c + r), Um = ld(q.f.U + c + r - sk);
            w[PL] = (double)(Um + cz * (U0 - Um));
        }
    };
    struct March : FaceRows<R> {
        __device__ __forceinline__ March(const DWX &q, int line, int by, int r0, int m, int n, const double *w, int PL)
        {
            R mu3, mu4;
            dw_stale_mu(q.g, q.f, this->mu1, this->mu2, mu3, mu4);
            this->begin(q.g, R(0.5) * q.g.ph.Cmu * ld(q.f.iRT + 4 * ix2(q.g, 1 + line, 1 + by) + 2), r0, m, n, w, PL);
        }
        __device__ __forceinline__ void row(const DWX &q, int r, bool last, const double *w, int PL, double &a, double &b, double &c, double &d)
        {
            this->rows(q.g, r, last, w, PL, a, b, c, d);
        }
    };
};

template <class R>
struct DWY {
    using Real = R;
    static constexpr int NRHS = 1;
    static constexpr int AHEAD = 2, TPS = 512, ROWS = 16, LGTI = 4;
    static constexpr bool LONG64 = false;
    GridT<R> g; FieldsT<R> f;
    __device__ bool skip() const { return blown(g); }
    __device__ int lines() const { return g.N1; }
    struct March {
        R z0, z1, mu3, mu4, dt, w, rdmx2;               // z0, z1: weights of planes k and N3-1; w: convection at the face below the row
        long long c, dk;
        int t4, t4k;
        __device__ __forceinline__ March(const DWY &q, int line, int by, int r0)
        {
            const GridT<R> &g = q.g;
            const int i = 1 + line, j = r0 + 1, k = 1 + by, km = g.N3 - 1;
            R mu1, mu2;
            dw_stale_mu(g, q.f, mu1, mu2, mu3, mu4);
            const R h = R(0.5) * ld(g.m3.rdmx + k);
            z0 = h * ld(g.m3.dx + km); z1 = h * ld(g.m3.dx + k);
            dt = R(g.scal[S_DT]);
            c = ix(g, i, j, k);
            dk = (long long)g.P1 * g.P2 * (km - k);
            t4 = 4 * ix2(g, j, k);
            t4k = 4 * g.P2 * (km - k);
            face(ld(q.f.V + c), ld(q.f.V + c + dk), ld(g.m2.rdmx + j));
        }
        __device__ __forceinline__ void face(R V, R Vk, R rd)
        {
            rdmx2 = rd;
            w = R(0.25) * (z0 * V + z1 * Vk) * rd;
        }
        struct In { R V, Vk, iR, iRk, rdx2, rdmx2, d; };
        __device__ __forceinline__ void load(const DWY &q, int r, In &n)
        {
            row_cell(q.g, c, t4);
            const long long sj = q.g.P1;
            TCS_OOB(q.g.scal, c + dk < 0 || c + sj + dk >= q.g.NP, (dk = 0, t4k = 0));
            n.V = ld(q.f.V + c + sj); n.Vk = ld(q.f.V + c + sj + dk);
            n.iR = ld(q.f.iRT + t4); n.iRk = ld(q.f.iRT + t4 + t4k);
            n.rdx2 = ld(q.g.m2.rdx + r + 1); n.rdmx2 = ld(q.g.m2.rdmx + r + 2);
            n.d = q.f.scr[c];
            c += sj;
            t4 += 4;
        }
        __device__ __forceinline__ void row(const DWY &q, int r, const In &n, double &a, double &b, double &cc, double *d)
        {
            const R w3 = w, m3 = mu3 * rdmx2, h = R(0.5) * q.g.ph.Cmu * (z0 * n.iR + z1 * n.iRk) * n.rdx2;
            face(n.V, n.Vk, n.rdmx2);
            const R am = -(h * m3 + w3) * dt, ap = (w - h * (mu4 * rdmx2)) * dt;
            a = r == 0 ? R(0) : am; cc = r == q.g.N2 - 1 ? R(0) : ap; b = 1.0 - ((double)am + (double)ap);
            d[0] = n.d;
        }
    };
    struct Out : PeriodicOut<R> {
        __device__ __forceinline__ Out(const DWY &q, int line, int by, int r) : PeriodicOut<R>(q.g, q.f.dW, 1 + line, r + 1, 1 + by) {}
        __device__ __forceinline__ void put(const DWY &q, const double *x) { PeriodicOut<R>::put(q.g, q.f.dW, R(x[0])); }
    };
};

template <class R>
static void launch_du_z(const Ctx<R> &cx, cudaStream_t s)
{
    launch_march(cx, DUZ<R>{cx.g, cx.f}, cx.g.N3, true, cx.g.N1, cx.g.N2, s, K_DU_Z);
}
template <class R>
static void launch_dv_z(const Ctx<R> &cx, cudaStream_t s)
{
    launch_march(cx, DVZ<R>{cx.g, cx.f}, cx.g.N3, true, cx.g.N1, cx.g.N2 - 1, s, K_DV_Z);
}
template <class R>
static void launch_dw_z(const Ctx<R> &cx, cudaStream_t s)
{
    launch_march(cx, DWZ<R>{cx.g, cx.f}, cx.g.N3, true, cx.g.N1, cx.g.N2, s, K_DW_Z);
}

template <class R>
static void launch_du_y(const Ctx<R> &cx, cudaStream_t s)
{
    launch_march(cx, DUY<R>{cx.g, cx.f}, cx.g.N2, false, cx.g.N1, cx.g.N3, s, K_DU_Y);
}

template <class R>
static void launch_dv_y(const Ctx<R> &cx, cudaStream_t s)
{
    launch_march(cx, DVY<R>{cx.g, cx.f}, cx.g.N2 - 1, false, cx.g.N1, cx.g.N3, s, K_DV_Y);
}

template <class R>
static void launch_dw_y(const Ctx<R> &cx, cudaStream_t s)
{
    launch_march(cx, DWY<R>{cx.g, cx.f}, cx.g.N2, false, cx.g.N1, cx.g.N3, s, K_DW_Y);
}

template <class R>
static void launch_du_x(const Ctx<R> &cx, cudaStream_t s)
{
    launch_xmarch(cx, DUX<R>{cx.g, cx.f}, cx.g.N1, cx.g.N2, cx.g.N3, s, K_DU_X);
}

template <class R>
static void launch_dv_x(const Ctx<R> &cx, cudaStream_t s)
{
    launch_xmarch(cx, DVX<R>{cx.g, cx.f}, cx.g.N1, cx.g.N2 - 1, cx.g.N3, s, K_DV_X);
}

template <class R>
static void launch_dw_x(const Ctx<R> &cx, cudaStream_t s)
{
    launch_xmarch(cx, DWX<R>{cx.g, cx.f}, cx.g.N1, cx.g.N2, cx.g.N3, s, K_DW_X);
}

template <class R>
void launch_solve_du(const Ctx<R> &cx, cudaStream_t s)
{
    launch_du_z(cx, s);
    launch_du_x(cx, s);
    launch_du_y(cx, s);
}

template <class R>
void launch_solve_dv(const Ctx<R> &cx, cudaStream_t s)
{
    launch_dv_z(cx, s);
    launch_dv_x(cx, s);
    launch_dv_y(cx, s);
}

template <class R>
void launch_solve_dw(const Ctx<R> &cx, cudaStream_t s)
{
    launch_dw_z(cx, s);
    launch_dw_x(cx, s);
    launch_dw_y(cx, s);
}

// ---------------------------------------------------------------------------
// blockLdV (:1278-1356): dV -= dt*M23 dW, j = 2..N2, then ghost(dV).
// ---------------------------------------------------------------------------
template <class R>
__device__ __forceinline__ R blockld_v_value(const GridT<R> &g, const FieldsT<R> &f, int i, int j, int k)
{
    const int jm = j - 1, kp = k + 1;
    const R *dx2 = g.m2.dx, *rdx3 = g.m3.rdx, *rdmx2 = g.m2.rdmx, *rdmx3 = g.m3.rdmx;
    const long long c = ix(g, i, j, k), sj = g.P1, sk = (long long)g.P1 * g.P2;
    const R dWc = ld(f.dW + c), dWym = ld(f.dW + c - sj), dWzp = ld(f.dW + c + sk), dWzpym = ld(f.dW + c + sk - sj);
    const R dwm5 = (dx2[jm] * dWc + dx2[j] * dWym) * rdmx2[j] * R(0.5);
    const R dwm6 = (dx2[jm] * dWzp + dx2[j] * dWzpym) * rdmx2[j] * R(0.5);
    const R ddwdy5 = (dWc - dWym) * rdmx2[j], ddwdy6 = (dWzp - dWzpym) * rdmx2[j];
    const R Vc = ld(f.V + c);
    const R dvdz5 = (Vc - ld(f.V + c - sk)) * rdmx3[k], dvdz6 = (ld(f.V + c + sk) - Vc) * rdmx3[kp];
    const int t4 = 4 * ix2(g, j, k);
    const R invRhoc = ld(f.iRT + t4 + 1), mu5 = ld(f.MuT + t4 + 3), mu6 = ld(f.MuT + t4 + 4 * g.P2 + 3);   // at the y face and the yz edges
    const R dt = g.scal[S_DT];
    return f.dV[c] - dt * (R(0.25) * (dwm5 * dvdz5 + dwm6 * dvdz6) - R(0.5) * g.ph.Cmu * invRhoc * rdx3[k] * (mu6 * ddwdy6 - mu5 * ddwdy5));
}

// Mu and invRho at the faces come from the table (MuT, iRT): 256^3 9.4 -> 7.6 ps
// per cell, FP32-mixed 7.6 -> 5.7, against forming them from the cells.
// KZ planes per thread: every input of the KZ cells is loaded before the first store
template <class R, int KZ>
__global__ void blockld_v_kernel(GridT<R> g, FieldsT<R> f)
{
    const int i = 1 + blockIdx.x * blockDim.x + threadIdx.x, j = 2 + blockIdx.y, k0 = 1 + KZ * blockIdx.z;
    if (i > g.N1 || blown(g)) return;
    R v[KZ];
#pragma unroll
    for (int q = 0; q < KZ; q++) v[q] = k0 + q <= g.N3 ? blockld_v_value(g, f, i, j, k0 + q) : R(0);
#pragma unroll
    for (int q = 0; q < KZ; q++)
        if (k0 + q <= g.N3) store_periodic(g, f.dV, i, j, k0 + q, v[q]);
}

template <class R>
void launch_blockld_v(const Ctx<R> &cx, cudaStream_t s)
{
    const GridT<R> &g = cx.g;
    probe_begin(cx, K_BLOCKLDV, s);
    blockld_v_kernel<R, 2><<<dim3((g.N1 + 127) / 128, g.N2 - 1, (g.N3 + 1) / 2), 128, 0, s>>>(g, cx.f);
    probe_end(cx, K_BLOCKLDV, s);
    record_launch_error("blockld_v");
}

// blockLdU (:1362-1460): dU -= dt*(M12 dV + M13 dW), j = 1..N2 (no ghost
// update follows in the driver; only interior dU is read afterwards).
template <class R>
__device__ __forceinline__ R blockld_u_value(const GridT<R> &g, const FieldsT<R> &f, int i, int j, int k)
{
    const int im = i - 1, jp = j + 1, kp = k + 1;
    const R *dx1 = g.m1.dx, *rdx2 = g.m2.rdx, *rdx3 = g.m3.rdx;
    const R *rdmx1 = g.m1.rdmx, *rdmx2 = g.m2.rdmx, *rdmx3 = g.m3.rdmx;
    const long long c = ix(g, i, j, k), sj = g.P1, sk = (long long)g.P1 * g.P2;
    const R jum = (j == 1) ? R(0.0) : R(1.0), jup = (j == g.N2) ? R(0.0) : R(1.0);
    // Mu and invRho are constant along i: the table's y and z faces
    const int t4 = 4 * ix2(g, j, k);
    const R invRhoc = ld(f.iRT + t4), mu3 = ld(f.MuT + t4 + 1), mu4 = ld(f.MuT + t4 + 5), mu5 = ld(f.MuT + t4 + 2), mu6 = ld(f.MuT + t4 + 4 * g.P2 + 2);
    const R dVc = ld(f.dV + c), dVxm = ld(f.dV + c - 1), dVyp = ld(f.dV + c + sj), dVxmyp = ld(f.dV + c - 1 + sj);
    const R dvm3 = (dx1[i] * dVxm + dx1[im] * dVc) * rdmx1[i] * R(0.5) * jum;
    const R dvm4 = (dx1[i] * dVxmyp + dx1[im] * dVyp) * rdmx1[i] * R(0.5) * jup;
    const R Uc = ld(f.U + c);
    const R dudy3 = (Uc - ld(f.U + c - sj)) * rdmx2[j], dudy4 = (ld(f.U + c + sj) - Uc) * rdmx2[jp];
    const R dvmdx3 = (dVc - dVxm) * rdmx1[i] * jum, dvmdx4 = (dVyp - dVxmyp) * rdmx1[i] * jup;
    const R dWc = ld(f.dW + c), dWxm = ld(f.dW + c - 1), dWzp = ld(f.dW + c + sk), dWxmzp = ld(f.dW + c - 1 + sk);
    const R dwm5 = (dx1[i] * dWxm + dx1[im] * dWc) * rdmx1[i] * R(0.5);
    const R dwm6 = (dx1[i] * dWxmzp + dx1[im] * dWzp) * rdmx1[i] * R(0.5);
    const R dudz5 = (Uc - ld(f.U + c - sk)) * rdmx3[k], dudz6 = (ld(f.U + c + sk) - Uc) * rdmx3[kp];
    const R dwmdx5 = (dWc - dWxm) * rdmx1[i], dwmdx6 = (dWzp - dWxmzp) * rdmx1[i];
    const R dt = g.scal[S_DT], Cmu = g.ph.Cmu;
    return f.dU[c]
        - dt * (R(0.25) * (dvm4 * dudy4 + dvm3 * dudy3) - R(0.5) * Cmu * invRhoc * rdx2[j] * (mu4 * dvmdx4 - mu3 * dvmdx3))
        - dt * (R(0.25) * (dwm6 * dudz6 + dwm5 * dudz5) - R(0.5) * Cmu * invRhoc * rdx3[k] * (mu6 * dwmdx6 - mu5 * dwmdx5));
}

// KZ planes per thread: every input of the KZ cells is loaded before the first store.
// Bound by its load latency.  With the face tables and no bound it ran slower than the
// kernel before the tables, which formed the faces: the FP32 form at 40 registers and 45
// warps per SM (us, before, unbounded, and with 16 blocks of 32 registers and 60 warps:
// 256^3 160, 162, 117; 400 x 200 x 384 306, 318, 220), the FP64 form at 48, too few to
// have a cell's loads on their way at once (256^3 216, 222 and, at up to 64, with 29 warps
// instead of 38, 195; 180 x 151 x 250 107, 111, 99).
template <class R, int KZ>
__global__ void __launch_bounds__(128, HasLo<R>::on ? 16 : 8) blockld_u_kernel(GridT<R> g, FieldsT<R> f)
{
    const int i = 1 + blockIdx.x * blockDim.x + threadIdx.x, j = 1 + blockIdx.y, k0 = 1 + KZ * blockIdx.z;
    if (i > g.N1 || blown(g)) return;
    R v[KZ];
#pragma unroll
    for (int q = 0; q < KZ; q++) v[q] = k0 + q <= g.N3 ? blockld_u_value(g, f, i, j, k0 + q) : R(0);
    const long long sk = (long long)g.P1 * g.P2;
#pragma unroll
    for (int q = 0; q < KZ; q++)
        if (k0 + q <= g.N3) f.dU[ix(g, i, j, k0) + q * sk] = v[q];
}

template <class R>
void launch_blockld_u(const Ctx<R> &cx, cudaStream_t s)
{
    const GridT<R> &g = cx.g;
    probe_begin(cx, K_BLOCKLDU, s);
    blockld_u_kernel<R, 2><<<dim3((g.N1 + 127) / 128, g.N2, (g.N3 + 1) / 2), 128, 0, s>>>(g, cx.f);
    probe_end(cx, K_BLOCKLDU, s);
    record_launch_error("blockld_u");
}

// Standalone mpi_momentum_pseudoupdateUVW (:178-208) + ghost(U,V,W): writes the
// second buffers; the caller swaps them in.  The step normally fuses this into
// the pressure right-hand side (tcs_pressure.cu).
template <class R>
__global__ void pseudo_update_kernel(GridT<R> g, FieldsT<R> f)
{
    const int i = 1 + blockIdx.x * blockDim.x + threadIdx.x, j = 1 + blockIdx.y, k = 1 + blockIdx.z;
    if (i > g.N1 || blown(g)) return;
    const long long c = ix(g, i, j, k);
    const R vmask = (j == 1) ? R(0.0) : R(1.0);     // dble(2 - j_indexS) on the lower plane
    if constexpr (HasLo<R>::on) {                    // FP32 form: FP64 sums of the high/low pairs
        float h, lo;
        split(join(f.U[c], f.Ulo[c]) + (double)f.dU[c], h, lo);
        store_periodic(g, f.Un, i, j, k, h); store_periodic(g, f.Unlo, i, j, k, lo);
        split(join(f.V[c], f.Vlo[c]) + (double)f.dV[c] * (double)vmask, h, lo);
        store_periodic(g, f.Vn, i, j, k, h); store_periodic(g, f.Vnlo, i, j, k, lo);
        split(join(f.W[c], f.Wlo[c]) + (double)f.dW[c], h, lo);
        store_periodic(g, f.Wn, i, j, k, h); store_periodic(g, f.Wnlo, i, j, k, lo);
    } else {
        store_periodic(g, f.Un, i, j, k, f.U[c] + f.dU[c]);
        store_periodic(g, f.Vn, i, j, k, f.V[c] + f.dV[c] * vmask);
        store_periodic(g, f.Wn, i, j, k, f.W[c] + f.dW[c]);
    }
}

template <class R>
void launch_pseudo_update(const Ctx<R> &cx, cudaStream_t s)
{
    const GridT<R> &g = cx.g;
    probe_begin(cx, K_PSEUDO, s);
    pseudo_update_kernel<<<dim3((g.N1 + 127) / 128, g.N2, g.N3), 128, 0, s>>>(g, cx.f);
    probe_end(cx, K_PSEUDO, s);
    record_launch_error("pseudo_update");
}

#undef MU

// The nine sweeps of solvedU, solvedV and solvedW for many cases, sweep by sweep (march_stage).
template <class R>
void launch_momentum_multi(const std::vector<Ctx<R> *> &cs, MultiArena &A, cudaStream_t s)
{
    march_stage(cs, A, s, launch_du_z<R>);
    march_stage(cs, A, s, launch_du_x<R>);
    march_stage(cs, A, s, launch_du_y<R>);
    march_stage(cs, A, s, launch_dv_z<R>);
    march_stage(cs, A, s, launch_dv_x<R>);
    march_stage(cs, A, s, launch_dv_y<R>);
    march_stage(cs, A, s, launch_dw_z<R>);
    march_stage(cs, A, s, launch_dw_x<R>);
    march_stage(cs, A, s, launch_dw_y<R>);
}

// the two forms
template void launch_momentum_multi<double>(const std::vector<Ctx<double> *> &, MultiArena &, cudaStream_t);
template void launch_momentum_multi<float>(const std::vector<Ctx<float> *> &, MultiArena &, cudaStream_t);
template void launch_momentum_coeffi<double>(const Ctx<double> &, cudaStream_t);
template void launch_momentum_coeffi<float>(const Ctx<float> &, cudaStream_t);
template void launch_solve_du<double>(const Ctx<double> &, cudaStream_t);
template void launch_solve_du<float>(const Ctx<float> &, cudaStream_t);
template void launch_solve_dv<double>(const Ctx<double> &, cudaStream_t);
template void launch_solve_dv<float>(const Ctx<float> &, cudaStream_t);
template void launch_solve_dw<double>(const Ctx<double> &, cudaStream_t);
template void launch_solve_dw<float>(const Ctx<float> &, cudaStream_t);
template void launch_blockld_v<double>(const Ctx<double> &, cudaStream_t);
template void launch_blockld_v<float>(const Ctx<float> &, cudaStream_t);
template void launch_blockld_u<double>(const Ctx<double> &, cudaStream_t);
template void launch_blockld_u<float>(const Ctx<float> &, cudaStream_t);
template void launch_pseudo_update<double>(const Ctx<double> &, cudaStream_t);
template void launch_pseudo_update<float>(const Ctx<float> &, cudaStream_t);

} // namespace tcs
