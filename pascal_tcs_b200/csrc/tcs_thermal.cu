// tcs_thermal.cu -- energy equation: mpi_thermal_coeffi + mpi_thermal_solver
// (module_solve_thermal.f90:116-532) as three fused kernels, one per ADI
// sweep (tcs_march.cuh).  Each evaluates the temperature-dependent properties
// at the stencil points it needs, builds the tridiagonal rows and solves its
// lines; only the sweep result goes to HBM.
//
//   z sweep  (:236-366) lines (i,j), rows k, cyclic   -> R
//   x sweep  (:388-434) lines (j,k), rows i, cyclic   R -> R
//   y sweep  (:456-524) lines (i,k), rows j           R -> Tn = T + R (+ ghosts)
//
// Divisions by metric quantities are multiplications by reciprocal tables.
#include "tcs_kernels.h"

namespace tcs {

template <class R>
struct ThermalZ {
    using Real = R;
    static constexpr int NRHS = 1;
    static constexpr int AHEAD = std::is_same<R, float>::value ? 1 : 0, TPS = 512, ROWS = 12, LGTI = 4;   // FP64 inputs of two rows do not fit the registers
    static constexpr bool LONG64 = std::is_same<R, double>::value;
    GridT<R> g; FieldsT<R> f;
    __device__ bool skip() const { return blown(g); }
    __device__ int lines() const { return g.N1; }
    // the rows of i that a plane needs in the column form
    static constexpr int NROW = 7, J0 = 1;
    static constexpr bool TABLES = false;
    __device__ static constexpr int row_dj(int q) { constexpr int v[] = {0, -1, 1, 0, 0, 1, 0}; return v[q]; }
    __device__ static constexpr int row_dk(int q) { constexpr int v[] = {1, 0, 0, 0, 0, 0, 1}; return v[q]; }
    __device__ __forceinline__ const R *row_src(int q) const
    {
        switch (q) {
        case 0: return f.T;
        case 1: return f.T;
        case 2: return f.T;
        case 3: return f.U;
        case 4: return f.V;
        case 5: return f.V;
        default: return f.W;
        }
    }
    // The right-hand side of :236-361 is the explicit operator minus the three
    // implicit operators applied to T.  Expanded, per direction d with faces
    // -/+ (kPP the face conductivity, ded the face gradient, u the face
    // velocity), the dK/dT products (e dkPP ded) of the explicit operator and
    // of the implicit one cancel, and so do the two dh Tc dv terms, leaving
    //   2 h rdx_d (kPP+ ded+ - kPP- ded-) - (u- ded- + u+ ded+) / 2.
    // On the two wall-adjacent planes (j = 1, N2) the jC_BC masks and the wall
    // terms break that in y; the difference is added there.  The z rows (am,
    // ac, ap) are the reference's, dK/dT terms included.
    struct March {
        R rdx1, rdx2, rdmx1, rdmx1p, rdmx2, rdmx2p, w1, w2, w3, w4, dt;   // w: weight of the neighbour at the x (1, 2) and y (3, 4) faces
        R Tc, Kc, dKc, F, G, s, q, w, dx3m, dx3;     // the cell; the face below it
        long long c;
        int j;
        __device__ __forceinline__ March(const ThermalZ &o, int line, int by, int r0)
        {
            const GridT<R> &g = o.g;
            const int i = 1 + line, k = r0 + 1;
            j = 1 + by;
            const R d1 = ld(g.m1.dx + i), d2 = ld(g.m2.dx + j);
            rdx1 = ld(g.m1.rdx + i); rdx2 = ld(g.m2.rdx + j);
            rdmx1 = ld(g.m1.rdmx + i); rdmx1p = ld(g.m1.rdmx + i + 1);
            rdmx2 = ld(g.m2.rdmx + j); rdmx2p = ld(g.m2.rdmx + j + 1);
            w1 = R(0.5) * rdmx1 * d1; w2 = R(0.5) * rdmx1p * d1; w3 = R(0.5) * rdmx2 * d2; w4 = R(0.5) * rdmx2p * d2;
            dt = R(g.scal[S_DT]);
            c = ix(g, i, j, k);
            dx3 = ld(g.m3.dx + k - 1);
            Tc = ld(o.f.T + c - (long long)g.P1 * g.P2);
            kpp_eval(g.ph, g.kdeg2 != 0, Tc, Kc, dKc);
            face(o, ld(o.f.T + c), ld(o.f.W + c), ld(g.m3.dx + k), ld(g.m3.rdmx + k));
        }
        // the z face between planes k-1 (Tc, Kc, dKc, dx3) and k, which becomes the current plane
        __device__ __forceinline__ void face(const ThermalZ &o, R Tp, R Wp, R dz, R rdmx3)
        {
            const GridT<R> &g = o.g;
            R Kp, dKp;
            kpp_eval(g.ph, g.kdeg2 != 0, Tp, Kp, dKp);
            dx3m = dx3;
            dx3 = dz;
            const R hm = R(0.5) * rdmx3, wm = hm * dx3m, de = (Tp - Tc) * rdmx3;
            const R kPP = Kc + wm * (Kp - Kc), dkPP = dKc + wm * (dKp - dKc);
            F = kPP * de;
            G = Wp * de;
            s = kPP * rdmx3;
            q = hm * (dkPP * de);
            w = R(0.25) * Wp * rdmx3;
            Tc = Tp; Kc = Kp; dKc = dKp;
        }
        struct In { R Txm, Txp, Tym, Typ, Tzp, Uc, Uxp, Vc, Vyp, Wzp, rdx3, dx3, rdmx3; };
        __device__ __forceinline__ void load(const ThermalZ &o, int r, In &n)
        {
            row_cell(o.g, c);
            const GridT<R> &g = o.g;
            const FieldsT<R> &f = o.f;
            const long long sj = g.P1, sk = (long long)g.P1 * g.P2;
            n.Txm = ld(f.T + c - 1); n.Txp = ld(f.T + c + 1); n.Tym = ld(f.T + c - sj); n.Typ = ld(f.T + c + sj); n.Tzp = ld(f.T + c + sk);
            n.Uc = ld(f.U + c); n.Uxp = ld(f.U + c + 1); n.Vc = ld(f.V + c); n.Vyp = ld(f.V + c + sj); n.Wzp = ld(f.W + c + sk);
            n.rdx3 = ld(g.m3.rdx + r + 1); n.dx3 = ld(g.m3.dx + r + 2); n.rdmx3 = ld(g.m3.rdmx + r + 2);
            c += sk;
        }
        // the same values from the ring: slot a holds plane k's rows, b the plane below's
        __device__ __forceinline__ void fill(const ThermalZ &o, int r, In &n, const double *a, const double *b, int w, int l)
        {
            const GridT<R> &g = o.g;
            const int s = w + 2;
            a += l + 1; b += l + 1;
            n.Txm = b[-1]; n.Txp = b[1]; n.Tzp = a[0]; n.Tym = a[s]; n.Typ = a[2 * s];
            n.Uc = a[3 * s]; n.Uxp = a[3 * s + 1]; n.Vc = a[4 * s]; n.Vyp = a[5 * s]; n.Wzp = a[6 * s];
            n.rdx3 = ld(g.m3.rdx + r + 1); n.dx3 = ld(g.m3.dx + r + 2); n.rdmx3 = ld(g.m3.rdmx + r + 2);
        }
        __device__ __forceinline__ void row(const ThermalZ &o, int r, const In &n, double &a, double &b, double &cc, double *d)
        {
            const GridT<R> &g = o.g;
            const PhysT<R> &p = g.ph;
            const bool d2 = g.kdeg2 != 0;
            const R Txm = n.Txm, Txp = n.Txp, Tym = n.Tym, Typ = n.Typ, Tzp = n.Tzp, Uc = n.Uc, Uxp = n.Uxp, Vc = n.Vc, Vyp = n.Vyp, Wzp = n.Wzp;
            const R rdx3 = n.rdx3;
            const R T0 = Tc, K0 = Kc, dK0 = dKc, F5 = F, G5 = G, s5 = s, q5 = q, w5 = w, d3m = dx3m, d3 = dx3;
            R irc, dirc;
            rhocp_eval(p, T0, irc, dirc);
            const R h = R(0.5) * p.Ct * irc, dh = R(0.5) * p.Ct * dirc;
            face(o, Tzp, Wzp, n.dx3, n.rdmx3);
            const R Kxm = kpp_only(p, d2, Txm), Kxp = kpp_only(p, d2, Txp);
            R Kym, Kyp, dKym = R(0), dKyp = R(0);
            const bool wall = j == 1 || j == g.N2;
            if (wall) { kpp_eval(p, d2, Tym, Kym, dKym); kpp_eval(p, d2, Typ, Kyp, dKyp); }
            else { Kym = kpp_only(p, d2, Tym); Kyp = kpp_only(p, d2, Typ); }
            const R dx1 = (T0 - Txm) * rdmx1, dx2 = (Txp - T0) * rdmx1p, dy3 = (T0 - Tym) * rdmx2, dy4 = (Typ - T0) * rdmx2p;
            const R kPP3 = K0 + w3 * (Kym - K0), kPP4 = K0 + w4 * (Kyp - K0);
            const R fx = (K0 + w2 * (Kxp - K0)) * dx2 - (K0 + w1 * (Kxm - K0)) * dx1, fy = kPP4 * dy4 - kPP3 * dy3;
            const R dv = fx * rdx1 + fy * rdx2 + (F - F5) * rdx3;
            R rhs = R(2) * h * dv - R(0.5) * ((Uc * dx1 + Uxp * dx2) + (Vc * dy3 + Vyp * dy4) + (G5 + G));
            if (wall) {
                const R h2 = h * rdx2;
                if (j == 1) {
                    const R qd = (dK0 + w3 * (dKym - dK0)) * dy3, am = -h2 * (kPP3 * rdmx2 - w3 * qd) - R(0.25) * Vc * rdmx2;
                    rhs = rhs + am * Tym + h2 * (R(1) - w3) * qd * T0 + (R(0.25) * Vc * rdmx2 + h2 * (kPP3 * rdmx2 - qd)) * p.Tbt;
                }
                if (j == g.N2) {
                    const R qd = (dK0 + w4 * (dKyp - dK0)) * dy4, ap = -h2 * (kPP4 * rdmx2p + w4 * qd) + R(0.25) * Vyp * rdmx2p;
                    rhs = rhs + ap * Typ - h2 * (R(1) - w4) * qd * T0 + (h2 * (kPP4 * rdmx2p + qd) - R(0.25) * Vyp * rdmx2p) * p.Tup;
                }
            }
            const R h3 = h * rdx3;
            a = (-h3 * (s5 - d3 * q5) - w5) * dt;
            cc = (w - h3 * (s + d3 * q)) * dt;
            b = 1.0 + (double)((h3 * (s + s5 - dx3 * q + d3m * q5) + (w5 - w) - R(0.5) * dh * dv) * dt);
            d[0] = rhs * dt;
        }
    };
    struct Out : ScratchOut<R> {
        __device__ __forceinline__ Out(const ThermalZ &q, int line, int by, int r) : ScratchOut<R>(q.g, q.f.scr, 1 + line, 1 + by, r + 1, (long long)q.g.P1 * q.g.P2) {}
        __device__ __forceinline__ void put(const ThermalZ &q, const double *x) { ScratchOut<R>::put(q.g, q.f.scr, R(x[0])); }
    };
};

// Stage 2 (:388-429): jm, jp, km, kp keep the values of the last stage-1
// iteration (N2-1, N2+1, N3-1, N3+1).  The whole row is built as it is staged,
// normalised by its diagonal (planes: d, c, a): keeping T, U, the right-hand side
// and the stale fluxes for the march instead takes a fourth plane, which halves
// the lines in flight (512 rows, FP64: 20 ps per cell against 27).
template <class R>
struct ThermalX {
    using Real = R;
    static constexpr int WORDS = 3, UNROLL = 2;
    GridT<R> g; FieldsT<R> f;
    __device__ bool skip() const { return blown(g); }
    __device__ int lines() const { return g.N2; }
    __device__ R *out(int line, int by) const { return f.scr + ix(g, 1, 1 + line, 1 + by); }
    struct Stage {
        long long c, cjm, cjp, ckm, ckp;
        R a3, b3, a4, b4, a5, b5, a6, b6, r2, r2p, r3, r3p, rdx2, rdx3, dt;   // stale faces: weights of the neighbour (a) and the cell (b)
        __device__ __forceinline__ Stage(const ThermalX &o, int line, int by)
        {
            const GridT<R> &g = o.g;
            const int j = 1 + line, k = 1 + by, jm = g.N2 - 1, jp = g.N2 + 1, km = g.N3 - 1, kp = g.N3 + 1;
            c = ix(g, 1, j, k); cjm = ix(g, 1, jm, k); cjp = ix(g, 1, jp, k); ckm = ix(g, 1, j, km); ckp = ix(g, 1, j, kp);
            r2 = ld(g.m2.rdmx + j); r2p = ld(g.m2.rdmx + jp); r3 = ld(g.m3.rdmx + k); r3p = ld(g.m3.rdmx + kp);
            a3 = R(0.5) * r2 * ld(g.m2.dx + j); b3 = R(0.5) * r2 * ld(g.m2.dx + jm);
            a4 = R(0.5) * r2p * ld(g.m2.dx + j); b4 = R(0.5) * r2p * ld(g.m2.dx + jp);
            a5 = R(0.5) * r3 * ld(g.m3.dx + k); b5 = R(0.5) * r3 * ld(g.m3.dx + km);
            a6 = R(0.5) * r3p * ld(g.m3.dx + k); b6 = R(0.5) * r3p * ld(g.m3.dx + kp);
            rdx2 = ld(g.m2.rdx + j); rdx3 = ld(g.m3.rdx + k);
            dt = R(g.scal[S_DT]);
        }
        __device__ __forceinline__ void put(const ThermalX &o, int r, double *w, int PL) const
        {
            TCS_OOB(o.g.scal, r < 0 || r >= o.g.N1, return);
            const GridT<R> &g = o.g;
            const PhysT<R> &p = g.ph;
            const bool d2 = g.kdeg2 != 0;
            const int i = r + 1;
            const R *const T = o.f.T + r, *const U = o.f.U + c + r;
            const R d = o.f.scr[c + r];
            const R Tc = ld(T + c), Txm = ld(T + c - 1), Txp = ld(T + c + 1), Tjm = ld(T + cjm), Tjp = ld(T + cjp), Tkm = ld(T + ckm), Tkp = ld(T + ckp);
            const R Uc = ld(U), Uxp = ld(U + 1);
            const R dxm = ld(g.m1.dx + i - 1), dx = ld(g.m1.dx + i), dxp = ld(g.m1.dx + i + 1), rdx1 = ld(g.m1.rdx + i);
            const R rd = ld(g.m1.rdmx + i), rdp = ld(g.m1.rdmx + i + 1);
            R K, dK, Km, dKm, Kp, dKp, irc, dirc;
            kpp_eval(p, d2, Tc, K, dK); kpp_eval(p, d2, Txm, Km, dKm); kpp_eval(p, d2, Txp, Kp, dKp);
            rhocp_eval(p, Tc, irc, dirc);
            const R h = R(0.5) * p.Ct * irc, h1 = h * rdx1;
            const R y = (a4 * kpp_only(p, d2, Tjp) + b4 * K) * ((Tjp - Tc) * r2p) - (a3 * kpp_only(p, d2, Tjm) + b3 * K) * ((Tc - Tjm) * r2);
            const R z = (a6 * kpp_only(p, d2, Tkp) + b6 * K) * ((Tkp - Tc) * r3p) - (a5 * kpp_only(p, d2, Tkm) + b5 * K) * ((Tc - Tkm) * r3);
            const R hm = R(0.5) * rd, hp = R(0.5) * rdp, g1 = (Tc - Txm) * rd, g2 = (Txp - Tc) * rdp;
            const R k1 = K + hm * dx * (Km - K), k2 = K + hp * dx * (Kp - K);
            const R q1 = hm * (dK + hm * dx * (dKm - dK)) * g1, q2 = hp * (dK + hp * dx * (dKp - dK)) * g2;
            const R s1 = k1 * rd, s2 = k2 * rdp, w1 = R(0.25) * Uc * rd, w2 = R(0.25) * Uxp * rdp;
            const R ac = h1 * (s2 + s1 - dxp * q2 + dxm * q1) + (w1 - w2) - R(0.5) * h * ((k2 * g2 - k1 * g1) * rdx1 + y * rdx2 + z * rdx3);
            const double rb = qrcp(1.0 + (double)(ac * dt));
            w[0] = (double)d * rb;
            w[PL] = (double)((w2 - h1 * (s2 + dx * q2)) * dt) * rb;
            w[2 * PL] = (double)((-h1 * (s1 - dx * q1) - w1) * dt) * rb;
        }
    };
    struct March {
        __device__ __forceinline__ March(const ThermalX &, int, int, int, int, int, const double *, int) {}
        __device__ __forceinline__ void row(const ThermalX &, int r, bool, const double *w, int PL, double &a, double &b, double &c, double &d)
        {
            a = w[2 * PL + r]; b = 1.0; c = w[PL + r]; d = w[r];
        }
    };
};

// Stage 3 (:456-507): km, kp stale (N3-1, N3+1); T += solution (:518-524).
template <class R>
struct ThermalY {
    using Real = R;
    static constexpr int NRHS = 1;
    static constexpr int AHEAD = 0, TPS = 512, ROWS = 16, LGTI = 4;
    static constexpr bool LONG64 = false;
    GridT<R> g; FieldsT<R> f;
    __device__ bool skip() const { return blown(g); }
    __device__ int lines() const { return g.N1; }
    struct March {
        R rdx1, rdmx1, rdmx1p, w1, w2, rdx3, rdmx3, rdmx3p, z5m, z5c, z6c, z6p, dt;   // weights along x (see ThermalZ) and of the stale z faces
        R Tc, Kc, dKc, F, s, q, w, dx2m, dx2;         // the cell; the face below it
        long long c, dkm, dkp;
        __device__ __forceinline__ March(const ThermalY &o, int line, int by, int r0)
        {
            const GridT<R> &g = o.g;
            const int i = 1 + line, j = r0 + 1, k = 1 + by, km = g.N3 - 1, kp = g.N3 + 1;
            const long long sk = (long long)g.P1 * g.P2;
            rdx1 = ld(g.m1.rdx + i); rdmx1 = ld(g.m1.rdmx + i); rdmx1p = ld(g.m1.rdmx + i + 1);
            w1 = R(0.5) * rdmx1 * ld(g.m1.dx + i); w2 = R(0.5) * rdmx1p * ld(g.m1.dx + i);
            rdx3 = ld(g.m3.rdx + k); rdmx3 = ld(g.m3.rdmx + k); rdmx3p = ld(g.m3.rdmx + kp);
            z5m = R(0.5) * rdmx3 * ld(g.m3.dx + k); z5c = R(0.5) * rdmx3 * ld(g.m3.dx + km);
            z6c = R(0.5) * rdmx3p * ld(g.m3.dx + kp); z6p = R(0.5) * rdmx3p * ld(g.m3.dx + k);
            dt = R(g.scal[S_DT]);
            c = ix(g, i, j, k);
            dkm = sk * (km - k); dkp = sk * (kp - k);
            dx2 = ld(g.m2.dx + j - 1);
            Tc = ld(o.f.T + c - g.P1);
            kpp_eval(g.ph, g.kdeg2 != 0, Tc, Kc, dKc);
            face(o, ld(o.f.T + c), ld(o.f.V + c), ld(g.m2.dx + j), ld(g.m2.rdmx + j));
        }
        // the y face between rows j-1 (Tc, Kc, dKc, dx2) and j, which becomes the current row
        __device__ __forceinline__ void face(const ThermalY &o, R Tp, R Vp, R dy, R rdmx2)
        {
            R Kp, dKp;
            kpp_eval(o.g.ph, o.g.kdeg2 != 0, Tp, Kp, dKp);
            dx2m = dx2;
            dx2 = dy;
            const R hm = R(0.5) * rdmx2, wm = hm * dx2m, de = (Tp - Tc) * rdmx2;
            const R kPP = Kc + wm * (Kp - Kc), dkPP = dKc + wm * (dKp - dKc);
            F = kPP * de;
            s = kPP * rdmx2;
            q = hm * (dkPP * de);
            w = R(0.25) * Vp * rdmx2;
            Tc = Tp; Kc = Kp; dKc = dKp;
        }
        struct In { R Txm, Txp, Typ, Tkm, Tkp, V, rdx2, dx2, rdmx2, d; };
        __device__ __forceinline__ void load(const ThermalY &o, int r, In &n)
        {
            row_cell(o.g, c);
            const GridT<R> &g = o.g;
            const R *const T = o.f.T;
            n.Txm = ld(T + c - 1); n.Txp = ld(T + c + 1); n.Typ = ld(T + c + g.P1);
            TCS_OOB(g.scal, c + dkm < 0 || c + dkp >= g.NP, dkm = dkp = 0);
            n.Tkm = ld(T + c + dkm); n.Tkp = ld(T + c + dkp);
            n.V = ld(o.f.V + c + g.P1);
            n.rdx2 = ld(g.m2.rdx + r + 1); n.dx2 = ld(g.m2.dx + r + 2); n.rdmx2 = ld(g.m2.rdmx + r + 2);
            n.d = o.f.scr[c];
            c += g.P1;
        }
        __device__ __forceinline__ void row(const ThermalY &o, int r, const In &n, double &a, double &b, double &cc, double *d)
        {
            const PhysT<R> &p = o.g.ph;
            const bool d2 = o.g.kdeg2 != 0;
            const R T0 = Tc, K0 = Kc, F3 = F, s3 = s, q3 = q, w3 = w, d2m = dx2m, d2c = dx2;
            R irc, dirc;
            rhocp_eval(p, T0, irc, dirc);
            const R h = R(0.5) * p.Ct * irc, h2 = h * n.rdx2;
            face(o, n.Typ, n.V, n.dx2, n.rdmx2);
            const R Kxm = kpp_only(p, d2, n.Txm), Kxp = kpp_only(p, d2, n.Txp), Kkm = kpp_only(p, d2, n.Tkm), Kkp = kpp_only(p, d2, n.Tkp);
            const R fx = (K0 + w2 * (Kxp - K0)) * ((n.Txp - T0) * rdmx1p) - (K0 + w1 * (Kxm - K0)) * ((T0 - n.Txm) * rdmx1);
            const R fz = (z6c * K0 + z6p * Kkp) * ((n.Tkp - T0) * rdmx3p) - (z5m * Kkm + z5c * K0) * ((T0 - n.Tkm) * rdmx3);
            const R jem = r == 0 ? R(0) : R(1), jep = r == o.g.N2 - 1 ? R(0) : R(1);
            const R ac = h2 * (s + s3 - dx2 * q * jep + d2m * q3 * jem) + (w3 - w) - R(0.5) * h * (fx * rdx1 + (F - F3) * n.rdx2 + fz * rdx3);
            a = (-h2 * (s3 - d2c * q3) - w3) * jem * dt;
            cc = (w - h2 * (s + d2c * q)) * jep * dt;
            b = 1.0 + (double)(ac * dt);
            d[0] = n.d;
        }
    };
    struct Out : PeriodicOut<R> {
        const R *T;
        __device__ __forceinline__ Out(const ThermalY &q, int line, int by, int r)
            : PeriodicOut<R>(q.g, q.f.Tn, 1 + line, r + 1, 1 + by), T(q.f.T + ix(q.g, 1 + line, r + 1, 1 + by)) {}
        __device__ __forceinline__ void put(const ThermalY &q, const double *x)
        {
            row_ptr(q.g, (const R *)q.f.T, T);
            PeriodicOut<R>::put(q.g, q.f.Tn, ld(T) + R(x[0]));
            T -= q.g.P1;
        }
    };
};

template <class R>
static void launch_thermal_z(const Ctx<R> &cx, cudaStream_t s)
{
    launch_march(cx, ThermalZ<R>{cx.g, cx.f}, cx.g.N3, true, cx.g.N1, cx.g.N2, s, K_THERMAL_Z);
}

template <class R>
static void launch_thermal_y(const Ctx<R> &cx, cudaStream_t s)
{
    launch_march(cx, ThermalY<R>{cx.g, cx.f}, cx.g.N2, false, cx.g.N1, cx.g.N3, s, K_THERMAL_Y);
}

template <class R>
static void launch_thermal_x(const Ctx<R> &cx, cudaStream_t s)
{
    launch_xmarch(cx, ThermalX<R>{cx.g, cx.f}, cx.g.N1, cx.g.N2, cx.g.N3, s, K_THERMAL_X);
}

template <class R>
void launch_thermal(const Ctx<R> &cx, cudaStream_t s)
{
    launch_thermal_z(cx, s);
    launch_thermal_x(cx, s);
    launch_thermal_y(cx, s);
}

// The same three sweeps for many cases, sweep by sweep (march_stage).
template <class R>
void launch_thermal_multi(const std::vector<Ctx<R> *> &cs, MultiArena &A, cudaStream_t s)
{
    march_stage(cs, A, s, launch_thermal_z<R>);
    march_stage(cs, A, s, launch_thermal_x<R>);
    march_stage(cs, A, s, launch_thermal_y<R>);
}

// the two forms
template void launch_thermal<double>(const Ctx<double> &, cudaStream_t);
template void launch_thermal<float>(const Ctx<float> &, cudaStream_t);
template void launch_thermal_multi<double>(const std::vector<Ctx<double> *> &, MultiArena &, cudaStream_t);
template void launch_thermal_multi<float>(const std::vector<Ctx<float> *> &, MultiArena &, cudaStream_t);

} // namespace tcs
