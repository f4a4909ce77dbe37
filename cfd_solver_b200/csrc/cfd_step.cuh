// cfd_step.cuh -- the arithmetic of one time step, cell by cell and tile by tile.
//
// Two forms of the step call it: the launch-per-phase kernels (cfd_kernels.cu, cfd_sweep.cu)
// and the team kernel (cfd_team.cu), which runs the phases of a case inside one launch. Both
// evaluate the same expressions in the same order, so a case gives the same bits in either.
#pragma once
#include <type_traits>

#include "cfd_common.cuh"
#include "cfd_kernels.cuh"

namespace cfd {

constexpr int JTW = TX + 4;   // 32 x 16 tile columns incl. a 2-cell halo
constexpr int JTH = TYJ + 4;  // 32 x 16 tile rows incl. a 2-cell halo

// A group of N threads that works on one tile: its members' index and its barrier. A whole
// CTA uses barrier 0; the groups of a CTA that holds several use a named barrier each.
template <int N_>
struct BlockGroup {
    static constexpr int N = N_;
    int tid;
    __device__ __forceinline__ BlockGroup() : tid(threadIdx.x) {}
    __device__ __forceinline__ void sync() const { __syncthreads(); }
};
template <int N_>
struct NamedGroup {
    static constexpr int N = N_;
    int tid, id;  // member index, group of the CTA
    __device__ __forceinline__ NamedGroup() : tid(threadIdx.x % N_), id(threadIdx.x / N_) {}
    __device__ __forceinline__ void sync() const {
        asm volatile("bar.sync %0, %1;" ::"r"(id + 1), "n"(N_) : "memory");
    }
};

// plane that holds the final multigrid V-cycle result of level l of case c (x on the
// case's coarsest level; otherwise fixed by the numbers of pre- and post-sweeps)
__device__ __forceinline__ int mg_result_plane(const BatchDev& b, const CaseDev& c, int l) {
    return l == c.nlev - 1 ? M_X : b.mg_res;
}

// ---------------------------------------------------------------------------
// convection and the five right-hand sides

// A field at a cell and two cells to each side, rows R apart. From shared memory (CrossAt)
// each value is read where it is used; from global memory (Cross) all loads come first and
// without a branch, and next to a wall the second cell along that axis is not read (it may
// lie outside).
struct CrossAt {
    const double* f;
    int R;
    __device__ __forceinline__ CrossAt(const double* F, int o, int R_, bool, bool) : f(F + o), R(R_) {}
    __device__ __forceinline__ double c() const { return f[0]; }
    __device__ __forceinline__ double e() const { return f[1]; }
    __device__ __forceinline__ double w() const { return f[-1]; }
    __device__ __forceinline__ double n() const { return f[R]; }
    __device__ __forceinline__ double s() const { return f[-R]; }
    __device__ __forceinline__ double ee() const { return f[2]; }
    __device__ __forceinline__ double ww() const { return f[-2]; }
    __device__ __forceinline__ double nn() const { return f[2 * R]; }
    __device__ __forceinline__ double ss() const { return f[-2 * R]; }
};
struct Cross {
    double v[9];
    __device__ __forceinline__ Cross(const double* F, int o, int R, bool near_i, bool near_j) {
        const int a = near_i ? 1 : 2, b = near_j ? R : 2 * R;
        v[0] = F[o]; v[1] = F[o + 1]; v[2] = F[o - 1]; v[3] = F[o + R]; v[4] = F[o - R];
        v[5] = F[o + a]; v[6] = F[o - a]; v[7] = F[o + b]; v[8] = F[o - b];
    }
    __device__ __forceinline__ double c() const { return v[0]; }
    __device__ __forceinline__ double e() const { return v[1]; }
    __device__ __forceinline__ double w() const { return v[2]; }
    __device__ __forceinline__ double n() const { return v[3]; }
    __device__ __forceinline__ double s() const { return v[4]; }
    __device__ __forceinline__ double ee() const { return v[5]; }
    __device__ __forceinline__ double ww() const { return v[6]; }
    __device__ __forceinline__ double nn() const { return v[7]; }
    __device__ __forceinline__ double ss() const { return v[8]; }
};

// One convective term ux df/dxi + ue df/deta of a field (PSolver.cpp:1110-1180): 4th-order
// central differences when the cell Peclet number is in (-2, 2] (and always in the rows /
// columns next to a wall, where the reference uses 2nd-order central), otherwise 3rd-order
// upwind. The reference forms du = (ux D1 + |ux| D4) / ux and multiplies by ux again; here
// the product is formed directly, and every division by a grid spacing is a multiplication
// by its reciprocal.
template <class S>
__device__ __forceinline__ double conv_one(const S& f, bool near_i, bool near_j, double ux, double ue, bool cen_i,
                                           bool cen_j, double rd0, double rd1) {
    const double fc = f.c(), fe = f.e(), fw = f.w();
    const double fn = f.n(), fs = f.s();
    double cx, cy;
    if (near_i) {
        cx = ux * (0.5 * (fe - fw) * rd0);
    } else {
        const double fee = f.ee(), fww = f.ww();
        if (near_j || cen_i) {
            cx = ux * ((1.0 / 12.0) * (8.0 * (fe - fw) - (fee - fww)) * rd0);
        } else {
            cx = (ux * ((1.0 / 12.0) * (-fee + 8.0 * fe - 8.0 * fw + fww)) +
                  fabs(ux) * (0.25 * (fee - 4.0 * fe + 6.0 * fc - 4.0 * fw + fww))) * rd0;
        }
    }
    if (near_j) {
        cy = ue * (0.5 * (fn - fs) * rd1);
    } else {
        const double fnn = f.nn(), fss = f.ss();
        if (near_i || cen_j) {
            cy = ue * ((1.0 / 12.0) * (8.0 * (fn - fs) - (fnn - fss)) * rd1);
        } else {
            cy = (ue * ((1.0 / 12.0) * (-fnn + 8.0 * fn - 8.0 * fs + fss)) +
                  fabs(ue) * (0.25 * (fnn - 4.0 * fn + 6.0 * fc - 4.0 * fs + fss))) * rd1;
        }
    }
    return cx + cy;
}

// Is the cell Peclet number n / a in (-2, 2]? Decided without the quotient: for a > 0, RN(n / a)
// is in (-2, 2] exactly when n is in (-2 a, 2 a] (2 a is exact, and the doubles next to it are
// more than half a unit in the last place of 2 away).
__device__ __forceinline__ bool peclet_central(double n, double a) { return n <= 2.0 * a && n > -2.0 * a; }

// what every cell's right-hand sides read of the case
struct RhsCase {
    const CaseDev& c;
    double rd0, rd1, dt, Red0, Red1, Pr, Ri;
    int n0, n1;
    bool cav;
    __device__ __forceinline__ explicit RhsCase(const CaseDev& c_) : c(c_) {
        rd0 = c.rd0; rd1 = c.rd1; dt = c.dt; Red0 = c.Re * c.d0; Red1 = c.Re * c.d1; Pr = c.Pr; Ri = c.Ri;
        n0 = c.n0; n1 = c.n1; cav = c.profile == CAVITY;
    }
};
struct RhsOut {
    double qu, qv, qt, qup, qvp;
};

// The five right-hand sides of cell (i, j) (PSolver.cpp:1063-1237). The fields are read at
// offset o with rows R apart; `be` points at the cell's beta (read next to an O-grid's walls).
template <class S>
__device__ __forceinline__ RhsOut rhs_cell(const RhsCase& a, int i, int j, const double* Us, const double* Vs,
                                           const double* Ts, const double* Ps, const double* UPs, const double* VPs,
                                           int o, int R, double xix, double xiy, double etx, double ety, double al,
                                           double ga, const double* bep) {
    const double dt = a.dt, rd0 = a.rd0, rd1 = a.rd1;
    const bool cav = a.cav;
    const bool near_j = (j == 1 || j == a.n1 - 2);
    const bool near_i = cav && (i == 1 || i == a.n0 - 2);
    const S fu(Us, o, R, near_i, near_j), fv(Vs, o, R, near_i, near_j), ft(Ts, o, R, near_i, near_j);
    const S fp(Ps, o, R, true, true);
    const double uc = fu.c(), vc = fv.c(), tc = ft.c();
    const double ux = xix * uc + xiy * vc;
    const double ue = etx * uc + ety * vc;
    // cell Peclet numbers ux Re dxi / alpha, ue Re deta / gamma (x Pr for T)
    const double pn1 = ux * a.Red0, pn2 = ue * a.Red1;
    const bool cu1 = peclet_central(pn1, al), cu2 = peclet_central(pn2, ga);
    const bool ct1 = peclet_central(pn1 * a.Pr, al), ct2 = peclet_central(pn2 * a.Pr, ga);
    const double cv0 = conv_one(fu, near_i, near_j, ux, ue, cu1, cu2, rd0, rd1);
    const double cv1 = conv_one(fv, near_i, near_j, ux, ue, cu1, cu2, rd0, rd1);
    const double cv2 = conv_one(ft, near_i, near_j, ux, ue, ct1, ct2, rd0, rd1);
    const double dp_dxi = (fp.e() - fp.w()) * (0.5 * rd0);
    const double dp_de = (fp.n() - fp.s()) * (0.5 * rd1);
    const double dp_dx = xix * dp_dxi + etx * dp_de;
    const double dp_dy = xiy * dp_dxi + ety * dp_de;
    RhsOut q;
    q.qu = dt * (-cv0 - dp_dx) + uc;
    q.qv = dt * (-cv1 - dp_dy + a.Ri * tc) + vc;
    q.qt = -dt * cv2 + tc;
    q.qup = q.qu + dt * dp_dx;
    q.qvp = q.qv + dt * dp_dy;
    if (!cav && near_j) {
        // folded wall-row couplings (PSolver.cpp:1195-1227)
        const CaseDev& c = a.c;
        const double be = *bep;
        const double g11 = div_by(ga, c.v11);
        const double bs = div_by(-dt * g11, c.vRe);
        const double bpos = div_by(dt * be, c.v01Re), bneg = -bpos;
        const double ts = div_by(-dt * g11, c.vRePr);
        const double tpos = div_by(dt * div_by(be, c.v01), c.vRePr), tneg = -tpos;
        int s0, s1, s2;
        double c1, c2, t1, t2;
        if (j == 1) {  // bus, buse (= ause), busw (= ausw)
            s0 = o - R; s1 = o - R + 1; s2 = o - R - 1;
            c1 = bneg; c2 = bpos; t1 = tneg; t2 = tpos;
        } else {       // bun, bune (= aune), bunw (= aunw)
            s0 = o + R; s1 = o + R + 1; s2 = o + R - 1;
            c1 = bpos; c2 = bneg; t1 = tpos; t2 = tneg;
        }
        double sumu = bs * Us[s0] + c1 * Us[s1] + c2 * Us[s2];
        q.qu = q.qu - sumu;
        double sumv = bs * Vs[s0] + c1 * Vs[s1] + c2 * Vs[s2];
        q.qv = q.qv - sumv;
        double sumt = ts * Ts[s0] + t1 * Ts[s1] + t2 * Ts[s2];
        q.qt = q.qt - sumt;
        sumu = bs * UPs[s0] + c1 * UPs[s1] + c2 * UPs[s2];
        q.qup = q.qup - sumu;
        sumv = bs * VPs[s0] + c1 * VPs[s1] + c2 * VPs[s2];
        q.qvp = q.qvp - sumv;
    }
    return q;
}

// Seeds the five solves' iterates at cell (i, j) (PSolver.cpp:1241-1337): u*, v*, T from the
// current fields, up / vp from the previous solution or zero (already chosen in `seed`). A
// solve predicted to stop after an odd number of sweeps (bit of `nextm`) starts in the scratch
// plane, so that its result ends in the iterate plane. Cells next to a boundary also write the
// boundary values the stencils read, into both iterate buffers. `fb` is plane 0 of the case.
// AHEAD: a boundary point's five loads are issued together (one latency instead of five, for
// more registers than k_rhs has to spare).
template <bool AHEAD>
__device__ __forceinline__ void rhs_seed(double* fb, long long ps, int nextm, int cur, int ld, int W, int per,
                                         bool cav, int n0, int n1, int i, int j, const double (&seed)[NFIELD]) {
    const int nxt = cur ^ 1;
    const double* U = fb + P_U * ps;
    const double* V = fb + P_V * ps;
    const double* T = fb + (P_T0 + cur) * ps;
    const double* UP = fb + (P_UP0 + cur) * ps;
    const double* VP = fb + (P_VP0 + cur) * ps;
    // iterate buffers of field f: A (the solution) and B (the Jacobi scratch)
    auto Ap = [&](int f) { return fb + (f < 2 ? P_US + f : P_T0 + 2 * (f - 2) + nxt) * ps; };
    auto Bp = [&](int f) { return fb + (P_BU + f) * ps; };
#pragma unroll
    for (int f = 0; f < NFIELD; f++)
        store_mirrored(((nextm >> f) & 1) ? Bp(f) : Ap(f), ld, i, j, W, per, seed[f]);
    auto put_bnd = [&](int bi, int bj) {
        const long long kb = (long long)bj * ld + bi;
        const bool zero_far = !cav && bj == n1 - 1;  // up/vp solves see zero on the far row
        if constexpr (AHEAD) {
            const double val[NFIELD] = {U[kb], V[kb], T[kb], zero_far ? 0.0 : UP[kb], zero_far ? 0.0 : VP[kb]};
#pragma unroll
            for (int f = 0; f < NFIELD; f++) {
                store_mirrored(Ap(f), ld, bi, bj, W, per, val[f]);
                store_mirrored(Bp(f), ld, bi, bj, W, per, val[f]);
            }
        } else {
#pragma unroll 1
            for (int f = 0; f < NFIELD; f++) {
                const double* src = f == F_U ? U : f == F_V ? V : f == F_T ? T : f == F_UP ? UP : VP;
                const double val = (zero_far && f >= F_UP) ? 0.0 : src[kb];
                store_mirrored(Ap(f), ld, bi, bj, W, per, val);
                store_mirrored(Bp(f), ld, bi, bj, W, per, val);
            }
        }
    };
    if (j == 1) put_bnd(i, 0);
    if (j == n1 - 2) put_bnd(i, n1 - 1);
    if (cav) {
        if (i == 1) {
            put_bnd(0, j);
            if (j == 1) put_bnd(0, 0);
            if (j == n1 - 2) put_bnd(0, n1 - 1);
        }
        if (i == n0 - 2) {
            put_bnd(n0 - 1, j);
            if (j == 1) put_bnd(n0 - 1, 0);
            if (j == n1 - 2) put_bnd(n0 - 1, n1 - 1);
        }
    }
}

// ---------------------------------------------------------------------------
// the u/v/T/up/vp sweeps (the operator and the Chebyshev recurrence: cfd_sweep.cu)

// FP64 plane of field f's iterate for state parity nxt (u*, v*, T, up, vp)
__device__ __forceinline__ int sw_iter_plane(int f, int nxt) { return f < 2 ? P_US + f : P_T0 + 2 * (f - 2) + nxt; }

// Off-centre sums of the u-type operator at a cell, x(dy, dx) giving the values around it: the
// 25-point (4th-order) rows and the 9-point near-wall rows.
template <typename ST, class X>
__device__ __forceinline__ ST sw_sum25(const X& x, ST E, ST G, ST B) {
    const ST ex = ST(-4.0 / 3.0) * (x(0, 1) + x(0, -1)) + ST(1.0 / 12.0) * (x(0, 2) + x(0, -2));
    const ST gy = ST(-4.0 / 3.0) * (x(1, 0) + x(-1, 0)) + ST(1.0 / 12.0) * (x(2, 0) + x(-2, 0));
    const ST bx = ST(8.0 / 9.0) * (x(1, 1) + x(-1, -1) - x(1, -1) - x(-1, 1)) +
                  ST(1.0 / 72.0) * (x(2, 2) + x(-2, -2) - x(2, -2) - x(-2, 2)) +
                  ST(1.0 / 9.0) * (x(2, -1) + x(-2, 1) + x(1, -2) + x(-1, 2) - x(2, 1) - x(-2, -1) - x(1, 2) - x(-1, -2));
    return E * ex + G * gy + B * bx;
}
template <typename ST, class X>
__device__ __forceinline__ ST sw_sum9(const X& x, ST E, ST G, ST B, bool drop_s, bool drop_n) {
    ST s = -E * (x(0, 1) + x(0, -1));
    const ST n = -G * x(1, 0) + ST(0.5) * B * (x(1, 1) - x(1, -1));
    const ST so = -G * x(-1, 0) + ST(0.5) * B * (x(-1, -1) - x(-1, 1));
    if (!drop_n) s += n;
    if (!drop_s) s += so;
    return s;
}

// residual of one cell for operator E, G, B; `scale` is 1/Pr for T
template <typename ST, class X>
__device__ __forceinline__ ST sw_residual(const X& x, ST E, ST G, ST B, bool nearw, bool drop_s, bool drop_n, bool tbug,
                                          ST scale, ST rhs) {
    // off-centre sum: the 25-point form, or the 9-point form on the near-wall cells
    ST sm = nearw ? sw_sum9<ST>(x, E, G, B, drop_s, drop_n) : sw_sum25<ST>(x, E, G, B);
    if (tbug && !nearw) sm -= B * x(2, -1);
    sm *= scale;
    const ST D = (nearw ? ST(2) : ST(2.5)) * (E + G);
    const ST ap = ST(1) + D * scale;
    return rhs - ap * x(0, 0) - sm;
}

// x_{k+1} from the residual (Chebyshev weight wgt on every sweep but the first)
template <typename ST>
__device__ __forceinline__ ST sw_next(ST xk, ST g, ST res, ST rap, bool weighted, ST wgt, ST xm) {
    ST xn = xk + g * res * rap;
    if (weighted) xn = wgt * (xn - xm) + xm;
    return xn;
}

// Chebyshev weight of the sweep after `sweep` (s2 of the bounds a, b; cw the weight of `sweep`)
__device__ __forceinline__ double cheb_s2(double ca, double cb) { return ((cb + ca) / (cb - ca)) * ((cb + ca) / (cb - ca)); }
__device__ __forceinline__ double cheb_next(int sweep, double cw, double s2) {
    return (sweep == 0) ? 1.0 / (1.0 - 1.0 / (2.0 * s2)) : 1.0 / (1.0 - cw / (4.0 * s2));
}

// ---------------------------------------------------------------------------
// continuity source

// far-field value of up / vp from its iterate (PSolver.cpp:1356-1382); k on the far row
__device__ __forceinline__ double upbc_out(const double* UP, long long k, int ld) {
    return (5.0 * UP[k - ld] - 4.0 * UP[k - 2LL * ld] + UP[k - 3LL * ld]) / 2.0;
}

struct FaceCase {
    double rd0, rd1, q0, q1, hdt, rdt;
    __device__ __forceinline__ explicit FaceCase(const CaseDev& c) {
        // the per-cell quotients as products (each within an ulp of the quotient; 1 / (4 d) is
        // 0.25 / d exactly)
        rd0 = c.rd0; rd1 = c.rd1; q0 = 0.25 * rd0; q1 = 0.25 * rd1;
        hdt = 0.5 * c.dt; rdt = c.rdt;
    }
};

// face velocities -> q of one cell (PSolver.cpp:1390-1449): pressure P, intermediate
// velocities U, V (their northern neighbours given as uN, vN) and the metrics X = xi_x,
// Y = xi_y, E = eta_x, G = eta_y at offset k, rows R apart
__device__ __forceinline__ double face_cell(const FaceCase& a, const double* P, const double* U, const double* V,
                                            const double* X, const double* Y, const double* E, const double* G, int k,
                                            int R, double uN, double vN) {
    const double rd0 = a.rd0, rd1 = a.rd1, q0 = a.q0, q1 = a.q1, hdt = a.hdt;
    const int kE = k + 1, kW = k - 1, kN = k + R, kS = k - R;
    double dpdxi_ip = (P[kE] - P[k]) * rd0;
    double dpde_ip = (P[kN + 1] + P[kN] - P[kS] - P[kS + 1]) * q1;
    double dpdxi_in = (P[k] - P[kW]) * rd0;
    double dpde_in = (P[kN] + P[kN - 1] - P[kS] - P[kS - 1]) * q1;
    double dpdxi_jp = (P[kN + 1] - P[kN - 1] + P[kE] - P[kW]) * q0;
    double dpde_jp = (P[kN] - P[k]) * rd1;
    double dpdxi_jn = (P[kE] - P[kW] + P[kS + 1] - P[kS - 1]) * q0;
    double dpde_jn = (P[k] - P[kS]) * rd1;
    double us_ip = 0.5 * (U[k] + U[kE]) - hdt * ((X[k] + X[kE]) * dpdxi_ip + (E[k] + E[kE]) * dpde_ip);
    double us_in = 0.5 * (U[k] + U[kW]) - hdt * ((X[k] + X[kW]) * dpdxi_in + (E[k] + E[kW]) * dpde_in);
    double us_jp = 0.5 * (U[k] + uN) - hdt * ((X[k] + X[kN]) * dpdxi_jp + (E[k] + E[kN]) * dpde_jp);
    double us_jn = 0.5 * (U[k] + U[kS]) - hdt * ((X[k] + X[kS]) * dpdxi_jn + (E[k] + E[kS]) * dpde_jn);
    double vs_ip = 0.5 * (V[k] + V[kE]) - hdt * ((Y[k] + Y[kE]) * dpdxi_ip + (G[k] + G[kE]) * dpde_ip);
    double vs_in = 0.5 * (V[k] + V[kW]) - hdt * ((Y[k] + Y[kW]) * dpdxi_in + (G[k] + G[kW]) * dpde_in);
    double vs_jp = 0.5 * (V[k] + vN) - hdt * ((Y[k] + Y[kN]) * dpdxi_jp + (G[k] + G[kN]) * dpde_jp);
    double vs_jn = 0.5 * (V[k] + V[kS]) - hdt * ((Y[k] + Y[kS]) * dpdxi_jn + (G[k] + G[kS]) * dpde_jn);
    double dusdxi = (us_ip - us_in) * rd0;
    double dusde = (us_jp - us_jn) * rd1;
    double dvsdxi = (vs_ip - vs_in) * rd0;
    double dvsde = (vs_jp - vs_jn) * rd1;
    double qq = (X[k] * dusdxi) + (E[k] * dusde) + (Y[k] * dvsdxi) + (G[k] * dvsde);
    return qq * a.rdt;
}

// ---------------------------------------------------------------------------
// pressure correction

// a 9-point stencil (a(0) .. a(8) in the order of the planes P_AP .. P_ASW) applied to the FP32
// field X at q, rows l0 apart; xc = X[q]
template <class A>
__device__ __forceinline__ double spmv_cell(const A& a, const float* X, long long q, int l0, double xc) {
    return a(0) * xc + a(1) * (double)X[q + 1] + a(2) * (double)X[q - 1] + a(3) * (double)X[q + l0] +
           a(4) * (double)X[q - l0] + a(5) * (double)X[q + l0 + 1] + a(6) * (double)X[q + l0 - 1] +
           a(7) * (double)X[q - l0 + 1] + a(8) * (double)X[q - l0 - 1];
}

// stored column of level column gi, gi in [-W, inf): the periodic wrap without a division
// in the common case (gi within one width of the level)
__device__ __forceinline__ int mg_wrap(int gi, int W) {
    int col = gi < 0 ? gi + W : gi;
    if (col >= W) col = col >= 2 * W ? col % W : col - W;
    return col;
}

__device__ __forceinline__ int mg_colour(int i, int j, int W, int periodic) {
    // 4 colours by parity; an odd periodic width gets 2 extra colours for its last column
    if (periodic && (W & 1) && i == W - 1) return 4 + (j & 1);
    return (i & 1) | ((j & 1) << 1);
}

// n / d rounded as the division rounds it, from y = the correctly rounded 1 / d: two residual
// corrections of n y (P. Markstein, Computation of elementary functions on the IBM RISC
// System/6000 processor, IBM J. Res. Dev. 34, 1990: with y correctly rounded, a quotient within
// an ulp is corrected to the rounded one). Five dependent operations instead of the twenty of a
// full division, which end every colour pass of a smoother whose diagonal never changes. For
// quotients outside 1e-30 .. 1e38 the last bit may differ.
__device__ __forceinline__ float mg_div(float n, float d, float y) {
    float q = n * y;
    q = fmaf(fmaf(-d, q, n), y, q);
    return fmaf(fmaf(-d, q, n), y, q);
}

// Pre-smoothing folded into the residual + restriction pass (schedule form `fused` = 2).
// One CTA per 32 x 8 tile of level l + 1. Its fine region E (the 65 x 17 fine points the
// restriction reads plus a one-cell ring: 67 x 19) is smoothed from zero in shared memory,
// zero outside E, by `inner` multicolour Gauss-Seidel sweeps; the residual is formed from
// that x and restricted into b_{l+1}; x is stored for the fine points the tile owns
// (columns 2 i0 .. 2 i0 + 63, rows 2 j0 - 1 .. 2 j0 + 14, and in the last tile row also the
// rows up to n1 - 2), where the post-smoother starts. Neighbouring regions overlap by up to
// three cells, and on a region's ring the residual uses the region's own smoothed x, not
// the owner's stored one. The V-cycle stays a fixed linear map (each CTA reads only level
// planes no CTA of the launch writes); it is a different map from form 1's, with the
// level's pre-smoothing pass and its read of the stencil saved.
constexpr int MPR_EW = 2 * TX + 3, MPR_EH = 2 * TY + 3;  // smoothed region E
constexpr int MPR_RW = 2 * TX + 1, MPR_RH = 2 * TY + 1;  // fine residual region
constexpr int MPR_BX = (MPR_EW + 1) / 2, MPR_BY = (MPR_EH + 1) / 2;  // 2 x 2 blocks of E: 34 x 10
// x of E with a zero ring (69 x 21 points), split by column parity; a parity half has rows
// of 40 words, and the second half starts 16 banks after the first
constexpr int MPR_XW = MPR_EW + 2, MPR_XH = MPR_EH + 2;
constexpr int MPR_XS = 40, MPR_XP = MPR_XH * MPR_XS + 8;
static_assert(MPR_XS >= (MPR_XW + 1) / 2 && MPR_XP % 32 == 16, "split layout of the region's x");
static_assert(MG_PRR_THREADS >= MPR_BX * MPR_BY && MG_PRR_THREADS >= TX * TY && MG_PRR_THREADS % 32 == 0,
              "one thread per 2 x 2 block of E, one per coarse point");

__device__ __forceinline__ int mpr_at(int xx, int ry) {  // point (xx, ry) of the ringed region
    return (xx & 1) * MPR_XP + ry * MPR_XS + (xx >> 1);
}
// the fine residual region (65 x 17 points), split by column parity like x: the blocks write
// it and the restriction reads it at column stride 2, which a plain row-major tile serves
// with two-way bank conflicts; split, consecutive threads touch consecutive words
constexpr int MPR_RS = 33, MPR_RP = MPR_RH * MPR_RS + 16;
__device__ __forceinline__ int mpr_rat(int x, int y) { return (x & 1) * MPR_RP + y * MPR_RS + (x >> 1); }

// Each thread owns one 2 x 2 block of E, which holds one point of each colour (E starts at
// an even column and row, and a level with a coarser one has an even width when periodic,
// so the colours are the four parity classes); its four stencils stay in registers.
template <bool WIDE, class Grp>
__device__ __forceinline__ void mg_prr_tile(const BatchDev& b, const CaseDev& c, int l, int i0, int j0, int dst,
                                            int inner, float* xs, float* rs, const Grp& g) {
    static_assert(Grp::N >= MPR_BX * MPR_BY && Grp::N >= TX * TY, "a thread per block of E, one per coarse point");
    const LevelDev& F = c.lev[l];
    const LevelDev& C = c.lev[l + 1];
    const int tid = g.tid;
    const int fl = F.ld, W = F.W, per = c.periodic, n1 = F.n1;
    if (per && (W & 1)) {  // a level with a coarser one has an even width
        if (tid == 0) atomicExch(b.error, 1);
        return;
    }
    const int ei0 = 2 * i0 - 2, ej0 = 2 * j0 - 2;  // level-l (column, row) of E's first point
    const bool own = tid < MPR_BX * MPR_BY;
    const int bx = own ? tid % MPR_BX : 0, by = own ? tid / MPR_BX : 0;
    const int gi0 = ei0 + 2 * bx;
    int c0, c1;  // stored columns of the block's two columns (c1 = c0 + 1 when both exist)
    if (per) {
        c0 = mg_wrap(gi0, W);
        c1 = c0 + 1;
    } else {
        c0 = (gi0 >= 0 && gi0 < W) ? gi0 : -1;
        c1 = (gi0 + 1 >= 0 && gi0 + 1 < W) ? gi0 + 1 : -1;
    }
    float a[2][2][10];  // [dy][dx][ap, ae, aw, an, as, ane, anw, ase, asw, b]
    bool ok[2][2];
#pragma unroll
    for (int dy = 0; dy < 2; dy++) {
        const int gj = ej0 + 2 * by + dy;
        const bool rowok = own && gj >= 1 && gj <= n1 - 2 && 2 * by + dy < MPR_EH;
        ok[dy][0] = rowok && c0 >= F.ilo && c0 <= F.ihi;
        ok[dy][1] = rowok && c1 >= F.ilo && c1 <= F.ihi && 2 * bx + 1 < MPR_EW;
        // the even column and its right neighbour, 8-byte aligned (safe row / column outside)
        const long long k = (long long)((gj >= 0 && gj < n1) ? gj : 1) * fl + (c0 >= 0 ? c0 : 0);
#pragma unroll
        for (int q = 0; q < 10; q++) {
            const float2 v = *reinterpret_cast<const float2*>(mplane(b, F, q < 9 ? M_AP + q : M_B) + k);
            a[dy][0][q] = v.x;
            a[dy][1][q] = v.y;
        }
    }
    float rdiag[2][2];  // reciprocals of the diagonals
#pragma unroll
    for (int dy = 0; dy < 2; dy++)
#pragma unroll
        for (int dx = 0; dx < 2; dx++) rdiag[dy][dx] = ok[dy][dx] ? __frcp_rn(a[dy][dx][0]) : 0.0f;
    for (int e = tid; e < 2 * MPR_XP; e += Grp::N) xs[e] = 0.0f;
    g.sync();
    // point of colour cc in the block: (dx, dy) = (cc & 1, cc >> 1); its ringed position is
    // (2 bx + dx + 1, 2 by + dy + 1)
    float xr[2][2] = {{0.0f, 0.0f}, {0.0f, 0.0f}};
    // the first sweep from zero: a colour's neighbours of the colours not yet relaxed are
    // still zero, so colour 0 reads none, colour 1 its E/W neighbours (colour 0), colour 2
    // its N/S (colour 0) and diagonal (colour 1) neighbours, colour 3 all eight
    auto relax0 = [&](auto cc_) {
        constexpr int cc = decltype(cc_)::value;
        constexpr int dx = cc & 1, dy = cc >> 1;
        if (ok[dy][dx]) {
            const float(&f)[10] = a[dy][dx];
            const int xx = 2 * bx + dx + 1, ry = 2 * by + dy + 1;
            float sm = 0.0f;
            if (cc == 1) sm = f[1] * xs[mpr_at(xx + 1, ry)] + f[2] * xs[mpr_at(xx - 1, ry)];
            if (cc == 2)
                sm = f[3] * xs[mpr_at(xx, ry + 1)] + f[4] * xs[mpr_at(xx, ry - 1)] +
                     f[5] * xs[mpr_at(xx + 1, ry + 1)] + f[6] * xs[mpr_at(xx - 1, ry + 1)] +
                     f[7] * xs[mpr_at(xx + 1, ry - 1)] + f[8] * xs[mpr_at(xx - 1, ry - 1)];
            if (cc == 3)
                sm = f[1] * xs[mpr_at(xx + 1, ry)] + f[2] * xs[mpr_at(xx - 1, ry)] +
                     f[3] * xs[mpr_at(xx, ry + 1)] + f[4] * xs[mpr_at(xx, ry - 1)] +
                     f[5] * xs[mpr_at(xx + 1, ry + 1)] + f[6] * xs[mpr_at(xx - 1, ry + 1)] +
                     f[7] * xs[mpr_at(xx + 1, ry - 1)] + f[8] * xs[mpr_at(xx - 1, ry - 1)];
            const float v = mg_div(f[9] - sm, f[0], rdiag[dy][dx]);
            xs[mpr_at(xx, ry)] = v;
            xr[dy][dx] = v;
        }
        g.sync();
    };
    auto relax = [&](auto cc_) {
        constexpr int cc = decltype(cc_)::value;
        constexpr int dx = cc & 1, dy = cc >> 1;
        if (ok[dy][dx]) {
            const float(&f)[10] = a[dy][dx];
            const int xx = 2 * bx + dx + 1, ry = 2 * by + dy + 1;
            const float sm = f[1] * xs[mpr_at(xx + 1, ry)] + f[2] * xs[mpr_at(xx - 1, ry)] +
                             f[3] * xs[mpr_at(xx, ry + 1)] + f[4] * xs[mpr_at(xx, ry - 1)] +
                             f[5] * xs[mpr_at(xx + 1, ry + 1)] + f[6] * xs[mpr_at(xx - 1, ry + 1)] +
                             f[7] * xs[mpr_at(xx + 1, ry - 1)] + f[8] * xs[mpr_at(xx - 1, ry - 1)];
            const float v = mg_div(f[9] - sm, f[0], rdiag[dy][dx]);
            xs[mpr_at(xx, ry)] = v;
            xr[dy][dx] = v;
        }
        g.sync();
    };
    using C0 = std::integral_constant<int, 0>;
    using C1 = std::integral_constant<int, 1>;
    using C2 = std::integral_constant<int, 2>;
    using C3 = std::integral_constant<int, 3>;
    if (inner > 0) {
        relax0(C0{}); relax0(C1{}); relax0(C2{}); relax0(C3{});
    }
    for (int n = 1; n < inner; n++) {
        relax(C0{}); relax(C1{}); relax(C2{}); relax(C3{});
    }
    // residual on the restriction's fine points (E without its ring), x of the owned points. The
    // block's four stencils read a 4 x 4 neighbourhood; WIDE holds it in registers (where one
    // CTA per SM leaves room: its latency is then one round of shared loads instead of four),
    // else every point reads its own eight neighbours
    float* OUT = mplane(b, F, dst);
    const int jhi = (j0 + TY > C.n1 - 2) ? n1 - 2 : min(2 * j0 + 14, n1 - 2);
    if (own) {
        float w[4][4] = {};
        if constexpr (WIDE) {
#pragma unroll
            for (int r = 0; r < 4; r++)
#pragma unroll
                for (int q = 0; q < 4; q++)
                    if (r >= 1 && r <= 2 && q >= 1 && q <= 2) w[r][q] = xr[r - 1][q - 1];
                    else w[r][q] = (2 * bx + q < MPR_XW && 2 * by + r < MPR_XH) ? xs[mpr_at(2 * bx + q, 2 * by + r)] : 0.0f;
        }
        auto nb = [&](int r, int q) -> float { return WIDE ? w[r][q] : xs[mpr_at(2 * bx + q, 2 * by + r)]; };
#pragma unroll
        for (int dy = 0; dy < 2; dy++) {
            const int y = 2 * by + dy, gj = ej0 + y;
            if (y < 1 || y > MPR_RH) continue;
            float v[2];
#pragma unroll
            for (int dx = 0; dx < 2; dx++) {
                const float(&f)[10] = a[dy][dx];
                float r = 0.0f;
                if (ok[dy][dx]) {
                    const float ax = f[0] * xr[dy][dx] + f[1] * nb(dy + 1, dx + 2) + f[2] * nb(dy + 1, dx) +
                                     f[3] * nb(dy + 2, dx + 1) + f[4] * nb(dy, dx + 1) + f[5] * nb(dy + 2, dx + 2) +
                                     f[6] * nb(dy + 2, dx) + f[7] * nb(dy, dx + 2) + f[8] * nb(dy, dx);
                    r = f[9] - ax;
                }
                const int x = 2 * bx + dx;
                if (x >= 1 && x <= MPR_RW) rs[mpr_rat(x - 1, y - 1)] = r;
                v[dx] = ok[dy][dx] ? xr[dy][dx] : 0.0f;
            }
            // owned: columns 2 i0 .. 2 i0 + 63 (E columns 2 .. 65, both of a block or none), rows up to jhi
            const int gi = ei0 + 2 * bx;
            if (bx < 1 || bx > TX || gj > jhi) continue;
            float* row = OUT + (long long)gj * fl;
            if (gi >= F.ilo && gi + 1 <= F.ihi) *reinterpret_cast<float2*>(row + gi) = make_float2(v[0], v[1]);
            else {
                if (gi >= F.ilo && gi <= F.ihi) row[gi] = v[0];
                if (gi + 1 >= F.ilo && gi + 1 <= F.ihi) row[gi + 1] = v[1];
            }
            if (per && gi == 0) { row[W] = v[0]; row[W + 1] = v[1]; }
            if (per && gi == W - 2) { row[-2] = v[0]; row[-1] = v[1]; }
        }
    }
    g.sync();
    if (tid >= TX * TY) return;
    const int li = tid % TX, lj = tid / TX;
    const int I = i0 + li, J = j0 + lj;
    if (I < C.ilo || I > C.ihi || J > C.n1 - 2) return;
    const int fx = 2 * li + 1, fy = 2 * lj + 1;  // fine (2I, 2J) in the residual region
    const float r4 = 0.0625f * (rs[mpr_rat(fx - 1, fy - 1)] + rs[mpr_rat(fx + 1, fy - 1)] + rs[mpr_rat(fx - 1, fy + 1)] +
                                rs[mpr_rat(fx + 1, fy + 1)]) +
                     0.125f * (rs[mpr_rat(fx, fy - 1)] + rs[mpr_rat(fx, fy + 1)] + rs[mpr_rat(fx - 1, fy)] +
                               rs[mpr_rat(fx + 1, fy)]) +
                     0.25f * rs[mpr_rat(fx, fy)];
    mplane(b, C, M_B)[(long long)J * C.ld + I] = r4;
}

// bilinear prolongation of the coarse result at fine point (i, j), i in [0, W): the four
// coarse points around it are loaded without a branch (an even index repeats its own point),
// since lanes of different parity would otherwise wait for one another's loads in turn: with
// that and one set of coarse loads per 2 x 2 block, k_mg_gs went from 279 to 218 us per step
// of the 256-case twin sweep
__device__ __forceinline__ float mg_prolong_at(const float* XC, int cl, int i, int j) {
    const int di = i & 1, dj = (j & 1) * cl;
    const float* q = XC + (long long)(j >> 1) * cl + (i >> 1);
    const float a = q[0], b = q[di], c = q[dj], d = q[dj + di];
    if (di && dj) return 0.25f * (a + b + c + d);
    if (di) return 0.5f * (a + b);
    if (dj) return 0.5f * (a + c);
    return a;
}

// Multicolour Gauss-Seidel sweeps of level l on a 32 x 16 tile (block Gauss-Seidel at tile
// edges: the halo ring holds the neighbouring tiles' values from before the first sweep).
// The sweeps read plane `src` and write plane `dst` != src, so nothing is read that another
// CTA writes.
//   mode 0: from x = 0, colours in order (first pre-sweep; src unused)
//   mode 1: from src, colours in order (further pre-sweeps)
//   mode 2: from src plus the prolonged result of level l + 1, colours reversed (first
//           post-sweep)
//   mode 3: from src, colours reversed (further post-sweeps)
// `inner` sweeps run back to back in shared memory (one launch and one read of the stencil
// for several sweeps, at the price of weaker coupling between tiles).
//
// A level with a coarser one has an even width when periodic, so its colours are the four
// parity classes. Tiles start at an even column and an odd row, so every 2 x 2 block of the
// tile holds one point of each colour: a thread owns one block (16 x 8 blocks, 128
// threads), keeps its four stencils in registers (loaded as column pairs) and relaxes one
// point per colour. x with its halo is held in shared memory split by column parity, rows
// padded so that a warp's two block rows fall in different banks: every read of a
// colour pass is free of bank conflicts.
constexpr int MG_GS_XW = TX + 2, MG_GS_XH = TYJ + 2;  // x halo region
constexpr int MG_GS_XS = 24;                           // row stride of a parity half
constexpr int MG_GS_XP = MG_GS_XH * MG_GS_XS;          // 432 = 16 mod 32 words
static_assert(MG_GS_XS >= (MG_GS_XW + 1) / 2 && (2 * MG_GS_XS) % 32 == 16 && MG_GS_XP % 32 == 16,
              "parity halves must keep a colour pass free of bank conflicts");
static_assert(MG_GS_THREADS == (TX / 2) * (TYJ / 2), "one thread per 2 x 2 block");
static_assert(MG_GS_THREADS >= 2 * (MG_GS_XW + TYJ), "one thread per point of the ring");

__device__ __forceinline__ int mg_gs_at(int xx, int ry) {  // halo point (xx, ry) in the split layout
    return (xx & 1) * MG_GS_XP + ry * MG_GS_XS + (xx >> 1);
}

template <class Grp>
__device__ __forceinline__ void mg_gs_tile(const BatchDev& b, const CaseDev& c, int l, int i0, int j0, int mode, int src,
                                           int dst, int inner, float* xs, const Grp& g) {
    static_assert(Grp::N == MG_GS_THREADS, "one thread per 2 x 2 block");
    const LevelDev& L = c.lev[l];
    const int tid = g.tid;
    const int ld = L.ld, W = L.W, per = c.periodic, n1 = L.n1;
    if (per && (W & 1)) {  // a level with a coarser one has an even width
        if (tid == 0) atomicExch(b.error, 1);
        return;
    }
    const bool zero = mode == 0, prolong = mode == 2, reverse = mode >= 2;
    const float* X = mplane(b, L, src);
    const float* XC = prolong ? mplane(b, c.lev[l + 1], mg_result_plane(b, c, l + 1)) : nullptr;
    const int cl = prolong ? c.lev[l + 1].ld : 0;
    // stored column of level column gi (periodic wrap), or -1 outside the level
    auto column = [&](int gi) -> int {
        if (per) return mg_wrap(gi, W);
        return (gi >= 0 && gi < W) ? gi : -1;
    };
    // this thread's 2 x 2 block: tile columns 2 bx, 2 bx + 1, rows 2 by, 2 by + 1
    const int bx = tid % (TX / 2), by = tid / (TX / 2);
    const int gi0 = i0 + 2 * bx;
    const int c0 = column(gi0), c1 = column(gi0 + 1);  // c1 = c0 + 1 whenever both are in the level
    float a[2][2][10];  // [dy][dx][ap^-1, ae, aw, an, as, ane, anw, ase, asw, b]
    bool ok[2][2];
#pragma unroll
    for (int dy = 0; dy < 2; dy++) {
        const int gj = j0 + 2 * by + dy;
        ok[dy][0] = gj >= 1 && gj <= n1 - 2 && c0 >= L.ilo && c0 <= L.ihi;
        ok[dy][1] = gj >= 1 && gj <= n1 - 2 && c1 >= L.ilo && c1 <= L.ihi;
        // an even column and its right neighbour, 8-byte aligned (safe row / column when outside)
        const long long k = (long long)((gj >= 0 && gj < n1) ? gj : 1) * ld + (c0 >= 0 ? c0 : 0);
#pragma unroll
        for (int q = 0; q < 10; q++) {
            const float2 v = *reinterpret_cast<const float2*>(mplane(b, L, q < 9 ? M_AP + q : M_B) + k);
            a[dy][0][q] = v.x;
            a[dy][1][q] = v.y;
        }
    }
    // x with the prolonged coarse correction (mode 2). The thread's own block starts at an even
    // column and an odd row, so the same four coarse points serve all of its four points;
    // the tile's ring of 100 points takes one thread each
    float xv[2][2] = {{0.0f, 0.0f}, {0.0f, 0.0f}}, xr = 0.0f;
    const bool ring = tid < 2 * (MG_GS_XW + TYJ);
    const int rx = tid < 2 * MG_GS_XW ? tid % MG_GS_XW : (tid & 1) * (MG_GS_XW - 1);
    const int ry0 = tid < MG_GS_XW ? 0 : tid < 2 * MG_GS_XW ? MG_GS_XH - 1 : 1 + (tid - 2 * MG_GS_XW) / 2;
    if (!zero) {
        const int ga = j0 + 2 * by;  // the block's odd row
        const int cc = c0 >= 0 ? c0 : 0, ra = ga < n1 ? ga : 1, rb = ga + 1 < n1 ? ga + 1 : 1;
        const float2 va = *reinterpret_cast<const float2*>(X + (long long)ra * ld + cc);
        const float2 vb = *reinterpret_cast<const float2*>(X + (long long)rb * ld + cc);
        const int gj = j0 - 1 + ry0, col = column(i0 - 1 + rx);
        const bool rin = ring && gj >= 0 && gj < n1 && col >= 0;
        const float vr = rin ? X[(long long)gj * ld + col] : 0.0f;
        float pa = 0.0f, pb = 0.0f, pc = 0.0f, pd = 0.0f, pr = 0.0f;
        if (prolong) {
            const float* q = XC + (long long)(ga <= n1 - 2 ? ga >> 1 : 0) * cl + (cc >> 1);
            const float A = q[0], B = q[1], C = q[cl], D = q[cl + 1];
            const bool run = rin && gj >= 1 && gj <= n1 - 2 && col >= L.ilo && col <= L.ihi;
            pr = mg_prolong_at(XC, cl, run ? col : L.ilo, run ? gj : 1);
            if (!run) pr = 0.0f;
            pa = 0.5f * (A + C);
            pb = 0.25f * (A + B + C + D);
            pc = C;
            pd = 0.5f * (C + D);
        }
        // a point outside the level is zero; a boundary point takes no correction
        const bool in0 = c0 >= 0, in1 = c1 >= 0;
        xv[0][0] = (in0 && ga < n1) ? (prolong && ok[0][0] ? va.x + pa : va.x) : 0.0f;
        xv[0][1] = (in1 && ga < n1) ? (prolong && ok[0][1] ? va.y + pb : va.y) : 0.0f;
        xv[1][0] = (in0 && ga + 1 < n1) ? (prolong && ok[1][0] ? vb.x + pc : vb.x) : 0.0f;
        xv[1][1] = (in1 && ga + 1 < n1) ? (prolong && ok[1][1] ? vb.y + pd : vb.y) : 0.0f;
        xr = vr + pr;
    }
#pragma unroll
    for (int dy = 0; dy < 2; dy++)
#pragma unroll
        for (int dx = 0; dx < 2; dx++) xs[mg_gs_at(2 * bx + dx + 1, 2 * by + dy + 1)] = xv[dy][dx];
    if (ring) xs[mg_gs_at(rx, ry0)] = xr;
#pragma unroll
    for (int dy = 0; dy < 2; dy++)
#pragma unroll
        for (int dx = 0; dx < 2; dx++) a[dy][dx][0] = ok[dy][dx] ? 1.0f / a[dy][dx][0] : 0.0f;
    g.sync();
    // point of colour cc in this thread's block: (dx, dy) = (cc & 1, 1 - (cc >> 1)) (the tile's
    // first row is odd); its halo position is (2 bx + dx + 1, 2 by + dy + 1)
    auto relax = [&](auto cc_) {
        constexpr int cc = decltype(cc_)::value;
        constexpr int dx = cc & 1, dy = 1 - (cc >> 1);
        if (ok[dy][dx]) {
            const float(&f)[10] = a[dy][dx];
            const int xx = 2 * bx + dx + 1, ry = 2 * by + dy + 1;
            const float sm = f[1] * xs[mg_gs_at(xx + 1, ry)] + f[2] * xs[mg_gs_at(xx - 1, ry)] +
                             f[3] * xs[mg_gs_at(xx, ry + 1)] + f[4] * xs[mg_gs_at(xx, ry - 1)] +
                             f[5] * xs[mg_gs_at(xx + 1, ry + 1)] + f[6] * xs[mg_gs_at(xx - 1, ry + 1)] +
                             f[7] * xs[mg_gs_at(xx + 1, ry - 1)] + f[8] * xs[mg_gs_at(xx - 1, ry - 1)];
            xs[mg_gs_at(xx, ry)] = (f[9] - sm) * f[0];
        }
        g.sync();
    };
    using C0 = std::integral_constant<int, 0>;
    using C1 = std::integral_constant<int, 1>;
    using C2 = std::integral_constant<int, 2>;
    using C3 = std::integral_constant<int, 3>;
    for (int n = 0; n < inner; n++) {
        if (reverse) { relax(C3{}); relax(C2{}); relax(C1{}); relax(C0{}); }
        else { relax(C0{}); relax(C1{}); relax(C2{}); relax(C3{}); }
    }
    float* OUT = mplane(b, L, dst);
#pragma unroll
    for (int dy = 0; dy < 2; dy++)
#pragma unroll
        for (int dx = 0; dx < 2; dx++) {
            const int i = gi0 + dx, j = j0 + 2 * by + dy;
            if (i < L.ilo || i > L.ihi || j > n1 - 2) continue;
            store_mirrored(OUT, ld, i, j, W, per, xs[mg_gs_at(2 * bx + dx + 1, 2 * by + dy + 1)]);
        }
}

// Galerkin coarse operator A_{l+1} = R A_l P at coarse point (I, J) (R full weighting, P
// bilinear, R = P^T / 4). Which coarse points a coupling reaches and with what weight depends
// only on the offsets, so the unrolled sums run over fixed registers; what is tested at run
// time is whether a point is an unknown.
__device__ __forceinline__ bool lev_unknown(const LevelDev& L, int periodic, int i, int j) {
    if (j < 1 || j > L.n1 - 2) return false;
    if (periodic) return true;
    return i >= L.ilo && i <= L.ihi;
}
__device__ __forceinline__ void mg_galerkin_point(const BatchDev& b, const CaseDev& c, int l, int I, int J) {
    const LevelDev& F = c.lev[l];
    const LevelDev& C = c.lev[l + 1];
    const int per = c.periodic, fl = F.ld;
    const float* A = mplane(b, F, M_AP);
    // stencil offsets in M_AP.. order: p, e, w, n, s, ne, nw, se, sw
    constexpr int ox[9] = {0, 1, -1, 0, 0, 1, -1, 1, -1};
    constexpr int oy[9] = {0, 0, 0, 1, -1, 1, 1, -1, -1};
    bool cu[3][3];  // coarse points around (I, J) that are unknowns
#pragma unroll
    for (int y = 0; y < 3; y++)
#pragma unroll
        for (int x = 0; x < 3; x++) cu[y][x] = lev_unknown(C, per, I + x - 1, J + y - 1);
    double acc[9];  // indexed (dy + 1) * 3 + (dx + 1)
#pragma unroll
    for (int m = 0; m < 9; m++) acc[m] = 0.0;
#pragma unroll
    for (int bj = -1; bj <= 1; bj++) {
#pragma unroll
        for (int bi = -1; bi <= 1; bi++) {
            const int fi = 2 * I + bi, fj = 2 * J + bj;
            if (!lev_unknown(F, per, fi, fj)) continue;
            const double wr = 0.25 * (bi == 0 ? 1.0 : 0.5) * (bj == 0 ? 1.0 : 0.5);
            const long long kf = (long long)fj * fl + fi;
#pragma unroll
            for (int m = 0; m < 9; m++) {
                const int sx = bi + ox[m], sy = bj + oy[m];  // fine point 2 (I, J) + (sx, sy)
                if (!lev_unknown(F, per, 2 * I + sx, 2 * J + sy)) continue;
                const double a = wr * (double)A[m * F.ps + kf];
                // its coarse parents: one along an even direction, two along an odd one
                const int nx = (sx & 1) ? 2 : 1, ny = (sy & 1) ? 2 : 1;
                const int px = (sx & 1) ? (sx - 1) / 2 : sx / 2, py = (sy & 1) ? (sy - 1) / 2 : sy / 2;
#pragma unroll
                for (int x = 0; x < 2; x++)
#pragma unroll
                    for (int y = 0; y < 2; y++) {
                        if (x >= nx || y >= ny || !cu[py + y + 1][px + x + 1]) continue;
                        acc[(py + y + 1) * 3 + px + x + 1] += a * (nx == 2 ? 0.5 : 1.0) * (ny == 2 ? 0.5 : 1.0);
                    }
            }
        }
    }
    constexpr int idx[9] = {4, 5, 3, 7, 1, 8, 6, 2, 0};  // p, e, w, n, s, ne, nw, se, sw
#pragma unroll
    for (int m = 0; m < 9; m++)
        store_mirrored(mplane(b, C, M_AP + m), C.ld, I, J, C.W, per, (float)acc[idx[m]]);
}

// Coarsest level: `sweeps` multicolour Gauss-Seidel sweeps by one group, x in shared memory
// (all rows, columns -H .. W+H-1). A thread holds the stencils of up to K points of each of the
// four parity colours in registers, so that every pass keeps all lanes busy; the last column
// of an odd periodic width has two colours of its own, whose few stencils are read where
// they are used. The points of a colour do not read one another, so the split over threads
// does not show in the result. A sweep is bound by the latency of its passes (a barrier,
// eight shared loads, eight multiply-adds, a quotient); through global memory, which levels
// of more than one unknown per thread used before, each pass paid L2 round trips instead: five
// steps of a 181 x 91 O-grid (90 x 44 unknowns on its coarsest level) took 5.75 ms, with the
// stencils in registers 2.68.
//
// mg_coarse_small: a level with no more unknowns than threads, one each (less set-up: 30
// against 38 us per step of the 256-case sweep).
template <class Grp>
__device__ __forceinline__ void mg_coarse_small(const BatchDev& b, const CaseDev& c, const LevelDev& L, int sweeps,
                                                float* xs, const Grp& g) {
    const int ld = L.ld, per = c.periodic, W = L.W;
    const int nx = L.ihi - L.ilo + 1, n = nx * (L.n1 - 2);
    const int ncol = (per && (W & 1)) ? 6 : 4;
    const int sw = W + 2 * H;
    for (int e = g.tid; e < L.n1 * sw; e += Grp::N) xs[e] = 0.0f;  // x = 0 (and boundaries)
    const bool in = g.tid < n;
    const int i = L.ilo + (in ? g.tid % nx : 0), j = 1 + (in ? g.tid / nx : 0);
    const long long p = (long long)j * ld + i;
    float f[9];
#pragma unroll
    for (int m = 0; m < 9; m++) f[m] = mplane(b, L, M_AP + m)[p];
    const float rhs = mplane(b, L, M_B)[p], rd = __frcp_rn(f[0]);
    const int col = in ? mg_colour(i, j, W, per) : -1;
    const int m = mirror_col(i, W, per);
    float* x = xs + j * sw + i + H;
    g.sync();
    for (int s = 0; s < sweeps; s++) {
        for (int cc = 0; cc < ncol; cc++) {
            if (col == cc) {
                const float sm = f[1] * x[1] + f[2] * x[-1] + f[3] * x[sw] + f[4] * x[-sw] + f[5] * x[sw + 1] +
                                 f[6] * x[sw - 1] + f[7] * x[-sw + 1] + f[8] * x[-sw - 1];
                const float v = mg_div(rhs - sm, f[0], rd);
                x[0] = v;
                if (m > -1000000) xs[j * sw + m + H] = v;
            }
            g.sync();
        }
    }
    if (in) store_mirrored(mplane(b, L, M_X), ld, i, j, W, per, x[0]);
}

struct MgColour {
    int fi, fj, nx, n;  // first column and row, points in a row, points
    __device__ __forceinline__ MgColour(const LevelDev& L, int per, int cc) {
        const int ie = per && (L.W & 1) ? L.W - 2 : L.ihi;
        fi = L.ilo + ((L.ilo ^ cc) & 1);
        fj = 1 + ((1 ^ (cc >> 1)) & 1);
        nx = ie >= fi ? (ie - fi) / 2 + 1 : 0;
        n = L.n1 - 2 >= fj ? nx * ((L.n1 - 2 - fj) / 2 + 1) : 0;
    }
};
template <int K, class Grp>
__device__ __forceinline__ void mg_coarse_regs(const BatchDev& b, const CaseDev& c, const LevelDev& L, int sweeps,
                                               float* xs, const Grp& g) {
    const int ld = L.ld, per = c.periodic, tid = g.tid, W = L.W;
    const int sw = W + 2 * H;
    float* X = mplane(b, L, M_X);
    const float* A = mplane(b, L, M_AP);
    const float* Bv = mplane(b, L, M_B);
    for (int e = tid; e < L.n1 * sw; e += Grp::N) xs[e] = 0.0f;  // x = 0 (and boundaries)
    float a[4][K][9], bv[4][K], y[4][K];
    int o[4][K];  // position in xs, and 1 / 2 in the top bits for a mirror W to the right / left; -1: none
#pragma unroll
    for (int cc = 0; cc < 4; cc++) {
        const MgColour q(L, per, cc);
#pragma unroll
        for (int k = 0; k < K; k++) {
            const int e = tid + k * Grp::N;
            const bool in = e < q.n;
            const int i = in ? q.fi + 2 * (e % q.nx) : L.ilo, j = in ? q.fj + 2 * (e / q.nx) : 1;
            const long long p = (long long)j * ld + i;
#pragma unroll
            for (int m = 0; m < 9; m++) a[cc][k][m] = A[m * L.ps + p];
            bv[cc][k] = Bv[p];
            y[cc][k] = __frcp_rn(a[cc][k][0]);
            o[cc][k] = in ? (j * sw + i + H) | ((per ? (i < 2 ? 1 : i >= W - 2 ? 2 : 0) : 0) << 28) : -1;
        }
    }
    auto relax = [&](int at, const float(&f)[9], float rhs, float rd) -> float {
        const float* x = xs + at;
        const float sm = f[1] * x[1] + f[2] * x[-1] + f[3] * x[sw] + f[4] * x[-sw] + f[5] * x[sw + 1] +
                         f[6] * x[sw - 1] + f[7] * x[-sw + 1] + f[8] * x[-sw - 1];
        return mg_div(rhs - sm, f[0], rd);
    };
    g.sync();
    for (int s = 0; s < sweeps; s++) {
#pragma unroll
        for (int cc = 0; cc < 4; cc++) {
#pragma unroll
            for (int k = 0; k < K; k++) {
                if (o[cc][k] < 0) continue;
                const int at = o[cc][k] & 0xfffffff, m = o[cc][k] >> 28;
                const float v = relax(at, a[cc][k], bv[cc][k], y[cc][k]);
                xs[at] = v;
                if (m) xs[m == 1 ? at + W : at - W] = v;
            }
            g.sync();
        }
        if (!(per && (W & 1))) continue;
        for (int cc = 0; cc < 2; cc++) {  // the last column's even rows, then its odd rows
            for (int j = 2 - cc + 2 * tid; j <= L.n1 - 2; j += 2 * Grp::N) {
                const long long p = (long long)j * ld + W - 1;
                float f[9];
#pragma unroll
                for (int m = 0; m < 9; m++) f[m] = A[m * L.ps + p];
                const int at = j * sw + W - 1 + H;
                const float v = relax(at, f, Bv[p], __frcp_rn(f[0]));
                xs[at] = v;
                xs[at - W] = v;
            }
            g.sync();
        }
    }
    const int nx = L.ihi - L.ilo + 1;
    for (int e = tid; e < nx * (L.n1 - 2); e += Grp::N) {
        const int i = L.ilo + e % nx, j = 1 + e / nx;
        store_mirrored(X, ld, i, j, W, per, xs[j * sw + i + H]);
    }
}

// The same sweeps for a level with more points of a colour than the threads hold: the stencils are
// read in every pass (from L2: a colour's are a quarter of the level's), four points per thread
// in flight at a time, and only the points of the pass's colour are visited. x is in shared
// memory where it fits, else in its own plane: `x` is point (0, 0), rows `xs` apart. Four steps of
// a 36 x 217 cavity (one level of 34 x 215 unknowns) take 14.7 ms with it, 33.0 with a visit of
// every point per pass and all of x in global memory.
template <class Grp>
__device__ __forceinline__ void mg_coarse_stream(const BatchDev& b, const CaseDev& c, const LevelDev& L, int sweeps,
                                                 float* x, int xs, const Grp& g) {
    constexpr int U = 4;
    const int ld = L.ld, per = c.periodic, W = L.W;
    const int nx = L.ihi - L.ilo + 1, n = nx * (L.n1 - 2);
    const float* A = mplane(b, L, M_AP);
    const float* Bv = mplane(b, L, M_B);
    for (int e = g.tid; e < n; e += Grp::N) store_mirrored(x, xs, L.ilo + e % nx, 1 + e / nx, W, per, 0.0f);
    g.sync();
    const bool odd = per && (W & 1);
    for (int s = 0; s < sweeps; s++) {
        for (int cc = 0; cc < (odd ? 6 : 4); cc++) {
            // colours 4 and 5: the last column's even and odd rows
            MgColour q(L, per, cc & 3);
            if (cc >= 4) {
                q.fi = W - 1;
                q.fj = 6 - cc;
                q.nx = 1;
                q.n = (L.n1 - 2 - q.fj) / 2 + 1;
            }
            for (int e0 = g.tid; e0 < q.n; e0 += U * Grp::N) {
                float f[U][9], rhs[U];
                int at[U], ii[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int e = e0 + u * Grp::N;
                    const int r = e < q.n ? e / q.nx : 0, i = e < q.n ? q.fi + 2 * (e - r * q.nx) : q.fi, j = q.fj + 2 * r;
                    const long long p = (long long)j * ld + i;
#pragma unroll
                    for (int m = 0; m < 9; m++) f[u][m] = A[m * L.ps + p];
                    rhs[u] = Bv[p];
                    at[u] = j * xs + i;
                    ii[u] = e < q.n ? i : -1;
                }
#pragma unroll
                for (int u = 0; u < U; u++) {
                    if (ii[u] < 0) continue;
                    float* v = x + at[u];
                    const float sm = f[u][1] * v[1] + f[u][2] * v[-1] + f[u][3] * v[xs] + f[u][4] * v[-xs] +
                                     f[u][5] * v[xs + 1] + f[u][6] * v[xs - 1] + f[u][7] * v[-xs + 1] +
                                     f[u][8] * v[-xs - 1];
                    const float r = (rhs[u] - sm) / f[u][0];
                    v[0] = r;
                    const int m = mirror_col(ii[u], W, per);
                    if (m > -1000000) v[m - ii[u]] = r;
                }
            }
            g.sync();
        }
    }
}

// KMAX: points of a colour per thread that the kernel's registers have room for
template <int KMAX, class Grp>
__device__ __forceinline__ void mg_coarse_solve(const BatchDev& b, const CaseDev& c, const LevelDev& L, int sweeps,
                                                float* xs, int xs_cap, const Grp& g) {
    // the odd rows' colours have at least as many points as the even rows', and one of the two
    // column parities the most
    const int most = max(MgColour(L, c.periodic, 2).n, MgColour(L, c.periodic, 3).n);
    const int sw = L.W + 2 * H, nx = L.ihi - L.ilo + 1, n = nx * (L.n1 - 2);
    const bool fits = L.n1 * sw <= xs_cap;
    float* X = mplane(b, L, M_X);
    if (fits && n <= Grp::N) {
        mg_coarse_small(b, c, L, sweeps, xs, g);
    } else if (fits && most <= Grp::N) {
        mg_coarse_regs<1>(b, c, L, sweeps, xs, g);
    } else if (fits && KMAX > 1 && most <= KMAX * Grp::N) {
        mg_coarse_regs<KMAX>(b, c, L, sweeps, xs, g);
    } else if (fits) {
        for (int e = g.tid; e < L.n1 * sw; e += Grp::N) xs[e] = 0.0f;
        g.sync();
        mg_coarse_stream(b, c, L, sweeps, xs + H, sw, g);
        for (int e = g.tid; e < n; e += Grp::N) {
            const int i = L.ilo + e % nx, j = 1 + e / nx;
            store_mirrored(X, L.ld, i, j, L.W, c.periodic, xs[j * sw + i + H]);
        }
    } else {
        mg_coarse_stream(b, c, L, sweeps, X, L.ld, g);
    }
}

// ---------------------------------------------------------------------------
// correction, boundaries and diagnostics

struct CorrOut {
    double un, vn, pn;
};

// velocity / pressure correction of one cell from pcor at it (pc) and its neighbours
// (PSolver.cpp:1471-1542); h0, h1 = 0.5 / dxi
__device__ __forceinline__ CorrOut correct_cell(double pc, double pN, double pS, double pE, double pW, double us,
                                                double vs, double xix, double xiy, double etx, double ety, double p0,
                                                double h0, double h1, double dt, double omega_p) {
    const double dpcor_dxi = (pE - pW) * h0;
    const double dpcor_de = (pN - pS) * h1;
    CorrOut o;
    o.un = us - dt * (xix * dpcor_dxi + etx * dpcor_de);
    o.vn = vs - dt * (xiy * dpcor_dxi + ety * dpcor_de);
    o.pn = (omega_p == 1.0) ? p0 + pc : p0 + omega_p * pc;
    return o;
}

// pcor on the boundary points beside cell (i, j) after its conditions (output only)
__device__ __forceinline__ void correct_bnd(double* PC, int ld, int W, int per, bool cav, int n0, int n1, int i, int j,
                                            double pc, double far) {
    const long long k = (long long)j * ld + i;
    if (j == 1) store_mirrored(PC, ld, i, 0, W, per, pc);
    if (j == n1 - 2) store_mirrored(PC, ld, i, n1 - 1, W, per, cav ? pc : far);
    if (cav) {
        if (i == 1) PC[k - 1] = pc;
        if (i == n0 - 2) PC[k + 1] = pc;
        if (i == 1 && j == 1) PC[0] = pc;
        if (i == n0 - 2 && j == 1) PC[n0 - 1] = pc;
        if (i == 1 && j == n1 - 2) PC[(long long)(n1 - 1) * ld] = pc;
        if (i == n0 - 2 && j == n1 - 2) PC[(long long)(n1 - 1) * ld + n0 - 1] = pc;
    }
}

struct DiagOut {
    double vort, dil;
};

// vorticity and dilatation of one interior cell (PSolver.cpp:1807-1853) from u, v at its four
// neighbours; h0, h1 = 0.5 / dxi (1 / (2 dxi) exactly)
__device__ __forceinline__ DiagOut diag_cell(double ue, double uw, double un, double us, double ve, double vw,
                                             double vn, double vs, double xix, double xiy, double etx, double ety,
                                             double h0, double h1) {
    DiagOut o;
    o.dil = xix * (ue - uw) * h0 + etx * (un - us) * h1 + ety * (vn - vs) * h1 + xiy * (ve - vw) * h0;
    const double dv_dxi = h0 * (ve - vw);
    const double dv_det = h1 * (vn - vs);
    const double du_dxi = h0 * (ue - uw);
    const double du_det = h1 * (un - us);
    o.vort = (xix * dv_dxi + etx * dv_det) - (xiy * du_dxi + ety * du_det);
    return o;
}

// the planes and constants of a case's boundary update
struct BcCase {
    const CaseDev& c;
    int ld, W, per, n1, n0, jf;
    double d0, d1, dt, Ri;
    double *U, *V, *Tn, *UPn, *VPn, *P, *VORT;
    const double *To, *X, *Yc, *XIX, *XIY, *ETX, *ETY, *ALPH, *BETA, *GAM, *JAC, *VEC;
    __device__ __forceinline__ BcCase(const BatchDev& b, const CaseDev& c_, int cur) : c(c_) {
        const int nxt = cur ^ 1;
        ld = c.ld; W = c.W; per = c.periodic; n1 = c.n1; n0 = c.n0; jf = n1 - 1;
        d0 = c.d0; d1 = c.d1; dt = c.dt; Ri = c.Ri;
        U = plane(b, c, P_U); V = plane(b, c, P_V); P = plane(b, c, P_P); VORT = plane(b, c, P_VORT);
        Tn = plane(b, c, P_T0 + nxt); UPn = plane(b, c, P_UP0 + nxt); VPn = plane(b, c, P_VP0 + nxt);
        To = plane(b, c, P_T0 + cur);
        X = plane(b, c, P_X); Yc = plane(b, c, P_Y);
        XIX = plane(b, c, P_XIX); XIY = plane(b, c, P_XIY); ETX = plane(b, c, P_ETX); ETY = plane(b, c, P_ETY);
        ALPH = plane(b, c, P_ALPH); BETA = plane(b, c, P_BETA); GAM = plane(b, c, P_GAM); JAC = plane(b, c, P_JAC);
        VEC = plane(b, c, P_VEC);
    }
};

// O-grid: circulation contribution of column i at j = n1-2 (PSolver.cpp:1568-1576); saves the
// far-field u, v before this update (uold of PSolver.cpp:1456) in s_old (2 (W + 1) doubles)
__device__ __forceinline__ double bc_circ(const BcCase& a, int i, double* s_old) {
    const double de = a.c.circ_de;
    const long long k = (long long)(a.n1 - 2) * a.ld + i, kp = k + 1;
    double f1 = (a.U[k] * a.ETY[k] - a.V[k] * a.ETX[k]) * fabs(a.JAC[k]);
    double f2 = (a.U[kp] * a.ETY[kp] - a.V[kp] * a.ETX[kp]) * fabs(a.JAC[kp]);
    const long long kf = (long long)a.jf * a.ld + i;
    s_old[i] = a.U[kf];
    s_old[a.W + 1 + i] = a.V[kf];
    return de * 0.5 * (f1 + f2);
}

// O-grid: far-field u, v, T of column i (PSolver.cpp:1549-1562, 1582-1609, 1632-1656)
struct FarOut {
    double u, v, T;
};
__device__ __forceinline__ FarOut bc_far(const BcCase& a, int i, double circ, const double* s_old) {
    const CaseDev& c = a.c;
    const double *U = a.U, *V = a.V, *X = a.X, *Yc = a.Yc;
    const long long kb = (long long)(a.jf - 1) * a.ld + i, k = (long long)a.jf * a.ld + i;
    const double costb = X[kb] / sqrt(X[kb] * X[kb] + Yc[kb] * Yc[kb]);
    const double sintb = Yc[kb] / sqrt(X[kb] * X[kb] + Yc[kb] * Yc[kb]);
    const double vr0 = U[kb] * costb + V[kb] * sintb;
    const double vth0 = -U[kb] * sintb + V[kb] * costb;
    const double cr = sqrt(X[kb] * X[kb] + Yc[kb] * Yc[kb]) / sqrt(X[k] * X[k] + Yc[k] * Yc[k]);
    const double costh = X[k] / sqrt(X[k] * X[k] + Yc[k] * Yc[k]);
    const double sinth = Yc[k] / sqrt(X[k] * X[k] + Yc[k] * Yc[k]);
    const double vrinf = c.uinf * costh + c.vinf * sinth;
    const double vtinf = -c.uinf * sinth + c.vinf * costh;
    const double cr2 = cr * cr;
    const double crk = fabs(circ) > 1e-2 ? cr : cr2;
    const double vr1 = vr0 * cr2 + vrinf * (1 - cr2);
    const double vth1 = vth0 * crk + vtinf * (1 - crk);
    const double vnn = c.uinf * a.VEC[2LL * a.ld + i] + c.vinf * a.VEC[3LL * a.ld + i];
    FarOut o;
    if (vnn >= 0) {
        o.u = c.uinf; o.v = c.vinf; o.T = 0.0;
    } else {
        o.u = costh * vr1 - sinth * vth1;
        o.v = sinth * vr1 + costh * vth1;
        const double uet_old = a.ETX[k] * s_old[i] + a.ETY[k] * s_old[a.W + 1 + i];
        o.T = a.To[k] - div_by(uet_old * a.dt, c.v1) * (a.To[k] - a.To[k - a.ld]);
    }
    store_mirrored(a.U, a.ld, i, a.jf, a.W, a.per, o.u);
    store_mirrored(a.V, a.ld, i, a.jf, a.W, a.per, o.v);
    store_mirrored(a.Tn, a.ld, i, a.jf, a.W, a.per, o.T);
    return o;
}

// O-grid: wall velocity of column i (PSolver.cpp:1617-1630). Rounded products: the team kernel
// forms a neighbour's value where k_bc reads it, so it must not melt into a later sum.
__device__ __forceinline__ double bc_wall_u(const BcCase& a, int i, double cwall) {
    return __dmul_rn(__dmul_rn(-a.c.speed_amp, cwall), a.Yc[i]);
}
__device__ __forceinline__ double bc_wall_v(const BcCase& a, int i, double cwall) {
    return __dmul_rn(__dmul_rn(a.c.speed_amp, cwall), a.X[i]);
}
__device__ __forceinline__ void bc_wall(const BcCase& a, int i, double uw, double vw) {
    store_mirrored(a.U, a.ld, i, 0, a.W, a.per, uw);
    store_mirrored(a.V, a.ld, i, 0, a.W, a.per, vw);
    store_mirrored(a.UPn, a.ld, i, 0, a.W, a.per, uw);
    store_mirrored(a.VPn, a.ld, i, 0, a.W, a.per, vw);
}

// cos and sin of the wall's phase 2 pi F t; exactly 1 and 0 for a wall at rest
__device__ __forceinline__ void bc_phase(const CaseDev& c, double t, double& cw, double& sw) {
    cw = 1.0;
    sw = 0.0;
    const double ang = 2.0 * c.Pi * c.F * t;
    if (ang != 0.0) {
        cw = cos(ang);
        sw = sin(ang);
    }
}

// u and v at a boundary point and its two neighbours along the boundary
struct Edge {
    double u, ue, uw, v, ve, vw;
};
__device__ __forceinline__ Edge edge_at(const BcCase& a, long long k) {
    return Edge{a.U[k], a.U[k + 1], a.U[k - 1], a.V[k], a.V[k + 1], a.V[k - 1]};
}

// One component of the boundary momentum balance lap(f) / Re - conv(f) at a boundary point: f at
// the point (f0), its neighbours along the boundary (fe, fw) and the two rows inside (f1, f2), the
// cross difference bd, the convection cy across the boundary. The callers subtract the
// acceleration of the boundary and add the buoyancy.
__device__ __forceinline__ double bc_force(const CaseDev& c, double f0, double fe, double fw, double f1, double f2,
                                           double bd, double al, double ga, double be, double uxi, double cy) {
    const double aa = div_by(al * (fe + fw - 2 * f0), c.v00);
    const double gg = div_by(ga * (f0 + f2 - 2 * f1), c.v11);
    const double bb = div_by(be * bd, c.v01);
    const double d2u = aa + gg - 2 * bb;
    double cv = div_by(uxi * 0.5 * (fe - fw), c.v0);
    cv = cv + cy;
    return div_by(1.0 * d2u, c.vRe) - cv;
}

// O-grid: wall pressure of column i (PSolver.cpp:1668-1725); swall = sin(2 pi F t). A moving wall
// makes the roundings of its velocity's products and of its acceleration show, so they are written
// out: which product melts into a sum would otherwise change with the code around it.
__device__ __forceinline__ double bc_wall_p(const BcCase& a, int i, const Edge& g, double swall) {
    const int ld = a.ld;
    const double *U = a.U, *V = a.V;
    const double d1 = a.d1;
    const long long k = i, k1 = k + ld, k2 = k + 2LL * ld;
    const double al = a.ALPH[k], ga = a.GAM[k], be = a.BETA[k], x = a.XIX[k], y = a.XIY[k], J = a.JAC[k];
    const double uxi = __fma_rn(x, g.u, __dmul_rn(y, g.v));
    const double uet = __fma_rn(a.ETX[k], g.u, __dmul_rn(a.ETY[k], g.v));
    const double u1 = U[k1], u2 = U[k2], ub = U[k1 + 1] + g.uw - U[k1 - 1] - g.ue;
    const double v1 = V[k1], v2 = V[k2], vb = V[k1 + 1] + g.vw - V[k1 - 1] - g.ve;
    const double acc = __dmul_rn(a.c.accn_amp, swall), T = a.Tn[k], p1 = a.P[k1];
    const double tu = bc_force(a.c, g.u, g.ue, g.uw, u1, u2, ub, al, ga, be, uxi, div_by(uet * (u1 - g.u), a.c.v1));
    const double tv = bc_force(a.c, g.v, g.ve, g.vw, v1, v2, vb, al, ga, be, uxi, div_by(uet * (v1 - g.v), a.c.v1));
    const double fu = __dsub_rn(tu, __dmul_rn(acc, a.Yc[k]));
    const double fv = __fma_rn(a.Ri, T, __fma_rn(acc, a.X[k], tv));
    const double pw = p1 - (fu * (-y * J) + fv * (x * J)) * d1;
    store_mirrored(a.P, ld, i, 0, a.W, a.per, pw);
    return pw;
}

// O-grid: far-field pressure of column i (PSolver.cpp:1726-1783); T = its temperature
__device__ __forceinline__ void bc_far_p(const BcCase& a, int i, const Edge& g, double T, const double* s_old) {
    const int ld = a.ld, W = a.W;
    const double *U = a.U, *V = a.V;
    const double d1 = a.d1;
    const long long k = (long long)a.jf * ld + i, k1 = k - ld, k2 = k - 2LL * ld;
    const double vnn = a.c.uinf * a.VEC[2LL * ld + i] + a.c.vinf * a.VEC[3LL * ld + i];
    const double ex = a.ETX[k], ey = a.ETY[k];
    const double u1 = U[k1], u2 = U[k2], v1 = V[k1], v2 = V[k2];
    double pf;
    if (vnn >= 0) {
        const double al = a.ALPH[k], ga = a.GAM[k], be = a.BETA[k], x = a.XIX[k], y = a.XIY[k], J = a.JAC[k];
        const double uxi = x * g.u + y * g.v;
        const double uet = ex * g.u + ey * g.v;
        const double ub = g.ue + U[k1 - 1] - U[k1 + 1] - g.uw, vb = g.ve + V[k1 - 1] - V[k1 + 1] - g.vw;
        const double alu = div_by(g.u - s_old[i], a.c.vdt), alv = div_by(g.v - s_old[W + 1 + i], a.c.vdt);
        const double nu = uet * (3.0 * g.u - 4 * u1 + u2), nv = uet * (3.0 * g.v - 4 * v1 + v2);
        const double fu = bc_force(a.c, g.u, g.ue, g.uw, u1, u2, ub, al, ga, be, uxi, div_by(nu, a.c.v1x2)) - alu;
        const double tv = bc_force(a.c, g.v, g.ve, g.vw, v1, v2, vb, al, ga, be, uxi, div_by(nv, a.c.v1x2)) - alv;
        const double fv = __fma_rn(a.Ri, T, tv);
        pf = a.P[k1] + (fu * (-y * J) + fv * (x * J)) * d1;
    } else {
        const double e0 = ex * g.u + ey * g.v;
        const double e1 = a.ETX[k1] * u1 + a.ETY[k1] * v1;
        const double e2 = a.ETX[k2] * u2 + a.ETY[k2] * v2;
        pf = 0.5 * a.c.vRe.y * div_by(3 * e0 - 4 * e1 + e2, a.c.v1);
    }
    store_mirrored(a.P, ld, i, a.jf, W, a.per, pf);
}

// vorticity of column i on boundary row j = 0 or n1-1 (PSolver.cpp:1855-1888)
__device__ __forceinline__ double bc_vort(const BcCase& a, int i, int j, const Edge& g) {
    const int ld = a.ld;
    const double *U = a.U, *V = a.V;
    const double hd0 = a.c.hd0, rd1 = a.c.rd1;
    const long long k = (long long)j * ld + i;
    const double dv_dxi = hd0 * (g.ve - g.vw);
    const double dv_det = (j == 0) ? rd1 * (V[k + ld] - g.v) : rd1 * (g.v - V[k - ld]);
    const double dv_dx = a.XIX[k] * dv_dxi + a.ETX[k] * dv_det;
    const double du_dxi = hd0 * (g.ue - g.uw);
    const double du_det = (j == 0) ? rd1 * (U[k + ld] - g.u) : rd1 * (g.u - U[k - ld]);
    const double du_dy = a.XIY[k] * du_dxi + a.ETY[k] * du_det;
    const double w = dv_dx - du_dy;
    store_mirrored(a.VORT, ld, i, j, a.W, a.per, w);
    return w;
}

// contributions of column i to the forces, moment and Nusselt number on j = 0
// (PSolver.cpp:1901-1983); P, VORT: row 0 of p and the vorticity
__device__ __forceinline__ void bc_integral(const BcCase& a, int i, const double* P, const double* VORT,
                                            double (&acc)[7]) {
    const int ld = a.ld;
    const double *JAC = a.JAC, *ETX = a.ETX, *ETY = a.ETY, *X = a.X, *Yc = a.Yc, *Tn = a.Tn;
    const double d0 = a.d0;
    const long long k = i, kp = i + 1;
    const double PJ1 = P[k] * JAC[k], pj2 = P[kp] * JAC[kp];
    const double VJ1 = VORT[k] * JAC[k], VJ2 = VORT[kp] * JAC[kp];
    acc[0] += 0.5 * d0 * (PJ1 * ETX[k] + pj2 * ETX[kp]);
    acc[1] += 0.5 * d0 * (PJ1 * ETY[k] + pj2 * ETY[kp]);
    acc[2] += 0.5 * d0 * (VJ1 * ETY[k] + VJ2 * ETY[kp]);
    acc[3] += 0.5 * d0 * (VJ1 * ETX[k] + VJ2 * ETX[kp]);
    const double TJ1 = JAC[k] * (ETX[k] * ETX[k] + ETY[k] * ETY[k]);
    const double TJ2 = JAC[kp] * (ETX[kp] * ETX[kp] + ETY[kp] * ETY[kp]);
    const double fp1 = PJ1 * (X[k] * ETY[k] - Yc[k] * ETX[k]);
    const double fp2 = pj2 * (X[kp] * ETY[kp] - Yc[kp] * ETX[kp]);
    const double fv1 = VJ1 * (X[k] * ETX[k] + Yc[k] * ETY[k]);
    const double fv2 = VJ2 * (X[kp] * ETX[kp] + Yc[kp] * ETY[kp]);
    const double fh1 = div_by(TJ1 * (4 * Tn[k + ld] - 3 * Tn[k] - Tn[k + 2LL * ld]), a.c.v1x2);
    const double fh2 = div_by(TJ2 * (4 * Tn[kp + ld] - 3 * Tn[kp] - Tn[kp + 2LL * ld]), a.c.v1x2);
    acc[4] += 0.5 * d0 * (fp1 + fp2);
    acc[5] += 0.5 * d0 * (fv1 + fv2);
    acc[6] += 0.5 * (fh1 + fh2) * d0;
}

// the case's wall integrals into its scalars (one thread)
__device__ __forceinline__ void bc_scalars(const CaseDev& c, const double (&acc)[7], double* sc) {
    const double Re = c.Re, Pi = c.Pi;
    const double pr_x = acc[0], pr_y = acc[1], vor_x = acc[2], vor_y = acc[3];
    const double cx = 2 * pr_x + (2.0 / Re) * vor_x;
    const double cy = 2 * pr_y - (2.0 / Re) * vor_y;
    const double sa = c.sa, ca = c.ca;
    sc[S_CLP] = 2 * pr_y * sa - 2 * pr_x * ca;
    sc[S_CDP] = 2 * pr_y * ca + 2 * pr_x * sa;
    sc[S_CLV] = -(2.0 / Re) * vor_y * sa - (2.0 / Re) * vor_x * ca;
    sc[S_CDV] = -(2.0 / Re) * vor_y * ca + (2.0 / Re) * vor_x * sa;
    sc[S_CL] = cy * sa - cx * ca;
    sc[S_CD] = cy * ca + cx * sa;
    sc[S_CM] = 2 * acc[4] - (2.0 / Re) * acc[5];
    const double ar = c.ar;
    if (c.profile != CAVITY)
        sc[S_NU] = (2 * acc[6]) / (Pi * (3 * (1 + (1.0 / ar)) - sqrt((3 + (1.0 / ar)) * ((3.0 / ar) + 1))));
    else
        sc[S_NU] = -acc[6];
}

// cavity: adiabatic side walls and zero normal pressure gradient (row j; column i; corners)
__device__ __forceinline__ void bc_cav_row(const BcCase& a, int j) {
    double *Tn = a.Tn, *P = a.P;
    const int n0 = a.n0;
    const long long r = (long long)j * a.ld;
    const DivBy three{3.0, 1.0 / 3.0};
    Tn[r] = div_by(4.0 * Tn[r + 1] - Tn[r + 2], three);
    Tn[r + n0 - 1] = div_by(4.0 * Tn[r + n0 - 2] - Tn[r + n0 - 3], three);
    P[r] = P[r + 1];
    P[r + n0 - 1] = P[r + n0 - 2];
}
__device__ __forceinline__ void bc_cav_col(const BcCase& a, int i) {
    a.P[i] = a.P[i + a.ld];
    a.P[(long long)a.jf * a.ld + i] = a.P[(long long)(a.jf - 1) * a.ld + i];
}
__device__ __forceinline__ void bc_cav_corners(const BcCase& a) {
    double* P = a.P;
    const int ld = a.ld, n0 = a.n0;
    P[0] = 0.5 * (P[1] + P[ld]);
    P[n0 - 1] = 0.5 * (P[n0 - 2] + P[ld + n0 - 1]);
    const long long r = (long long)a.jf * ld;
    P[r] = 0.5 * (P[r + 1] + P[r - ld]);
    P[r + n0 - 1] = 0.5 * (P[r + n0 - 2] + P[r - ld + n0 - 1]);
}

}  // namespace cfd
