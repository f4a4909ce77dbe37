// cfd_kernels.cu -- sm_100a kernels of one projection time step, batched over a case table.
//
// Reference mapping (mhsuhail00/CFD_Solver, PSolver.cpp):
//   k_assemble_p     pressure 9-point stencil            PSolver.cpp:944-1040
//   k_rhs            contravariant velocities,           PSolver.cpp:1063-1069
//                    convection + predictor RHS          PSolver.cpp:1075-1237
//   k_sweep_*        the five gauss() systems            PSolver.cpp:1241-1350, 2280-2446
//   (cfd_sweep.cu)   (u/v/T coefficients assembled in     PSolver.cpp:752-940
//                     shared memory from alpha, beta, gamma; k_sweep_fin, k_mom_fix,
//                     k_mom_update finish each sweep / solve)
//   k_upbc           up/vp far-field condition           PSolver.cpp:1356-1382
//   k_face_q         face velocities -> continuity q     PSolver.cpp:1390-1449
//   k_bicg_* / k_mg_*  pressure correction (replaces      PSolver.cpp:1453-1466, 2067-2278
//                    sip9p): BiCGStab on the stored 9-point stencil, preconditioned by a
//                    Galerkin multigrid V-cycle with multicolour Gauss-Seidel smoothing
//   k_correct        pcor BCs + velocity / p correction  PSolver.cpp:1471-1542
//   k_bc             far-field / wall BCs, circulation,  PSolver.cpp:1549-1783
//                    boundary pressure, wall integrals   PSolver.cpp:1901-1983
//   k_diag           dilatation, vorticity, dmax         PSolver.cpp:1807-1853
//   k_si             stream function (output only)       PSolver.cpp:1789-1801
#include "cfd_common.cuh"
#include "cfd_reduce.cuh"
#include "cfd_kernels.cuh"
#include "cfd_bulk.cuh"
#include "cfd_step.cuh"

namespace cfd {

// ---------------------------------------------------------------------------
// The 9-point pressure stencil at one cell (PSolver.cpp:944-1040) from the four metric
// planes X = xi_x, Y = xi_y, E = eta_x, G = eta_y at the cell and its four neighbours,
// in the order ap, ae, aw, an, as, ane, anw, ase, asw. c1 = 1 / (2 dxi0^2), c2 = 1 / (8 dxi0
// dxi1), c3 = 1 / (2 dxi1^2) (the reference divides by these; multiplying by reciprocals
// moves each coefficient by at most a unit in the last place). The stencil is stored
// once (k_assemble_p): rebuilding it inside the SpMV was measured slower (about 100 FP64
// operations per cell against 40 bytes saved).
template <typename T>
struct P9In {
    T x, xe, xw, xn, xs, y, ye, yw, yn, ys, e, ee, ew, en, es, g, ge, gw, gn, gs;
};

template <typename T>
__device__ __forceinline__ void p9_coefs(const P9In<T>& m, T c1, T c2, T c3, T (&a)[9]) {
    const T X = m.x, Y = m.y, E = m.e, G = m.g;
    a[1] = (X * c1) * (X + m.xe) + (E * c2) * (m.xn - m.xs) + (Y * c1) * (Y + m.ye) + (G * c2) * (m.yn - m.ys);
    a[2] = (X * c1) * (X + m.xw) + (E * c2) * (m.xs - m.xn) + (Y * c1) * (Y + m.yw) + (G * c2) * (m.ys - m.yn);
    a[3] = (X * c2) * (m.ee - m.ew) + (E * c3) * (E + m.en) + (Y * c2) * (m.ge - m.gw) + (G * c3) * (G + m.gn);
    a[4] = (X * c2) * (m.ew - m.ee) + (E * c3) * (E + m.es) + (Y * c2) * (m.gw - m.ge) + (G * c3) * (G + m.gs);
    a[5] = (X * c2) * (E + m.ee) + (E * c2) * (X + m.xn) + (Y * c2) * (G + m.ge) + (G * c2) * (Y + m.yn);
    a[8] = (X * c2) * (E + m.ew) + (E * c2) * (X + m.xs) + (Y * c2) * (G + m.gw) + (G * c2) * (Y + m.ys);
    a[6] = -((X * c2) * (E + m.ew)) - (E * c2) * (X + m.xn) - (Y * c2) * (G + m.gw) - (G * c2) * (Y + m.yn);
    a[7] = -((X * c2) * (E + m.ee)) - (E * c2) * (X + m.xs) - (Y * c2) * (G + m.ge) - (G * c2) * (Y + m.ys);
    a[0] = (-X * (T(2) * X + m.xw + m.xe)) * c1 + (-E * (T(2) * E + m.es + m.en)) * c3 +
           (-Y * (T(2) * Y + m.yw + m.ye)) * c1 + (-G * (T(2) * G + m.gs + m.gn)) * c3;
}

// the metrics around flat index k of planes X, Y, E, G with row pitch ld
template <typename T, typename S>
__device__ __forceinline__ P9In<T> p9_load(const S* X, const S* Y, const S* E, const S* G, long long k, int ld) {
    P9In<T> m;
    m.x = X[k]; m.xe = X[k + 1]; m.xw = X[k - 1]; m.xn = X[k + ld]; m.xs = X[k - ld];
    m.y = Y[k]; m.ye = Y[k + 1]; m.yw = Y[k - 1]; m.yn = Y[k + ld]; m.ys = Y[k - ld];
    m.e = E[k]; m.ee = E[k + 1]; m.ew = E[k - 1]; m.en = E[k + ld]; m.es = E[k - ld];
    m.g = G[k]; m.ge = G[k + 1]; m.gw = G[k - 1]; m.gn = G[k + ld]; m.gs = G[k - ld];
    return m;
}

// pressure stencil assembly, also the set-up of multigrid level 0 (stencil and the FP32
// metric copies its matrix-free sweeps read)
__global__ void __launch_bounds__(NT) k_assemble_p(BatchDev b, int toff) {
    const Tile t = b.ftiles[toff + blockIdx.x];
    const CaseDev& c = b.cases[t.c];
    const int i = t.i0 + (int)(threadIdx.x % TX), j = t.j0 + (int)(threadIdx.x / TX);
    if (i < c.ilo || i > c.ihi || j > c.n1 - 2) return;
    const int ld = c.ld, W = c.W, per = c.periodic;
    const long long k = (long long)j * ld + i;
    const P9In<double> m = p9_load<double>(plane(b, c, P_XIX), plane(b, c, P_XIY), plane(b, c, P_ETX),
                                           plane(b, c, P_ETY), k, ld);
    double vals[9];
    p9_coefs<double>(m, c.pc1, c.pc2, c.pc3, vals);
    const LevelDev& L0 = c.lev[0];
    const int ld0 = L0.ld;
#pragma unroll
    for (int q = 0; q < 9; q++) {
        store_mirrored(plane(b, c, P_AP + q), ld, i, j, W, per, vals[q]);
        store_mirrored(mplane(b, L0, M_AP + q), ld0, i, j, W, per, (float)vals[q]);
    }
}

// ---------------------------------------------------------------------------
// contravariant velocities + convection + the five right-hand sides
// (PSolver.cpp:1063-1237); also seeds the five solves' iterates. A CTA owns a 32 x 16 tile
// (two cells per thread); u, v, T, p, up, vp with a 2-cell halo and the seven metric
// planes of the tile arrive by tensor TMA into shared memory.
constexpr int RHS_HALO = 6, RHS_INT = 7;
constexpr size_t RHS_SMEM = (size_t)(RHS_HALO * JTW * JTH + RHS_INT * TX * TYJ) * sizeof(double) + 128;
const size_t kRhsSmem = RHS_SMEM;

// Three CTAs per SM (80 registers, 40 bytes of spills; the 63 KB staged per CTA fits three
// times): while one CTA computes, two others' copies are in flight. Two CTAs per SM at 122
// registers left the SM idle between a CTA's copies and its arithmetic (431 vs 373 us per
// step on the 256-case twin sweep).
__global__ void __launch_bounds__(NT, 3) k_rhs(BatchDev b) {
    after_previous();
    extern __shared__ __align__(128) unsigned char rraw[];
    __shared__ __align__(8) uint64_t bar;
    double* sm = reinterpret_cast<double*>((reinterpret_cast<uintptr_t>(rraw) + 127) & ~uintptr_t(127));
    const Tile t = b.jtiles[blockIdx.x];
    const CaseDev& c = b.cases[t.c];
    const int tid = threadIdx.x;
    const int cur = b.cur;
    // halo tiles: u, v, T, p, up, vp; interior tiles: xix, xiy, etx, ety, alpha, gamma, beta
    double* SI = sm + RHS_HALO * JTW * JTH;
    const bool active = b.iscal[(long long)t.c * NISCAL + I_ACTIVE] != 0;
    if (tid == 0 && t.k == 0) {
        int* is = b.iscal + (long long)t.c * NISCAL;
        int word = active ? (1 << NFIELD) - 1 : 0;
        for (int f = 0; f < NFIELD; f++) {
            is[I_MDONE0 + f] = active ? 0 : 1;
            is[I_MIT0 + f] = 0;
            is[I_MODD0 + f] = 0;
            is[I_MFLIP0 + f] = b.mixed ? 0 : is[I_MNEXT0 + f];
            word |= (is[I_MFLIP0 + f] != 0) << (NFIELD + f);
        }
        is[I_MWORD] = word;
        if (active) atomicAdd(b.mactive, NFIELD);
        else is[I_PDONE] = 1;  // an empty slot takes no part in the step
    }
    if (tid == 0) {  // the sweep kernel's word for this tile (I_MWORD of the case)
        int word = active ? (1 << NFIELD) - 1 : 0;
        if (active && !b.mixed)
            for (int f = 0; f < NFIELD; f++)
                word |= (b.iscal[(long long)t.c * NISCAL + I_MNEXT0 + f] != 0) << (NFIELD + f);
        b.tword[blockIdx.x] = word;
    }
    if (!active) return;
    if (tid == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
        const char* maps = b.tmaps + (size_t)t.c * TMAP_STRIDE;
        mbar_arrive_expect_tx(&bar, (RHS_HALO * JTW * JTH + RHS_INT * TX * TYJ) * sizeof(double));
        const int hp[RHS_HALO] = {P_U, P_V, P_T0 + cur, P_P, P_UP0 + cur, P_VP0 + cur};
        const int ip[RHS_INT] = {P_XIX, P_XIY, P_ETX, P_ETY, P_ALPH, P_GAM, P_BETA};
        for (int m = 0; m < RHS_HALO; m++) tma_load_3d(sm + m * JTW * JTH, maps, t.i0, t.j0 - 2, hp[m], &bar);
        for (int m = 0; m < RHS_INT; m++) tma_load_3d(SI + m * TX * TYJ, maps + 128, t.i0 + 2, t.j0, ip[m], &bar);
    }
    // the case's constants and planes, loaded while the copies are in flight
    const int ld = c.ld, W = c.W, per = c.periodic, n1 = c.n1, n0 = c.n0, ilo = c.ilo, ihi = c.ihi;
    const bool cav = c.profile == CAVITY;
    const RhsCase rc(c);
    double* const fb = b.f64 + c.base + H;  // plane 0 of the case; plane k at fb + k * ps
    const long long ps = c.ps;
    const bool warm = c.warm_up != 0;
    int nextm = 0;  // fields whose first iterate goes into the scratch plane (FP64 form)
    if (!b.mixed)
        for (int f = 0; f < NFIELD; f++) nextm |= (b.iscal[(long long)t.c * NISCAL + I_MNEXT0 + f] != 0) << f;
    __syncthreads();
    const bool ok = __syncthreads_and(mbar_wait_bounded(&bar, 0, b.wait_polls));
    if (!ok) {
        if (tid == 0) {
            atomicExch(b.error, 1);
            mbar_wait_bounded(&bar, 0);  // the copies land before the CTA leaves
        }
        return;
    }
    const double *Us = sm, *Vs = sm + JTW * JTH, *Ts = sm + 2 * JTW * JTH, *Ps = sm + 3 * JTW * JTH,
                 *UPs = sm + 4 * JTW * JTH, *VPs = sm + 5 * JTW * JTH;
    const int li = tid % TX, lj = tid / TX;
    const int i = t.i0 + li;
#pragma unroll 1
    for (int h = 0; h < 2; h++) {
        const int j = t.j0 + lj + h * TY;
        if (i < ilo || i > ihi || j > n1 - 2) continue;
        const int o = (lj + h * TY + 2) * JTW + (li + 2);
        const int oi = (lj + h * TY) * TX + li;
        const long long k = (long long)j * ld + i;
        const RhsOut r = rhs_cell<CrossAt>(rc, i, j, Us, Vs, Ts, Ps, UPs, VPs, o, JTW, SI[oi], SI[TX * TYJ + oi],
                                  SI[2 * TX * TYJ + oi], SI[3 * TX * TYJ + oi], SI[4 * TX * TYJ + oi],
                                  SI[5 * TX * TYJ + oi], SI + 6 * TX * TYJ + oi);
        fb[P_RU * ps + k] = r.qu;
        fb[P_RV * ps + k] = r.qv;
        fb[P_RT * ps + k] = r.qt;
        fb[P_RUP * ps + k] = r.qup;
        fb[P_RVP * ps + k] = r.qvp;
        const double seed[NFIELD] = {Us[o], Vs[o], Ts[o], warm ? UPs[o] : 0.0, warm ? VPs[o] : 0.0};
        rhs_seed<false>(fb, ps, nextm, cur, ld, W, per, cav, n0, n1, i, j, seed);
    }
}

// ---------------------------------------------------------------------------
// up/vp far-field condition (PSolver.cpp:1356-1382), one CTA per O-grid case
__global__ void __launch_bounds__(BC_THREADS) k_upbc(BatchDev b) {
    after_previous();
    const CaseDev& c = b.cases[blockIdx.x];
    if (c.profile != OGRID || !b.iscal[(long long)blockIdx.x * NISCAL + I_ACTIVE]) return;
    const int ld = c.ld, j = c.n1 - 1, nxt = b.cur ^ 1;
    double* UP = plane(b, c, P_UP0 + nxt);
    double* VP = plane(b, c, P_VP0 + nxt);
    const double* U = plane(b, c, P_U);
    const double* V = plane(b, c, P_V);
    const double* VEC = plane(b, c, P_VEC);
    for (int i = threadIdx.x; i < c.W; i += blockDim.x) {
        const double vnn = c.uinf * VEC[2LL * ld + i] + c.vinf * VEC[3LL * ld + i];
        const long long k = (long long)j * ld + i;
        double a, bb;
        if (vnn >= 0) {
            a = U[k];
            bb = V[k];
        } else {
            a = upbc_out(UP, k, ld);
            bb = upbc_out(VP, k, ld);
        }
        store_mirrored(UP, ld, i, j, c.W, 1, a);
        store_mirrored(VP, ld, i, j, c.W, 1, bb);
    }
}

// ---------------------------------------------------------------------------
// face velocities -> continuity source q (PSolver.cpp:1390-1449) with the
// mass-residual reductions; seeds the BiCGStab residual. 32 x 16 tiles, two cells per
// thread; p, up, vp and the four metric planes with their halo arrive by tensor TMA.
constexpr int FQ_HALO = 7;
constexpr size_t FQ_SMEM = (size_t)FQ_HALO * JTW * JTH * sizeof(double) + 128;
const size_t kFaceQSmem = FQ_SMEM;

__global__ void __launch_bounds__(NT, 4) k_face_q(BatchDev b) {
    after_previous();
    extern __shared__ __align__(128) unsigned char fraw[];
    __shared__ __align__(8) uint64_t bar;
    double* sm = reinterpret_cast<double*>((reinterpret_cast<uintptr_t>(fraw) + 127) & ~uintptr_t(127));
    const Tile t = b.jtiles[blockIdx.x];
    const CaseDev& c = b.cases[t.c];
    const int tid = threadIdx.x;
    const int nxt = b.cur ^ 1;
    if (!b.iscal[(long long)t.c * NISCAL + I_ACTIVE]) return;  // uniform over the case
    if (tid == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
        const char* maps = b.tmaps + (size_t)t.c * TMAP_STRIDE;
        mbar_arrive_expect_tx(&bar, FQ_HALO * JTW * JTH * sizeof(double));
        const int hp[FQ_HALO] = {P_P, P_UP0 + nxt, P_VP0 + nxt, P_XIX, P_XIY, P_ETX, P_ETY};
        for (int m = 0; m < FQ_HALO; m++) tma_load_3d(sm + m * JTW * JTH, maps, t.i0, t.j0 - 2, hp[m], &bar);
    }
    // the case's constants and output planes, loaded while the copies are in flight
    const int ld = c.ld, ilo = c.ilo, ihi = c.ihi, n1 = c.n1, ld0 = c.lev[0].ld;
    double* QP = plane(b, c, P_Q);
    double* KRP = plane(b, c, P_KR);
    float* B0 = mplane(b, c.lev[0], M_B);
    const FaceCase fc(c);
    __syncthreads();
    const bool ok = __syncthreads_and(mbar_wait_bounded(&bar, 0, b.wait_polls));
    if (!ok) {
        if (tid == 0) {
            atomicExch(b.error, 1);
            mbar_wait_bounded(&bar, 0);  // the copies land before the CTA leaves
        }
        return;
    }
    const double *P = sm, *U = sm + JTW * JTH, *V = sm + 2 * JTW * JTH, *X = sm + 3 * JTW * JTH,
                 *Y = sm + 4 * JTW * JTH, *E = sm + 5 * JTW * JTH, *G = sm + 6 * JTW * JTH;
    const int li = tid % TX, lj = tid / TX;
    const int i = t.i0 + li;
    double red[3] = {0.0, 0.0, 0.0};
    for (int h = 0; h < 2; h++) {
        const int j = t.j0 + lj + h * TY;
        if (!ok || i < ilo || i > ihi || j > n1 - 2) continue;
        const int k = (lj + h * TY + 2) * JTW + (li + 2);
        const double q = face_cell(fc, P, U, V, X, Y, E, G, k, JTW, U[k + JTW], V[k + JTW]);
        // q doubles as BiCGStab's shadow residual r_hat; p, v and the iterate pcor are
        // initialised by the first iteration's kernels (beta = 0, x = 0)
        const long long kg = (long long)j * ld + i;
        QP[kg] = q;
        KRP[kg] = q;
        // the first iteration's p = r_0 = q, as the preconditioner's right-hand side (k_bicg_p
        // has nothing to do in the first iteration; the second reads p_1 from the q plane)
        B0[(long long)j * ld0 + i] = (float)q;
        red[0] += fabs(q);
        red[1] += q * q;
        red[2] = fmax(red[2], fabs(q));
    }
    tile_partial<3, 0x4u>(b, blockIdx.x, 0, red);
}

// ---------------------------------------------------------------------------
// BiCGStab, right-preconditioned, FP64 vectors; per-case scalars live on the device
// The BiCGStab kernels run on the 32 x 16 tiles, two cells per thread (rows lj and
// lj + 8), every load of both cells issued before the arithmetic.
__global__ void __launch_bounds__(NT, 3) k_bicg_p(BatchDev b) {
    after_previous();
    const Tile t = b.jtiles[blockIdx.x];
    if (b.iscal[(long long)t.c * NISCAL + I_PDONE]) return;
    // p_{k+1} = r_k + beta (p_k - omega v_k), launched at the end of iteration k (after
    // k_bicg_x has counted it and formed beta). p_1 = r_0 = q is k_face_q's, written as the
    // preconditioner's right-hand side, so after the first iteration p_1 is read from the q
    // plane. Before any iteration (it == 0) there is nothing to do.
    const int it = b.iscal[(long long)t.c * NISCAL + I_PIT];
    if (it == 0) return;
    const CaseDev& c = b.cases[t.c];
    const int i = t.i0 + (int)(threadIdx.x % TX), j0 = t.j0 + (int)(threadIdx.x / TX);
    const double* sc = b.scal + (long long)t.c * NSCAL;
    const double beta = sc[S_BETA], omega = sc[S_OMEGA];
    double* Pv = plane(b, c, P_KP);
    const double* Pold = it == 1 ? plane(b, c, P_Q) : Pv;
    const double* R = plane(b, c, P_KR);
    const double* Vv = plane(b, c, P_KV);
    const LevelDev& L = c.lev[0];
    bool in[2];
    long long k[2];
    double r[2], po[2], v[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int j = j0 + h * TY;
        in[h] = i >= c.ilo && i <= c.ihi && j <= c.n1 - 2;
        k[h] = in[h] ? (long long)j * c.ld + i : (long long)c.ld + c.ilo;
        r[h] = R[k[h]];
        po[h] = Pold[k[h]];
        v[h] = Vv[k[h]];
    }
#pragma unroll
    for (int h = 0; h < 2; h++) {
        if (!in[h]) continue;
        const int j = j0 + h * TY;
        const double p = r[h] + beta * (po[h] - omega * v[h]);
        Pv[k[h]] = p;
        mplane(b, L, M_B)[(long long)j * L.ld + i] = (float)p;
    }
}

// y = A * x with x = (double) MG level-0 result; mode 0: p_hat, v, (r_hat, v) -> alpha
//                                               mode 1: s_hat, t, (t, s), (t, t) -> omega
__global__ void __launch_bounds__(NT, 5) k_spmv(BatchDev b, int mode) {
    after_previous();
    const Tile t = b.jtiles[blockIdx.x];
    if (b.iscal[(long long)t.c * NISCAL + I_PDONE]) return;
    const CaseDev& c = b.cases[t.c];
    const int i = t.i0 + (int)(threadIdx.x % TX), j0 = t.j0 + (int)(threadIdx.x / TX);
    const int ld = c.ld;
    const LevelDev& L = c.lev[0];
    const int l0 = L.ld;
    const float* X = mplane(b, L, mg_result_plane(b, c, 0));
    const double* DOT = plane(b, c, mode == 0 ? P_Q : P_KS);
    bool in[2];
    long long k[2];
    double y[2], xc[2], dv[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int j = j0 + h * TY;
        in[h] = i >= c.ilo && i <= c.ihi && j <= c.n1 - 2;
        const int jj = in[h] ? j : 1, ii = in[h] ? i : c.ilo;
        const long long kk = (long long)jj * ld + ii, q = (long long)jj * l0 + ii;
        k[h] = kk;
        xc[h] = (double)X[q];
        y[h] = spmv_cell([&](int m) { return plane(b, c, P_AP + m)[kk]; }, X, q, l0, xc[h]);
        dv[h] = DOT[kk];
    }
    double red[2] = {0.0, 0.0};
#pragma unroll
    for (int h = 0; h < 2; h++) {
        if (!in[h]) continue;
        if (mode == 0) {
            plane(b, c, P_KV)[k[h]] = y[h];
            red[0] += dv[h] * y[h];
        } else {
            plane(b, c, P_KT)[k[h]] = y[h];
            red[0] += y[h] * dv[h];
            red[1] += y[h] * y[h];
        }
    }
    if (mode == 0) {
        const double one[1] = {red[0]};
        tile_partial<1, 0u>(b, blockIdx.x, 0, one);
    } else {
        tile_partial<2, 0u>(b, blockIdx.x, 0, red);
    }
}

// s = r - alpha v, and the half step x += alpha p_hat; when |s| already meets the stop rule
// the solve ends here (the standard early exit: x + alpha p_hat is the iterate whose
// residual is s) and the second preconditioner application of the iteration is skipped
__global__ void __launch_bounds__(NT, 5) k_bicg_s(BatchDev b) {
    after_previous();
    const Tile t = b.jtiles[blockIdx.x];
    if (b.iscal[(long long)t.c * NISCAL + I_PDONE]) return;
    const bool first = b.iscal[(long long)t.c * NISCAL + I_PIT] == 0;
    const CaseDev& c = b.cases[t.c];
    const int i = t.i0 + (int)(threadIdx.x % TX), j0 = t.j0 + (int)(threadIdx.x / TX);
    const double alpha = b.scal[(long long)t.c * NSCAL + S_ALPHA];
    double* X = plane(b, c, P_PCOR);
    const double *R = plane(b, c, P_KR), *Vv = plane(b, c, P_KV);
    const LevelDev& L = c.lev[0];
    const float* PH = mplane(b, L, mg_result_plane(b, c, 0));  // p_hat, as the V-cycle left it
    bool in[2];
    long long k[2];
    double x0[2], r[2], v[2], ph[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int j = j0 + h * TY;
        in[h] = i >= c.ilo && i <= c.ihi && j <= c.n1 - 2;
        k[h] = in[h] ? (long long)j * c.ld + i : (long long)c.ld + c.ilo;
        x0[h] = first ? 0.0 : X[k[h]];
        r[h] = R[k[h]];
        v[h] = Vv[k[h]];
        ph[h] = (double)PH[in[h] ? (long long)j * L.ld + i : (long long)L.ld + c.ilo];
    }
    double red[1] = {0.0};
#pragma unroll
    for (int h = 0; h < 2; h++) {
        if (!in[h]) continue;
        const int j = j0 + h * TY;
        const double s = r[h] - alpha * v[h];
        const double x = x0[h] + alpha * ph[h];
        plane(b, c, P_KS)[k[h]] = s;
        store_mirrored(X, c.ld, i, j, c.W, c.periodic, x);
        mplane(b, L, M_B)[(long long)j * L.ld + i] = (float)s;
        red[0] += fabs(s);
    }
    tile_partial<1, 0u>(b, blockIdx.x, 0, red);
}

__global__ void __launch_bounds__(NT, 5) k_bicg_x(BatchDev b) {
    after_previous();
    const Tile t = b.jtiles[blockIdx.x];
    if (b.iscal[(long long)t.c * NISCAL + I_PDONE]) return;
    const CaseDev& c = b.cases[t.c];
    const int i = t.i0 + (int)(threadIdx.x % TX), j0 = t.j0 + (int)(threadIdx.x / TX);
    const double* sc0 = b.scal + (long long)t.c * NSCAL;
    const double omega = sc0[S_OMEGA];
    const int ld = c.ld;
    double* X = plane(b, c, P_PCOR);
    const LevelDev& L = c.lev[0];
    const float* SH = mplane(b, L, mg_result_plane(b, c, 0));  // s_hat, as the V-cycle left it
    const double *S = plane(b, c, P_KS), *T = plane(b, c, P_KT), *Q = plane(b, c, P_Q);
    bool in[2];
    long long k[2];
    double x0[2], sh[2], s[2], tt[2], q[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int j = j0 + h * TY;
        in[h] = i >= c.ilo && i <= c.ihi && j <= c.n1 - 2;
        k[h] = in[h] ? (long long)j * ld + i : (long long)ld + c.ilo;
        x0[h] = X[k[h]];
        sh[h] = (double)SH[in[h] ? (long long)j * L.ld + i : (long long)L.ld + c.ilo];
        s[h] = S[k[h]];
        tt[h] = T[k[h]];
        q[h] = Q[k[h]];
    }
    double red[2] = {0.0, 0.0};
#pragma unroll
    for (int h = 0; h < 2; h++) {
        if (!in[h]) continue;
        const int j = j0 + h * TY;
        // x already carries the half step alpha p_hat (k_bicg_s)
        store_mirrored(X, ld, i, j, c.W, c.periodic, x0[h] + omega * sh[h]);
        const double r = s[h] - omega * tt[h];
        plane(b, c, P_KR)[k[h]] = r;
        red[0] += q[h] * r;
        red[1] += fabs(r);
    }
    tile_partial<2, 0u>(b, blockIdx.x, 0, red);
}

// ---------------------------------------------------------------------------
// multigrid preconditioner, FP32, level tiles.
//
// One V-cycle: on the way down, level l is pre-smoothed from zero and its residual formed
// and restricted into b_{l+1} -- either by k_mg_gs (mode 0: writes x_l) followed by
// k_mg_rr, or (schedule form 2) by k_mg_prr in one pass over overlapping regions; then one
// k_mg_coarse launch smooths every case's coarsest level (one CTA per case, in place in x);
// on the way up, k_mg_gs (mode 2) adds the prolonged coarse result and post-smooths,
// writing the level's result into its r plane. No kernel reads a plane that another CTA of
// the same launch writes, so the V-cycle is a fixed linear map (the same bits whatever the
// CTA schedule), as the Krylov method needs. The level's final result lives in r (x for a
// case whose coarsest level it is).

// Residual r = b - A x of level l on the fine points a coarse tile of level l + 1 needs,
// in shared memory, then full-weighting restriction into b_{l+1} (tiles of level l + 1;
// levels start from x = 0 on their own). Fine points that are not unknowns contribute 0.
__global__ void __launch_bounds__(NT) k_mg_rr(BatchDev b, int l, int src) {
    after_previous();
    constexpr int RW = 2 * TX + 1, RH = 2 * TY + 1;  // fine residual region
    constexpr int XW = RW + 2, XH = RH + 2;          // fine x region (one-cell halo)
    __shared__ float xs[XH * XW];
    __shared__ float rs[RH * RW];
    const Tile t = b.atiles[l + 1][blockIdx.x];
    if (b.iscal[(long long)t.c * NISCAL + I_PDONE]) return;
    const CaseDev& c = b.cases[t.c];
    const LevelDev& F = c.lev[l];
    const LevelDev& C = c.lev[l + 1];
    const int tid = threadIdx.x;
    const int fl = F.ld, per = c.periodic;
    const int fi0 = 2 * t.i0 - 1, fj0 = 2 * t.j0 - 1;
    const float* X = mplane(b, F, src);
    for (int e = tid; e < XH * XW; e += NT) {
        const int gj = fj0 - 1 + e / XW, gi = fi0 - 1 + e % XW;
        float v = 0.0f;
        if (gj >= 0 && gj < F.n1 && gi >= -H && gi < F.W + H) v = X[(long long)gj * fl + gi];
        xs[e] = v;
    }
    __syncthreads();
    // fine unknown columns in stored form: periodic -1 .. W (halo mirrors), else ilo .. ihi
    const int clo = per ? -1 : F.ilo, chi = per ? F.W : F.ihi;
    for (int e = tid; e < RH * RW; e += NT) {
        const int rj = e / RW, ri = e % RW;
        const int gj = fj0 + rj, gi = fi0 + ri;
        float r = 0.0f;
        if (gj >= 1 && gj <= F.n1 - 2 && gi >= clo && gi <= chi) {
            const long long k = (long long)gj * fl + gi;
            const int o = (rj + 1) * XW + (ri + 1);
            const float ax = mplane(b, F, M_AP)[k] * xs[o] + mplane(b, F, M_AE)[k] * xs[o + 1] +
                             mplane(b, F, M_AW)[k] * xs[o - 1] + mplane(b, F, M_AN)[k] * xs[o + XW] +
                             mplane(b, F, M_AS)[k] * xs[o - XW] + mplane(b, F, M_ANE)[k] * xs[o + XW + 1] +
                             mplane(b, F, M_ANW)[k] * xs[o + XW - 1] + mplane(b, F, M_ASE)[k] * xs[o - XW + 1] +
                             mplane(b, F, M_ASW)[k] * xs[o - XW - 1];
            r = mplane(b, F, M_B)[k] - ax;
        }
        rs[e] = r;
    }
    __syncthreads();
    const int li = tid % TX, lj = tid / TX;
    const int I = t.i0 + li, J = t.j0 + lj;
    if (I < C.ilo || I > C.ihi || J > C.n1 - 2) return;
    const int f = (2 * lj + 1) * RW + (2 * li + 1);  // fine (2I, 2J) in the residual region
    const float v = 0.0625f * (rs[f - RW - 1] + rs[f - RW + 1] + rs[f + RW - 1] + rs[f + RW + 1]) +
                    0.125f * (rs[f - RW] + rs[f + RW] + rs[f - 1] + rs[f + 1]) + 0.25f * rs[f];
    const long long kc = (long long)J * C.ld + I;
    mplane(b, C, M_B)[kc] = v;
}

// pre-smoothing folded into the residual + restriction pass (mg_prr_tile): one CTA per
// 32 x 8 tile of level l + 1
__global__ void __launch_bounds__(MG_PRR_THREADS, 3) k_mg_prr(BatchDev b, int l, int dst, int inner) {
    after_previous();
    __shared__ float xs[2 * MPR_XP];
    __shared__ float rs[2 * MPR_RP];
    const Tile t = b.atiles[l + 1][blockIdx.x];
    if (b.iscal[(long long)t.c * NISCAL + I_PDONE]) return;
    const CaseDev& c = b.cases[t.c];
    mg_prr_tile<false>(b, c, l, t.i0, t.j0, dst, inner, xs, rs, BlockGroup<MG_PRR_THREADS>());
}

// multicolour Gauss-Seidel sweeps of level l on a 32 x 16 tile (mg_gs_tile)
__global__ void __launch_bounds__(MG_GS_THREADS, 8) k_mg_gs(BatchDev b, int l, int mode, int src, int dst, int inner) {
    after_previous();
    __shared__ float xs[2 * MG_GS_XP];
    const Tile t = b.mtiles[l][blockIdx.x];
    if (b.iscal[(long long)t.c * NISCAL + I_PDONE]) return;
    const CaseDev& c = b.cases[t.c];
    mg_gs_tile(b, c, l, t.i0, t.j0, mode, src, dst, inner, xs, BlockGroup<MG_GS_THREADS>());
}

// coarsest level: `sweeps` multicolour GS sweeps by one CTA per case (mg_coarse_solve)
constexpr int MGC_THREADS = 1024, MGC_SMEM = 12000;  // x of the level: 46.9 KB
__global__ void __launch_bounds__(MGC_THREADS) k_mg_coarse(BatchDev b, int l, int sweeps) {
    after_previous();
    __shared__ float xs[MGC_SMEM];
    // l < 0: one launch for every case, each on its own coarsest level (the case lists of
    // all levels are stored back to back from ccases[0])
    const int cid = l >= 0 ? b.ccases[l][blockIdx.x] : b.ccases[0][blockIdx.x];
    if (b.iscal[(long long)cid * NISCAL + I_PDONE]) return;
    const CaseDev& c = b.cases[cid];
    mg_coarse_solve<1>(b, c, c.lev[l >= 0 ? l : c.nlev - 1], sweeps, xs, MGC_SMEM, BlockGroup<MGC_THREADS>());
}

// Galerkin coarse operator of level l + 1 (mg_galerkin_point): one thread per coarse point
__global__ void __launch_bounds__(NT) k_mg_galerkin(BatchDev b, int l, int toff) {
    const Tile t = b.atiles[l + 1][toff + blockIdx.x];
    const CaseDev& c = b.cases[t.c];
    const LevelDev& C = c.lev[l + 1];
    const int I = t.i0 + (int)(threadIdx.x % TX), J = t.j0 + (int)(threadIdx.x / TX);
    if (I < C.ilo || I > C.ihi || J > C.n1 - 2) return;
    mg_galerkin_point(b, c, l, I, J);
}

// ---------------------------------------------------------------------------
// pcor boundary conditions + velocity / pressure correction (PSolver.cpp:1471-1542);
// also the momentum part of the steady residual, sum |u^{n+1} - u^n| + |v^{n+1} - v^n|
__global__ void __launch_bounds__(NT, 4) k_correct(BatchDev b) {
    after_previous();
    // a 32 x 16 tile, two cells per thread (rows lj and lj + 8): every load of both cells
    // is issued before any arithmetic
    const Tile t = b.jtiles[blockIdx.x];
    const CaseDev& c = b.cases[t.c];
    const int* isc = b.iscal + (long long)t.c * NISCAL;
    if (!isc[I_ACTIVE]) return;  // uniform over the case
    // no pressure iteration ran (q vanished or broke down at once): pcor = 0
    const bool none = isc[I_PIT] == 0;
    const int ld = c.ld, W = c.W, per = c.periodic, n1 = c.n1, n0 = c.n0;
    const bool cav = c.profile == CAVITY;
    double* PC = plane(b, c, P_PCOR);
    double* U = plane(b, c, P_U);
    double* V = plane(b, c, P_V);
    double* P = plane(b, c, P_P);
    const double* US = plane(b, c, P_US);
    const double* VS = plane(b, c, P_VS);
    const double* XIX = plane(b, c, P_XIX);
    const double* XIY = plane(b, c, P_XIY);
    const double* ETX = plane(b, c, P_ETX);
    const double* ETY = plane(b, c, P_ETY);
    const double* VEC = plane(b, c, P_VEC);
    const int i = t.i0 + (int)(threadIdx.x % TX);
    bool in[2];
    double pc0[2], pn0[2], ps0[2], pe0[2], pw0[2], us[2], vs[2], xix[2], etx[2], xiy[2], ety[2], u0[2], v0[2],
        p0[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int j = t.j0 + (int)(threadIdx.x / TX) + h * TY;
        in[h] = i >= c.ilo && i <= c.ihi && j <= n1 - 2;
        const long long k = in[h] ? (long long)j * ld + i : (long long)ld + c.ilo;  // a safe cell when out
        pc0[h] = PC[k]; pn0[h] = PC[k + ld]; ps0[h] = PC[k - ld]; pe0[h] = PC[k + 1]; pw0[h] = PC[k - 1];
        us[h] = US[k]; vs[h] = VS[k];
        xix[h] = XIX[k]; etx[h] = ETX[k]; xiy[h] = XIY[k]; ety[h] = ETY[k];
        u0[h] = U[k]; v0[h] = V[k]; p0[h] = P[k];
    }
    const double vnn = c.uinf * VEC[2LL * ld + i] + c.vinf * VEC[3LL * ld + i];
    const double h0 = c.hd0, h1 = c.hd1, dt = c.dt;  // the gradients' quotients as products
    double red[1] = {0.0};
#pragma unroll
    for (int h = 0; h < 2; h++) {
        if (!in[h]) continue;
        const int j = t.j0 + (int)(threadIdx.x / TX) + h * TY;
        const double pc = none ? 0.0 : pc0[h];
        // pcor on the boundary after its conditions: wall copy, far field 0 / copy at inflow
        const double far = (!cav && vnn >= 0) ? pc : 0.0;
        const double pN = none ? 0.0 : (j == n1 - 2) ? (cav ? pc : far) : pn0[h];
        const double pS = none ? 0.0 : (j == 1) ? pc : ps0[h];
        const double pE = none ? 0.0 : (cav && i == n0 - 2) ? pc : pe0[h];
        const double pW = none ? 0.0 : (cav && i == 1) ? pc : pw0[h];
        const CorrOut r = correct_cell(pc, pN, pS, pE, pW, us[h], vs[h], xix[h], xiy[h], etx[h], ety[h], p0[h], h0, h1,
                                       dt, c.omega_p);
        red[0] += fabs(r.un - u0[h]) + fabs(r.vn - v0[h]);
        store_mirrored(U, ld, i, j, W, per, r.un);
        store_mirrored(V, ld, i, j, W, per, r.vn);
        store_mirrored(P, ld, i, j, W, per, r.pn);
        if (none) store_mirrored(PC, ld, i, j, W, per, 0.0);
        // record the boundary pcor (output only)
        correct_bnd(PC, ld, W, per, cav, n0, n1, i, j, pc, far);
    }
    tile_partial<1, 0u>(b, blockIdx.x, 3, red);  // column 3: k_diag has 0 .. 2, one k_fin sums all
}

// ---------------------------------------------------------------------------
// boundary update, boundary pressure and wall integrals: one CTA per case
// (O-grid: PSolver.cpp:1549-1783 and 1855-1983; cavity: this project's walls)
__global__ void __launch_bounds__(BC_THREADS, 2) k_bc(BatchDev b) {
    after_previous();
    const int cid = blockIdx.x;
    const CaseDev& c = b.cases[cid];
    if (!b.iscal[(long long)cid * NISCAL + I_ACTIVE]) return;
    const BcCase a(b, c, b.cur);
    const int W = c.W, n1 = c.n1, n0 = c.n0;
    const bool cav = c.profile == CAVITY;
    __shared__ double red[16 * 32];
    __shared__ double s_circ;
    int* is = b.iscal + (long long)cid * NISCAL;
    double* sc = b.scal + (long long)cid * NSCAL;
    const int time_new = (int)((double)is[I_TIME] + c.dt);
    // the time the wall motion sees: the reference's int (PSolver.cpp:186), or t = n dt
    const double t_new = c.time_accurate ? sc[S_TIME] + c.dt : (double)time_new;
    extern __shared__ double s_old[];  // 2 * (W + 1); W <= 4096

    if (!cav) {
        {
            double acc[1] = {0.0};
            for (int i = threadIdx.x; i < W; i += blockDim.x) acc[0] += bc_circ(a, i, s_old);
            block_sum<1>(acc, red);
            if (threadIdx.x == 0) s_circ = acc[0];
            __syncthreads();
        }
        const double circ = s_circ;
        double cwall, swall;
        bc_phase(c, t_new, cwall, swall);
        for (int i = threadIdx.x; i < W; i += blockDim.x) {
            bc_far(a, i, circ, s_old);
            bc_wall(a, i, bc_wall_u(a, i, cwall), bc_wall_v(a, i, cwall));
        }
        __syncthreads();
        for (int i = threadIdx.x; i < W; i += blockDim.x) {
            bc_wall_p(a, i, edge_at(a, i), swall);
            const long long kf = (long long)a.jf * a.ld + i;
            bc_far_p(a, i, edge_at(a, kf), a.Tn[kf], s_old);
        }
    } else {
        // static walls
        for (int j = 1 + threadIdx.x; j <= n1 - 2; j += blockDim.x) bc_cav_row(a, j);
        for (int i = 1 + threadIdx.x; i <= n0 - 2; i += blockDim.x) bc_cav_col(a, i);
        __syncthreads();
        if (threadIdx.x == 0) bc_cav_corners(a);
    }
    __syncthreads();
    const int nb = c.ihi - c.ilo + 1;
    for (int e = threadIdx.x; e < 2 * nb; e += blockDim.x) {
        const int i = c.ilo + e % nb, j = (e < nb) ? 0 : n1 - 1;
        bc_vort(a, i, j, edge_at(a, (long long)j * a.ld + i));
    }
    __syncthreads();
    double acc[7] = {0, 0, 0, 0, 0, 0, 0};
    for (int i = threadIdx.x; i <= n0 - 2; i += blockDim.x) bc_integral(a, i, a.P, a.VORT, acc);
    block_sum<7>(acc, red);
    if (threadIdx.x == 0) {
        bc_scalars(c, acc, sc);
        sc[S_CIRC] = cav ? 0.0 : s_circ;
        is[I_TIME] = time_new;
        sc[S_TIME] = t_new;
    }
}

// ---------------------------------------------------------------------------
// dilatation, interior vorticity, dmax and the energy residual (PSolver.cpp:1807-1853)
__global__ void __launch_bounds__(NT, 3) k_diag(BatchDev b) {
    after_previous();
    // a 32 x 16 tile, two cells per thread; all loads of both cells first
    const Tile t = b.jtiles[blockIdx.x];
    const CaseDev& c = b.cases[t.c];
    if (!b.iscal[(long long)t.c * NISCAL + I_ACTIVE]) return;  // uniform over the case
    const int ld = c.ld, W = c.W, per = c.periodic;
    const int i = t.i0 + (int)(threadIdx.x % TX);
    const double* U = plane(b, c, P_U);
    const double* V = plane(b, c, P_V);
    const double* XIX = plane(b, c, P_XIX);
    const double* XIY = plane(b, c, P_XIY);
    const double* ETX = plane(b, c, P_ETX);
    const double* ETY = plane(b, c, P_ETY);
    const double* TN = plane(b, c, P_T0 + (b.cur ^ 1));
    const double* TO = plane(b, c, P_T0 + b.cur);
    bool in[2];
    double ue[2], uw[2], un[2], us[2], ve[2], vw[2], vn[2], vs[2], xix[2], xiy[2], etx[2], ety[2], tn[2], to[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int j = t.j0 + (int)(threadIdx.x / TX) + h * TY;
        in[h] = i >= c.ilo && i <= c.ihi && j <= c.n1 - 2;
        const long long k = in[h] ? (long long)j * ld + i : (long long)ld + c.ilo;  // a safe cell when out
        ue[h] = U[k + 1]; uw[h] = U[k - 1]; un[h] = U[k + ld]; us[h] = U[k - ld];
        ve[h] = V[k + 1]; vw[h] = V[k - 1]; vn[h] = V[k + ld]; vs[h] = V[k - ld];
        xix[h] = XIX[k]; xiy[h] = XIY[k]; etx[h] = ETX[k]; ety[h] = ETY[k];
        tn[h] = TN[k]; to[h] = TO[k];
    }
    // 0.5 / d is 1 / (2 d) exactly: the dilatation's quotients become products
    const double h0 = c.hd0, h1 = c.hd1;
    double red[3] = {-1.0e300, 0.0, 0.0};
#pragma unroll
    for (int h = 0; h < 2; h++) {
        if (!in[h]) continue;
        const int j = t.j0 + (int)(threadIdx.x / TX) + h * TY;
        const DiagOut d = diag_cell(ue[h], uw[h], un[h], us[h], ve[h], vw[h], vn[h], vs[h], xix[h], xiy[h], etx[h],
                                    ety[h], h0, h1);
        store_mirrored(plane(b, c, P_VORT), ld, i, j, W, per, d.vort);
        store_mirrored(plane(b, c, P_DIL), ld, i, j, W, per, d.dil);
        const double dT = fabs(tn[h] - to[h]);
        red[0] = fmax(red[0], d.dil);
        red[1] += dT;
        red[2] = fmax(red[2], dT);
    }
    tile_partial<3, 0x5u>(b, blockIdx.x, 0, red);
}

// The case's totals of the tile kernel just launched and what follows from them: one CTA per
// case. `maxit` is the pressure solve's cap.
template <int WHAT>
__device__ __forceinline__ void fin_case(const BatchDev& b, int cid, int maxit) {
    const CaseDev& c = b.cases[cid];
    int* is = b.iscal + (long long)cid * NISCAL;
    double* sc = b.scal + (long long)cid * NSCAL;
    if (WHAT == FIN_FACE_Q || WHAT == FIN_STEP) {
        if (!is[I_ACTIVE]) return;
    } else if (is[I_PDONE]) {
        return;
    }
    const int tb = c.jt_begin, tn = c.jt_count;
    if constexpr (WHAT == FIN_FACE_Q) {
        double red[3];
        case_total<3, 0x4u>(b, tb, tn, red);
        if (threadIdx.x != 0) return;
        sc[S_QL1] = red[0];
        sc[S_QL2] = sqrt(red[1]);
        if (is[I_NSTEP] == 0) sc[S_QL2_0] = sqrt(red[1]);
        sc[S_QMAX] = red[2];
        sc[S_RHO] = red[1];
        sc[S_ALPHA] = 1.0;
        sc[S_OMEGA] = 1.0;
        sc[S_BETA] = 0.0;
        sc[S_NB1] = red[0];
        sc[S_RL1] = red[0];
        is[I_PIT] = 0;
        // this step's solver status starts with the momentum / energy solves: a field still
        // iterating when their loop ended stopped at the sweep cap
        is[I_PSTATUS] = (is[I_MWORD] & ((1 << NFIELD) - 1)) ? ST_MAXITER : 0;
        if (red[0] == 0.0 || !isfinite(red[0])) {
            is[I_PDONE] = 1;
            if (!isfinite(red[0])) is[I_STATUS] |= ST_NAN;
        } else {
            is[I_PDONE] = 0;
            atomicAdd(b.active, 1);
        }
    } else if constexpr (WHAT == FIN_SPMV0) {
        double red[1];
        case_total<1, 0u>(b, tb, tn, red);
        if (threadIdx.x != 0) return;
        if (red[0] == 0.0 || !isfinite(red[0])) {
            is[I_PSTATUS] |= ST_BREAKDOWN;
            is[I_PDONE] = 1;
            atomicSub(b.active, 1);
        } else {
            sc[S_ALPHA] = sc[S_RHO] / red[0];
        }
    } else if constexpr (WHAT == FIN_SPMV1) {
        double red[2];
        case_total<2, 0u>(b, tb, tn, red);
        if (threadIdx.x == 0) sc[S_OMEGA] = red[1] > 0.0 ? red[0] / red[1] : 0.0;
    } else if constexpr (WHAT == FIN_BICG_S) {
        double red[1];
        case_total<1, 0u>(b, tb, tn, red);
        if (threadIdx.x != 0) return;
        const bool conv = red[0] <= c.tol_p * sc[S_NB1] || red[0] <= c.atol_p;
        if (conv || !isfinite(red[0])) {
            is[I_PIT] += 1;
            sc[S_RL1] = red[0];
            if (!isfinite(red[0])) is[I_STATUS] |= ST_NAN;
            is[I_PDONE] = 1;
            atomicSub(b.active, 1);
        }
    } else if constexpr (WHAT == FIN_BICG_X) {
        double red[2];
        case_total<2, 0u>(b, tb, tn, red);
        if (threadIdx.x != 0) return;
        const double alpha = sc[S_ALPHA], omega = sc[S_OMEGA];
        const int it = ++is[I_PIT];
        const double rho_new = red[0];
        sc[S_RL1] = red[1];
        const bool conv = red[1] <= c.tol_p * sc[S_NB1] || red[1] <= c.atol_p;
        bool stop = conv;
        if (!isfinite(red[1])) { is[I_STATUS] |= ST_NAN; stop = true; }
        else if (!conv && (omega == 0.0 || rho_new == 0.0)) { is[I_PSTATUS] |= ST_BREAKDOWN; stop = true; }
        else if (!conv && it >= maxit) { is[I_PSTATUS] |= ST_MAXITER; stop = true; }
        if (!stop) {
            sc[S_BETA] = (rho_new / sc[S_RHO]) * (alpha / omega);
            sc[S_RHO] = rho_new;
        } else {
            is[I_PDONE] = 1;
            atomicSub(b.active, 1);
        }
    } else {  // the step's residuals: k_diag's columns 0 .. 2, k_correct's 3
        double red[4];
        case_total<4, 0x5u>(b, tb, tn, red);
        if (threadIdx.x != 0) return;
        sc[S_DMAX] = fmax(red[0], 0.0);
        sc[S_DTL1] = red[1];
        sc[S_DTMAX] = red[2];
        sc[S_DUL1] = red[3];
        // steady residual: mean (|du| + |dv| + |dT|) / dt over the unknown cells
        const double ncell = (double)(c.ihi - c.ilo + 1) * (c.n1 - 2);
        sc[S_SR] = (red[3] + red[1]) / (c.dt * ncell);
        if (is[I_NSTEP] == 0) sc[S_SR0] = sc[S_SR];
        is[I_NSTEP] += 1;
    }
}
__global__ void __launch_bounds__(NT) k_fin(BatchDev b, FinKernel what, int maxit) {
    after_previous();
    switch (what) {
        case FIN_FACE_Q: fin_case<FIN_FACE_Q>(b, blockIdx.x, maxit); break;
        case FIN_SPMV0: fin_case<FIN_SPMV0>(b, blockIdx.x, maxit); break;
        case FIN_SPMV1: fin_case<FIN_SPMV1>(b, blockIdx.x, maxit); break;
        case FIN_BICG_S: fin_case<FIN_BICG_S>(b, blockIdx.x, maxit); break;
        case FIN_BICG_X: fin_case<FIN_BICG_X>(b, blockIdx.x, maxit); break;
        case FIN_STEP: fin_case<FIN_STEP>(b, blockIdx.x, maxit); break;
    }
}

// stream function, a scan along j per column (PSolver.cpp:1789-1801)
__global__ void __launch_bounds__(BC_THREADS) k_si(BatchDev b) {
    const CaseDev& c = b.cases[blockIdx.x];
    const int ld = c.ld;
    double* SI = plane(b, c, P_SI);
    const double* U = plane(b, c, P_U);
    const double* V = plane(b, c, P_V);
    const double* XIX = plane(b, c, P_XIX);
    const double* XIY = plane(b, c, P_XIY);
    const double* JAC = plane(b, c, P_JAC);
    const int ncol = c.periodic ? c.W : c.n0;
    for (int i = threadIdx.x; i < ncol; i += blockDim.x) {
        double s = 0.0;
        store_mirrored(SI, ld, i, 0, c.W, c.periodic, 0.0);
        for (int j = 1; j < c.n1; j++) {
            const long long k = (long long)j * ld + i, kb = k - ld;
            const double ca = (XIX[k] * U[k] * fabs(JAC[k]) + XIX[kb] * U[kb] * fabs(JAC[kb]));
            const double cb = (XIY[k] * V[k] * fabs(JAC[k]) + XIY[kb] * V[kb] * fabs(JAC[kb]));
            s = s + (ca + cb) * 0.5 * c.d1;
            store_mirrored(SI, ld, i, j, c.W, c.periodic, s);
        }
    }
}

// condition of a graph while-loop: keep looping while `*flag > 0` and fewer than `maxc`
// iterations ran this step; `total` accumulates iterations over all steps
__global__ void k_loop_cond(cudaGraphConditionalHandle h, const int* flag, int* counter, int maxc,
                            int* total) {
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        const int n = ++(*counter);
        atomicAdd(total, 1);
        cudaGraphSetConditional(h, (*flag > 0 && n < maxc) ? 1u : 0u);
    }
}

// condition of a graph if-node: run the body when `*flag > 0`; `total` counts the runs
__global__ void k_if_cond(cudaGraphConditionalHandle h, const int* flag, int* total) {
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        const bool go = *flag > 0;
        if (go) atomicAdd(total, 1);
        cudaGraphSetConditional(h, go ? 1u : 0u);
    }
}

// ---------------------------------------------------------------------------
// Resident state <-> one contiguous staging buffer (so a state snapshot crosses PCIe as one
// copy per direction). Per case: the six state planes u, v, p, T, up, vp, each n1 rows of the
// stored columns (n0 for the cavity, W = n0 - 1 for the periodic O-grid), then 16 doubles:
// int time and int steps taken, then the first-step steady residual and continuity norm (the
// references of the relative residuals), then the time as a double. Unpacking writes the periodic halo mirrors too.
// blockIdx.x = case * 7 + m (m = 6: the counter slot), blockIdx.y = STATE_ROWS rows of the plane;
// one warp per row. The call is bound by PCIe (55.7 GB/s) once the packing keeps up: with one CTA
// per plane a 1025 x 1025 case (50 MB) kept six SMs busy and its snapshot took 2,562 us, 944 in
// row blocks; 64 cases (87 MB) 1,680 and 1,587, 256 cases (396 MB) 7,164 and 7,108.
__global__ void __launch_bounds__(256) k_state_pack(BatchDev b, double* stage, const long long* off, int to_stage) {
    const int c = blockIdx.x / 7, m = blockIdx.x % 7;
    const CaseDev& d = b.cases[c];
    const int nc = d.periodic ? d.W : d.n0;
    double* dst = stage + off[c] + (long long)m * d.n1 * nc;
    if (m == 6) {
        // the case's counters: the reference's int time, the steps taken, and the
        // first-step references of the relative residuals
        int* is = b.iscal + (long long)c * NISCAL;
        double* sc = b.scal + (long long)c * NSCAL;
        int* di = reinterpret_cast<int*>(dst);
        if (threadIdx.x == 0 && blockIdx.y == 0) {
            if (to_stage) {
                di[0] = is[I_TIME];
                di[1] = is[I_NSTEP];
                dst[1] = sc[S_SR0];
                dst[2] = sc[S_QL2_0];
                dst[3] = sc[S_TIME];
                for (int k = 4; k < 16; k++) dst[k] = 0.0;
            } else {
                is[I_TIME] = di[0];
                is[I_NSTEP] = di[1];
                sc[S_SR0] = dst[1];
                sc[S_QL2_0] = dst[2];
                sc[S_TIME] = dst[3];
            }
        }
        return;
    }
    const int ids[6] = {P_U, P_V, P_P, P_T0 + b.cur, P_UP0 + b.cur, P_VP0 + b.cur};
    double* P = plane(b, d, ids[m]);
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    const int jend = min(d.n1, ((int)blockIdx.y + 1) * STATE_ROWS);
    for (int j = blockIdx.y * STATE_ROWS + (threadIdx.x >> 5); j < jend; j += nw) {
        double* row = P + (long long)j * d.ld;
        double* srow = dst + (long long)j * nc;
        if (to_stage) {
#pragma unroll 4
            for (int i = lane; i < nc; i += 32) srow[i] = row[i];
        } else {
#pragma unroll 4
            for (int i = lane; i < nc; i += 32) store_mirrored(row, 0, i, 0, d.W, d.periodic, srow[i]);
        }
    }
}

}  // namespace cfd
