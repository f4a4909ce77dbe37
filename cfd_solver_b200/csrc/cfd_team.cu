// cfd_team.cu -- whole time steps of a case inside one launch.
//
// The launch-per-phase step (cfd_api.cu) runs 28 to 74 kernels a step. A case of 65 x 65 to
// a few hundred points a side does not fill the chip in any of them: each launch costs its
// own start, its chain of dependent loads (tile, case, flags, data) and its drain, 5-7 us
// whatever the work. Here a team of CTAs owns one case and runs all phases of its steps,
// with a barrier between phases, and several steps per launch. The case's descriptor
// and its solver state sit in shared memory, every CTA forms the per-case sums itself (from
// the same partials in the same order), so all CTAs take the same decisions and no flag
// crosses CTAs; a case stops its sweeps and pressure iterations on its own, whatever the
// other cases of the batch need.
//
// A team is a thread-block cluster of up to 16 CTAs (hardware barrier, without a limit; any number of
// teams in waves), or, for one larger case, a share of a cooperative grid with a counter
// barrier whose polls are bounded. One CTA has 512 threads: four groups of 128 for the
// sweeps and the post-smoother, two groups of 256 for the cell kernels, the whole CTA for
// k_rhs's cells and the pre-smoothing regions. The arithmetic is cfd_step.cuh's, the partial
// sums and their order are those of the launch-per-phase kernels, so a case gives the same
// bits in either form.
//
// Memory order: a phase's plain stores are read by other CTAs only after the next barrier
// (release by every CTA, acquire by every CTA); no phase reads what another CTA writes in
// the same phase. Partial sums have four regions, and a region is not written again before every
// CTA has read it: 0 / 1 alternate between sweeps and between the halves of a pressure iteration
// (a barrier lies between a region's readers and its next writer), 2 is the continuity
// source's alone, 3 the correction's and the diagnostics'.
#include "cfd_bulk.cuh"
#include "cfd_common.cuh"
#include "cfd_reduce.cuh"
#include "cfd_step.cuh"
#include "cfd_sweep.cuh"
#include "cfd_team.cuh"

namespace cfd {

namespace {

constexpr int NT5 = TEAM_THREADS;
constexpr int TAIL_TILES = 1;  // levels of at most this many regions run in one CTA

// the case's solver state, one copy per CTA, the same in all of them
struct TeamState {
    int mnext, flip, mask, modd, mdone, status, pdone, pit, pstatus, itime, nstep;
    int mit[NFIELD];
    double mr0[NFIELD], mr[NFIELD], cw[2];
    double s2[2], g[2];  // constants of the Chebyshev recurrence (u-type, T systems)
    double alpha, omega, beta, rho, nb1, rl1, ql1, ql2, qmax, ql2_0, sr, sr0, dul1, dtl1, dtmax, dmax, time;
    double wall[7];      // the step's wall integrals (first CTA)
    unsigned long long work[4];
};

// Shared memory: the case, its state and reduction scratch; the four sweep groups'
// operators; a work area of the phase. The phases are functions of their own (not inlined):
// each has the registers to itself, and what they share lives here.
struct TeamSh {
    TeamArgs a;        // the launch's arguments: a reference to the kernel parameter would be read
                       // through global memory, a round trip at the start of every phase
    CaseDev c;
    TeamState ts;
    double red[16 * 32];
    double sred[(NT5 / SW_THREADS) * SW_WARPS * NFIELD];
    double* fb;        // plane 0 of the case; plane k at fb + k * c.ps
    unsigned* bar;     // grid form: the team's arrival counter
    unsigned target;   // its value after the next barrier
    int cid, rank, tail;
    int ops_tile[NT5 / SW_THREADS];  // tile whose operator each sweep group holds
};
constexpr int OPS_BYTES = 3 * TX * TYJ * 8 + 2 * TX * TYJ * 4;  // one sweep group's operator
constexpr int OPS_OFF = (sizeof(TeamSh) + 127) / 128 * 128;
constexpr int WORK_OFF = OPS_OFF + (NT5 / SW_THREADS) * OPS_BYTES;
constexpr int COARSE_WORDS = 12000;
constexpr int WORK_MIN = COARSE_WORDS * 4;
static_assert((2 * MPR_XP + 2 * MPR_RP) * 4 <= WORK_MIN && 4 * 2 * MG_GS_XP * 4 <= WORK_MIN, "work area");

extern __shared__ __align__(128) unsigned char team_dsm[];
__device__ __forceinline__ TeamSh& sh() { return *reinterpret_cast<TeamSh*>(team_dsm); }

struct Tiling {  // 32-column tiles of the unknown cells, `ty` rows each, row-major
    int ncx, n;
    __device__ __forceinline__ Tiling(int ihi, int n1, int ty) {
        ncx = ihi / TX + 1;
        n = ncx * ((n1 - 2 + ty - 1) / ty);
    }
    __device__ __forceinline__ int i0(int t) const { return (t % ncx) * TX; }
    __device__ __forceinline__ int j0(int t, int ty) const { return 1 + (t / ncx) * ty; }
};
__device__ __forceinline__ Tiling cell_tiles() { return Tiling(sh().c.ihi, sh().c.n1, TYJ); }

// partial rows of the case, in one of four regions
__device__ __forceinline__ double* part(int region) {
    return sh().a.b.partial + ((long long)region * sh().a.b.njtiles + sh().c.jt_begin) * PSTRIDE;
}

// all CTAs of the team have finished the phase, and its stores are visible to all of them;
// false when the counter barrier gave up
__device__ __noinline__ bool team_barrier() {
    if (sh().a.cluster) {
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        return true;
    }
    __syncthreads();
    bool got = true;
    if (threadIdx.x == 0) {
        unsigned* bar = sh().bar;
        const unsigned target = sh().target += sh().a.nr, limit = sh().a.polls;
        __threadfence();
        atomicAdd(bar, 1u);
        got = false;
        for (unsigned n = 0; n < limit && !got; n++) {
            unsigned v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
            got = (int)(v - target) >= 0;
        }
        __threadfence();
        if (!got) atomicExch(sh().a.b.error, 1);
    }
    return __syncthreads_and(got);
}
#define TEAM_SYNC()                       \
    do {                                  \
        if (!team_barrier()) return false; \
    } while (0)

template <bool MAX>
__device__ __forceinline__ double warp_tree(double x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double y = __shfl_down_sync(0xffffffffu, x, o);
        x = MAX ? fmax(x, y) : x + y;
    }
    return x;
}

// block_reduce_mixed() over a group of threads; result in its thread 0
template <int NV, unsigned MAXMASK, class Grp>
__device__ __forceinline__ void group_reduce(double (&v)[NV], double* smem, const Grp& g) {
    const int lane = g.tid & 31, warp = g.tid >> 5, nw = Grp::N >> 5;
#pragma unroll
    for (int k = 0; k < NV; k++) {
        const double x = ((MAXMASK >> k) & 1u) ? warp_tree<true>(v[k]) : warp_tree<false>(v[k]);
        if (lane == 0) smem[k * 32 + warp] = x;
    }
    g.sync();
    if (warp == 0) {
#pragma unroll
        for (int k = 0; k < NV; k++) {
            const bool mx = (MAXMASK >> k) & 1u;
            const double x = lane < nw ? smem[k * 32 + lane] : (mx ? -1.0e300 : 0.0);
            v[k] = mx ? warp_tree<true>(x) : warp_tree<false>(x);
        }
    }
    g.sync();
}

// The case's totals from its tiles' partial rows (row t at part + t * PSTRIDE), in thread 0: the
// sum k_fin and k_sweep_fin form with `nthr` threads. The threads above add nothing
// (adding their zeros changes no bit); up to 32 rows one warp holds every term, and the
// block's second stage would only add zeros to its sum.
template <int NV, unsigned MAXMASK>
__device__ __forceinline__ void team_total(const double* part, int count, int nthr, double (&v)[NV]) {
#pragma unroll
    for (int k = 0; k < NV; k++) v[k] = ((MAXMASK >> k) & 1u) ? -1.0e300 : 0.0;
    if (count <= 32) {
        if (threadIdx.x >= 32) return;
        if ((int)threadIdx.x < count) {
            const double* src = part + (long long)threadIdx.x * PSTRIDE;
#pragma unroll
            for (int k = 0; k < NV; k++) v[k] = ((MAXMASK >> k) & 1u) ? fmax(v[k], src[k]) : v[k] + src[k];
        }
#pragma unroll
        for (int k = 0; k < NV; k++)
            v[k] = ((MAXMASK >> k) & 1u) ? fmax(warp_tree<true>(v[k]), -1.0e300) : warp_tree<false>(v[k]);
        return;
    }
    if ((int)threadIdx.x < nthr)
        for (int t = threadIdx.x; t < count; t += nthr) {
            const double* src = part + (long long)t * PSTRIDE;
#pragma unroll
            for (int k = 0; k < NV; k++) {
                const double x = src[k];
                v[k] = ((MAXMASK >> k) & 1u) ? fmax(v[k], x) : v[k] + x;
            }
        }
    group_reduce<NV, MAXMASK>(v, sh().red, BlockGroup<NT5>());
}

// ---- contravariant velocities, convection, right-hand sides; iterates seeded (k_rhs)
template <bool MX>
__device__ __noinline__ void team_rhs(int cur) {
    const CaseDev& c = sh().c;
    const Tiling jt = cell_tiles();
    const int tid = threadIdx.x, ld = c.ld;
    const long long ps = c.ps;
    double* const fb = sh().fb;
    if (tid == 0) {
        TeamState& ts = sh().ts;
        ts.flip = MX ? 0 : ts.mnext;
        ts.mask = (1 << NFIELD) - 1;
        ts.modd = ts.mdone = 0;
    }
    __syncthreads();
    const RhsCase rc(c);
    const bool warm = c.warm_up != 0;
    const int nextm = sh().ts.flip;
    const double *U = fb + P_U * ps, *V = fb + P_V * ps, *T = fb + (P_T0 + cur) * ps, *P = fb + P_P * ps,
                 *UP = fb + (P_UP0 + cur) * ps, *VP = fb + (P_VP0 + cur) * ps;
    for (int t = sh().rank; t < jt.n; t += sh().a.nr) {
        const int i = jt.i0(t) + tid % TX, j = jt.j0(t, TYJ) + tid / TX;
        if (i < c.ilo || i > c.ihi || j > c.n1 - 2) continue;
        const int k = j * ld + i;
        const double up = UP[k], vp = VP[k];
        const RhsOut r = rhs_cell<Cross>(rc, i, j, U, V, T, P, UP, VP, k, ld, fb[P_XIX * ps + k], fb[P_XIY * ps + k],
                                         fb[P_ETX * ps + k], fb[P_ETY * ps + k], fb[P_ALPH * ps + k],
                                         fb[P_GAM * ps + k], fb + P_BETA * ps + k);
        const double seed[NFIELD] = {U[k], V[k], T[k], warm ? up : 0.0, warm ? vp : 0.0};
        fb[P_RU * ps + k] = r.qu;
        fb[P_RV * ps + k] = r.qv;
        fb[P_RT * ps + k] = r.qt;
        fb[P_RUP * ps + k] = r.qup;
        fb[P_RVP * ps + k] = r.qvp;
        rhs_seed<true>(fb, ps, nextm, cur, ld, c.W, c.periodic, c.profile == CAVITY, c.n0, c.n1, i, j, seed);
    }
}

template <int MODE>
struct TeamSweepTypes {
    using T = double;
};
template <>
struct TeamSweepTypes<SW_MX> {
    using T = float;
};

// One sweep of the team's case: every task is one tile and the fields of one part. A group
// of 128 threads reads its windows straight from global memory (they meet in L1), four
// rows and one column per thread as in cfd_sweep.cu. The operator of the group's last tile
// stays in shared memory: with at least as many groups as tasks it is built once per launch.
template <int MODE>
__device__ __noinline__ void team_sweep(int sweep, int nxt) {
    using ST = typename TeamSweepTypes<MODE>::T;
    const BatchDev& b = sh().a.b;
    const CaseDev& c = sh().c;
    const TeamState& ts = sh().ts;
    const Tiling jt = cell_tiles();
    const NamedGroup<SW_THREADS> g;
    const int lane = g.tid & 31, wrp = g.tid >> 5, mask = ts.mask;
    const int slots = (NT5 / SW_THREADS) * sh().a.nr;
    const int parts = min((int)NFIELD, max(1, slots / jt.n));
    double* OPS = reinterpret_cast<double*>(team_dsm + OPS_OFF + g.id * OPS_BYTES);
    float* RAP = reinterpret_cast<float*>(team_dsm + OPS_OFF + g.id * OPS_BYTES + 3 * TX * TYJ * 8);
    double* sred = sh().sred + g.id * SW_WARPS * NFIELD;
    double* prt = part(sweep & 1);
    const bool weighted = MODE == SW_MX ? true : sweep > 0;
    const bool has_prev = MODE == SW_MX ? sweep > 1 : (MODE == SW_F64 && sweep > 0);
    const int ld = c.ld, W = c.W, per = c.periodic, n1 = c.n1;
    double* const fb = sh().fb;
    float* const xb = b.f32 + c.xbase + H32;
    for (int task = g.id * sh().a.nr + sh().rank; task < jt.n * parts; task += slots) {
        const int t = task % jt.n, part_id = task / jt.n;
        int fm = 0;
        for (int f = part_id; f < NFIELD; f += parts) fm |= 1 << f;
        fm &= mask;
        if (fm == 0) continue;  // uniform over the group
        const int i0 = jt.i0(t), j0 = jt.j0(t, TYJ);
        const int i = i0 + lane, jw = j0 + wrp * SW_ROWS;
        const int ic = min(i, c.ihi);  // lanes past the last column read a safe one
        bool inq[SW_ROWS], nearw[SW_ROWS], drop_s[SW_ROWS], drop_n[SW_ROWS];
#pragma unroll
        for (int q = 0; q < SW_ROWS; q++) {
            const int j = jw + q;
            inq[q] = i >= c.ilo && i <= c.ihi && j <= n1 - 2;
            nearw[q] = j == 1 || j == n1 - 2 || (c.profile == CAVITY && (i == 1 || i == c.n0 - 2));
            drop_s[q] = c.profile == OGRID && j == 1;
            drop_n[q] = c.profile == OGRID && j == n1 - 2;
        }
        if (sh().ops_tile[g.id] != t) {  // uniform over the group
            const double kE = c.swk[0], kG = c.swk[1], kB = c.swk[2], rPr = c.rPr;
#pragma unroll
            for (int q = 0; q < SW_ROWS; q++) {
                const int o = (wrp * SW_ROWS + q) * TX + lane;
                const long long k = (long long)min(jw + q, n1 - 1) * ld + ic;
                const double E = kE * fb[P_ALPH * c.ps + k], B = kB * fb[P_BETA * c.ps + k], G = kG * fb[P_GAM * c.ps + k];
                const double D = (nearw[q] ? 2.0 : 2.5) * (E + G);
                OPS[o] = E;
                OPS[TX * TYJ + o] = G;
                OPS[2 * TX * TYJ + o] = B;
                RAP[o] = (float)__drcp_rn(1.0 + D);
                RAP[TX * TYJ + o] = (float)__drcp_rn(1.0 + D * rPr);
            }
        }
        const int mcol = mirror_col(i, W, per);
        const int sld = MODE == SW_MX ? c.xld : ld;  // pitch of the swept planes
        const int dld = MODE == SW_F64 ? ld : c.xld;
        for (int fr = fm; fr; fr &= fr - 1) {
            const int f = __ffs(fr) - 1;
            const bool isT = f == F_T;
            const ST* X;
            const ST* R;
            double* dst64 = nullptr;
            float* dst32 = nullptr;
            float* res32 = nullptr;
            if constexpr (MODE == SW_MX) {
                X = xb + (long long)(((sweep & 1) == 0 ? X_DA : X_DB) + f) * c.xps;
                R = xb + (long long)(X_R + f) * c.xps;
                dst32 = xb + (long long)(((sweep & 1) == 0 ? X_DB : X_DA) + f) * c.xps;
            } else {
                double* it = fb + sw_iter_plane(f, nxt) * c.ps;
                double* sc = fb + (P_BU + f) * c.ps;
                R = fb + (P_RU + f) * c.ps;
                if (MODE == SW_F64) {
                    const bool to_scratch = ((sweep & 1) == 0) != (((ts.flip >> f) & 1) != 0);
                    X = to_scratch ? it : sc;
                    dst64 = to_scratch ? sc : it;
                } else {
                    X = it;
                    dst32 = xb + (long long)(X_DB + f) * c.xps;
                    res32 = xb + (long long)(X_R + f) * c.xps;
                }
            }
            // the thread's window: rows jw - 2 .. jw + 5 (clamped: a row outside is read by no
            // cell's sum), columns i - 2 .. i + 2
            ST w[8][5], rhs[SW_ROWS], xm[SW_ROWS];
#pragma unroll
            for (int rr = 0; rr < 8; rr++) {
                const ST* row = X + (long long)min(max(jw + rr - 2, 0), n1 - 1) * sld + ic;
#pragma unroll
                for (int cl = 0; cl < 5; cl++) w[rr][cl] = row[cl - 2];
            }
#pragma unroll
            for (int q = 0; q < SW_ROWS; q++) {
                const long long jr = min(jw + q, n1 - 1);
                rhs[q] = R[jr * sld + ic];
                if (MODE == SW_F64) xm[q] = has_prev ? (ST)dst64[jr * dld + ic] : ST(0);
                else if (MODE == SW_MX) xm[q] = has_prev ? (ST)dst32[jr * dld + ic] : ST(0);
                else xm[q] = ST(0);
            }
            const ST gg = (ST)ts.g[isT];
            const ST wgt = weighted ? (ST)ts.cw[isT] : ST(1);
            const ST scale = isT ? (ST)c.rPr : ST(1);
            const bool tbug = isT && !c.fix_T_annw;
            const int rapoff = isT ? TX * TYJ : 0;
            double racc = 0.0;
#pragma unroll
            for (int q = 0; q < SW_ROWS; q++) {
                const int o = (wrp * SW_ROWS + q) * TX + lane;
                const ST E = (ST)OPS[o], G = (ST)OPS[TX * TYJ + o], B = (ST)OPS[2 * TX * TYJ + o];
                const auto x = [&](int dy, int dx) { return w[q + 2 + dy][2 + dx]; };
                const ST res = sw_residual<ST>(x, E, G, B, nearw[q], drop_s[q], drop_n[q], tbug, scale, rhs[q]);
                const ST rap = (ST)RAP[rapoff + o];
                const ST xk = w[q + 2][2];
                racc += inq[q] ? fabs((double)res) : 0.0;
                const long long kk = (long long)(jw + q) * dld;
                if (MODE == SW_MX0) {
                    const float d1 = (float)(gg * res * rap), rr = (float)res;
                    if (inq[q]) {
                        dst32[kk + i] = d1;
                        res32[kk + i] = rr;
                        if (mcol > -1000000) {
                            dst32[kk + mcol] = d1;
                            res32[kk + mcol] = rr;
                        }
                    }
                } else {
                    const ST xn = sw_next<ST>(xk, gg, res, rap, weighted, wgt, xm[q]);
                    if (inq[q]) {
                        if (MODE == SW_F64) {
                            dst64[kk + i] = (double)xn;
                            if (mcol > -1000000) dst64[kk + mcol] = (double)xn;
                        } else {
                            dst32[kk + i] = (float)xn;
                            if (mcol > -1000000) dst32[kk + mcol] = (float)xn;
                        }
                    }
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) racc += __shfl_down_sync(0xffffffffu, racc, o);
            if (lane == 0) sred[wrp * NFIELD + f] = racc;
        }
        g.sync();
        if (g.tid < NFIELD && ((fm >> g.tid) & 1)) {
            double x = 0.0;
#pragma unroll
            for (int w = 0; w < SW_WARPS; w++) x += sred[w * NFIELD + g.tid];
            prt[(long long)t * PSTRIDE + g.tid] = x;
            sh().ops_tile[g.id] = t;
        }
        g.sync();
    }
}

// After a sweep, in every CTA: the case's residuals, the stop rule and the next Chebyshev
// weights (k_sweep_fin), one lane per field
__device__ __noinline__ void team_mom_rule(int sweep) {
    TeamState& ts = sh().ts;
    const CaseDev& c = sh().c;
    double v[NFIELD];
    const int n = cell_tiles().n;
    team_total<NFIELD, 0u>(part(sweep & 1), n, sweep_sum_threads(n), v);
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x, mask = ts.mask, flip = ts.flip;
        double x = 0.0;
#pragma unroll
        for (int f = 0; f < NFIELD; f++) {
            const double vf = __shfl_sync(0xffffffffu, v[f], 0);
            if (lane == f) x = vf;
        }
        bool done = false, nan = false;
        if (lane < NFIELD && ((mask >> lane) & 1)) {
            const double mr0 = sweep == 0 ? ((x != 0.0) ? x : 1.0) : ts.mr0[lane];
            ts.mr0[lane] = mr0;
            ts.mr[lane] = x;
            ts.mit[lane] = sweep + 1;
            nan = !isfinite(x);
            done = (x / mr0 < c.tol_mom) || (x <= c.atol_mom) || nan;
        }
        if (lane >= 8 && lane < 10) ts.cw[lane - 8] = cheb_next(sweep, ts.cw[lane - 8], ts.s2[lane - 8]);
        const int dm = (int)__ballot_sync(0xffffffffu, done), nm = (int)__ballot_sync(0xffffffffu, nan);
        if (lane == 0) {
            if (sweep == 0) ts.mnext &= ~mask;
            if (nm) ts.status |= ST_NAN;
            // the result is in the scratch plane when the sweep's parity equals the solve's start
            // plane flag; the next step's start is predicted from this parity
            ts.mdone |= dm;
            ts.modd |= dm & ((sweep & 1) ? flip : ~flip);
            if ((sweep & 1) == 0) ts.mnext |= dm;
            ts.mask = mask & ~dm;
            const unsigned long long ncell = (unsigned long long)(c.ihi - c.ilo + 1) * (c.n1 - 2);
            const unsigned long long nf = (unsigned long long)__popc(mask) * ncell;
            ts.work[0] += nf;
            ts.work[1] += ncell;
            if (sweep == 0) ts.work[2] += nf;
            if (sweep == 1) ts.work[3] += nf;
        }
    }
    __syncthreads();
}

// precision form: x = x0 + d (k_mom_update)
__device__ __noinline__ void team_mom_update(int nxt) {
    const CaseDev& c = sh().c;
    const Tiling jt = cell_tiles();
    const int tid = threadIdx.x, modd = sh().ts.modd;
    for (int t = sh().rank; t < jt.n; t += sh().a.nr) {
        const int i = jt.i0(t) + tid % TX, j = jt.j0(t, TYJ) + tid / TX;
        if (i < c.ilo || i > c.ihi || j > c.n1 - 2) continue;
        const long long k = (long long)j * c.ld + i, kx = (long long)j * c.xld + i;
        double x[NFIELD];
        float d[NFIELD];
#pragma unroll
        for (int f = 0; f < NFIELD; f++) {
            x[f] = sh().fb[sw_iter_plane(f, nxt) * c.ps + k];
            d[f] = xplane(sh().a.b, c, (((modd >> f) & 1) ? X_DB : X_DA) + f)[kx];
        }
#pragma unroll
        for (int f = 0; f < NFIELD; f++)
            store_mirrored(sh().fb + sw_iter_plane(f, nxt) * c.ps, c.ld, i, j, c.W, c.periodic, x[f] + (double)d[f]);
    }
}

// ---- continuity source (k_face_q), with the far-field up / vp (k_upbc) formed where they are
// read and results left in a scratch plane copied home (k_mom_fix): neighbours read the
// plane the solve ended in, and only its owner writes a cell of the other
template <bool MX>
__device__ __noinline__ void team_face(int nxt) {
    const CaseDev& c = sh().c;
    const TeamState& ts = sh().ts;
    const Tiling jt = cell_tiles();
    const NamedGroup<256> g;
    const int ld = c.ld, n1 = c.n1;
    const long long ps = c.ps;
    const bool cav = c.profile == CAVITY;
    double* const fb = sh().fb;
    const FaceCase fc(c);
    // solves whose result is in the scratch plane: stopped there, or ran to the cap from there
    const int odd = MX ? 0 : ((ts.modd & ts.mdone) | (ts.flip & ~ts.mdone));
    double* UPi = fb + sw_iter_plane(F_UP, nxt) * ps;
    double* VPi = fb + sw_iter_plane(F_VP, nxt) * ps;
    const double* UP = ((odd >> F_UP) & 1) ? fb + P_BUP * ps : UPi;
    const double* VP = ((odd >> F_VP) & 1) ? fb + P_BVP * ps : VPi;
    const double *P = fb + P_P * ps, *X = fb + P_XIX * ps, *Y = fb + P_XIY * ps, *E = fb + P_ETX * ps,
                 *G = fb + P_ETY * ps, *VEC = fb + P_VEC * ps;
    const LevelDev& L0 = c.lev[0];
    float* B0 = mplane(sh().a.b, L0, M_B);
    for (int t = g.id * sh().a.nr + sh().rank; t < jt.n; t += 2 * sh().a.nr) {
        const int i = jt.i0(t) + g.tid % TX, j0 = jt.j0(t, TYJ) + g.tid / TX;
        double r[3] = {0.0, 0.0, 0.0};
#pragma unroll 1
        for (int h = 0; h < 2; h++) {
            const int j = j0 + h * TY;
            if (i < c.ilo || i > c.ihi || j > n1 - 2) continue;
            const int k = j * ld + i;
            const bool farrow = !cav && j == n1 - 2;
            double uN = UP[k + ld], vN = VP[k + ld];
            if (farrow) {
                const long long kf = k + ld;
                const double vnn = c.uinf * VEC[2LL * ld + i] + c.vinf * VEC[3LL * ld + i];
                const double uo = upbc_out(UP, kf, ld), vo = upbc_out(VP, kf, ld);
                const double ui = fb[P_U * ps + kf], vi = fb[P_V * ps + kf];
                uN = vnn >= 0 ? ui : uo;
                vN = vnn >= 0 ? vi : vo;
            }
            const double q = face_cell(fc, P, UP, VP, X, Y, E, G, k, ld, uN, vN);
            fb[P_Q * ps + k] = q;
            fb[P_KR * ps + k] = q;
            B0[(long long)j * L0.ld + i] = (float)q;
            r[0] += fabs(q);
            r[1] += q * q;
            r[2] = fmax(r[2], fabs(q));
            if (farrow) {
                store_mirrored(UPi, ld, i, n1 - 1, c.W, c.periodic, uN);
                store_mirrored(VPi, ld, i, n1 - 1, c.W, c.periodic, vN);
            }
            if (odd) {
                double x[NFIELD];
#pragma unroll
                for (int f = 0; f < NFIELD; f++) x[f] = fb[(P_BU + f) * ps + k];
#pragma unroll
                for (int f = 0; f < NFIELD; f++)
                    if ((odd >> f) & 1)
                        store_mirrored(fb + sw_iter_plane(f, nxt) * ps, ld, i, j, c.W, c.periodic, x[f]);
            }
        }
        group_reduce<3, 0x4u>(r, sh().red + g.id * 256, g);
        if (g.tid == 0)
            for (int q = 0; q < 3; q++) part(2)[(long long)t * PSTRIDE + q] = r[q];
    }
}

__device__ __noinline__ void team_face_total() {  // also the sip seam's start: its `mask` is 0
    TeamState& ts = sh().ts;
    double v[3];
    team_total<3, 0x4u>(part(2), cell_tiles().n, NT, v);
    if (threadIdx.x == 0) {
        ts.ql1 = v[0];
        ts.ql2 = sqrt(v[1]);
        if (ts.nstep == 0) ts.ql2_0 = ts.ql2;
        ts.qmax = v[2];
        ts.rho = v[1];
        ts.alpha = 1.0;
        ts.omega = 1.0;
        ts.beta = 0.0;
        ts.nb1 = ts.rl1 = v[0];
        ts.pit = 0;
        // a field still iterating when its loop ended stopped at the sweep cap
        ts.pstatus = ts.mask ? ST_MAXITER : 0;
        ts.pdone = (v[0] == 0.0 || !isfinite(v[0])) ? 1 : 0;
        if (!isfinite(v[0])) ts.status |= ST_NAN;
    }
    __syncthreads();
}

// first level whose pre-smoothing has few regions: from there one CTA runs the V-cycle
__device__ __forceinline__ int team_tail(const CaseDev& c) {
    int tail = 0;
    for (int l = 0; l + 1 < c.nlev; l++)
        if (Tiling(c.lev[l + 1].ihi, c.lev[l + 1].n1, TY).n > TAIL_TILES) tail = l + 1;
    return tail;
}

// ---- one V-cycle from M_B of level 0 into its result plane (form 2 of run_vcycle)
__device__ __noinline__ void team_prr(int l, int first, int stride) {
    const CaseDev& c = sh().c;
    float* xs = reinterpret_cast<float*>(team_dsm + WORK_OFF);
    const Tiling tl(c.lev[l + 1].ihi, c.lev[l + 1].n1, TY);
#pragma unroll 1
    for (int t = first; t < tl.n; t += stride)
        mg_prr_tile<true>(sh().a.b, c, l, tl.i0(t), tl.j0(t, TY), M_X, sh().a.nu_pre, xs, xs + 2 * MPR_XP, BlockGroup<NT5>());
}
__device__ __noinline__ void team_gs(int l, int first, int stride) {
    const CaseDev& c = sh().c;
    const NamedGroup<MG_GS_THREADS> g;
    float* xs = reinterpret_cast<float*>(team_dsm + WORK_OFF) + g.id * 2 * MG_GS_XP;
    const Tiling tl(c.lev[l].ihi, c.lev[l].n1, TYJ);
#pragma unroll 1
    for (int t = first; t < tl.n; t += stride) {
        mg_gs_tile(sh().a.b, c, l, tl.i0(t), tl.j0(t, TYJ), 2, M_X, M_R, sh().a.nu_post, xs, g);
        g.sync();  // the group's x tile is read out before the next tile overwrites it
    }
}
__device__ __noinline__ void team_coarse() {
    const CaseDev& c = sh().c;
    mg_coarse_solve<2>(sh().a.b, c, c.lev[c.nlev - 1], sh().a.coarse_sweeps, reinterpret_cast<float*>(team_dsm + WORK_OFF),
                    COARSE_WORDS, BlockGroup<NT5>());
}
__device__ __noinline__ bool team_vcycle() {
    constexpr int G = NT5 / MG_GS_THREADS;
    const int nlev = sh().c.nlev, tail = sh().tail, rank = sh().rank, gid = threadIdx.x / MG_GS_THREADS;
    for (int l = 0; l < tail; l++) {
        team_prr(l, rank, sh().a.nr);
        TEAM_SYNC();
    }
    if (rank == 0) {
        for (int l = tail; l + 1 < nlev; l++) {
            team_prr(l, 0, 1);
            __syncthreads();
        }
        team_coarse();
        __syncthreads();
        for (int l = nlev - 2; l >= tail; l--) {
            team_gs(l, gid, G);
            __syncthreads();
        }
    }
    TEAM_SYNC();
    for (int l = tail - 1; l >= 0; l--) {
        team_gs(l, gid * sh().a.nr + rank, G * sh().a.nr);
        TEAM_SYNC();
    }
    return true;
}

// ---- BiCGStab on the case; p_hat and s_hat are read where the V-cycle left them
// y = A x of the V-cycle's result: mode 0 v = A p_hat and (r_hat, v); mode 1 t = A s_hat,
// (t, s), (t, t) (k_spmv)
__device__ __noinline__ void team_spmv(int mode) {
    const CaseDev& c = sh().c;
    const Tiling jt = cell_tiles();
    const NamedGroup<256> g;
    const LevelDev& L0 = c.lev[0];
    const int ld = c.ld, l0 = L0.ld;
    double* const fb = sh().fb;
    const float* X = mplane(sh().a.b, L0, mg_result_plane(sh().a.b, c, 0));
    const double* DOT = fb + (mode == 0 ? P_Q : P_KS) * c.ps;
    double* Y = fb + (mode == 0 ? P_KV : P_KT) * c.ps;
    for (int t = g.id * sh().a.nr + sh().rank; t < jt.n; t += 2 * sh().a.nr) {
        const int i = jt.i0(t) + g.tid % TX, j0 = jt.j0(t, TYJ) + g.tid / TX;
        double r[2] = {0.0, 0.0}, y[2], dv[2];
        bool in[2];
        long long k[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int j = j0 + h * TY;
            in[h] = i >= c.ilo && i <= c.ihi && j <= c.n1 - 2;
            const int jj = in[h] ? j : 1, ii = in[h] ? i : c.ilo;
            k[h] = (long long)jj * ld + ii;
            const long long q = (long long)jj * l0 + ii;
            y[h] = spmv_cell([&](int m) { return fb[(P_AP + m) * c.ps + k[h]]; }, X, q, l0, (double)X[q]);
            dv[h] = DOT[k[h]];
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            if (!in[h]) continue;
            Y[k[h]] = y[h];
            if (mode == 0) {
                r[0] += dv[h] * y[h];
            } else {
                r[0] += y[h] * dv[h];
                r[1] += y[h] * y[h];
            }
        }
        group_reduce<2, 0u>(r, sh().red + g.id * 256, g);
        if (g.tid == 0) {
            part(0)[(long long)t * PSTRIDE] = r[0];
            part(0)[(long long)t * PSTRIDE + 1] = r[1];
        }
    }
}
__device__ __noinline__ void team_spmv_total(int mode) {
    TeamState& ts = sh().ts;
    double v[2];
    team_total<2, 0u>(part(0), cell_tiles().n, NT, v);
    if (threadIdx.x == 0) {
        if (mode == 1) {
            ts.omega = v[1] > 0.0 ? v[0] / v[1] : 0.0;
        } else if (v[0] == 0.0 || !isfinite(v[0])) {
            ts.pstatus |= ST_BREAKDOWN;
            ts.pdone = 1;
        } else {
            ts.alpha = ts.rho / v[0];
        }
    }
    __syncthreads();
}

// s = r - alpha v and the half step x += alpha p_hat (k_bicg_s)
__device__ __noinline__ void team_bicg_s() {
    const CaseDev& c = sh().c;
    const Tiling jt = cell_tiles();
    const NamedGroup<256> g;
    const LevelDev& L0 = c.lev[0];
    double* const fb = sh().fb;
    const long long ps = c.ps;
    const double alpha = sh().ts.alpha;
    const bool first = sh().ts.pit == 0;
    double* X = fb + P_PCOR * ps;
    const double *R = fb + P_KR * ps, *Vv = fb + P_KV * ps;
    const float* PH = mplane(sh().a.b, L0, mg_result_plane(sh().a.b, c, 0));
    float* B0 = mplane(sh().a.b, L0, M_B);
    for (int t = g.id * sh().a.nr + sh().rank; t < jt.n; t += 2 * sh().a.nr) {
        const int i = jt.i0(t) + g.tid % TX, j0 = jt.j0(t, TYJ) + g.tid / TX;
        double r[1] = {0.0}, x0[2], rr[2], vv[2], ph[2];
        bool in[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int j = j0 + h * TY;
            in[h] = i >= c.ilo && i <= c.ihi && j <= c.n1 - 2;
            const int jj = in[h] ? j : 1, ii = in[h] ? i : c.ilo;
            const long long k = (long long)jj * c.ld + ii;
            x0[h] = first ? 0.0 : X[k];
            rr[h] = R[k];
            vv[h] = Vv[k];
            ph[h] = (double)PH[(long long)jj * L0.ld + ii];
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            if (!in[h]) continue;
            const int j = j0 + h * TY;
            const double s = rr[h] - alpha * vv[h];
            const double x = x0[h] + alpha * ph[h];
            fb[P_KS * ps + (long long)j * c.ld + i] = s;
            store_mirrored(X, c.ld, i, j, c.W, c.periodic, x);
            B0[(long long)j * L0.ld + i] = (float)s;
            r[0] += fabs(s);
        }
        group_reduce<1, 0u>(r, sh().red + g.id * 256, g);
        if (g.tid == 0) part(1)[(long long)t * PSTRIDE] = r[0];
    }
}

// x += omega s_hat, r = s - omega t (k_bicg_x)
__device__ __noinline__ void team_bicg_x() {
    const CaseDev& c = sh().c;
    const Tiling jt = cell_tiles();
    const NamedGroup<256> g;
    const LevelDev& L0 = c.lev[0];
    double* const fb = sh().fb;
    const long long ps = c.ps;
    const double omega = sh().ts.omega;
    double* X = fb + P_PCOR * ps;
    const double *S = fb + P_KS * ps, *T = fb + P_KT * ps, *Q = fb + P_Q * ps;
    const float* SH = mplane(sh().a.b, L0, mg_result_plane(sh().a.b, c, 0));
    for (int t = g.id * sh().a.nr + sh().rank; t < jt.n; t += 2 * sh().a.nr) {
        const int i = jt.i0(t) + g.tid % TX, j0 = jt.j0(t, TYJ) + g.tid / TX;
        double r[2] = {0.0, 0.0}, x0[2], s[2], tt[2], q[2], hh[2];
        bool in[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int j = j0 + h * TY;
            in[h] = i >= c.ilo && i <= c.ihi && j <= c.n1 - 2;
            const int jj = in[h] ? j : 1, ii = in[h] ? i : c.ilo;
            const long long k = (long long)jj * c.ld + ii;
            x0[h] = X[k];
            s[h] = S[k];
            tt[h] = T[k];
            q[h] = Q[k];
            hh[h] = (double)SH[(long long)jj * L0.ld + ii];
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            if (!in[h]) continue;
            const int j = j0 + h * TY;
            store_mirrored(X, c.ld, i, j, c.W, c.periodic, x0[h] + omega * hh[h]);
            const double rn = s[h] - omega * tt[h];
            fb[P_KR * ps + (long long)j * c.ld + i] = rn;
            r[0] += q[h] * rn;
            r[1] += fabs(rn);
        }
        group_reduce<2, 0u>(r, sh().red + g.id * 256, g);
        if (g.tid == 0) {
            part(1)[(long long)t * PSTRIDE] = r[0];
            part(1)[(long long)t * PSTRIDE + 1] = r[1];
        }
    }
}

// the next direction (k_bicg_p)
__device__ __noinline__ void team_bicg_p() {
    const CaseDev& c = sh().c;
    const Tiling jt = cell_tiles();
    const LevelDev& L0 = c.lev[0];
    double* const fb = sh().fb;
    const long long ps = c.ps;
    const double beta = sh().ts.beta, omega = sh().ts.omega;
    double* Pv = fb + P_KP * ps;
    const double* Pold = sh().ts.pit == 1 ? fb + P_Q * ps : Pv;
    const double *R = fb + P_KR * ps, *Vv = fb + P_KV * ps;
    float* B0 = mplane(sh().a.b, L0, M_B);
    for (int t = sh().rank; t < jt.n; t += sh().a.nr) {
        const int i = jt.i0(t) + (int)threadIdx.x % TX, j = jt.j0(t, TYJ) + (int)threadIdx.x / TX;
        if (i < c.ilo || i > c.ihi || j > c.n1 - 2) continue;
        const long long k = (long long)j * c.ld + i;
        const double p = R[k] + beta * (Pold[k] - omega * Vv[k]);
        Pv[k] = p;
        B0[(long long)j * L0.ld + i] = (float)p;
    }
}

// the solve: up to maxit_p iterations of two V-cycles, the half-step exit after the first
__device__ __noinline__ bool team_pressure() {
    TeamState& ts = sh().ts;
    const CaseDev& c = sh().c;
    for (int it = 0; it < sh().a.p_iters && !ts.pdone; it++) {
        if (!team_vcycle()) return false;
        team_spmv(0);
        TEAM_SYNC();
        team_spmv_total(0);
        if (ts.pdone) break;
        team_bicg_s();
        TEAM_SYNC();
        {
            double v[1];
            team_total<1, 0u>(part(1), cell_tiles().n, NT, v);
            if (threadIdx.x == 0) {
                const bool conv = v[0] <= c.tol_p * ts.nb1 || v[0] <= c.atol_p;
                if (conv || !isfinite(v[0])) {
                    ts.pit += 1;
                    ts.rl1 = v[0];
                    if (!isfinite(v[0])) ts.status |= ST_NAN;
                    ts.pdone = 1;
                }
            }
            __syncthreads();
        }
        if (ts.pdone) break;
        if (!team_vcycle()) return false;
        team_spmv(1);
        TEAM_SYNC();
        team_spmv_total(1);
        team_bicg_x();
        TEAM_SYNC();
        {
            double v[2];
            team_total<2, 0u>(part(1), cell_tiles().n, NT, v);
            if (threadIdx.x == 0) {
                const int itn = ++ts.pit;
                ts.rl1 = v[1];
                const bool conv = v[1] <= c.tol_p * ts.nb1 || v[1] <= c.atol_p;
                bool stop = conv;
                if (!isfinite(v[1])) { ts.status |= ST_NAN; stop = true; }
                else if (!conv && (ts.omega == 0.0 || v[0] == 0.0)) { ts.pstatus |= ST_BREAKDOWN; stop = true; }
                else if (!conv && itn >= sh().a.maxit_p) { ts.pstatus |= ST_MAXITER; stop = true; }
                if (!stop) {
                    ts.beta = (v[0] / ts.rho) * (ts.alpha / ts.omega);
                    ts.rho = v[0];
                } else {
                    ts.pdone = 1;
                }
            }
            __syncthreads();
        }
        if (ts.pdone) break;
        team_bicg_p();
        TEAM_SYNC();
    }
    return true;
}

// ---- velocity / pressure correction (k_correct)
__device__ __noinline__ void team_correct() {
    const CaseDev& c = sh().c;
    const Tiling jt = cell_tiles();
    const NamedGroup<256> g;
    const int ld = c.ld, W = c.W, per = c.periodic, n0 = c.n0, n1 = c.n1;
    const long long ps = c.ps;
    const bool cav = c.profile == CAVITY;
    double* const fb = sh().fb;
    const bool none = sh().ts.pit == 0;  // no pressure iteration ran: pcor = 0
    double *PC = fb + P_PCOR * ps, *U = fb + P_U * ps, *V = fb + P_V * ps, *P = fb + P_P * ps;
    const double* VEC = fb + P_VEC * ps;
    const double h0 = c.hd0, h1 = c.hd1, dt = c.dt;
    for (int t = g.id * sh().a.nr + sh().rank; t < jt.n; t += 2 * sh().a.nr) {
        const int i = jt.i0(t) + g.tid % TX, j0 = jt.j0(t, TYJ) + g.tid / TX;
        double r[1] = {0.0};
        bool in[2];
        double pc0[2], pn0[2], ps0[2], pe0[2], pw0[2], us[2], vs[2], m[2][4], u0[2], v0[2], p0[2];
        const int ic = min(i, c.ihi);
        const double vnn = c.uinf * VEC[2LL * ld + ic] + c.vinf * VEC[3LL * ld + ic];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int j = j0 + h * TY;
            in[h] = i >= c.ilo && i <= c.ihi && j <= n1 - 2;
            const long long k = in[h] ? (long long)j * ld + i : (long long)ld + c.ilo;  // a safe cell when out
            pc0[h] = PC[k]; pn0[h] = PC[k + ld]; ps0[h] = PC[k - ld]; pe0[h] = PC[k + 1]; pw0[h] = PC[k - 1];
            us[h] = fb[P_US * ps + k]; vs[h] = fb[P_VS * ps + k];
            m[h][0] = fb[P_XIX * ps + k]; m[h][1] = fb[P_XIY * ps + k];
            m[h][2] = fb[P_ETX * ps + k]; m[h][3] = fb[P_ETY * ps + k];
            u0[h] = U[k]; v0[h] = V[k]; p0[h] = P[k];
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            if (!in[h]) continue;
            const int j = j0 + h * TY;
            const double pc = none ? 0.0 : pc0[h];
            // pcor on the boundary after its conditions: wall copy, far field 0 / copy at inflow
            const double far = (!cav && vnn >= 0) ? pc : 0.0;
            const double pN = none ? 0.0 : (j == n1 - 2) ? (cav ? pc : far) : pn0[h];
            const double pS = none ? 0.0 : (j == 1) ? pc : ps0[h];
            const double pE = none ? 0.0 : (cav && i == n0 - 2) ? pc : pe0[h];
            const double pW = none ? 0.0 : (cav && i == 1) ? pc : pw0[h];
            const CorrOut o = correct_cell(pc, pN, pS, pE, pW, us[h], vs[h], m[h][0], m[h][1], m[h][2], m[h][3], p0[h],
                                           h0, h1, dt, c.omega_p);
            r[0] += fabs(o.un - u0[h]) + fabs(o.vn - v0[h]);
            store_mirrored(U, ld, i, j, W, per, o.un);
            store_mirrored(V, ld, i, j, W, per, o.vn);
            store_mirrored(P, ld, i, j, W, per, o.pn);
            if (none) store_mirrored(PC, ld, i, j, W, per, 0.0);
            correct_bnd(PC, ld, W, per, cav, n0, n1, i, j, pc, far);
        }
        group_reduce<1, 0u>(r, sh().red + g.id * 256, g);
        // column 3 of the step's region (team_diag has 0 .. 2): a solve with nothing to do passes no
        // barrier between team_face_total's reads of part(2) and this store
        if (g.tid == 0) part(3)[(long long)t * PSTRIDE + 3] = r[0];
    }
}

// ---- boundaries (k_bc). The O-grid's wall and far field share no value, so two CTAs do them
// side by side.
// The far field: circulation, u, v, T, then p and vorticity from the new row (held in shared
// memory, where neighbouring columns meet)
__device__ __noinline__ void team_bc_far(int cur) {
    const CaseDev& c = sh().c;
    const BcCase bc(sh().a.b, c, cur);
    const int tid = threadIdx.x, W = c.W;
    double* s_old = reinterpret_cast<double*>(team_dsm + WORK_OFF);
    double* un = s_old + 2 * (W + 1);
    double* vn = un + W + 1;
    double* red = sh().red;
    double acc[1] = {0.0};
    if (tid < BC_THREADS)
        for (int i = tid; i < W; i += BC_THREADS) acc[0] += bc_circ(bc, i, s_old);
    block_sum<1>(acc, red);
    if (tid == 0) {
        sh().a.b.scal[(long long)sh().cid * NSCAL + S_CIRC] = acc[0];
        red[0] = acc[0];
    }
    __syncthreads();
    const double circ = red[0];
    for (int i = tid; i < W; i += NT5) {
        const FarOut o = bc_far(bc, i, circ, s_old);
        un[i] = o.u;
        vn[i] = o.v;
    }
    __syncthreads();
    for (int i = tid; i < W; i += NT5) {
        const int e = i + 1 == W ? 0 : i + 1, w = i == 0 ? W - 1 : i - 1;
        const Edge g{un[i], un[e], un[w], vn[i], vn[e], vn[w]};
        bc_far_p(bc, i, g, bc.Tn[(long long)bc.jf * bc.ld + i], s_old);
        bc_vort(bc, i, bc.jf, g);
    }
    __syncthreads();
}

// The wall: velocity (from the coordinates, so a neighbour's needs no exchange), pressure and
// vorticity of each column; then the integrals along it. The cavity's static walls likewise.
__device__ __noinline__ void team_bc_wall(int cur, double t_new) {
    const CaseDev& c = sh().c;
    const BcCase bc(sh().a.b, c, cur);
    const int tid = threadIdx.x, W = c.W, n0 = c.n0, n1 = c.n1;
    double acc[7] = {0, 0, 0, 0, 0, 0, 0};
    if (c.profile != CAVITY) {
        double* pw = reinterpret_cast<double*>(team_dsm + WORK_OFF);
        double* vw = pw + W + 1;
        double cwall, swall;
        bc_phase(c, t_new, cwall, swall);
        for (int i = tid; i < W; i += NT5) {
            const Edge g{bc_wall_u(bc, i, cwall), bc_wall_u(bc, i + 1, cwall), bc_wall_u(bc, i - 1, cwall),
                         bc_wall_v(bc, i, cwall), bc_wall_v(bc, i + 1, cwall), bc_wall_v(bc, i - 1, cwall)};
            const double p = bc_wall_p(bc, i, g, swall), w = bc_vort(bc, i, 0, g);
            bc_wall(bc, i, g.u, g.v);
            pw[i] = p;
            vw[i] = w;
            if (i == 0) {
                pw[W] = p;
                vw[W] = w;
            }
        }
        __syncthreads();
        if (tid < BC_THREADS)
            for (int i = tid; i <= n0 - 2; i += BC_THREADS) bc_integral(bc, i, pw, vw, acc);
    } else {
        for (int j = 1 + tid; j <= n1 - 2; j += NT5) bc_cav_row(bc, j);
        for (int i = 1 + tid; i <= n0 - 2; i += NT5) {
            bc_cav_col(bc, i);
            bc_vort(bc, i, 0, edge_at(bc, i));
            bc_vort(bc, i, n1 - 1, edge_at(bc, (long long)(n1 - 1) * bc.ld + i));
        }
        __syncthreads();
        if (tid == 0) bc_cav_corners(bc);
        __syncthreads();
        if (tid < BC_THREADS)
            for (int i = tid; i <= n0 - 2; i += BC_THREADS) bc_integral(bc, i, bc.P, bc.VORT, acc);
    }
    block_sum<7>(acc, sh().red);
    if (tid == 0)
        for (int k = 0; k < 7; k++) sh().ts.wall[k] = acc[k];
}

// vorticity, dilatation and the energy residual (k_diag) of the tiles in tile rows [r0, r1) and
// [r2, r3), spread over `nw` CTAs of which this is the wrank-th
__device__ __noinline__ void team_diag(int cur, int r0, int r1, int r2, int r3, int wrank, int nw) {
    const CaseDev& c = sh().c;
    const Tiling jt = cell_tiles();
    const NamedGroup<256> g;
    const int ld = c.ld;
    const long long ps = c.ps;
    double* const fb = sh().fb;
    const double *U = fb + P_U * ps, *V = fb + P_V * ps, *TN = fb + (P_T0 + (cur ^ 1)) * ps, *TO = fb + (P_T0 + cur) * ps;
    const double h0 = c.hd0, h1 = c.hd1;
    const int na = (r1 - r0) * jt.ncx, nb = (r3 - r2) * jt.ncx;
    for (int e = g.id * nw + wrank; e < na + nb; e += 2 * nw) {
        const int t = e < na ? r0 * jt.ncx + e : r2 * jt.ncx + e - na;
        const int i = jt.i0(t) + g.tid % TX, j0 = jt.j0(t, TYJ) + g.tid / TX;
        double r[3] = {-1.0e300, 0.0, 0.0};
        bool in[2];
        double ue[2], uw[2], un[2], us[2], ve[2], vw[2], vn[2], vs[2], m[2][4], tn[2], to[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int j = j0 + h * TY;
            in[h] = i >= c.ilo && i <= c.ihi && j <= c.n1 - 2;
            const long long k = in[h] ? (long long)j * ld + i : (long long)ld + c.ilo;  // a safe cell when out
            ue[h] = U[k + 1]; uw[h] = U[k - 1]; un[h] = U[k + ld]; us[h] = U[k - ld];
            ve[h] = V[k + 1]; vw[h] = V[k - 1]; vn[h] = V[k + ld]; vs[h] = V[k - ld];
            m[h][0] = fb[P_XIX * ps + k]; m[h][1] = fb[P_XIY * ps + k];
            m[h][2] = fb[P_ETX * ps + k]; m[h][3] = fb[P_ETY * ps + k];
            tn[h] = TN[k]; to[h] = TO[k];
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            if (!in[h]) continue;
            const int j = j0 + h * TY;
            const DiagOut d = diag_cell(ue[h], uw[h], un[h], us[h], ve[h], vw[h], vn[h], vs[h], m[h][0], m[h][1],
                                        m[h][2], m[h][3], h0, h1);
            store_mirrored(fb + P_VORT * ps, ld, i, j, c.W, c.periodic, d.vort);
            store_mirrored(fb + P_DIL * ps, ld, i, j, c.W, c.periodic, d.dil);
            const double dT = fabs(tn[h] - to[h]);
            r[0] = fmax(r[0], d.dil);
            r[1] += dT;
            r[2] = fmax(r[2], dT);
        }
        group_reduce<3, 0x5u>(r, sh().red + g.id * 256, g);
        if (g.tid == 0)
            for (int q = 0; q < 3; q++) part(3)[(long long)t * PSTRIDE + q] = r[q];
    }
}

// the step's residual sums (only one CTA's copy is reported)
__device__ __noinline__ void team_step_total() {
    TeamState& ts = sh().ts;
    const CaseDev& c = sh().c;
    double v[4];
    team_total<4, 0x5u>(part(3), cell_tiles().n, NT, v);
    if (threadIdx.x == 0) {
        ts.dmax = fmax(v[0], 0.0);
        ts.dtl1 = v[1];
        ts.dtmax = v[2];
        ts.dul1 = v[3];
        // steady residual: mean (|du| + |dv| + |dT|) / dt over the unknown cells
        const double ncell = (double)(c.ihi - c.ilo + 1) * (c.n1 - 2);
        ts.sr = (v[3] + v[1]) / (c.dt * ncell);
        if (ts.nstep == 0) ts.sr0 = ts.sr;
    }
}

// one time step; false when a barrier gave up
template <bool MX>
__device__ __forceinline__ bool team_step(int cur) {
    const TeamState& ts = sh().ts;
    const int nxt = cur ^ 1, rank = sh().rank, nr = sh().a.nr, last = nr - 1;
    team_rhs<MX>(cur);
    TEAM_SYNC();
    for (int sweep = 0;; sweep++) {
        if (!MX) team_sweep<SW_F64>(sweep, nxt);
        else if (sweep == 0) team_sweep<SW_MX0>(sweep, nxt);
        else team_sweep<SW_MX>(sweep, nxt);
        TEAM_SYNC();
        team_mom_rule(sweep);
        if (ts.mask == 0 || sweep + 1 >= sh().a.sweep_cap) break;
    }
    if (MX) {
        team_mom_update(nxt);
        TEAM_SYNC();
    }
    team_face<MX>(nxt);
    TEAM_SYNC();
    team_face_total();
    if (!team_pressure()) return false;
    team_correct();
    TEAM_SYNC();
    // the first CTA has the wall, the last the far field; the others meanwhile do the
    // diagnostics of the tiles that read no boundary row (every tile in the cavity, whose walls
    // do not move)
    const CaseDev& c = sh().c;
    const bool cav = c.profile == CAVITY;
    const int time_new = (int)((double)ts.itime + c.dt);
    // the time the wall motion sees: the reference's int (PSolver.cpp:186), or t = n dt
    const double t_new = c.time_accurate ? ts.time + c.dt : (double)time_new;
    if (!cav && rank == last) team_bc_far(cur);
    if (rank == 0) {
        team_bc_wall(cur, t_new);
        __syncthreads();
    }
    const Tiling jt = cell_tiles();
    const int ncy = jt.n / jt.ncx;
    const bool spare = nr > 2;  // CTAs without a boundary
    if (!spare || (rank != 0 && rank != last))
        team_diag(cur, cav ? 0 : 1, cav ? ncy : max(ncy - 1, 1), 0, 0, spare ? rank - 1 : rank, spare ? nr - 2 : nr);
    if (!cav) {
        TEAM_SYNC();
        team_diag(cur, 0, 1, max(ncy - 1, 1), ncy, rank, nr);
    }
    TEAM_SYNC();
    if (rank == last) team_step_total();
    __syncthreads();
    if (threadIdx.x == 0) {
        sh().ts.nstep += 1;
        sh().ts.itime = time_new;
        sh().ts.time = t_new;
    }
    __syncthreads();
    return true;
}

template <bool MX>
__device__ __forceinline__ void team_run(const TeamArgs& a) {
    const BatchDev& b = a.b;
    const int tid = threadIdx.x, nr = a.nr;
    const int team = blockIdx.x / nr, rank = blockIdx.x - team * nr;
    const int cid = a.ids[team];
    int* is = b.iscal + (long long)cid * NISCAL;
    double* sc = b.scal + (long long)cid * NSCAL;
    // a launch queued behind one whose barrier gave up leaves the batch as it is
    if (!a.cluster && *b.error) return;
    if (!is[I_ACTIVE]) {  // an empty slot takes no part in the step (uniform over the team)
        if (rank == 0 && tid == 0) {
            int word = 0;
            for (int f = 0; f < NFIELD; f++) {
                is[I_MDONE0 + f] = 1;
                is[I_MIT0 + f] = 0;
                is[I_MODD0 + f] = 0;
                is[I_MFLIP0 + f] = MX ? 0 : is[I_MNEXT0 + f];
                word |= (is[I_MFLIP0 + f] != 0) << (NFIELD + f);
            }
            is[I_MWORD] = word;
            is[I_PDONE] = 1;
        }
        return;
    }
    TeamSh& s = sh();
    TeamState& ts = s.ts;
    for (int k = tid; k < (int)(sizeof(TeamArgs) / 4); k += NT5)
        reinterpret_cast<int*>(&s.a)[k] = reinterpret_cast<const int*>(&a)[k];
    for (int k = tid; k < (int)(sizeof(CaseDev) / 4); k += NT5)
        reinterpret_cast<int*>(&s.c)[k] = reinterpret_cast<const int*>(b.cases + cid)[k];
    if (tid == 0) {
        ts.mnext = 0;
        for (int f = 0; f < NFIELD; f++) ts.mnext |= (is[I_MNEXT0 + f] != 0) << f;
        ts.status = is[I_STATUS];
        ts.itime = is[I_TIME];
        ts.nstep = is[I_NSTEP];
        ts.ql2_0 = sc[S_QL2_0];
        ts.sr0 = sc[S_SR0];
        ts.time = sc[S_TIME];
        ts.cw[0] = sc[S_CW0];
        ts.cw[1] = sc[S_CW1];
        for (int k = 0; k < 4; k++) ts.work[k] = 0;
        for (int k = 0; k < NT5 / SW_THREADS; k++) s.ops_tile[k] = -1;
        s.cid = cid;
        s.rank = rank;
        s.bar = a.bar + team;
        s.target = 0;
    }
    __syncthreads();
    const CaseDev& c = s.c;
    if (tid < 2) {
        ts.s2[tid] = cheb_s2(c.cheb_a[tid], c.cheb_b[tid]);
        ts.g[tid] = 2.0 / (c.cheb_a[tid] + c.cheb_b[tid]);
    }
    if (tid == 0) {
        s.fb = b.f64 + c.base + H;
        s.tail = team_tail(c);
    }
    __syncthreads();
    int cur = b.cur;
    for (int step = 0; step < a.nsteps; step++, cur ^= 1)
        if (!team_step<MX>(cur)) return;
    // the state the host reads and the next launch starts from
    if (rank == nr - 1 && tid == 0) {
        sc[S_DUL1] = ts.dul1; sc[S_DMAX] = ts.dmax; sc[S_DTL1] = ts.dtl1; sc[S_DTMAX] = ts.dtmax;
        sc[S_SR] = ts.sr; sc[S_SR0] = ts.sr0;
    }
    if (rank == 0 && tid == 0) {
        int word = ts.mask;
        for (int f = 0; f < NFIELD; f++) {
            is[I_MDONE0 + f] = (ts.mdone >> f) & 1;
            is[I_MIT0 + f] = ts.mit[f];
            is[I_MODD0 + f] = (ts.modd >> f) & 1;
            is[I_MFLIP0 + f] = (ts.flip >> f) & 1;
            is[I_MNEXT0 + f] = (ts.mnext >> f) & 1;
            word |= ((ts.flip >> f) & 1) << (NFIELD + f);
            sc[S_MR0 + f] = ts.mr0[f];
            sc[S_MR + f] = ts.mr[f];
        }
        is[I_MWORD] = word;
        is[I_PDONE] = 1;
        is[I_PIT] = ts.pit;
        is[I_PSTATUS] = ts.pstatus;
        is[I_STATUS] = ts.status;
        is[I_TIME] = ts.itime;
        is[I_NSTEP] = ts.nstep;
        sc[S_TIME] = ts.time;
        sc[S_CW0] = ts.cw[0];
        sc[S_CW1] = ts.cw[1];
        sc[S_RHO] = ts.rho; sc[S_ALPHA] = ts.alpha; sc[S_OMEGA] = ts.omega; sc[S_BETA] = ts.beta;
        sc[S_NB1] = ts.nb1; sc[S_RL1] = ts.rl1;
        sc[S_QL1] = ts.ql1; sc[S_QL2] = ts.ql2; sc[S_QMAX] = ts.qmax; sc[S_QL2_0] = ts.ql2_0;
        bc_scalars(c, ts.wall, sc);
        if (c.profile == CAVITY) sc[S_CIRC] = 0.0;
        for (int k = 0; k < 4; k++) atomicAdd(&b.work[k], ts.work[k]);
    }
}

// ---- the sip9p() seam (cfd_sip_solve, PSolver.cpp:2067-2278): the step's pressure solve on the
// caller's stencil, for the correction e of A (phi0 + e) = q with e = 0 on the boundary rows
// (and, without periodic xi, the boundary columns), as sip9p holds them.
//
// One pass over the unknown cells: the caller's stencil into the case's planes and multigrid
// level 0, r0 = q - A phi0 (phi0's boundary values enter through the stencil) as right-hand
// side, shadow residual and first preconditioner input, and its sums; the V-cycle's x planes
// start from zero
__device__ __noinline__ void sip_start(const SipArgs& p) {
    const CaseDev& c = sh().c;
    const Tiling jt = cell_tiles();
    const NamedGroup<256> g;
    const LevelDev& L0 = c.lev[0];
    double* const fb = sh().fb;
    const int n0 = c.n0, nr = sh().a.nr, W = c.W;
    for (int l = 0; l < c.nlev; l++) {
        const LevelDev& L = c.lev[l];
        for (int q = 0; q < 2; q++) {
            float* x = mplane(sh().a.b, L, q == 0 ? M_X : M_R) - H;
            const long long n = (long long)L.n1 * L.ld;
            for (long long e = (long long)sh().rank * NT5 + threadIdx.x; e < n; e += (long long)nr * NT5) x[e] = 0.0f;
        }
    }
    for (int t = g.id * nr + sh().rank; t < jt.n; t += 2 * nr) {
        const int i = jt.i0(t) + g.tid % TX, j0 = jt.j0(t, TYJ) + g.tid / TX;
        double r[3] = {0.0, 0.0, 0.0};
#pragma unroll 1
        for (int h = 0; h < 2; h++) {
            const int j = j0 + h * TY;
            if (i < c.ilo || i > c.ihi || j > c.n1 - 2) continue;
            const long long k = (long long)j * c.ld + i, s = (long long)j * n0 + i;
            // the caller's columns to both sides (column n0 - 1 of a periodic array repeats column 0)
            const int e = c.periodic && i + 1 == W ? 1 - W : 1, w = c.periodic && i == 0 ? W - 1 : -1;
            const double* X = p.phi + s;
            double a[9];
#pragma unroll
            for (int q = 0; q < 9; q++) a[q] = p.a[q][s];
            const double ax = a[0] * X[0] + a[1] * X[e] + a[2] * X[w] + a[3] * X[n0] + a[4] * X[-n0] + a[5] * X[n0 + e] +
                              a[6] * X[n0 + w] + a[7] * X[-n0 + e] + a[8] * X[-n0 + w];
            const double res = p.q[s] - ax;
#pragma unroll
            for (int q = 0; q < 9; q++) {
                fb[(P_AP + q) * c.ps + k] = a[q];
                store_mirrored(mplane(sh().a.b, L0, M_AP + q), L0.ld, i, j, W, c.periodic, (float)a[q]);
            }
            fb[P_Q * c.ps + k] = res;
            fb[P_KR * c.ps + k] = res;
            mplane(sh().a.b, L0, M_B)[(long long)j * L0.ld + i] = (float)res;
            r[0] += fabs(res);
            r[1] += res * res;
            r[2] = fmax(r[2], fabs(res));
        }
        group_reduce<3, 0x4u>(r, sh().red + g.id * 256, g);
        if (g.tid == 0)
            for (int q = 0; q < 3; q++) part(2)[(long long)t * PSTRIDE + q] = r[q];
    }
}

__device__ __noinline__ void sip_galerkin(int l) {
    const CaseDev& c = sh().c;
    const LevelDev& C = c.lev[l + 1];
    const int nx = C.ihi - C.ilo + 1, n = nx * (C.n1 - 2);
    for (int e = sh().rank * NT5 + threadIdx.x; e < n; e += sh().a.nr * NT5)
        mg_galerkin_point(sh().a.b, c, l, C.ilo + e % nx, 1 + e / nx);
}

// phi = phi0 + e on the unknown cells (the seam column repeats column 0)
__device__ __noinline__ void sip_out(const SipArgs& p) {
    const CaseDev& c = sh().c;
    const int nx = c.ihi - c.ilo + 1, n = nx * (c.n1 - 2);
    const double* E = sh().fb + P_PCOR * c.ps;
    if (sh().ts.pit == 0) return;  // no iteration ran: e = 0
    for (int q = sh().rank * NT5 + threadIdx.x; q < n; q += sh().a.nr * NT5) {
        const int i = c.ilo + q % nx, j = 1 + q / nx;
        double* x = p.phi + (long long)j * c.n0 + i;
        const double v = *x + E[(long long)j * c.ld + i];
        *x = v;
        if (c.periodic && i == 0) x[c.n0 - 1] = v;
    }
}

__device__ __forceinline__ bool sip_run(const SipArgs& p) {
    TeamSh& s = sh();
    const int tid = threadIdx.x;
    for (int k = tid; k < (int)(sizeof(TeamArgs) / 4); k += NT5)
        reinterpret_cast<int*>(&s.a)[k] = reinterpret_cast<const int*>(&p.t)[k];
    for (int k = tid; k < (int)(sizeof(CaseDev) / 4); k += NT5)
        reinterpret_cast<int*>(&s.c)[k] = reinterpret_cast<const int*>(&p.c)[k];
    static_assert(sizeof(TeamState) <= kSipStateBytes && sizeof(TeamState) % 4 == 0, "state between launches");
    for (int k = tid; k < (int)(sizeof(TeamState) / 4); k += NT5)
        reinterpret_cast<int*>(&s.ts)[k] = p.first ? 0 : reinterpret_cast<const int*>(p.state)[k];
    if (tid == 0) {
        s.rank = blockIdx.x;
        s.bar = p.t.bar;
        s.target = 0;
        s.fb = p.t.b.f64 + p.c.base + H;
        s.tail = team_tail(p.c);
    }
    __syncthreads();
    if (p.first) {
        sip_start(p);
        TEAM_SYNC();
        for (int l = 0; l + 1 < s.c.nlev; l++) {
            sip_galerkin(l);
            TEAM_SYNC();
        }
        team_face_total();
    }
    if (!team_pressure()) return false;
    const bool over = s.ts.pdone || s.ts.pit >= p.t.maxit_p;
    if (over) sip_out(p);
    TEAM_SYNC();
    if (blockIdx.x == 0) {
        for (int k = tid; k < (int)(sizeof(TeamState) / 4); k += NT5)
            reinterpret_cast<int*>(p.state)[k] = reinterpret_cast<const int*>(&s.ts)[k];
        if (tid == 0) {
            p.out[0] = over;
            p.out[1] = s.ts.pit;
            p.out[2] = s.ts.status;
            p.out[3] = s.ts.pstatus;
        }
    }
    return true;
}
#undef TEAM_SYNC

}  // namespace

__global__ void __launch_bounds__(TEAM_THREADS, 1) k_team_f64(const __grid_constant__ TeamArgs a) { team_run<false>(a); }
__global__ void __launch_bounds__(TEAM_THREADS, 1) k_team_mx(const __grid_constant__ TeamArgs a) { team_run<true>(a); }

__global__ void __launch_bounds__(TEAM_THREADS, 1) k_team_sip(const __grid_constant__ SipArgs p) { sip_run(p); }

size_t sip_smem() { return (size_t)WORK_OFF + WORK_MIN; }

size_t team_smem(int max_W) {
    const size_t rows = 4 * (size_t)(max_W + 1) * sizeof(double);  // the far field's rows
    return (size_t)WORK_OFF + (rows > (size_t)WORK_MIN ? rows : (size_t)WORK_MIN);
}

}  // namespace cfd
