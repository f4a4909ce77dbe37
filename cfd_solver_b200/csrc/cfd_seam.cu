// cfd_seam.cu -- the fine-grained gauss() seam: one stored-coefficient system solve.
//
// The reference's gauss() (PSolver.cpp:2280-2446) takes the 25 coefficient planes
// of one momentum / energy system, the iterate phi (initial guess, boundary values)
// and the right-hand side q, and runs relative-L1-stopped lexicographic Gauss-Seidel.
// cfd_gauss_solve() takes the same planes as device arrays in the reference's
// argument order and solves with Chebyshev-accelerated Jacobi sweeps instead (the
// spectrum bounds of D^-1 A come from the coefficients: smooth modes at 1/max(ap),
// Gershgorin on top). Layout: n1*n0 float64, [j][i]; with `periodic` the seam
// column n0-1 duplicates column 0 as in the reference, unknowns i = 0..n0-2;
// otherwise columns 0 and n0-1 are fixed. 9-point rows: j = 1, n1-2 (and, when not
// periodic, i = 1, n0-2).
//
// The whole solve is one cooperative launch: the bounds, the sweeps and the stop rule, with a
// counter barrier between them whose polls are bounded. The host reads the outcome once (per
// kSeamSweeps sweeps). Every CTA sums the partial residuals itself in the same order, so all
// take the same decision. The pass that finds the bounds also forms the first sweep's Jacobi
// corrections, which need only the step length 2 / (a + b) from it: the first sweep then adds
// them without reading the 25 planes again. Bound by the coefficient planes' bytes on large
// grids (1025^2: 41 us a sweep of 28 planes, 5.7 TB/s; 24 sweeps 2.73 -> 1.05 ms a call) and by
// the launch, the barriers and the loads' latency on small ones (257^2, 4 sweeps: 772 -> 50 us;
// before, a cudaMalloc, a launch per sweep, a host wait per pair and a cudaFree).
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <mutex>

#include "../../include/cfd_b200.h"
#include "cfd_scratch.cuh"
#include "cfd_share.cuh"

namespace cfd_seam {

constexpr int BS = 256;
constexpr int MAX_BLOCKS = 2048;         // rows of a partial buffer
constexpr int kSeamSweeps = 512;         // sweeps of one launch at most

// scratch layout (doubles): scalars, two partial buffers of three columns, the second iterate
enum { SC_A, SC_B, SC_R0, SC_W, SC_DONE, SC_SWEEPS, SC_FAIL, SC_CNT, NSC };
constexpr int SCRATCH_HEAD = 8 + 4096;
static_assert(NSC <= 8 && 8 + 2 * MAX_BLOCKS <= SCRATCH_HEAD, "scratch layout");

struct Sys {
    int n0, n1, periodic;
    const double* c[25];  // gauss() argument order
    double* x0;           // caller's phi
    double* x1;           // scratch iterate
    const double* q;
    double* sc;           // scalars
    double* part;         // per-block partials, two buffers of MAX_BLOCKS
    unsigned int* cnt;    // barrier arrivals, zero at launch
    unsigned polls;       // of a barrier before it gives up
};

// gauss() argument order: ap, ae, as, an, aw, ase, asw, ane, anw, ass, assee, assww, asse,
// assw, asee, asww, ann, annee, annww, anne, annw, anee, anww, aee, aww
__host__ __device__ constexpr int dx_of(int m) {
    constexpr int d[25] = {0, 1, 0, 0, -1, 1, -1, 1, -1, 0, 2, -2, 1, -1, 2, -2, 0, 2, -2, 1, -1, 2, -2, 2, -2};
    return d[m];
}
__host__ __device__ constexpr int dy_of(int m) {
    constexpr int d[25] = {0, 0, -1, 1, 0, -1, -1, 1, 1, -2, -2, -2, -2, -2, -1, -1, 2, 2, 2, 2, 2, 1, 1, 0, 0};
    return d[m];
}

// all CTAs have arrived and see one another's stores; false when the polls ran out
__device__ __forceinline__ bool seam_barrier(const Sys& s, unsigned& target) {
    target += gridDim.x;
    __syncthreads();
    bool got = true;
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(s.cnt, 1u);
        got = false;
        for (unsigned n = 0; n < s.polls && !got; n++) {
            unsigned v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(s.cnt) : "memory");
            got = (int)(v - target) >= 0;
        }
        __threadfence();
        if (!got) s.sc[SC_FAIL] = 1.0;
    }
    return __syncthreads_and(got);
}

template <bool MAX>
__device__ __forceinline__ double block_fold(double v, double* sm) {
    for (int o = 16; o > 0; o >>= 1) {
        const double y = __shfl_down_sync(0xffffffffu, v, o);
        v = MAX ? fmax(v, y) : v + y;
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = v;
    __syncthreads();
    double r = sm[0];
    for (int w = 1; w < BS / 32; w++) r = MAX ? fmax(r, sm[w]) : r + sm[w];
    return r;  // in every thread
}
// fold of one value per CTA over the grid, the same bits in every CTA
template <bool MAX>
__device__ __forceinline__ double grid_fold(const double* part, double* sm) {
    double v = 0.0;
    for (int m = threadIdx.x; m < (int)gridDim.x; m += BS) v = MAX ? fmax(v, part[m]) : v + part[m];
    return block_fold<MAX>(v, sm);
}

struct Cell {
    int i, j;
    int col[5];  // array column of i - 2 .. i + 2, less i (the periodic wrap without a branch)
    long long k;
    bool near9;
    __device__ __forceinline__ Cell(const Sys& s, int e, int ilo, int nx) {
        j = 1 + e / nx;
        i = ilo + (e - (j - 1) * nx);
        k = (long long)j * s.n0 + i;
        near9 = j == 1 || j == s.n1 - 2 || (!s.periodic && (i == 1 || i == s.n0 - 2));
        const int P = s.n0 - 1;
#pragma unroll
        for (int d = -2; d <= 2; d++) {
            const int ii = i + d;
            col[d + 2] = s.periodic ? (ii < 0 ? d + P : ii >= P ? d - P : d) : d;
        }
    }
};

// sum of the off-centre couplings of `src` at the cell, in gauss()'s order; with ABS also the
// sum of the couplings' magnitudes
template <bool ABS>
__device__ __forceinline__ double couplings(const Sys& s, const Cell& t, const double* src, double& off) {
    double a[8], x[8], sum = 0.0;
#pragma unroll
    for (int b = 0; b < 3; b++) {  // eight at a time: their loads in flight together
        if (b > 0 && t.near9) break;
#pragma unroll
        for (int m = 0; m < 8; m++) {
            const int q = 1 + 8 * b + m;
            a[m] = s.c[q][t.k];
            x[m] = src[t.k + (long long)dy_of(q) * s.n0 + t.col[dx_of(q) + 2]];
        }
#pragma unroll
        for (int m = 0; m < 8; m++) {
            sum += a[m] * x[m];
            if (ABS) off += fabs(a[m]);
        }
    }
    return sum;
}

__device__ __forceinline__ void put(const Sys& s, double* dst, const Cell& t, double v) {
    dst[t.k] = v;
    if (s.periodic && t.i == 0) dst[(long long)t.j * s.n0 + s.n0 - 1] = v;  // seam column
}

// sweeps [first, first + nsweeps) of the solve (an even number); first == 0 also finds the bounds
__global__ void __launch_bounds__(BS, 2) k_seam_solve(const __grid_constant__ Sys s, int first, int nsweeps, double tol) {
    __shared__ double sm[BS / 32];
    unsigned target = 0;
    const int ilo = s.periodic ? 0 : 1, nx = s.n0 - 2 - ilo + 1, ncell = nx * (s.n1 - 2);
    const int stride = gridDim.x * BS, e0 = blockIdx.x * BS + threadIdx.x;
    double a, b, r0, w;
    int sweep = first;
    if (first == 0) {
        // bounds; the first sweep's corrections xj - x into x1; its residual
        double ap_most = 0.0, off_most = 0.0, r = 0.0;
        for (int e = e0; e < ncell; e += stride) {
            const Cell t(s, e, ilo, nx);
            const double ap = s.c[0][t.k], rhs = s.q[t.k], xk = s.x0[t.k];
            double off = 0.0;
            const double sum = couplings<true>(s, t, s.x0, off);
            const double xj = (rhs - sum) / ap;
            s.x1[t.k] = xj - xk;
            r += fabs(rhs - ap * xk - sum);
            ap_most = fmax(ap_most, fabs(ap));
            off_most = fmax(off_most, off / fabs(ap));
        }
        // boundary values of the second iterate
        for (int e = e0; e < s.n0; e += stride) {
            s.x1[e] = s.x0[e];
            const long long k = (long long)(s.n1 - 1) * s.n0 + e;
            s.x1[k] = s.x0[k];
        }
        if (!s.periodic)
            for (int e = e0; e < s.n1; e += stride) {
                const long long k = (long long)e * s.n0;
                s.x1[k] = s.x0[k];
                s.x1[k + s.n0 - 1] = s.x0[k + s.n0 - 1];
            }
        double* p = s.part;
        ap_most = block_fold<true>(ap_most, sm);
        off_most = block_fold<true>(off_most, sm);
        r = block_fold<false>(r, sm);
        const int G = gridDim.x;
        if (threadIdx.x == 0) {
            p[blockIdx.x] = ap_most;
            p[G + blockIdx.x] = off_most;
            p[2 * G + blockIdx.x] = r;
        }
        if (!seam_barrier(s, target)) return;
        ap_most = grid_fold<true>(p, sm);
        off_most = grid_fold<true>(p + G, sm);
        r = grid_fold<false>(p + 2 * G, sm);
        a = 0.9 / ap_most;
        b = 1.05 * (1.0 + off_most);
        r0 = r != 0.0 ? r : 1.0;
        const double g = 2.0 / (a + b), s2 = ((b + a) / (b - a)) * ((b + a) / (b - a));
        w = 1.0 / (1.0 - 1.0 / (2.0 * s2));
        for (int e = e0; e < ncell; e += stride) {
            const Cell t(s, e, ilo, nx);
            put(s, s.x1, t, s.x0[t.k] + g * s.x1[t.k]);
        }
        if (!seam_barrier(s, target)) return;
        sweep = 1;
    } else {
        a = s.sc[SC_A];
        b = s.sc[SC_B];
        r0 = s.sc[SC_R0];
        w = s.sc[SC_W];
    }
    const double g = 2.0 / (a + b), s2 = ((b + a) / (b - a)) * ((b + a) / (b - a));
    double done = 0.0;
    for (; sweep < first + nsweeps; sweep++) {
        // x_{k+1} overwrites x_{k-1}: even sweeps from the caller's array into the scratch
        const bool to_scratch = (sweep & 1) == 0;
        const double* src = to_scratch ? s.x0 : s.x1;
        double* dst = to_scratch ? s.x1 : s.x0;
        double r = 0.0, unused = 0.0;
        for (int e = e0; e < ncell; e += stride) {
            const Cell t(s, e, ilo, nx);
            const double ap = s.c[0][t.k], rhs = s.q[t.k], xk = src[t.k], xm = dst[t.k];
            const double sum = couplings<false>(s, t, src, unused);
            const double xj = (rhs - sum) / ap;
            put(s, dst, t, w * (xk + g * (xj - xk) - xm) + xm);
            r += fabs(rhs - ap * xk - sum);
        }
        w = 1.0 / (1.0 - w / (4.0 * s2));
        // pairs end in the caller's array; the stop is decided on the second sweep of a pair
        double* p = s.part + ((sweep >> 1) & 1) * MAX_BLOCKS;
        if (!to_scratch) {
            r = block_fold<false>(r, sm);
            if (threadIdx.x == 0) p[blockIdx.x] = r;
        }
        if (!seam_barrier(s, target)) return;
        if (to_scratch) continue;
        const double t = grid_fold<false>(p, sm);
        if (t / r0 < tol || !isfinite(t)) {
            done = isfinite(t) ? 1.0 : 2.0;
            sweep++;
            break;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        s.sc[SC_A] = a;
        s.sc[SC_B] = b;
        s.sc[SC_R0] = r0;
        s.sc[SC_W] = w;
        s.sc[SC_DONE] = done;
        s.sc[SC_SWEEPS] = (double)sweep;
    }
}

// CTAs that are resident together on the current device, and its SMs (0: the query failed)
struct Resident {
    int dev, all, sms;
};
Resident resident_blocks() {
    static std::atomic<int> known[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return {0, 0, 0};
    int v = known[dev].load();
    if (v == 0) {
        int sms = 0, per = 0;
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_seam_solve, BS, 0) != cudaSuccess)
            return {0, 0, 0};
        v = sms << 16 | std::min(sms * per, MAX_BLOCKS / 3);
        known[dev].store(v);
    }
    return {dev, v & 0xffff, v >> 16};
}

}  // namespace cfd_seam

void cfd_internal_set_error(const char* msg);

// shared driver on `scratch` (cfd_seam_scratch_doubles() doubles, 16-byte aligned)
int cfd_seam_solve(int n0, int n1, int periodic, const double* const* coef, double* phi, const double* q,
                   double tol, int maxit, int* sweeps, void* stream, double* scratch, unsigned polls) {
    using namespace cfd_seam;
    cudaStream_t st = (cudaStream_t)stream;
    Sys s;
    s.n0 = n0; s.n1 = n1; s.periodic = periodic;
    for (int m = 0; m < 25; m++) s.c[m] = coef[m];
    const int nx = periodic ? n0 - 1 : n0 - 2, ny = n1 - 2;
    s.sc = scratch;
    s.cnt = reinterpret_cast<unsigned int*>(scratch + SC_CNT);
    s.part = scratch + 8;
    s.x0 = phi;
    s.x1 = scratch + SCRATCH_HEAD;
    s.q = q;
    s.polls = polls;
    const Resident most = resident_blocks();
    if (most.all <= 0) {
        cfd_internal_set_error("gauss seam: no usable device");
        return CFD_E_CUDA;
    }
    const int grid = (int)std::min<long long>(most.all, ((long long)nx * ny + BS - 1) / BS);
    const cfd::ChipShare share(most.dev, std::min(grid, most.sms));  // a step beside this call may give way
    // sweeps run in pairs (the pair ends in the caller's array), so at most maxit rounded
    // down to even sweeps are taken; the outcome is read once per launch
    double sc[8] = {};
    if (cudaMemsetAsync(scratch, 0, sizeof(sc), st) != cudaSuccess) {
        cfd_internal_set_error("gauss seam: scratch initialisation failed");
        return CFD_E_CUDA;
    }
    int done = 0;
    for (int first = 0; first + 2 <= maxit && !done; first += kSeamSweeps) {
        int nsweeps = std::min(kSeamSweeps, (maxit - first) / 2 * 2);
        if (first > 0 && cudaMemsetAsync(s.cnt, 0, sizeof(double), st) != cudaSuccess) {
            cfd_internal_set_error("gauss seam: stream error");
            return CFD_E_CUDA;
        }
        void* args[] = {&s, &first, &nsweeps, &tol};
        if (cudaLaunchCooperativeKernel((const void*)k_seam_solve, dim3(grid), dim3(BS), args, 0, st) != cudaSuccess) {
            cfd_internal_set_error("gauss seam: kernel launch failed");
            return CFD_E_CUDA;
        }
        if (cudaMemcpyAsync(sc, scratch, sizeof(sc), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
            cudaStreamSynchronize(st) != cudaSuccess) {
            cfd_internal_set_error("gauss seam: stream error");
            return CFD_E_CUDA;
        }
        if (sc[SC_FAIL] != 0.0) {
            cfd_internal_set_error("gauss seam: a bounded wait inside the kernel timed out");
            return CFD_E_CUDA;
        }
        if (sweeps) *sweeps = (int)sc[SC_SWEEPS];
        done = sc[SC_DONE] != 0.0;
    }
    if (sc[SC_DONE] == 2.0) {
        cfd_internal_set_error("gauss seam: residual not finite");
        return CFD_E_DIVERGED;
    }
    if (!done) cfd_internal_set_error("gauss seam: maxit reached");
    return done ? CFD_OK : CFD_E_MAXITER;
}

size_t cfd_seam_scratch_doubles(int n0, int n1, int periodic) {
    (void)periodic;
    return (size_t)cfd_seam::SCRATCH_HEAD + (size_t)n0 * n1;
}

// ---- the library's scratch pool (cfd_scratch.cuh)
namespace cfd {
namespace {
constexpr int kMaxDevices = 64;
struct DevicePool {
    cudaMemPool_t pool;
    unsigned long long context;
};
std::mutex g_pool_mu;
DevicePool g_pool[kMaxDevices] = {};

cudaMemPool_t scratch_pool() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
    const unsigned long long id = context_id();
    std::lock_guard<std::mutex> lock(g_pool_mu);
    DevicePool& d = g_pool[dev];
    if (!d.pool || d.context != id) {  // the pool of a context that is gone went with it
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t p = nullptr;
        if (cudaMemPoolCreate(&p, &props) != cudaSuccess) return nullptr;
        unsigned long long keep = kScratchKeep;
        cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep);
        d = {p, id};
    }
    return d.pool;
}
}  // namespace

unsigned long long context_id() {
    using GetId = CUresult (*)(CUcontext, unsigned long long*);
    static const GetId get = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuCtxGetId", &f, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            f = nullptr;
        return reinterpret_cast<GetId>(f);
    }();
    unsigned long long id = 0;
    // cudaFree(nullptr) makes the device's context current where the thread has none yet
    if (cudaFree(nullptr) != cudaSuccess || !get || get(nullptr, &id) != CUDA_SUCCESS) return 0;
    return id;
}

void* scratch_take(size_t bytes, cudaStream_t st) {
    void* p = nullptr;
    cudaMemPool_t pool = scratch_pool();
    if (!pool || cudaMallocFromPoolAsync(&p, bytes, pool, st) != cudaSuccess) {
        cudaGetLastError();  // the failure is reported by the caller
        return nullptr;
    }
    return p;
}

void scratch_give(void* p, cudaStream_t st) {
    if (p) cudaFreeAsync(p, st);
}
}  // namespace cfd

extern "C" int cfd_internal_gauss_solve(int n0, int n1, int periodic, const double* const* coef, double* phi,
                                        const double* q, double tol, int maxit, int* sweeps, void* stream,
                                        unsigned polls) {
    if (n0 < 8 || n1 < 6 || !coef || !phi || !q || maxit < 2) {
        cfd_internal_set_error("cfd_gauss_solve: bad arguments");
        return CFD_E_ARG;
    }
    for (int m = 0; m < 25; m++)
        if (!coef[m]) {
            cfd_internal_set_error("cfd_gauss_solve: null coefficient plane");
            return CFD_E_ARG;
        }
    double* scratch = (double*)cfd::scratch_take(cfd_seam_scratch_doubles(n0, n1, periodic) * sizeof(double),
                                                 (cudaStream_t)stream);
    if (!scratch) {
        cfd_internal_set_error("cfd_gauss_solve: no device memory for the scratch");
        return CFD_E_OOM;
    }
    const int rc = cfd_seam_solve(n0, n1, periodic, coef, phi, q, tol, maxit, sweeps, stream, scratch, polls);
    if (rc == CFD_E_CUDA) cudaStreamSynchronize((cudaStream_t)stream);
    cfd::scratch_give(scratch, (cudaStream_t)stream);
    return rc;
}

extern "C" int cfd_gauss_solve(int n0, int n1, int periodic, const double* const* coef, double* phi,
                               const double* q, double tol, int maxit, int* sweeps, void* stream) {
    return cfd_internal_gauss_solve(n0, n1, periodic, coef, phi, q, tol, maxit, sweeps, stream, cfd::kSeamPolls);
}
