// cfd_team.cuh -- the team kernel: whole time steps of a case by one team of CTAs (cfd_team.cu).
#pragma once
#include "cfd_common.cuh"

namespace cfd {

constexpr int TEAM_THREADS = 512;
constexpr unsigned TEAM_POLLS = 1u << 24;  // polls of a grid-form barrier before it gives up (about 10 s)

struct TeamArgs {
    BatchDev b;           // b.cur: state parity before the first step
    const int* ids;       // case of each team
    unsigned* bar;        // grid form: per team arrival counter, zero at launch
    int nr;               // CTAs per team
    int cluster;          // 1: a team is a thread-block cluster; 0: a share of a cooperative grid
    int nsteps;
    int sweep_cap;        // sweeps of one momentum / energy solve
    int maxit_p;          // iteration cap of the pressure solve
    int p_iters;          // iterations of it in this launch
    int nu_pre, nu_post, coarse_sweeps;
    unsigned polls;       // limit of the grid form's barrier waits
};

// The sip9p() seam: one pressure-correction solve by one team (a cooperative grid). The caller's
// nine planes (in the order P_AP .. P_ASW), phi0 and q are n1 x n0 arrays.
struct SipArgs {
    TeamArgs t;
    CaseDev c;
    const double* a[9];
    double* phi;
    const double* q;
    int first;      // 1: the solve's first launch; 0: continues it
    void* state;    // solver state between launches (kSipStateBytes)
    int* out;       // done, iterations, status, pressure status
};
constexpr size_t kSipStateBytes = 1024;
constexpr int kSipOut = 4;

__global__ void k_team_f64(const __grid_constant__ TeamArgs a);
__global__ void k_team_mx(const __grid_constant__ TeamArgs a);
__global__ void k_team_sip(const __grid_constant__ SipArgs p);
size_t sip_smem();
// dynamic shared memory of a team CTA for cases of at most max_W stored columns
size_t team_smem(int max_W);
}  // namespace cfd
