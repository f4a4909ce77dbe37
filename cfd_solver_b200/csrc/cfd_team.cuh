// cfd_team.cuh -- the team kernel: whole time steps of a case by one team of CTAs (cfd_team.cu).
#pragma once
#include "cfd_common.cuh"

namespace cfd {

constexpr int TEAM_THREADS = 512;
constexpr int TEAM_MAX_CLUSTER = 16;

struct TeamArgs {
    BatchDev b;           // b.cur: state parity before the first step
    const int* ids;       // case of each team
    unsigned* bar;        // grid form: per team arrival counter, zero at launch
    int nr;               // CTAs per team
    int cluster;          // 1: a team is a thread-block cluster; 0: a share of a cooperative grid
    int nsteps;
    int sweep_cap;        // sweeps of one momentum / energy solve
    int maxit_p;
    int fin_threads;      // threads that sum a sweep's partial residuals (as k_sweep_fin)
    int nu_pre, nu_post, coarse_sweeps;
};

__global__ void k_team_f64(const __grid_constant__ TeamArgs a);
__global__ void k_team_mx(const __grid_constant__ TeamArgs a);
// dynamic shared memory of a team CTA for cases of at most max_W stored columns
size_t team_smem(int max_W);
}  // namespace cfd
