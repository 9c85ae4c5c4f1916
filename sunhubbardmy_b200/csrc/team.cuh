// Teams: the CTAs of one thread-block cluster that work on one chain.
//
// A kernel that is launched with a cluster of several CTAs per chain splits the
// chain's tiles or columns over them and exchanges results through global
// memory (the L2), with the cluster barrier's release and acquire in place of
// __syncthreads().  Launched without a cluster the team is one CTA and sync()
// is __syncthreads().
#pragma once
#include "common.cuh"

struct Team {
    int rank, size;
    // every thread of every CTA of the team calls it; global and shared writes
    // before it are visible to the team after it
    DQ_DEV void sync() const {
        if (size == 1) {
            __syncthreads();
        } else {
            __syncwarp();
            asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
        }
    }
    // width of the column chunks that n columns are dealt out in (chunk i to
    // rank i mod size): everything for one CTA, else multiples of 16
    DQ_DEV int chunk(int n) const { return size == 1 ? n : ((n + size - 1) / size + 15) & ~15; }
};

DQ_DEV Team this_team() {
    unsigned r, s;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(s));
    return Team{(int)r, (int)s};
}

#define TEAM_SMEM_MAX (200 * 1024)    // dynamic shared memory allowed to the team kernels

static inline void team_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* at, int nchains, int team, size_t smem,
                               cudaStream_t st) {
    cfg.gridDim = dim3(nchains * team);
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = team;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = team > 1 ? 1 : 0;
}

// k with a cluster of `team` CTAs per chain: grid nchains x team, chain blockIdx.x / team
template <class... P, class... A>
static inline void launch_team(void (*k)(P...), int nchains, int team, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    team_config(cfg, at, nchains, team, smem, st);
    cudaLaunchKernelEx(&cfg, k, (P)args...);
}
