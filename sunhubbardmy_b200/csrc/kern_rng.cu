// SFMT-19937 on the device, one warp per chain.
//
// Reference: lib/m_spring.f90:187-379 (spring_sfmt_init/_source/_kernel/_core);
// spring_sfmt_stream maps the 32-bit output u to (u + 0.5) / 2^32.  The
// generator state (624 words + read index) lives in the chain's device memory
// and advances exactly as the reference's does, so the draws of a chain are
// the reference's draws for the same seed.  The draws of a whole half sweep
// (two per site and slice) are produced ahead of the update kernels, which read
// them in visiting order.
#include "chain_access.cuh"
#include "kernels.h"

#define SFMT_N 156
#define SFMT_N32 624
#define SFMT_POS1 122

// The next 156 words of 128 bits, by one warp on the state in shared memory.  Word i
// is r(i) = t(i) ^ (r(i-2) >> 8) ^ (r(i-1) << 18 per lane), where
// t(i) = a ^ (a << 8) ^ ((b >> 11) & mask) needs only a = w(i) and b = w(i + 122) of the old
// state or r(i - 34): the lanes form 32 of the t at once, and the serial part that is
// left is a few shifts a word, which every lane runs (keeping its own word).  The
// state is a serial chain of 25,600 words a half sweep for 256 sites and 200 slices.  With
// 100 slices the draws, copies and wrap checks of a sweep take 4.23 ms, and 5.72 with the
// whole recursion in one lane.
__device__ void sfmt_gen_all(uint4* st, uint4* tb) {
    const int lane = threadIdx.x & 31;
    uint4 r1 = st[SFMT_N - 2], r2 = st[SFMT_N - 1];
    for (int i0 = 0; i0 < SFMT_N; i0 += 32) {
        const int i = i0 + lane, n = min(32, SFMT_N - i0);
        if (i < SFMT_N) {
            const uint4 a = st[i], b = st[i + SFMT_POS1 < SFMT_N ? i + SFMT_POS1 : i + SFMT_POS1 - SFMT_N];
            uint4 t;
            t.x = a.x ^ (a.x << 8) ^ ((b.x >> 11) & 0xdfffffefU);
            t.y = a.y ^ __funnelshift_l(a.x, a.y, 8) ^ ((b.y >> 11) & 0xddfecb7fU);
            t.z = a.z ^ __funnelshift_l(a.y, a.z, 8) ^ ((b.z >> 11) & 0xbffaffffU);
            t.w = a.w ^ __funnelshift_l(a.z, a.w, 8) ^ ((b.w >> 11) & 0xbffffff6U);
            tb[lane] = t;
        }
        __syncwarp();
        uint4 mine = make_uint4(0, 0, 0, 0);
#pragma unroll 4
        for (int q = 0; q < n; ++q) {
            uint4 r = tb[q];
            r.x ^= __funnelshift_r(r1.x, r1.y, 8) ^ (r2.x << 18);
            r.y ^= __funnelshift_r(r1.y, r1.z, 8) ^ (r2.y << 18);
            r.z ^= __funnelshift_r(r1.z, r1.w, 8) ^ (r2.z << 18);
            r.w ^= (r1.w >> 8) ^ (r2.w << 18);
            r1 = r2;
            r2 = r;
            if (q == lane) mine = r;
        }
        __syncwarp();
        if (i < SFMT_N) st[i] = mine;
        __syncwarp();
    }
}

// count = slices * rps draws per chain (slices > 0; rps = words per time slice
// of the chain's model), or exactly -slices draws.  One warp per chain: the
// state is held in shared memory, and the warp copies each block of 624 outputs to the chain's draw
// buffer with coalesced stores.
#define SFMT_WARPS 4
__global__ void __launch_bounds__(32 * SFMT_WARPS) k_sfmt_fill(const ChainDev* __restrict__ chains, int ch0,
                                                               int nchains, int slices) {
    __shared__ uint4 sst[SFMT_WARPS][SFMT_N];
    __shared__ uint4 stb[SFMT_WARPS][32];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ch = ch0 + blockIdx.x * SFMT_WARPS + w;
    if (ch >= ch0 + nchains) return;      // whole warps; no block barrier below
    const int count = slices > 0 ? slices * chains[ch].md->rps : -slices;
    uint32_t* gst = chains[ch].sfmt;
    uint32_t* out = chains[ch].rnd;
    uint32_t* s = (uint32_t*)sst[w];
    for (int e = lane; e < SFMT_N32; e += 32) s[e] = gst[e];
    int idx = (int)gst[SFMT_N32];
    __syncwarp();
    for (int k = 0; k < count;) {
        if (idx >= SFMT_N32) {
            sfmt_gen_all(sst[w], stb[w]);
            idx = 0;
        }
        const int n = min(SFMT_N32 - idx, count - k);
        for (int e = lane; e < n; e += 32) out[k + e] = s[idx + e];
        k += n;
        idx += n;
        __syncwarp();                     // the block is read before it is regenerated
    }
    for (int e = lane; e < SFMT_N32; e += 32) gst[e] = s[e];
    if (lane == 0) gst[SFMT_N32] = (uint32_t)idx;
}

void launch_sfmt(const ChainDev* chains, int nchains, int slices, cudaStream_t st) {
    k_sfmt_fill<<<(nchains + SFMT_WARPS - 1) / SFMT_WARPS, 32 * SFMT_WARPS, 0, st>>>(chains, 0, nchains, slices);
}

void launch_sfmt_raw(const ChainDev* chains, int chain, int count, cudaStream_t st) {
    k_sfmt_fill<<<1, 32 * SFMT_WARPS, 0, st>>>(chains, chain, 1, -count);
}
