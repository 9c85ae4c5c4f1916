// Local Hubbard-Stratonovich updates of one time slice, a team of CTAs (team.cuh) per
// chain, or one CTA where chains are many or small.
//
// Reference: src/dqmc_config_u/dqmc_update_delay.f90:1-137 (delayed update),
// dqmc_update.f90 (fast update) and dqmc_update_submatrix.f90 (submatrix
// update).  All three visit the sites in order with two SFMT draws per site
// and accept with |Re(R phase)/Re(phase)| > r; they differ only in how the
// accepted rank-1 changes are folded into G.  This kernel runs all of them as
// one scheme: the accept walk of a window of consecutive sites needs only the
// window's block of G plus the window's own new columns (the submatrix
// update's observation), all in shared memory and walked by one warp; the
// rank-1 changes are carried as delayed columns (A, B), G' = G + A B^T, and
// flushed after nublock accepted sites as one DMMA tensor-core GEMM (the
// delayed update's blocking).  The accept/reject sequence equals the
// reference's in exact arithmetic.
#include "chain_access.cuh"
#include "kernels.h"
#include "flush.cuh"
#include "team.cuh"

#define UPD_NT 256                 // threads per CTA

DQ_DEV double u32_to_stream(uint32_t u) { return ((double)u + 0.5) * (1.0 / 4294967296.0); }

// ph times a power of two that brings its larger part near 1 (the quotient of the parts keeps
// its bits), where it has left 2^-100 .. 2^100
DQ_DEV double2 near_one(double2 ph) {
    const int e = max(__double2hiint(ph.x) & 0x7fffffff, __double2hiint(ph.y) & 0x7fffffff) >> 20;
    if (abs(e - 1023) <= 100 || e == 2047) return ph;
    return cscale(ph, __hiloint2double((2046 - e) << 20, 0));
}

// Window of UPD_L consecutive sites, walked by warp 0 (lane p owns site
// w0 + p).  Its state overlays the GEMM staging buffer, which is only used by
// the flush after the window has been closed.
#define UPD_L 32
#define UPD_LP (UPD_L + 1)       // odd pitch: rows and columns of gW are both conflict-free
#define UPD_SP (UPD_L + 2)       // pitch of the staged rows: 2 (mod 8), conflict-free DMMA fragments
#define UPD_CH 4                 // window columns extended to all rows per pass (one CTA per chain)
struct UpdWalk {
    double2 gW[UPD_L * UPD_LP];  // G'(w0 + p, w0 + q) at gW[q * UPD_LP + p], G' = G + A B^T
    double2 aW[UPD_L][UPD_L];    // [m][p]: window row p of the window's m-th new column of A
    double2 bW[UPD_L][UPD_L];    // the same for B
};
struct UpdWin {
    double2 sg[UPD_L];           // scale of the m-th accepted flip (delta / ratio)
    int pm[UPD_L];               // window position of the m-th accepted site (0 from r on)
    int r, wend;                 // accepted sites; sites the walk consumed
    int pad[2];
};
static_assert(sizeof(UpdWin) % 16 == 0 && sizeof(UpdWalk) % 16 == 0, "window state alignment");
// Dynamic shared memory of the update kernel: the window state, then
//  * one CTA per chain: the walk's state and a chunk's rows of the delayed columns;
//  * teams: the walk's state or (after the walk) the window's rows of the delayed
//    columns, and the two triangles of upd_extend_tile;
// or the flush staging, whichever is larger.
__host__ __device__ inline size_t upd_rows_elems(int nb) { return (size_t)2 * ((nb + 3) & ~3) * UPD_SP; }
__host__ __device__ inline size_t upd_walk_elems(int nb, bool team) {
    const size_t w = sizeof(UpdWalk) / sizeof(double2), r = upd_rows_elems(nb);
    return team && r > w ? r : w;
}
static size_t upd_smem_bytes(int nb, bool team) {
    const size_t tail = team ? 2 * UPD_L * UPD_LP : (size_t)2 * UPD_CH * nb;
    const size_t w = sizeof(UpdWin) + (upd_walk_elems(nb, team) + tail) * sizeof(double2);
    return w > UpdGemm::SMEM_ELEMS * sizeof(double2) ? w : UpdGemm::SMEM_ELEMS * sizeof(double2);
}

// The window's new columns on all rows are
//   a_m = s_m (c_m + sum_{m' < m} a_m' b_m'(f_m)),      c_m = G'(:,f_m),
//   b_m = c_m + sum_{m' < m} b_m' a_m'(f_m),            c_m = G'(f_m,:)^T - e_(f_m),
// with b_m'(f_m), a_m'(f_m) known from the walk: [a] = [c] Ta, [b] = [c] Tb with
// upper triangular matrices that are the same for every row, so the walk of a team
// forms them as it goes (lane = row j, T(j, m) at j * UPD_LP + m) and the columns are
// two products on the tensor pipe.
//
// One 8-row tile (rows i0..) of the window's new columns of a side (0: A, 1: B), by
// one warp: the columns c as accumulators (column 8 f + 2 (lane & 3) + h in register
// [f][h]), G' = G + A B^T over the k delayed columns being the tile's rows of X times
// the staged rows F of the other factor (pitch UPD_SP); then c T into the columns
// k.. of X.  An accumulator register is the second product's left operand as it
// stands when the four k rows of a step are taken as the columns 8 f + 2 q + h, q = 0..3.
DQ_DEV void upd_extend_tile(const UpdWin* W, const double2* G, double2* X, const double2* F, const double2* T, int side, int N,
                            int k, int w0, int r, int i0) {
    const int lane = threadIdx.x & 31, q4 = lane & 3, row = i0 + (lane >> 2);
    const bool ok = row < N;
    double cr[4][2], ci[4][2];
    int pb[4];
#pragma unroll
    for (int f = 0; f < 4; ++f) {
        pb[f] = W->pm[8 * f + (lane >> 2)];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int m = 8 * f + 2 * q4 + h, site = w0 + W->pm[m];
            double2 g = cmk(0, 0);
            if (ok && m < r) {
                g = side ? G[MIDX(site, row, N)] : G[MIDX(row, site, N)];
                if (side && row == site) g.x -= 1.0;
            }
            cr[f][h] = g.x; ci[f][h] = g.y;
        }
    }
#pragma unroll 4
    for (int kk = 0; kk < k; kk += 4) {
        const int kr = kk + q4;
        const double2 a = (ok && kr < k) ? X[MIDX(row, kr, N)] : cmk(0, 0);
#pragma unroll
        for (int f = 0; f < 4; ++f)
            if (8 * f < r) zdmma(cr[f], ci[f], a, F[kr * UPD_SP + pb[f]]);
    }
#pragma unroll
    for (int g = 0; g < 4; ++g) {
        if (8 * g >= r) break;
        double orr[2] = {0.0, 0.0}, oi[2] = {0.0, 0.0};
#pragma unroll
        for (int f = 0; f <= g; ++f)
#pragma unroll
            for (int h = 0; h < 2; ++h)
                zdmma(orr, oi, cmk(cr[f][h], ci[f][h]), T[(8 * f + 2 * q4 + h) * UPD_LP + 8 * g + (lane >> 2)]);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int m = 8 * g + 2 * q4 + h;
            if (ok && m < r) X[MIDX(row, k + m, N)] = cmk(orr[h], oi[h]);
        }
    }
}

// The same by one CTA for all rows, a thread per row: with every row in one CTA the
// products above would cost half of the flush on the tensor pipe (padding of r to 8
// and the product with T), where the row's own recursion costs a fifth on the FMA pipe.
DQ_DEV void upd_extend_rows(const UpdWin* W, const UpdWalk* Y, const double2* G, double2* A, double2* B, double2* As, int N,
                            int nb, int k, int w0, int r) {
    const int tid = threadIdx.x, nth = blockDim.x;
    double2* Bs = As + UPD_CH * nb;                 // [UPD_CH][nb]: rows A(f_m, :) and B(f_m, :) of a chunk of columns
    for (int m0 = 0; m0 < r; m0 += UPD_CH) {
        const int mc = min(UPD_CH, r - m0);
        for (int e = tid; e < mc * k; e += nth) {
            const int mm = e % mc, m2 = e / mc, sm = w0 + W->pm[m0 + mm];
            As[mm * nb + m2] = A[MIDX(sm, m2, N)];
            Bs[mm * nb + m2] = B[MIDX(sm, m2, N)];
        }
        __syncthreads();
        for (int i = tid; i < N; i += nth) {
            double2 c1[UPD_CH], c2[UPD_CH];
            int pmm[UPD_CH];
#pragma unroll
            for (int mm = 0; mm < UPD_CH; ++mm) {
                pmm[mm] = W->pm[m0 + min(mm, mc - 1)];
                c1[mm] = G[MIDX(i, w0 + pmm[mm], N)];
                c2[mm] = G[MIDX(w0 + pmm[mm], i, N)];
            }
            // delayed columns since the last flush: G' = G + A B^T
#pragma unroll 4
            for (int m2 = 0; m2 < k; ++m2) {
                const double2 ai = A[MIDX(i, m2, N)], bi = B[MIDX(i, m2, N)];
#pragma unroll
                for (int mm = 0; mm < UPD_CH; ++mm) {
                    c1[mm] = cfma(ai, Bs[mm * nb + m2], c1[mm]);
                    c2[mm] = cfma(As[mm * nb + m2], bi, c2[mm]);
                }
            }
            // this window's earlier chunks
#pragma unroll 2
            for (int m1 = 0; m1 < m0; ++m1) {
                const double2 a1 = A[MIDX(i, k + m1, N)], b1 = B[MIDX(i, k + m1, N)];
#pragma unroll
                for (int mm = 0; mm < UPD_CH; ++mm) {
                    c1[mm] = cfma(Y->bW[m1][pmm[mm]], a1, c1[mm]);
                    c2[mm] = cfma(Y->aW[m1][pmm[mm]], b1, c2[mm]);
                }
            }
            // this chunk, in order
#pragma unroll
            for (int mm = 0; mm < UPD_CH; ++mm) {
                if (mm >= mc) break;
#pragma unroll
                for (int m1 = 0; m1 < mm; ++m1) {
                    c1[mm] = cfma(Y->bW[m0 + m1][pmm[mm]], c1[m1], c1[mm]);
                    c2[mm] = cfma(Y->aW[m0 + m1][pmm[mm]], c2[m1], c2[mm]);
                }
                c1[mm] = cmul(c1[mm], W->sg[m0 + mm]);
                if (i == w0 + pmm[mm]) c2[mm].x -= 1.0;
                A[MIDX(i, k + m0 + mm, N)] = c1[mm];
                B[MIDX(i, k + m0 + mm, N)] = c2[mm];
            }
        }
        __syncthreads();
    }
}

// A team of CTAs per chain; the slice's sites are visited in windows of UPD_L:
//   1. the window block of the current G' = G + A B^T (k delayed columns since
//      the last flush) is formed in shared memory;
//   2. warp 0 walks the window: lane p tests site w0 + p against its running
//      diagonal, the first passing lane (a ballot) is accepted, every lane
//      updates the phase identically and appends its row of the new window
//      columns (a = s (G'(:,f) + Aw Bw(f,:)^T), b = G'(f,:)^T + Bw Aw(f,:)^T - e_f
//      restricted to the window) -- no block barrier per accepted site;
//   3. A and B are extended by the window's columns on all rows (upd_extend_tile
//      on 8-row tiles, or upd_extend_rows);
//   4. after nublock delayed columns (and at the end of the slice) the
//      factors are flushed, G += A B^T, on the FP64 tensor pipe.
// A window also ends at the accepted site that fills the nublock columns.
// Every CTA of a team forms the window block and walks it for itself (the same
// operations on the same values, so the same decisions), which saves an exchange
// on the serial path; rank 0 alone writes the field and the statistics.  The
// tiles of steps 3 and 4 are dealt out over the team, which meets after each, and
// before a flush that no accepted site of the last window precedes: no CTA
// stores a tile of G while another may still read its window block from it.
//
// forced = 1: the global block move's forced flips of slice nt (sites with
// blk[i] != 0 go to the next field value, no random test, chains whose block
// did not pass the first stage do nothing); the log of the product of the
// flips' ratios is accumulated in stats[ST_BLK_LR_*].
template <bool TEAM>
__global__ void __launch_bounds__(UPD_NT, 2) k_update_delay(const ChainDev* __restrict__ chains, int nt, int visit, int forced,
                                                            int dir) {
    extern __shared__ double2 dsm[];
    const Team tm = TEAM ? this_team() : Team{0, 1};
    const ChainDev& c = chains[blockIdx.x / tm.size];
    const ModelDev& md = *c.md;
    const int N = c.N, nb = md.nublock, lc = md.lcomp, nflr = md.nflr;
    if (forced && c.blk[N] == 0) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nth = blockDim.x;
    cplx* gsm = dsm;                                   // GEMM staging
    UpdWin* W = (UpdWin*)dsm;                          // window state (same memory)
    UpdWalk* Y = (UpdWalk*)(W + 1);
    // teams: rows A(w0 + p, m), B(w0 + p, m) at m * UPD_SP + p, over the walk's state, then Ta and Tb
    double2* sA = (double2*)(W + 1);
    double2* sB = sA + upd_rows_elems(nb) / 2;
    double2* Ta = sA + upd_walk_elems(nb, TEAM);      // one CTA: the chunk's rows
    double2* Tb = Ta + UPD_L * UPD_LP;
    int32_t* cf = c.conf + (size_t)(nt - 1) * N;
    const uint32_t* rw = c.rnd + (size_t)visit * md.rps + md.rw_u[dir];
    double2* G = c.G;
    double2* A = c.A;
    double2* B = c.B;

    // walk state, kept by warp 0
    double2 ph = cmk(c.stats[ST_PHASE_RE], c.stats[ST_PHASE_IM]);
    double acc = 0.0, lr_re = 0.0, lr_im = 0.0;
    if (forced && tid == 0) { lr_re = c.stats[ST_BLK_LR_RE]; lr_im = c.stats[ST_BLK_LR_IM]; }

    int k = 0, s = 0;
    while (s < N) {
        const int w0 = s, L = min(UPD_L, N - w0);
        // 1. warp w forms the 8 x 8 tiles w and w + 8 of the window block
        {
            const int p = 8 * (warp & 3) + (lane >> 2), q0 = 8 * (warp >> 2), q4 = lane & 3;
            double cr[2][2], ci[2][2];
#pragma unroll
            for (int t = 0; t < 2; ++t)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int q = q0 + 16 * t + 2 * q4 + h;
                    const double2 g = (p < L && q < L) ? G[MIDX(w0 + p, w0 + q, N)] : cmk(0, 0);
                    cr[t][h] = g.x; ci[t][h] = g.y;
                }
            if (TEAM)
                for (int e = tid; e < 2 * UPD_L * UPD_LP; e += nth) Ta[e] = cmk(0, 0);
            const int qb = q0 + (lane >> 2);
#pragma unroll 4
            for (int kk = 0; kk < k; kk += 4) {
                const int m = kk + q4;
                const double2 a = (p < L && m < k) ? A[MIDX(w0 + p, m, N)] : cmk(0, 0);
#pragma unroll
                for (int t = 0; t < 2; ++t)
                    zdmma(cr[t], ci[t], a, (qb + 16 * t < L && m < k) ? B[MIDX(w0 + qb + 16 * t, m, N)] : cmk(0, 0));
            }
#pragma unroll
            for (int t = 0; t < 2; ++t)
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    Y->gW[(q0 + 16 * t + 2 * q4 + h) * UPD_LP + p] = cmk(cr[t][h], ci[t][h]);
        }
        __syncthreads();
        // 2. walk (dqmc_update_delay.f90:52-60 per site)
        bool flip = false;
        int nvv = 0;
        if (warp == 0) {
            const int p = lane, j = w0 + p;
            bool cand = false;
            double2 dl = cmk(0, 0), phr = cmk(0, 0), dW = cmk(0, 0);
            double gam = 0.0, thr = 0.0;
            if (p < L) {
                const int is = cf[j];
                const int iflip = forced ? 1 : (int)ceil(u32_to_stream(rw[2 * j]) * (lc - 1));
                const int kk = (is - 1) * (lc - 1) + (iflip - 1);
                dl = md.delta[kk];
                gam = md.gam_ratio[kk];
                phr = md.phase_ratio[kk];
                thr = forced ? 0.0 : u32_to_stream(rw[2 * j + 1]);
                nvv = (is + iflip - 1) % lc + 1;
                cand = !forced || c.blk[j] != 0;
                dW = Y->gW[p * UPD_LP + p];
            }
            W->pm[lane] = 0;
            __syncwarp();
            // FP64 divides and square roots are dependent chains of 75 to 125 cycles, so
            // the loop has only delta / ratio: the test multiplies out Re(phase), and the
            // phase, whose modulus the test does not see, is normalised after the walk
            // (1.7 k cycles per accepted site, 2.3 k before).  Until then near_one keeps it in
            // range: a flip's ratio may be anything whose square FP64 holds (ratio^nflr).
            int r = 0, pc = 0, wend = L, nties = 0;
            while (pc < L) {
                const double2 ratio1 = cadd(cmul(csub(cmk(1, 0), dW), dl), cmk(1, 0));
                double2 rr = ratio1;
                for (int f = 1; f < nflr; ++f) rr = cmul(rr, ratio1);
                double2 rt = cmul(cscale(rr, gam), phr);
                const double num = fabs(cmul(rt, ph).x), ax = fabs(ph.x), lim = thr * ax;
                const bool open = cand && p >= pc;
                const bool pass = open && (forced || num > lim);
                double2 sscl = cmk(0, 0);
                if (pass) sscl = cdiv(dl, ratio1);
                const bool tie = open && !forced && fabs(num - lim) < DQ_NEAR_TIE * ax;
                const unsigned bal = __ballot_sync(0xffffffffu, pass);
                // this iteration decides the lanes up to the first passing one
                // (all remaining lanes when none passes); later lanes are
                // tested again with the updated diagonal
                nties += tie && (bal == 0 || p <= __ffs(bal) - 1);
                if (bal == 0) break;
                const int pf = __ffs(bal) - 1;
                rt.x = __shfl_sync(0xffffffffu, rt.x, pf);
                rt.y = __shfl_sync(0xffffffffu, rt.y, pf);
                sscl.x = __shfl_sync(0xffffffffu, sscl.x, pf);
                sscl.y = __shfl_sync(0xffffffffu, sscl.y, pf);
                ph = cmul(ph, rt);
                if (lane == 0) {
                    acc += 1.0;
                    if (forced) {
                        const double2 l = clog_(rt);
                        lr_re += l.x;
                        lr_im += l.y;
                    }
                    W->pm[r] = pf;
                    W->sg[r] = sscl;
                }
                if (p == pf) { cand = false; flip = true; }
                double2 a = Y->gW[pf * UPD_LP + p];          // G'(p, f)
                double2 b = Y->gW[p * UPD_LP + pf];          // G'(f, p)
                double2 ta = cmk(p == r ? 1.0 : 0.0, 0.0), tb = ta;
                const double2 *Tap = Ta + p * UPD_LP, *Tbp = Tb + p * UPD_LP;
                int m = 0;
                for (; m + 1 < r; m += 2) {        // two steps' loads under way together
                    const double2 cb = Y->bW[m][pf], ca = Y->aW[m][pf], cb1 = Y->bW[m + 1][pf], ca1 = Y->aW[m + 1][pf];
                    const double2 x0 = Y->aW[m][p], y0 = Y->bW[m][p], x1 = Y->aW[m + 1][p], y1 = Y->bW[m + 1][p];
                    a = cfma(cb1, x1, cfma(cb, x0, a));
                    b = cfma(ca1, y1, cfma(ca, y0, b));
                    if (TEAM) {
                        ta = cfma(cb1, Tap[m + 1], cfma(cb, Tap[m], ta));
                        tb = cfma(ca1, Tbp[m + 1], cfma(ca, Tbp[m], tb));
                    }
                }
                if (m < r) {
                    const double2 cb = Y->bW[m][pf], ca = Y->aW[m][pf];
                    a = cfma(cb, Y->aW[m][p], a);
                    b = cfma(ca, Y->bW[m][p], b);
                    if (TEAM) {
                        ta = cfma(cb, Tap[m], ta);
                        tb = cfma(ca, Tbp[m], tb);
                    }
                }
                a = cmul(a, sscl);
                if (p == pf) b.x -= 1.0;
                dW = cfma(a, b, dW);
                Y->aW[r][p] = a;
                Y->bW[r][p] = b;
                if (TEAM) {
                    Ta[p * UPD_LP + r] = cmul(ta, sscl);
                    Tb[p * UPD_LP + r] = tb;
                }
                ph = near_one(ph);
                ++r;
                pc = pf + 1;
                __syncwarp();
                if (k + r == nb) { wend = pc; break; }
            }
            if (r) ph = cscale(ph, 1.0 / sqrt(cabs2(ph)));
            if (lane == 0) { W->r = r; W->wend = wend; }
            nties = warp_sum(nties);
            if (lane == 0 && nties && tm.rank == 0) c.stats[ST_NEAR_TIE] += (double)nties;
        }
        __syncthreads();
        // 3. the window's columns on all rows
        const int r = W->r, wend = W->wend;
        const bool flush = k + r == nb || (w0 + wend >= N && k + r > 0);
        if (r) {
            if (TEAM) {
                for (int e = tid; e < UPD_L * ((k + 3) & ~3); e += nth) {
                    const int p = e % UPD_L, m = e / UPD_L;
                    const bool v = p < L && m < k;
                    sA[m * UPD_SP + p] = v ? A[MIDX(w0 + p, m, N)] : cmk(0, 0);
                    sB[m * UPD_SP + p] = v ? B[MIDX(w0 + p, m, N)] : cmk(0, 0);
                }
                __syncthreads();
                const int nt8 = (N + 7) / 8;
                for (int t = tm.rank * (UPD_NT / 32) + warp; t < 2 * nt8; t += tm.size * (UPD_NT / 32)) {
                    const int side = t >= nt8;
                    upd_extend_tile(W, G, side ? B : A, side ? sA : sB, side ? Tb : Ta, side, N, k, w0, r, 8 * (t - side * nt8));
                }
            } else {
                upd_extend_rows(W, Y, G, A, B, Ta, N, nb, k, w0, r);
            }
            tm.sync();           // the columns are complete; every CTA has read the window's field
            if (tm.rank == 0 && flip) cf[w0 + lane] = nvv;
        } else if (flush) {
            tm.sync();           // every CTA has read the window block of G
        } else {
            __syncthreads();
        }
        k += r;
        s = w0 + wend;
        if (flush) {
            flush_addto(G, A, B, N, k, gsm, tm.rank, tm.size);
            tm.sync();
            k = 0;
        }
    }
    if (tm.rank == 0 && tid == 0) {
        c.stats[ST_PHASE_RE] = ph.x;
        c.stats[ST_PHASE_IM] = ph.y;
        if (forced) {
            c.stats[ST_BLK_LR_RE] = lr_re;
            c.stats[ST_BLK_LR_IM] = lr_im;
        } else {
            c.stats[ST_ACC] += acc;
            c.stats[ST_PROP] += N;
        }
    }
}

// The flush alone, G += A B^T over the model's nublock delayed columns, one
// CTA per chain with the staging of k_update_delay: the delayed-update GEMM's
// own rate (dqmc_gpu_time_op 6).  Modifies G.
__global__ void __launch_bounds__(UPD_NT, 2) k_update_flush(const ChainDev* __restrict__ chains) {
    extern __shared__ double2 dsm[];
    const ChainDev& c = chains[blockIdx.x];
    flush_addto(c.G, c.A, c.B, c.N, c.md->nublock, dsm, 0, 1);
}

// The t-V bond field's updates of one family nf at slice nt, delayed
// (src/dqmc_config_v/dqmc_update_delay.f90:30-112): a team of CTAs per chain, the
// bonds in nnlf_list order.  The accepted rank-2 changes are carried as
// columns of (A, B), G' = G + A B^T: bond b's 2 x 2 block of G' is
// G(P,P) + A(P,:) B(P,:)^T (warp 0, lanes over the delayed columns), the ratio
// det(I + (1 - G')(P,P) Delta) and S = Delta (I + ...)^-1 are thread 0's, and an
// accepted bond appends the columns a_q = sum_p G'(:,P_p) S(p,q) and
// b_q = G'(P_q,:)^T - e_(P_q) (whole CTA).  After nublock columns (rounded down
// to even) and at the family's end the factors are flushed, G += A B^T, on the
// FP64 tensor pipe.  Iflip is 1 for the two-valued field; bond k uses the
// words 2k (iflip) and 2k + 1 (accept test) of the family's draws (0b layout:
// families ascending after the plaquette words; b0: descending after the U
// field's).  The rows of the columns and the flush's tiles are dealt out over the
// chain's team, which meets after each accepted bond and before a flush that a
// rejected one precedes; every CTA takes the decisions for itself.  The flush is two
// thirds of the kernel with one CTA per chain: a family of honeycomb 12 x 12 takes
// 2.39 ms for 16 chains with one CTA each, 1.22 ms on teams.
template <bool TEAM>
__global__ void __launch_bounds__(UPD_NT, 2) k_vbond_delay(const ChainDev* __restrict__ chains, int nt, int nf, int visit,
                                                           int dir) {
    extern __shared__ double2 dsm[];                  // flush staging
    __shared__ double2 s_ap[2][64], s_bp[2][64];      // A(P_q, m), B(P_q, m) of the current bond
    __shared__ double2 s_mat[4];
    __shared__ int s_pc[2], s_acc;
    const Team team = TEAM ? this_team() : Team{0, 1};
    const ChainDev& c = chains[blockIdx.x / team.size];
    const ModelDev& md = *c.md;
    if (!md.lwrapv || !c.vconf) return;
    const int N = c.N, lf = md.nn_lf, nnf = md.nn_nf, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nbv = min(md.nublock, 64) & ~1;         // delayed columns per flush (even)
    double2 *G = c.G, *A = c.A, *B = c.B;
    int32_t* cf = c.vconf + ((size_t)(nt - 1) * nnf + (nf - 1)) * N;
    const int* rows = md.vrows + (size_t)(nf - 1) * 2 * lf;
    const uint32_t* rw = c.rnd + (size_t)visit * md.rps + md.rw_v[dir] + (size_t)(dir ? nnf - nf : nf - 1) * 2 * lf;
    double2 ph = cmk(c.stats[ST_PHASE_RE], c.stats[ST_PHASE_IM]);
    double acc = 0.0, nties = 0.0;
    int k = 0;
    for (int b = 0; b < lf; ++b) {
        // every thread is done with the previous bond's shared values
        __syncthreads();
        const int i1 = rows[2 * b], i2 = rows[2 * b + 1];
        int newval = 0;
        if (warp == 0) {
            // the bond's rows of the delayed factors, and G'(P,P)
            double2 g[4] = {cmk(0, 0), cmk(0, 0), cmk(0, 0), cmk(0, 0)};   // (0,0) (1,0) (0,1) (1,1)
            for (int m = lane; m < k; m += 32) {
                const double2 a0 = A[MIDX(i1, m, N)], a1 = A[MIDX(i2, m, N)];
                const double2 b0 = B[MIDX(i1, m, N)], b1 = B[MIDX(i2, m, N)];
                s_ap[0][m] = a0; s_ap[1][m] = a1; s_bp[0][m] = b0; s_bp[1][m] = b1;
                g[0] = cfma(a0, b0, g[0]); g[1] = cfma(a1, b0, g[1]);
                g[2] = cfma(a0, b1, g[2]); g[3] = cfma(a1, b1, g[3]);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                g[e].x = warp_sum(g[e].x);
                g[e].y = warp_sum(g[e].y);
            }
            if (lane == 0) {
                s_pc[0] = i1; s_pc[1] = i2;
                const double2 g11 = cadd(G[MIDX(i1, i1, N)], g[0]), g21 = cadd(G[MIDX(i2, i1, N)], g[1]);
                const double2 g12 = cadd(G[MIDX(i1, i2, N)], g[2]), g22 = cadd(G[MIDX(i2, i2, N)], g[3]);
                const int is = cf[b];
                const double2 d0 = md.vdp[is - 1], d1 = md.vdm[is - 1];
                const double2 v00 = cadd(cmk(1, 0), cmul(cmk(1.0 - g11.x, -g11.y), d0));
                const double2 v10 = cmul(cmk(-g21.x, -g21.y), d0);
                const double2 v01 = cmul(cmk(-g12.x, -g12.y), d1);
                const double2 v11 = cadd(cmk(1, 0), cmul(cmk(1.0 - g22.x, -g22.y), d1));
                const double2 det = csub(cmul(v00, v11), cmul(v01, v10));
                const double2 id = cdiv(cmk(1, 0), det);
                s_mat[0] = cmul(d0, cmul(v11, id));              // S = Delta vukmat^-1, column-major
                s_mat[1] = cmul(d1, cmul(cmk(-v10.x, -v10.y), id));
                s_mat[2] = cmul(d0, cmul(cmk(-v01.x, -v01.y), id));
                s_mat[3] = cmul(d1, cmul(v00, id));
                const double ra = fabs(cmul(det, ph).x / ph.x), r = u32_to_stream(rw[2 * b + 1]);
                if (fabs(ra - r) < DQ_NEAR_TIE) nties += 1.0;
                s_acc = ra > r;
                if (s_acc) {
                    acc += 1.0;
                    ph = cscale(cmul(ph, det), 1.0 / sqrt(cmulc(det, det).x));
                    newval = is % 2 + 1;
                }
            }
        }
        __syncthreads();
        const bool accepted = s_acc;
        if (accepted) {
            const int p0 = s_pc[0], p1 = s_pc[1];
            const double2 S00 = s_mat[0], S10 = s_mat[1], S01 = s_mat[2], S11 = s_mat[3];
            for (int i = team.rank * blockDim.x + tid; i < N; i += team.size * blockDim.x) {
                double2 c0 = G[MIDX(i, p0, N)], c1 = G[MIDX(i, p1, N)];      // G'(i, P)
                double2 r0 = G[MIDX(p0, i, N)], r1 = G[MIDX(p1, i, N)];      // G'(P, i)
#pragma unroll 4
                for (int m = 0; m < k; ++m) {
                    const double2 ai = A[MIDX(i, m, N)], bi = B[MIDX(i, m, N)];
                    c0 = cfma(ai, s_bp[0][m], c0); c1 = cfma(ai, s_bp[1][m], c1);
                    r0 = cfma(s_ap[0][m], bi, r0); r1 = cfma(s_ap[1][m], bi, r1);
                }
                if (i == p0) r0.x -= 1.0;
                if (i == p1) r1.x -= 1.0;
                A[MIDX(i, k, N)] = cadd(cmul(c0, S00), cmul(c1, S10));
                A[MIDX(i, k + 1, N)] = cadd(cmul(c0, S01), cmul(c1, S11));
                B[MIDX(i, k, N)] = r0;
                B[MIDX(i, k + 1, N)] = r1;
            }
            k += 2;
            team.sync();         // the columns are complete; every CTA has read the bond's value
            if (team.rank == 0 && tid == 0) cf[b] = newval;
        }
        if (k > 0 && (k + 2 > nbv || b == lf - 1)) {
            // the last bond rejected: every CTA has read G(P,P) before one stores to G
            if (TEAM && !accepted) team.sync();
            flush_addto(G, A, B, N, k, dsm, team.rank, team.size);
            if (TEAM) team.sync();      // one CTA: the next bond's barrier
            k = 0;
        }
    }
    if (team.rank == 0 && tid == 0) {
        c.stats[ST_PHASE_RE] = ph.x;
        c.stats[ST_PHASE_IM] = ph.y;
        c.stats[ST_ACCV] += acc;
        c.stats[ST_PROPV] += lf;
        c.stats[ST_NEAR_TIE] += nties;
    }
}

void setup_update() {
    for (const void* k : {(const void*)k_update_delay<false>, (const void*)k_update_delay<true>, (const void*)k_vbond_delay<false>,
                          (const void*)k_vbond_delay<true>}) {
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, TEAM_SMEM_MAX);
        cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    }
    cudaFuncSetAttribute(k_update_flush, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
}

// the delayed bond updates when the flush depth allows two columns, else the
// rank-2 updates straight on G (kern_plqu.cu)
int launch_vbond_delay(const ChainDev* chains, int nchains, int nublock, int team, int nt, int nf, int visit, int dir,
                       cudaStream_t st) {
    if ((min(nublock, 64) & ~1) < 2) return 0;
    const size_t smem = UpdGemm::SMEM_ELEMS * sizeof(double2);
    launch_team(team > 1 ? k_vbond_delay<true> : k_vbond_delay<false>, nchains, team, smem, st, chains, nt, nf, visit, dir);
    return 1;
}

// tiles: the window's columns by upd_extend_tile, else by upd_extend_rows (team 1).  The two differ in
// rounding, so a handle keeps one of them whatever the team of a run is.
void launch_update(const ChainDev* chains, int nchains, int nublock, int team, int tiles, int nt, int visit, cudaStream_t st,
                   int forced, int dir) {
    launch_team(tiles ? k_update_delay<true> : k_update_delay<false>, nchains, team, upd_smem_bytes(nublock, tiles), st, chains,
                nt, visit, forced, dir);
}

void launch_update_flush(const ChainDev* chains, int nchains, cudaStream_t st) {
    size_t smem = UpdGemm::SMEM_ELEMS * sizeof(double2);
    k_update_flush<<<nchains, UPD_NT, smem, st>>>(chains);
}
