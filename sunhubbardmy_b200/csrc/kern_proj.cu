// Projective (ground-state) DQMC: updates, stabilisation and Green's function
// of the projector path: one CTA per walker for the update's walk, a team of CTAs
// (team.cuh) for the QR factorisations.
//
// State per walker: UR = B(tau,0) P (N x ne), UL = P^H B(beta,tau) (ne x N,
// stored transposed as ULT = UL^T, N x ne), ULRINV = (UL UR)^-1 (ne x ne) and
// the stack Ust(0:nst) of N x ne matrices (src/dqmc_proj_core.f90:11-19).
//
// Reference routines:
//  * k_proj_update: dqmc_proj_update_submatrix_LR (src/dqmc_config_v/
//    dqmc_proj_update_submatrix_LR.f90:1-298 for the bond field,
//    src/dqmc_config_u/dqmc_proj_update_submatrix_LR.f90:1-282 for the site
//    field).  Units (bonds of one family, or sites) are visited in order in
//    windows of `wrows` rows (nustock): the window's rows of R = UR ULRINV and
//    of F = R UL are formed by two GEMMs, the accept/reject sequence runs on
//    the F block in shared memory while Gamma^-1 = (I + Delta F_AA)^-1 Delta
//    is built up one accepted unit at a time, and the window is flushed with
//    ULRINV -= (ULRINV UL_A)(Gamma^-1 R_A) and UR_A <- (I + Delta) UR_A.
//    Instead of re-evaluating F_rr - F_rA Gamma^-1 F_Ar for each unit, the
//    walk keeps the Schur complement of F as a sum of products (pwin_walk),
//    which gives the same numbers in exact arithmetic.
//  * k_proj_qr: s_zgeQR_pqmc (lib/s_matrix.f90:1822-1996) as used by
//    dqmc_proj_stablize_0b_qr / _b0_qr: Q of a tall N x ne matrix with an
//    even number of negative R diagonal entries (else column 1 is negated)
//    and log |det R|.  The wide UL is factored through its transpose, which
//    is the stored layout.
//  * k_proj_ulr: ULR = UL UR and its inverse (s_invlu_z /
//    s_inv_logdet_lu_z); the inverse is taken through a Householder QR, and
//    log det ULR = log det Q + sum log R_ii.
//  * k_proj_t1 + k_proj_gmat: green_equaltime (src/dqmc_proj_core/
//    green_equaltime.f90): G = I - (UR ULRINV) UL, several CTAs per walker.
#include "chain_access.cuh"
#include "kernels.h"
#include "linalg.cuh"

#define PW_MAXR 32          // largest update window (rows)
#define PW_LD (PW_MAXR + 1)
#define PW_LS (PW_MAXR + 2)   // pitch of what the DMMA fragments read: 2 (mod 8)

struct ProjSmem {
    LinalgSmem L;
    double red[64];
};

DQ_DEV LinalgScratch proj_scratch(const ChainDev& c) {
    LinalgScratch s;
    s.Vs = c.W[5];
    s.Ws = c.smallw;
    s.Ws2 = c.smallw + (size_t)QR_NB2 * c.N;
    s.T = c.T;
    s.tau = c.tau;
    s.T64 = c.T64;
    return s;
}

static size_t proj_la_smem(int maxN) {
    size_t a = QR_PANEL_ELEMS(maxN);
    size_t b = GemmBig::SMEM_ELEMS;
    if ((size_t)GemmWide::SMEM_ELEMS > b) b = GemmWide::SMEM_ELEMS;
    return (a > b ? a : b) * sizeof(double2) + sizeof(ProjSmem) + 64;
}

// ---------------------------------------------------------------------------
// s_zgeQR_pqmc on the N x ne matrix mat_id, in place (X <- Q); the log of
// |det R| goes to logwDV[dst] = logwDV[add] + log|det R| (add < 0: nothing added;
// dst < 0: not recorded).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_proj_qr(const ChainDev* __restrict__ chains, int mat_id, int dst, int add) {
    extern __shared__ double2 ssm[];
    const Team tm = this_team();
    const ChainDev c = chains[blockIdx.x / tm.size];
    const ModelDev& md = *c.md;
    const int N = c.N, ne = md.ne, tid = threadIdx.x, nth = blockDim.x;
    double2* buf = ssm;
    ProjSmem* S = (ProjSmem*)(ssm + ((QR_PANEL_ELEMS(N) > (size_t)GemmBig::SMEM_ELEMS) ? QR_PANEL_ELEMS(N) : (size_t)GemmBig::SMEM_ELEMS));
    LinalgScratch sc = proj_scratch(c);
    double2* X = chain_mat(c, mat_id);
    double2* A = c.W[1];
    for (int e = tm.rank * nth + tid; e < N * ne; e += tm.size * nth) A[e] = X[e];
    tm.sync();
    cta_qr64(A, N, sc, buf, buf, &S->L, tm, ne);
    cta_form_q64(N, X, sc, buf, tm, ne);
    tm.sync();
    if (tm.rank) return;
    double lg = 0.0, neg = 0.0;
    for (int i = tid; i < ne; i += nth) {
        double r = A[MIDX(i, i, N)].x;
        lg += log(fabs(r));
        neg += (r < 0.0) ? 1.0 : 0.0;
    }
    lg = block_sum(lg, S->red);
    neg = block_sum(neg, S->red);
    if (((long long)llround(neg)) & 1)
        for (int i = tid; i < N; i += nth) X[i] = cmk(-X[i].x, -X[i].y);
    if (tid == 0 && dst >= 0) c.logwDV[dst] = (add >= 0 ? c.logwDV[add] : 0.0) + lg;
}

// ---------------------------------------------------------------------------
// out = (ULT^T UR)^-1; with logdet, stats[LOGDETM] = logwDV[ia] (+ logwDV[ib]) +
// log det(UL UR), the logweightf of the sweep routines.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_proj_ulr(const ChainDev* __restrict__ chains, int out_id, int logdet, int ia, int ib) {
    extern __shared__ double2 ssm[];
    const Team tm = this_team();
    const ChainDev c = chains[blockIdx.x / tm.size];
    const ModelDev& md = *c.md;
    const int N = c.N, ne = md.ne, tid = threadIdx.x, nth = blockDim.x;
    double2* buf = ssm;
    ProjSmem* S = (ProjSmem*)(ssm + ((QR_PANEL_ELEMS(N) > (size_t)GemmBig::SMEM_ELEMS) ? QR_PANEL_ELEMS(N) : (size_t)GemmBig::SMEM_ELEMS));
    LinalgScratch sc = proj_scratch(c);
    double2* M = c.W[2];
    ZGemmArgs g;
    g.M = ne; g.N = ne; g.K = N; g.alpha = cmk(1, 0); g.beta = cmk(0, 0);
    g.A = c.ULT; g.lda = N; g.opA = OP_T; g.B = c.UR; g.ldb = N; g.opB = OP_N; g.C = M; g.ldc = ne;
    team_zgemm(g, tm, buf);
    tm.sync();
    cta_qr64(M, ne, sc, buf, buf, &S->L, tm);
    double2 ld = cmk(0, 0);
    int bad = 0;
    if (tm.rank == 0) {
        for (int i = tid; i < ne; i += nth) {
            const double r = M[MIDX(i, i, ne)].x;
            bad |= (r == 0.0 || !isfinite(r));
        }
        // a zero or non-finite pivot of UL UR: zgetrf's info > 0 in s_inv_logdet_lu_z
        bad = __syncthreads_or(bad);
        if (bad && tid == 0) chain_raise(c, DQ_FAIL_SINGULAR);
    }
    if (logdet && tm.rank == 0) {
        ld = cta_logdet_q(sc.tau, ne, S->red);
        double2 lr = cmk(0, 0);
        for (int i = tid; i < ne; i += nth) {
            double r = M[MIDX(i, i, ne)].x;
            lr = cadd(lr, cmk(log(fabs(r)), r < 0.0 ? M_PI : 0.0));
        }
        lr = block_csum(lr, S->red);
        ld = cadd(ld, lr);
    }
    double2* X = chain_mat(c, out_id);
    const int w = tm.chunk(ne);
    for (int c0 = tm.rank * w; c0 < ne; c0 += tm.size * w) {
        const int nc = min(w, ne - c0);
        for (int e = tid; e < ne * nc; e += nth) X[e + c0 * ne] = cmk((e % ne) == c0 + e / ne ? 1.0 : 0.0, 0.0);
        __syncthreads();
        cta_apply_qh64(ne, X, c0, nc, sc, buf);
        cta_trsm_upper64(M, ne, X, c0, nc, buf, &S->L);
    }
    if (logdet && tm.rank == 0 && tid == 0) {
        double w = c.logwDV[ia] + (ib >= 0 ? c.logwDV[ib] : 0.0);
        c.stats[ST_LOGDETM_RE] = ld.x + w;
        c.stats[ST_LOGDETM_IM] = ld.y;
        c.stats[ST_GINFO] = (bad || !isfinite(ld.x + w) || !isfinite(ld.y)) ? (double)DQ_FAIL_SINGULAR : 0.0;
    }
}

// T1 = UR * INV (N x ne), tiles shared by gridDim.x CTAs per walker
__global__ void __launch_bounds__(256) k_proj_t1(const ChainDev* __restrict__ chains, int inv_id) {
    extern __shared__ double2 ssm[];
    const ChainDev c = chains[blockIdx.y];
    const int N = c.N, ne = c.md->ne;
    ZGemmArgs g;
    g.M = N; g.N = ne; g.K = ne; g.alpha = cmk(1, 0); g.beta = cmk(0, 0);
    g.A = c.UR; g.lda = N; g.opA = OP_N; g.B = chain_mat(c, inv_id); g.ldb = ne; g.opB = OP_N;
    g.C = c.W[0]; g.ldc = N;
    zgemm_cta<GemmBig>(g, blockIdx.x, gridDim.x, ssm);
}

// dst = I - T1 * ULT^T (N x N)
__global__ void __launch_bounds__(256) k_proj_gmat(const ChainDev* __restrict__ chains, int dst_id) {
    extern __shared__ double2 ssm[];
    const ChainDev c = chains[blockIdx.y];
    const int N = c.N, ne = c.md->ne;
    double2* D = chain_mat(c, dst_id);
    ZGemmArgs g;
    g.M = N; g.N = N; g.K = ne; g.alpha = cmk(-1, 0); g.beta = cmk(0, 0);
    g.A = c.W[0]; g.lda = N; g.opA = OP_N; g.B = c.ULT; g.ldb = N; g.opB = OP_T;
    g.C = D; g.ldc = N;
    zgemm_cta<GemmBig>(g, blockIdx.x, gridDim.x, ssm);
    // the diagonal of the tiles this CTA wrote
    const int tm = (N + GemmBig::BM - 1) / GemmBig::BM, tn = (N + GemmBig::BN - 1) / GemmBig::BN;
    for (int t = blockIdx.x; t < tm * tn; t += gridDim.x) {
        int m0 = (t % tm) * GemmBig::BM, n0 = (t / tm) * GemmBig::BN;
        int lo = max(m0, n0), hi = min(min(m0 + GemmBig::BM, n0 + GemmBig::BN), N);
        for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) D[MIDX(i, i, N)].x += 1.0;
    }
}

// copy of an N x ne matrix (conj = 1: complex conjugate)
__global__ void k_tall_copy(const ChainDev* __restrict__ chains, int dst_id, int src_id) {
    const ChainDev c = chains[blockIdx.y];
    const size_t n = (size_t)c.N * c.md->ne;
    double2* d = chain_mat(c, dst_id);
    const double2* s = chain_mat(c, src_id);
    for (size_t e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) d[e] = s[e];
}

// ---------------------------------------------------------------------------
// projective local update (submatrix-LR), see the file header.  One window of
// one bond family (or of the sites) is three launches:
//   k_pwin_rg    (several CTAs per walker)  Rg = UR(rows,:) ULRINV  [nr x ne]
//                                           Ut = ULRINV UL(:,rows)  [ne x nr]
//   k_pwin_seq   (one CTA per walker)       F = Rg UL(:,rows), the accept /
//                reject sequence with Gamma bordering, Vt = Gamma Rg,
//                UR(A,:) *= 1 + Delta
//   k_pwin_flush (several CTAs per walker)  ULRINV -= Ut Vt
// so the window GEMMs use all SMs while the sequential part runs one CTA per
// walker.  Scratch per walker in pw: Rg, Ut and Vt (32 x ne each); F and Gamma stay in shared memory.
// ---------------------------------------------------------------------------
struct PUpdSmem {
    double2 F[PW_MAXR * PW_LD];     // F(x, y) of the window at x + y * PW_LD (window-start values)
    // vectors of the accepted rows m, element of window row x at m * PW_LS + x (see pwin_walk)
    double2 aP[PW_MAXR * PW_LS], bP[PW_MAXR * PW_LS], al[PW_MAXR * PW_LS], be[PW_MAXR * PW_LS];
    double2 Gm[PW_MAXR * PW_LS];    // Gamma(x, y) at x + y * PW_LS (zero off the accepted rows)
    double2 dl[PW_MAXR];            // Delta of the accepted rows, else 0
    int rows[PW_MAXR];
    int nacc;                       // accepted rows
};

DQ_DEV double u32_stream(uint32_t u) { return ((double)u + 0.5) * (1.0 / 4294967296.0); }

// window geometry of one walker: returns false when window w is past the end
struct PWin {
    int bond, b, nunits, R, upw, u0, nu, nr;
    const int* rows;     // global row list of the window (bond field), nullptr for sites
};
DQ_DEV bool pwin(const ChainDev& c, int nf, int w, PWin& p) {
    const ModelDev& md = *c.md;
    p.bond = nf > 0;
    p.b = p.bond ? 2 : 1;
    p.nunits = p.bond ? md.nn_lf : c.N;
    int R = min(md.nublock, PW_MAXR);
    R -= R % p.b;
    if (R < p.b) R = p.b;
    p.R = R;
    p.upw = R / p.b;
    p.u0 = w * p.upw;
    if (p.u0 >= p.nunits) return false;
    p.nu = min(p.upw, p.nunits - p.u0);
    p.nr = p.nu * p.b;
    p.rows = p.bond ? md.vrows + (size_t)(nf - 1) * 2 * md.nn_lf + 2 * p.u0 : nullptr;
    return true;
}

DQ_DEV void pw_ptrs(const ChainDev& c, int R, double2*& Rg, double2*& Ut, double2*& Vt) {
    const int ne = c.md->ne;
    Rg = c.pw;
    Ut = Rg + (size_t)R * ne;
    Vt = Ut + (size_t)ne * R;
}

// Rg = UR(rows,:) ULRINV and Ut = ULRINV UL(:,rows) = ULRINV ULT(rows,:)^T
__global__ void __launch_bounds__(256) k_pwin_rg(const ChainDev* __restrict__ chains, int nf, int w) {
    extern __shared__ double2 ssm[];
    const ChainDev& c = chains[blockIdx.y];
    PWin p;
    if (!pwin(c, nf, w, p)) return;
    const int N = c.N, ne = c.md->ne;
    double2 *Rg, *Ut, *Vt;
    pw_ptrs(c, p.R, Rg, Ut, Vt);
    ZGemmArgs ga;   // Rg
    ga.M = p.nr; ga.N = ne; ga.K = ne; ga.alpha = cmk(1, 0); ga.beta = cmk(0, 0);
    ga.A = p.rows ? c.UR : c.UR + p.u0; ga.lda = N; ga.opA = OP_N; ga.arow = p.rows;
    ga.B = c.ULRINV; ga.ldb = ne; ga.opB = OP_N; ga.C = Rg; ga.ldc = p.nr;
    ZGemmArgs gb;   // Ut
    gb.M = ne; gb.N = p.nr; gb.K = ne; gb.alpha = cmk(1, 0); gb.beta = cmk(0, 0);
    gb.A = c.ULRINV; gb.lda = ne; gb.opA = OP_N;
    gb.B = p.rows ? c.ULT : c.ULT + p.u0; gb.ldb = N; gb.opB = OP_T; gb.brow = p.rows;
    gb.C = Ut; gb.ldc = ne;
    const int ca = zt_pick(ga.M, ga.N), cb = zt_pick(gb.M, gb.N);
    const int ta = zt_tiles(ca, ga.M, ga.N), tb = zt_tiles(cb, gb.M, gb.N);
    for (int t = blockIdx.x; t < ta + tb; t += gridDim.x) {
        if (t < ta) zgemm_tile(ga, ca, t, ssm);
        else zgemm_tile(gb, cb, t - ta, ssm);
    }
}

// ULRINV -= Ut Vt (skipped when the window accepted nothing)
__global__ void __launch_bounds__(256) k_pwin_flush(const ChainDev* __restrict__ chains, int nf, int w) {
    extern __shared__ double2 ssm[];
    const ChainDev& c = chains[blockIdx.y];
    PWin p;
    if (!pwin(c, nf, w, p)) return;
    if (c.pw_flag[0] == 0) return;
    const int ne = c.md->ne;
    double2 *Rg, *Ut, *Vt;
    pw_ptrs(c, p.R, Rg, Ut, Vt);
    ZGemmArgs g;
    g.M = ne; g.N = ne; g.K = p.nr; g.alpha = cmk(-1, 0); g.beta = cmk(1, 0);
    g.A = Ut; g.lda = ne; g.opA = OP_N; g.B = Vt; g.ldb = p.nr; g.opB = OP_N; g.C = c.ULRINV; g.ldc = ne;
    const int cl = zt_pick(g.M, g.N), nt = zt_tiles(cl, g.M, g.N);
    for (int t = blockIdx.x; t < nt; t += gridDim.x) zgemm_tile(g, cl, t, ssm);
}

// The accept / reject walk of a window, by one warp: lane x holds row x of the
// window and the b x b diagonal block of its unit in
//   P = F - F Gamma F = F - sum_m a_m b_m,
// so every remaining unit is tested at once and the first that passes (a ballot)
// is accepted, as the sequential visit does.  An accepted unit with rows r and
// g = (I + Delta P_rr)^-1 Delta appends, per row,
//   a = P(:, r) g, b = P(r, :),  al = (e_r - Gamma F(:, r)) g, be = e_r - F(r, :) Gamma,
// all four by the same recursion over the m accepted rows (coefficients b_m(r) and
// a_m(r)), and Gamma = sum_m al_m be_m.  No block barrier inside the walk: with two of
// them a unit and one thread's divisions a family of 64 walkers (288 sites, ne = 144, nine
// windows of 32 rows, updates included) took 1.54 ms, and 1.31 ms this way.
template <int B>
DQ_DEV void pwin_walk(PUpdSmem* S, const ChainDev& c, const ModelDev& md, const uint32_t* rnd, int32_t* cf, int u0, int nu) {
    const int lane = threadIdx.x & 31, k = lane / B, x = lane, lc = B == 2 ? 2 : md.lcomp;
    const bool live = k < nu, lead = live && lane % B == 0;
    double2 ph = cmk(c.stats[ST_PHASE_RE], c.stats[ST_PHASE_IM]);
    double2 d1 = cmk(0, 0), d2 = cmk(0, 0), phr = cmk(1, 0), p0 = cmk(0, 0), p1 = cmk(0, 0);
    double thr = 0.0, gam = 1.0;
    int isp = 0;
    bool cand = live;
    if (live) {
        const int u = u0 + k, is = cf[u];
        const int iflip = (int)ceil(u32_stream(rnd[2 * u]) * (lc - 1));
        isp = (is + iflip - 1) % lc + 1;
        thr = u32_stream(rnd[2 * u + 1]);
        if (B == 2) {
            d1 = md.vdp[is - 1];
            d2 = md.vdm[is - 1];
            p1 = S->F[x + (x ^ 1) * PW_LD];
        } else {
            const int kk = (is - 1) * (lc - 1) + (iflip - 1);
            d1 = md.delta[kk];
            gam = md.gam_ratio[kk];
            phr = md.phase_ratio[kk];
        }
        p0 = S->F[x + x * PW_LD];
    }
    S->dl[lane] = cmk(0, 0);
    double accm = 0.0;
    int pc = 0, nm = 0, nties = 0;
    while (pc < nu) {
        // the unit's ratio and g, in every lane of the unit
        double2 det, g11, g12 = cmk(0, 0), g21 = cmk(0, 0), g22 = cmk(0, 0);
        if (B == 2) {
            const double2 o0 = cmk(__shfl_xor_sync(0xffffffffu, p0.x, 1), __shfl_xor_sync(0xffffffffu, p0.y, 1));
            const double2 o1 = cmk(__shfl_xor_sync(0xffffffffu, p1.x, 1), __shfl_xor_sync(0xffffffffu, p1.y, 1));
            const bool first = (lane & 1) == 0;
            const double2 prr = first ? p0 : o0, pr1 = first ? p1 : o1, p1r = first ? o1 : p1, p11 = first ? o0 : p0;
            const double2 v11 = cadd(cmk(1, 0), cmul(prr, d1)), v21 = cmul(p1r, d1);
            const double2 v12 = cmul(pr1, d2), v22 = cadd(cmk(1, 0), cmul(p11, d2));
            det = csub(cmul(v11, v22), cmul(v12, v21));
            const double2 id = cdiv(cmk(1, 0), det);
            g11 = cmul(cmul(v22, d1), id);
            g12 = cmul(cmul(cmk(-v12.x, -v12.y), d1), id);
            g21 = cmul(cmul(cmk(-v21.x, -v21.y), d2), id);
            g22 = cmul(cmul(v11, d2), id);
        } else {
            const double2 ratio1 = cadd(cmk(1, 0), cmul(p0, d1));
            double2 r = ratio1;
            for (int f = 1; f < md.nflr; ++f) r = cmul(r, ratio1);
            det = cmul(cscale(r, gam), phr);
            g11 = cdiv(d1, ratio1);
        }
        const double num = fabs(cmul(det, ph).x), ax = fabs(ph.x), lim = thr * ax;
        const bool open = cand && k >= pc;
        const bool pass = open && num > lim;
        const unsigned bal = __ballot_sync(0xffffffffu, pass);
        const int kf = bal ? (__ffs(bal) - 1) / B : nu;
        nties += lead && open && k <= kf && fabs(num - lim) < DQ_NEAR_TIE * ax;
        if (!bal) break;
        const int r = kf * B;
        auto from = [&](double2 v) { return cmk(__shfl_sync(0xffffffffu, v.x, r), __shfl_sync(0xffffffffu, v.y, r)); };
        det = from(det);
        g11 = from(g11);
        if (B == 2) { g12 = from(g12); g21 = from(g21); g22 = from(g22); }
        ph = cmul(ph, det);
        ph = cscale(ph, 1.0 / sqrt(cabs2(ph)));
        accm += 1.0;
        if (k == kf) {
            cand = false;
            S->dl[lane] = lane % B == 0 ? d1 : d2;
            if (lane % B == 0) cf[u0 + k] = isp;
        }
        // P(x, r + q), P(r + q, x), (e - Gamma F)(x, r + q), (e - F Gamma)(r + q, x)
        double2 cc[B], rr[B], aa[B], bb[B];
#pragma unroll
        for (int q = 0; q < B; ++q) {
            cc[q] = S->F[x + (r + q) * PW_LD];
            rr[q] = S->F[r + q + x * PW_LD];
            aa[q] = bb[q] = cmk(x == r + q ? 1.0 : 0.0, 0.0);
        }
#pragma unroll 2
        for (int m = 0; m < nm; ++m) {
            const double2 am = S->aP[m * PW_LS + x], bm = S->bP[m * PW_LS + x], lm = S->al[m * PW_LS + x], em = S->be[m * PW_LS + x];
#pragma unroll
            for (int q = 0; q < B; ++q) {
                const double2 fb = S->bP[m * PW_LS + r + q], fa = S->aP[m * PW_LS + r + q];
                const double2 nb = cmk(-fb.x, -fb.y), na = cmk(-fa.x, -fa.y);
                cc[q] = cfma(am, nb, cc[q]);
                aa[q] = cfma(lm, nb, aa[q]);
                rr[q] = cfma(na, bm, rr[q]);
                bb[q] = cfma(na, em, bb[q]);
            }
        }
        __syncwarp();
        double2 an[B], ln[B];
        if (B == 2) {
            an[0] = cfma(cc[0], g11, cmul(cc[B - 1], g21)); an[B - 1] = cfma(cc[0], g12, cmul(cc[B - 1], g22));
            ln[0] = cfma(aa[0], g11, cmul(aa[B - 1], g21)); ln[B - 1] = cfma(aa[0], g12, cmul(aa[B - 1], g22));
        } else {
            an[0] = cmul(cc[0], g11);
            ln[0] = cmul(aa[0], g11);
        }
#pragma unroll
        for (int q = 0; q < B; ++q) {
            S->aP[(nm + q) * PW_LS + x] = an[q];
            S->bP[(nm + q) * PW_LS + x] = rr[q];
            S->al[(nm + q) * PW_LS + x] = ln[q];
            S->be[(nm + q) * PW_LS + x] = bb[q];
            p0 = cfma(cmk(-an[q].x, -an[q].y), rr[q], p0);
            if (B == 2) {
                const double2 o = cmk(__shfl_xor_sync(0xffffffffu, rr[q].x, 1), __shfl_xor_sync(0xffffffffu, rr[q].y, 1));
                p1 = cfma(cmk(-an[q].x, -an[q].y), o, p1);
            }
        }
        nm += B;
        pc = kf + 1;
        __syncwarp();
    }
    // the steps of four accepted rows that Gamma's product takes
    for (int m = nm; m < ((nm + 3) & ~3); ++m) S->al[m * PW_LS + x] = S->be[m * PW_LS + x] = cmk(0, 0);
    nties = warp_sum(nties);
    if (lane == 0) {
        S->nacc = nm;
        c.pw_flag[0] = nm > 0;
        c.stats[ST_PHASE_RE] = ph.x;
        c.stats[ST_PHASE_IM] = ph.y;
        c.stats[B == 2 ? ST_ACCV : ST_ACC] += accm;
        c.stats[ST_NEAR_TIE] += (double)nties;
        c.stats[B == 2 ? ST_PROPV : ST_PROP] += (double)nu;
    }
}

// visit: slices already updated in this half sweep; dir 0 = 0b (bond families
// 1..nn_nf, then sites), 1 = b0 (sites, then families nn_nf..1) fixes where
// this call's draws sit in the half sweep's random words; rnd_off >= 0
// overrides that offset.  The products around the walk are too small for the
// general GEMM's tiles (32 x 32 and 32 x ne): their k range (F) or columns (Vt)
// are split over the eight warps, with fragments read from global memory.
__global__ void __launch_bounds__(256) k_pwin_seq(const ChainDev* __restrict__ chains, int nt, int nf, int w, int visit,
                                                  int dir, int rnd_off) {
    extern __shared__ double2 ssm[];
    const ChainDev& c = chains[blockIdx.x];
    const ModelDev& md = *c.md;
    const int N = c.N, ne = md.ne, tid = threadIdx.x, nth = blockDim.x;
    PWin p;
    if (!pwin(c, nf, w, p)) {
        if (tid == 0) c.pw_flag[0] = 0;
        return;
    }
    PUpdSmem* S = (PUpdSmem*)ssm;
    const int bond = p.bond, nr = p.nr, u0 = p.u0;
    const int lane = tid & 31, warp = tid >> 5, q4 = lane & 3, l4 = lane >> 2;
    if (rnd_off < 0) {
        const int vw = md.lwrapv ? 2 * md.nn_lf * md.nn_nf : 0, uw = md.lwrapu ? 2 * N : 0;
        int within;
        if (dir == 0) within = md.rw_pre0 + (bond ? (nf - 1) * 2 * md.nn_lf : vw);
        else within = bond ? uw + (md.nn_nf - nf) * 2 * md.nn_lf : 0;
        rnd_off = visit * md.rps + within;
    }
    const uint32_t* rnd = c.rnd + rnd_off;
    int32_t* cf = bond ? c.vconf + ((size_t)(nt - 1) * md.nn_nf + (nf - 1)) * N : c.conf + (size_t)(nt - 1) * N;
    double2 *Rg, *Ut, *Vt;
    pw_ptrs(c, p.R, Rg, Ut, Vt);
    for (int x = tid; x < nr; x += nth) S->rows[x] = p.rows ? p.rows[x] : u0 + x;
    __syncthreads();
    {   // F = Rg UL(:,rows) = Rg ULT(rows,:)^T: warp w the columns 16 (w & 1).. and every fourth k step
        double cr[4][2][2], ci[4][2][2];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) { cr[i][j][0] = cr[i][j][1] = ci[i][j][0] = ci[i][j][1] = 0.0; }
        int ry[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int y = 16 * (warp & 1) + 8 * j + l4;
            ry[j] = y < nr ? S->rows[y] : -1;
        }
#pragma unroll 2
        for (int s = warp >> 1; 4 * s < ne; s += 4) {
            const int l = 4 * s + q4;
            double2 va[4], vb[2];
#pragma unroll
            for (int i = 0; i < 4; ++i) va[i] = (l < ne && 8 * i + l4 < nr) ? Rg[8 * i + l4 + (size_t)l * nr] : cmk(0, 0);
#pragma unroll
            for (int j = 0; j < 2; ++j) vb[j] = (l < ne && ry[j] >= 0) ? c.ULT[MIDX(ry[j], l, N)] : cmk(0, 0);
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j) zdmma(cr[i][j], ci[i][j], va[i], vb[j]);
        }
        // partial products over the walk's vectors: warp w at w * 512, element x + 32 (y mod 16)
        double2* part = S->aP;
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    part[warp * 512 + 8 * i + l4 + 32 * (8 * j + 2 * q4 + h)] = cmk(cr[i][j][h], ci[i][j][h]);
        __syncthreads();
        for (int e = tid; e < PW_MAXR * PW_MAXR; e += nth) {
            const int x = e & 31, y = e >> 5, o = x + 32 * (y & 15), h = y >> 4;
            double2 v = part[h * 512 + o];
#pragma unroll
            for (int q = 1; q < 4; ++q) v = cadd(v, part[(h + 2 * q) * 512 + o]);
            S->F[x + y * PW_LD] = v;
        }
    }
    __syncthreads();
    if (warp == 0) {
        if (bond) pwin_walk<2>(S, c, md, rnd, cf, u0, p.nu);
        else pwin_walk<1>(S, c, md, rnd, cf, u0, p.nu);
    }
    __syncthreads();
    const int nm = S->nacc;
    if (nm == 0) return;
    {   // Gamma = al be, tiles w and w + 8
        const int x = 8 * (warp & 3) + l4, y0 = 8 * (warp >> 2);
        double cr[2][2] = {{0, 0}, {0, 0}}, ci[2][2] = {{0, 0}, {0, 0}};
        for (int m = q4; m < ((nm + 3) & ~3); m += 4) {
            const double2 a = S->al[m * PW_LS + x];
#pragma unroll
            for (int t = 0; t < 2; ++t) zdmma(cr[t], ci[t], a, S->be[m * PW_LS + y0 + 16 * t + l4]);
        }
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
            for (int h = 0; h < 2; ++h) S->Gm[x + (y0 + 16 * t + 2 * q4 + h) * PW_LS] = cmk(cr[t][h], ci[t][h]);
    }
    __syncthreads();
    // Vt = Gamma Rg, 8 columns of Rg per warp and step
    for (int l0 = 8 * warp; l0 < ne; l0 += 64) {
        double cr[4][2], ci[4][2];
#pragma unroll
        for (int i = 0; i < 4; ++i) { cr[i][0] = cr[i][1] = ci[i][0] = ci[i][1] = 0.0; }
        double2 vb[8];
#pragma unroll
        for (int s = 0; s < 8; ++s)
            vb[s] = (l0 + l4 < ne && 4 * s + q4 < nr) ? Rg[4 * s + q4 + (size_t)(l0 + l4) * nr] : cmk(0, 0);
#pragma unroll
        for (int s = 0; s < 8; ++s)
#pragma unroll
            for (int i = 0; i < 4; ++i) zdmma(cr[i], ci[i], S->Gm[8 * i + l4 + (4 * s + q4) * PW_LS], vb[s]);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int x = 8 * i + l4, l = l0 + 2 * q4 + h;
                if (x < nr && l < ne) Vt[x + (size_t)l * nr] = cmk(cr[i][h], ci[i][h]);
            }
    }
    for (int e = tid; e < nr * ne; e += nth) {
        const int x = e % nr, l = e / nr;
        const double2 d = S->dl[x];
        if (d.x != 0.0 || d.y != 0.0) {
            double2* q = c.UR + MIDX(S->rows[x], l, N);
            const double2 v = *q;
            *q = cadd(v, cmul(d, v));
        }
    }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
static constexpr size_t PUPD_SMEM = sizeof(PUpdSmem);
static_assert(offsetof(PUpdSmem, dl) - offsetof(PUpdSmem, aP) >= 8 * 512 * sizeof(double2), "partial products of F");

void setup_proj() {
    for (const void* k : {(const void*)k_proj_qr, (const void*)k_proj_ulr}) {
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, TEAM_SMEM_MAX);
        cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    }
    cudaFuncSetAttribute(k_pwin_seq, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PUPD_SMEM);
    cudaFuncSetAttribute(k_pwin_rg, cudaFuncAttributeMaxDynamicSharedMemorySize, ZT_SMEM_ELEMS * (int)sizeof(double2));
    cudaFuncSetAttribute(k_pwin_flush, cudaFuncAttributeMaxDynamicSharedMemorySize, ZT_SMEM_ELEMS * (int)sizeof(double2));
    cudaFuncSetAttribute(k_proj_t1, cudaFuncAttributeMaxDynamicSharedMemorySize, GemmBig::SMEM_ELEMS * (int)sizeof(double2));
    cudaFuncSetAttribute(k_proj_gmat, cudaFuncAttributeMaxDynamicSharedMemorySize, GemmBig::SMEM_ELEMS * (int)sizeof(double2));
}

void launch_proj_qr(const ChainDev* chains, int nchains, int maxN, int team, int mat_id, int dst, int add, cudaStream_t st) {
    launch_team(k_proj_qr, nchains, team, proj_la_smem(maxN), st, chains, mat_id, dst, add);
}

void launch_proj_ulr(const ChainDev* chains, int nchains, int maxN, int team, int out_id, int logdet, int ia, int ib, cudaStream_t st) {
    launch_team(k_proj_ulr, nchains, team, proj_la_smem(maxN), st, chains, out_id, logdet, ia, ib);
}

void launch_proj_green(const ChainDev* chains, int nchains, int inv_id, int dst_id, int ctas, cudaStream_t st) {
    size_t sm = (size_t)GemmBig::SMEM_ELEMS * sizeof(double2);
    k_proj_t1<<<dim3(ctas, nchains), 256, sm, st>>>(chains, inv_id);
    k_proj_gmat<<<dim3(ctas, nchains), 256, sm, st>>>(chains, dst_id);
}

void launch_tall_copy(const ChainDev* chains, int nchains, int dst_id, int src_id, cudaStream_t st) {
    k_tall_copy<<<dim3(8, nchains), 256, 0, st>>>(chains, dst_id, src_id);
}

// one family (nf >= 1) or the site field (nf = 0) of slice nt: nwin windows,
// g_rg / g_fl CTAs per walker for the window GEMMs
void launch_proj_update(const ChainDev* chains, int nchains, int nt, int nf, int visit, int dir, int rnd_off,
                        int nwin, int g_rg, int g_fl, cudaStream_t st) {
    size_t sm = (size_t)ZT_SMEM_ELEMS * sizeof(double2);
    for (int w = 0; w < nwin; ++w) {
        k_pwin_rg<<<dim3(g_rg, nchains), 256, sm, st>>>(chains, nf, w);
        k_pwin_seq<<<nchains, 256, PUPD_SMEM, st>>>(chains, nt, nf, w, visit, dir, rnd_off);
        k_pwin_flush<<<dim3(g_fl, nchains), 256, sm, st>>>(chains, nf, w);
    }
}
