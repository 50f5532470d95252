// Persistent DLR energy-step kernel: fixed-rank integrator
// (SolverCSD.jl SolveFirstCollisionSourceDLR, :891-1120).
//
// Each energy step is a fixed sequence of phases separated by team barriers:
//   A  boundary inflow (PsiBeam, :977-988) + dose half-steps (:990-997, :1104-1111)
//   B  uncollided upwind sweep (:1000-1005, solveFluxUpwind! :388-463)
//      + streaming Grams X^T L_d X, W^T A_d W (:1022-1025, :1035-1038)
//   C  K = XS - dE sum L_d K C_d, L = WS^T - dE sum A_d L G_d^T (:1027, :1040)
//   D,E,F  rank-revealing orthonormal bases of K and L (svd!(K).U, :1029/:1042)
//   G  S-step Grams with the new bases (:1053-1063)
//   H..K out-scattering (:1066-1074)
//   L..O in-scattering K/L/S (:1076-1102)
// The range finder: Jacobi eig of A^T A -> V; Gram of A V -> Jacobi -> V2, nu;
// C = A V V2_J / nu_J materialised; CholQR on C. Directions with
// nu_j <= tol nu_0 are null; rank-deficient bases are completed with the
// candidate canonical vectors in index order (boundary cells for X, moments for W).
// What bounds a step is latency: its products would take 10 us of the FP64 pipes
// (100 x 100 cells, P_21, r = 20), but it is a chain of some 30 team barriers
// (2 us each, 55 us), reductions through L2 (35 us), six pairs of Cholesky
// factorisations (49 us) and, between them, short passes over a CTA's rows
// (150 us; 290 us in all, 1060 before). So a row pass is one tile of up to TR rows
// whose loads are one 16-byte load per thread, its products and Grams are 8 x 8
// blocks on the FP64 tensor pipe, one per warp, and 512 threads fill those
// blocks (256 threads with one product chain per thread took 1060 us).
#pragma once
#include "dlr_device.cuh"

namespace titus {

constexpr int NSLOT = 24;

struct SmemLayout {
    double slot[NSLOT][KK];
    double ja[KK], jv[KK];
    double lamK[KM], lamL[KM];
    double acc[PMAX];
    double tA[TR * KM];
    double tL[4][TR * KM];
    double tO[TR * KM];
    double tP[TR * QM];
    double vec[4 * KM + QM];
    double wnrm[KM];
    int wcand[KM];
    int misc[8];
};

// slot indices
enum {
    SL_S = 0, SL_G0 = 1, SL_C0 = 5, SL_P0 = 9,
    SL_VK = 13, SL_VL = 14, SL_TK = 15, SL_TL = 16, SL_RK = 17, SL_RL = 18,
    SL_RIK = 19, SL_RIL = 20, SL_M = 21, SL_N = 22, SL_WC = 23
};

struct Ctx {
    DevProblem P;
    TeamState st;
    SmemLayout* sm;
    int G, b;
    int c0, c1, m0, m1;  // own cells / moments
    int k;               // current basis width (rank)
    double* psi_in;
    double* psi_out;
    double* CX;          // n x KM scratch (materialised C of the X-side range finder)
    double* CW;          // N x KM scratch
    int rhoK, rhoL;
    unsigned long long* prof;  // non-null only on the profiled CTA
    unsigned gen;              // team barrier generation
    int parity;                // partial buffer in use (double-buffered)
    int cur_n;                 // energy index of the current step (diagnostics)
};

constexpr int kDirectReduceMax = 16;  // teams up to this size sum partials directly

__device__ __forceinline__ bool is_bnd(const DevProblem& P, int c) {
    int i = c / P.ny, j = c - (c / P.ny) * P.ny;
    return i == 0 || j == 0 || i == P.nx - 1 || j == P.ny - 1;
}

// ------------------------------------------------------------- reductions ---
__device__ __forceinline__ void acc_zero(Ctx& x, int count) {
    for (int e = threadIdx.x; e < count; e += NT) x.sm->acc[e] = 0.0;
    __syncthreads();
}
// Partials are double-buffered by parity: a CTA may publish the next
// reduction while slower CTAs still read the previous one.
__device__ __forceinline__ double* part_base(const Ctx& x, int g) {
    return x.st.part + ((size_t)x.parity * x.G + g) * PMAX;
}
__device__ __forceinline__ void acc_publish(Ctx& x, int count) {
    x.parity ^= 1;
    double* dst = part_base(x, x.b);
    for (int e = threadIdx.x; e < count; e += NT) dst[e] = x.sm->acc[e];
}
// entries [off, off+m*n) of the team's sums (publish_sync leaves them in acc) as a
// matrix of KM stride
__device__ inline void reduce_into(Ctx& x, int off, int m, int n, double* dst) {
    for (int e = threadIdx.x; e < m * n; e += NT) dst[(e / n) * KM + e % n] = x.sm->acc[off + e];
    __syncthreads();
}

// acc[off + i*kb + j] += sum_{r < nr} tA[r][i] tB[r][j]; `rot` as for for_blocks.
// Two accumulators halve the chain of products, which a block waits for.
__device__ __forceinline__ void gram_acc(double* acc, int off, const double* tA, int lda, int ka,
                                         const double* tB, int ldb, int kb, int nr, int rot = 0) {
    for_blocks(ka, kb, rot, [&](int i, int j, int o) {
        const int kr = threadIdx.x & 3;
        double d0[2] = {0.0, 0.0}, d1[2] = {0.0, 0.0};
#pragma unroll 1
        for (int r0 = kr; r0 < nr + kr; r0 += 16) {
            double av[4], bv[4];
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                const bool in = r0 + 4 * s < nr;
                av[s] = in ? tA[(r0 + 4 * s) * lda + i] : 0.0;
                bv[s] = in ? tB[(r0 + 4 * s) * ldb + j] : 0.0;
            }
            w_mma(d0, av[0], bv[0]);
            w_mma(d1, av[1], bv[1]);
            w_mma(d0, av[2], bv[2]);
            w_mma(d1, av[3], bv[3]);
        }
        if (i < ka) {
            if (o < kb) acc[off + i * kb + o] += d0[0] + d1[0];
            if (o + 1 < kb) acc[off + i * kb + o + 1] += d0[1] + d1[1];
        }
    });
}

// ------------------------------------------------------------ row helpers ---
// Tiles hold at most TR rows; thread t owns the columns j, j + 1 of row r of
// such a tile, so that one load of 16 bytes a thread fetches it.
static_assert(TR % 8 == 0 && TR * KM / 2 <= NT, "a pair of columns per thread");
static_assert(QMAX <= KM && KM % 2 == 0 && QM % 2 == 0, "rows of the ordinates by the same pairs");
struct Pair {
    int r, j;
    __device__ Pair() : r(threadIdx.x / (KM / 2)), j(2 * (threadIdx.x % (KM / 2))) {}
};
// rows of a tile such that `rows` rows take tiles of nearly the same height
__device__ __forceinline__ int tile_rows(int rows) {
    const int tiles = max(1, (rows + TR - 1) / TR);
    return max(1, (rows + tiles - 1) / tiles);
}
__device__ __forceinline__ double2 ldcg2(const double* p) { return __ldcg(reinterpret_cast<const double2*>(p)); }
__device__ __forceinline__ void st2(double* p, double2 v) { *reinterpret_cast<double2*>(p) = v; }

// rows [r0, r0+nr) of A (row length `ld` in memory and in t), columns < k
__device__ __forceinline__ void load_rows(double* t, const double* A, int r0, int nr, int k, int ld = KM) {
    const Pair p;
    if (p.r < nr && p.j < k) st2(t + p.r * ld + p.j, ldcg2(A + (size_t)(r0 + p.r) * ld + p.j));
}
// the pair of columns o, o + 1 of one row, of a tile and of its matrix in memory
__device__ __forceinline__ void put_pair(double* t, double* A, int k, int o, double v0, double v1) {
    t[o] = v0;
    t[o + 1] = v1;
    if (o + 1 < k) st2(A + o, make_double2(v0, v1));
    else if (o < k) A[o] = v0;
}

// tO = tA M, also stored to rows [r0, r0+nr) of D unless D is null (tA: nr x ka, M: ka x kb)
__device__ __forceinline__ void tile_mm(double* tO, const double* tA, const double* M, int nr, int ka, int kb,
                                        double* D = nullptr, int r0 = 0) {
    for_blocks(nr, kb, 0, [&](int r, int j, int o) {
        double d[2] = {0.0, 0.0};
        mma_dot(d, ka, tA + r * KM, 1, M + j, KM);
        if (D && r < nr) put_pair(tO + r * KM, D + (size_t)(r0 + r) * KM, kb, o, d[0], d[1]);
        else tO[r * KM + o] = d[0], tO[r * KM + o + 1] = d[1];
    });
}

// Matrix-free stencils (stencils.jl:26-128) applied to rows [r0, r0+nr) of A:
// t[0] = L2x A, t[1] = L2y A and, unless `central`, t[2] = L1x A, t[3] = L1y A;
// zero on boundary rows. `tA`, if given, receives the rows of A themselves.
__device__ inline void stencil_tile(const Ctx& x, const double* A, int r0, int nr, int k, double (*t)[TR * KM],
                                    double* tA, bool central) {
    const DevProblem& P = x.P;
    const double hx = 0.5 / P.dx, hy = 0.5 / P.dy;
    const Pair p;
    if (p.r >= nr || p.j >= k) return;
    const int c = r0 + p.r, e = p.r * KM + p.j;
    const double* a = A + (size_t)c * KM + p.j;
    double2 l2x = {0.0, 0.0}, l2y = l2x, l1x = l2x, l1y = l2x;
    const bool in = !is_bnd(P, c);
    const int sx = in ? P.ny : 0, sy = in ? 1 : 0;
    const double2 v0 = ldcg2(a), vxm = ldcg2(a - (ptrdiff_t)sx * KM), vxp = ldcg2(a + (ptrdiff_t)sx * KM),
                  vym = ldcg2(a - sy * KM), vyp = ldcg2(a + sy * KM);
    const double r_0 = P.rinv[c], rxm = P.rinv[c - sx], rxp = P.rinv[c + sx], rym = P.rinv[c - sy],
                 ryp = P.rinv[c + sy];
    if (in) {
        const auto one = [&](double a0, double xm, double xp, double ym, double yp, double& x2, double& y2,
                             double& x1, double& y1) {
            const double b0 = a0 * r_0, axm = xm * rxm, axp = xp * rxp, aym = ym * rym, ayp = yp * ryp;
            x2 = (axp - axm) * hx;
            y2 = (ayp - aym) * hy;
            x1 = b0 / P.dx - hx * axm - hx * axp;
            y1 = b0 / P.dy - hy * aym - hy * ayp;
        };
        one(v0.x, vxm.x, vxp.x, vym.x, vyp.x, l2x.x, l2y.x, l1x.x, l1y.x);
        one(v0.y, vxm.y, vxp.y, vym.y, vyp.y, l2x.y, l2y.y, l1x.y, l1y.y);
    }
    if (tA) st2(tA + e, v0);
    st2(t[0] + e, l2x);
    st2(t[1] + e, l2y);
    if (!central) {
        st2(t[2] + e, l1x);
        st2(t[3] + e, l1y);
    }
}

// Sparse P_N operators applied to rows [r0, r0+nr) of B (N x KM): t[d] = A_d B
// for the first `nops` operators (Ax, Az, |Ax|, |Az|). Four entries of a row are
// in flight at a time; those past its end repeat the first one with weight zero.
__device__ inline void spmm_tile(const Ctx& x, const double* B, int r0, int nr, int k, double (*t)[TR * KM],
                                 int nops = NOPS) {
    const int kp = (k + 1) >> 1;
    for (int e = threadIdx.x; e < nops * nr * kp; e += NT) {
        const int d = e / (nr * kp), rem = e - d * nr * kp;
        const int r = rem / kp, j = 2 * (rem - r * kp);
        const Csr& A = x.P.op[d];
        const int p0 = A.rowptr[r0 + r], p1 = A.rowptr[r0 + r + 1];
        double2 s = {0.0, 0.0};
#pragma unroll 1
        for (int p = p0; p < p1; p += 4) {
            int col[4];
            double val[4];
            double2 b[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                col[u] = A.col[p + u < p1 ? p + u : p];
                val[u] = p + u < p1 ? A.val[p + u] : 0.0;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) b[u] = ldcg2(B + (size_t)col[u] * KM + j);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                s.x = fma(val[u], b[u].x, s.x);
                s.y = fma(val[u], b[u].y, s.y);
            }
        }
        st2(t[d] + r * KM + j, s);
    }
}

// ----------------------------------------------------- range finder parts ---
// After G0 (Gram of A) is reduced into sm->ja: Jacobi -> V slot.
__device__ inline void rf_eig0(Ctx& x, double* V, double* lam, int k) {
    {
        ProfScope ps(x.prof, PF_JACOBI);
        jacobi_eig(x.sm->ja, x.sm->jv, lam, k, x.st.status);
    }
    sm_copy(V, x.sm->jv, k, k);
}
// After G1 (Gram of A V) in sm->ja: Jacobi -> V2 ; T1 = V V2_J diag(1/nu_J); returns rho.
__device__ inline int rf_eig1(Ctx& x, const double* V, double* T1, int k, double tol) {
    __shared__ double s_nu[KM];
    __shared__ int s_rho;
    {
        ProfScope ps(x.prof, PF_JACOBI);
        jacobi_eig(x.sm->ja, x.sm->jv, s_nu, k, x.st.status);
    }
    if (threadIdx.x == 0) {
        double nu0 = sqrt(fmax(s_nu[0], 0.0));
        int rho = 0;
        if (nu0 > 0.0) {
            for (int j = 0; j < k; ++j) {
                double nj = sqrt(fmax(s_nu[j], 0.0));
                if (nj > tol * nu0) rho = j + 1; else break;
            }
        }
        s_rho = rho;
        for (int j = 0; j < k; ++j) s_nu[j] = sqrt(fmax(s_nu[j], 0.0));
    }
    __syncthreads();
    int rho = s_rho;
    // T1 = V * V2[:, :rho] / nu
    for (int e = threadIdx.x; e < k * rho; e += NT) {
        int i = e / rho, j = e - (e / rho) * rho;
        double s = 0.0;
        for (int l = 0; l < k; ++l) s = fma(V[i * KM + l], x.sm->jv[l * KM + j], s);
        T1[i * KM + j] = s / s_nu[j];
    }
    __syncthreads();
    return rho;
}

// W-side completion in the small space (see oracle.linalg._complete):
// candidate c is accepted when 1 - ||P[c,:]||^2 > 1/4, P = [B, v_1..v_a],
// B = CW Ri. Stores per accepted vector its candidate, norm and coefficients
// w_a = P_{a-1}[c_a, :] in slot SL_WC (row a).
static __device__ __noinline__ void w_complete(Ctx& x, int rho, int need) {
    ProfScope ps(x.prof, PF_COMPLETE);
    SmemLayout* sm = x.sm;
    double* wc = sm->slot[SL_WC];
    double* Ri = sm->slot[SL_RIL];
    double* brow = sm->vec;           // B[c,:] (rho)
    __shared__ int s_acc, s_next;
    if (threadIdx.x == 0) { s_acc = 0; s_next = 0; }
    __syncthreads();
    while (true) {
        int acc = s_acc, it = s_next;
        if (acc >= need) break;
        if (it >= x.P.nwcomp || it >= NCAND) {
            if (threadIdx.x == 0) set_status(x.st.status, ST_COMPLETION);
            __syncthreads();
            break;
        }
        int c = x.P.wcomp[it];
        for (int j = threadIdx.x; j < rho; j += NT) {
            double s = 0.0;
            for (int l = 0; l <= j; ++l) s = fma(ldcg(x.CW + (size_t)c * KM + l), Ri[l * KM + j], s);
            brow[j] = s;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            double* prow = sm->vec + KM;  // [B[c,:], v_1[c], ..., v_acc[c]]
            for (int j = 0; j < rho; ++j) prow[j] = brow[j];
            for (int a = 0; a < acc; ++a) {
                const double* w = wc + a * KM;
                double v = (c == sm->wcand[a]) ? 1.0 : 0.0;
                for (int j = 0; j < rho + a; ++j) v -= prow[j] * w[j];
                prow[rho + a] = v / sm->wnrm[a];
            }
            double ss = 0.0;
            for (int j = 0; j < rho + acc; ++j) ss += prow[j] * prow[j];
            double nv2 = 1.0 - ss;
            if (nv2 > 0.25) {
                for (int j = 0; j < rho + acc; ++j) wc[acc * KM + j] = prow[j];
                sm->wcand[acc] = c;
                sm->wnrm[acc] = sqrt(nv2);
                s_acc = acc + 1;
            }
            s_next = it + 1;
        }
        __syncthreads();
    }
}

// Materialise rows [r0, r0+nr) of the new W-side basis into tile t and of `old`,
// if given, into tile tB: columns :rho = C Ri, columns rho+a = completion vector a.
__device__ inline void w_basis_tile(Ctx& x, int r0, int nr, int rho, int need, double* t, const double* old = nullptr,
                                    double* tB = nullptr, int k = 0) {
    SmemLayout* sm = x.sm;
    load_rows(sm->tA, x.CW, r0, nr, rho);
    if (old) load_rows(tB, old, r0, nr, k);
    __syncthreads();
    if (need > 0) {
        tile_mm(t, sm->tA, sm->slot[SL_RIL], nr, rho, rho);
        __syncthreads();
        const double* wc = sm->slot[SL_WC];
        for (int r = threadIdx.x; r < nr; r += NT) {
            int m = r0 + r;
            double* row = t + r * KM;
            for (int a = 0; a < need; ++a) {
                const double* w = wc + a * KM;
                double v = (m == sm->wcand[a]) ? 1.0 : 0.0;
                for (int j = 0; j < rho + a; ++j) v -= row[j] * w[j];
                row[rho + a] = v / sm->wnrm[a];
            }
        }
        __syncthreads();
        const Pair p;
        if (p.r < nr && p.j < rho + need)
            put_pair(t + p.r * KM, x.st.W + (size_t)(r0 + p.r) * KM, rho + need, p.j, t[p.r * KM + p.j],
                     t[p.r * KM + p.j + 1]);
    } else {
        tile_mm(t, sm->tA, sm->slot[SL_RIL], nr, rho, rho, x.st.W, r0);
    }
    __syncthreads();
}

// Materialise rows of the new X-side basis into tile t and X, and the old ones
// into tile tB: C Ri, then completion cells.
__device__ inline void x_basis_tile(Ctx& x, int r0, int nr, int rho, int k, double* t, double* tB) {
    SmemLayout* sm = x.sm;
    load_rows(sm->tA, x.CX, r0, nr, rho);
    load_rows(tB, x.st.X, r0, nr, k);
    __syncthreads();
    for_blocks(nr, k, 0, [&](int r, int j, int o) {
        double d[2] = {0.0, 0.0};
        mma_dot(d, rho, sm->tA + r * KM, 1, sm->slot[SL_RIK] + j, KM);
        if (r >= nr) return;
        // completion failures are reported through the status flag; keep reads in bounds
        for (int h = 0; h < 2; ++h) {
            const int ci = o + h - rho;
            if (ci >= 0) d[h] = (ci < x.P.nxcomp && r0 + r == x.P.xcomp[ci]) ? 1.0 : 0.0;
        }
        put_pair(t + r * KM, x.st.X + (size_t)(r0 + r) * KM, k, o, d[0], d[1]);
    });
    __syncthreads();
}

}  // namespace titus
