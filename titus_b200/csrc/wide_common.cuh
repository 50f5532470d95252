// Building blocks of the rank-adaptive DLR kernel (parallel and BUG-rejection
// integrators, SolverCSD.jl :1726-2008 and :2011-2374).
//
// Widths: the rank entering a step is at most RA; augmented bases [X X~] hold
// up to KA = 2 RA columns. Tall factors are row-major in global memory (L2
// resident) with leading dimension KA (X, W) or RA (K, L and their projected /
// range-finder copies). Every reduction over rows goes through per-CTA partial
// buffers and a two-stage sum into the team's reduced buffer `red`, which all
// CTAs then read; small-matrix algebra is repeated bit-identically by every CTA
// in shared memory and in a per-CTA scratch area of global memory, so all CTAs
// take the same control decisions (ranks, rejections) without a broadcast.
#pragma once
#include "dlr_device.cuh"
#include "umma.cuh"
#include "wide_state.h"

// The rank-adaptive kernels are compiled twice: for the reference's 2D
// problems (four streaming pairs, namespace titus::wide) and for 3D problems
// (six pairs, the z pair appended; namespace titus::wide3, titus_adaptive3d.cu).
#ifndef TITUS_WIDE_NOPS
#define TITUS_WIDE_NOPS 4
#endif
#ifndef TITUS_WIDE_NS
#define TITUS_WIDE_NS wide
#endif

namespace titus {
namespace TITUS_WIDE_NS {

// streaming pairs (stencil L_d, P_N matrix A_d): (L2x, Ax), (L2y, Az), (L1x, |Ax|),
// (L1y, |Az|) and, for 3D problems, (L2z, Ay), (L1z, |Ay|)
constexpr int NOPS_W = TITUS_WIDE_NOPS;
constexpr bool kThreeD = NOPS_W == 6;
static_assert(NOPS_W == 4 || NOPS_W == 6, "four (2D) or six (3D) streaming pairs");

// Threads per CTA. 512 against 256 (the same code, 148 CTAs unless stated): 200 x 200,
// P29, ranks 8 to 20: 2616 and 2607 us a step; 128 x 128, P21: 2118 and 2316, on
// one CTA (the batched form) 31.6 and 38.3 ms; 48 x 48, P7, ranks 2 to 9: 540 and
// 521. The row work and the wide factorisations gain, the barriers lose a little.
constexpr int NT = 512;
constexpr int RA = titus::WIDE_RA;   // max rank entering a step
constexpr int KA = 2 * RA;      // max augmented width
constexpr int LDS = KA + 1;     // row stride of the truncation SVD's column arrays (odd: no bank conflicts)
constexpr int QW = titus::QM;   // psi leading dimension (reduced ordinates <= QW)
constexpr int TRW = 8;          // rows per staged tile (minimum layout)
constexpr int TRMAX = 512;      // rows per staged tile when the phase's free shared memory allows
constexpr int PMAXW = 2 * NOPS_W * KA * KA;   // largest reduction (BUG S-step Grams): 51200 doubles in 2D
constexpr int WORKD = 20480;    // shared work area (doubles)
constexpr int ACCW = 16384;     // accumulator chunk (doubles), inside the work area
constexpr int FLD = 10 * RA;    // feature-tile leading dimension (doubles)
constexpr int SCRW = kThreeD ? 90112 : 81920;   // per-CTA scratch (doubles, global)
constexpr int WCS = 3 * RA;     // row stride of the W-side completion coefficients

// extra device status codes (titus::ST_* holds 1..4)
constexpr int ST_LIMIT = 5;        // rank would exceed RA
constexpr int ST_UNSUPPORTED = 6;  // angular basis lost orthonormality (cannot complete)
constexpr int ST_SVD = 7;          // Jacobi SVD did not converge
constexpr int ST_REF_SHAPE = 8;    // the reference's next step raises DimensionMismatch (parallel-rejection loop)

using WideState = titus::WideState;

// Per-CTA scratch layout (offsets in doubles). r x r matrices use ld RA.
enum : int {
    SO_SC = 0,                            // stacked S C_d          (NOPS_W RA x RA)
    SO_SG = SO_SC + NOPS_W * RA * RA,     // stacked S^T G_d^T      (NOPS_W RA x RA)
    SO_SBAR = SO_SG + NOPS_W * RA * RA,   // S after the streaming / in-scattering S update (RA x RA)
    SO_SIDE = SO_SBAR + RA * RA,     // per-side blocks, SIDE_STRIDE each
};
// per-side block offsets (relative to SO_SIDE + side * SIDE_STRIDE)
enum : int {
    SS_F1 = 0,                 // Q1 = A F1 (range part), r x rho1
    SS_P1 = SS_F1 + RA * RA,   // F1 F1^T
    SS_T = SS_P1 + RA * RA,    // projection coefficients / range-finder transform
    SS_M1 = SS_T + RA * RA,    // Q1^T A (BUG: top block of X1^T X)
    SS_R0 = SS_M1 + RA * RA,   // inverse Cholesky factor of the range-finder Gram
    SS_RI = SS_R0 + RA * RA,   // inverse Cholesky factor of C^T C (basis = C RI)
    SS_V0 = SS_RI + RA * RA,   // slow path: eigenvectors of G0
    SS_WC = SS_V0 + RA * RA,   // W-side completion coefficients (RA rows, stride WCS)
    SIDE_STRIDE = SS_WC + RA * 3 * RA,
};
constexpr int SO_XTPSI = SO_SIDE + 2 * SIDE_STRIDE;  // KA x QW   X^T psi
constexpr int SO_MTDW = SO_XTPSI + KA * QW;          // QW x KA   MRed^T diag(Dvec) W
constexpr int SO_TMP = SO_MTDW + QW * KA;            // 3 x KA x KA general temporaries
constexpr int SO_DBG = SO_TMP + 3 * KA * KA;           // KA x KA: input of the last truncation SVD
constexpr int SO_S0 = SO_DBG + KA * KA;                 // RA x RA: S entering the energy (parallel-rejection loop)
constexpr int SO_END = SO_S0 + RA * RA;
static_assert(SO_END <= SCRW, "per-CTA scratch too small");

struct WSmem {
    double S[KA * KA];     // state S (ld KA)
    double work[WORKD];    // phase-dependent union
    double vec[6 * KA + 2 * QW];
    double dmisc[32];
    int imisc[32];
    int wcand[RA];
    double wnrm[RA];
    int perm[KA];
    double sig[KA];
    unsigned long long mbar[2];   // MIXED mode: completion barriers of the two tensor-core chunk buffers
    unsigned tmem_slot;           // MIXED mode: TMEM base address written by tcgen05.alloc
};

// Per-side bookkeeping of one augmentation (identical in every CTA).
struct SideInfo {
    int rho1;      // numerical rank of the old basis (range part of Q1)
    int fast1;     // 1: Q1 = A R1^{-1} (certified); 0: Jacobi (F1 = V diag(lambda^-1/2))
    int rho2;      // numerical rank of the projected new directions
    int fast2;     // 1: certified CholQR2 path
    int need2;     // completion vectors appended after the range part of Q2
    int cand0;     // first X candidate used by Q2's completion
    double scale;  // Frobenius norm of [A B]
};

struct WCtx {
    DevProblem P;
    WideState st;
    WSmem* sm;
    double* scr;    // this CTA's scratch
    int G, b;
    int c0, c1, m0, m1;
    int r;          // current rank
    double* psi_in;
    double* psi_out;
    unsigned gen;
    int parity;
    const double* redp;  // reduced buffer of the latest reduction
    int cur_n;
    unsigned long long* prof;
    SideInfo side[2];
    int mixed;           // 1: MIXED precision (tensor-core operator Grams where the width >= 32)
    umma::TcCtx tc;      // tensor-core state (MIXED only)
};

// Widths from which the MIXED mode forms the operator Grams on the tensor cores.
constexpr int kTcMinWidth = 32;

// Rows per tile that fit `avail` doubles of shared memory at `per_row` doubles a row.
__device__ __forceinline__ int rows_fit(int avail, int per_row) {
    const int r = avail / per_row;
    return r < 1 ? 1 : (r > TRMAX ? TRMAX : r);
}

__device__ __forceinline__ bool is_bnd_w(const DevProblem& P, int c) {
    if constexpr (kThreeD) {
        // 3D: cell (i, j, k) at row (k nx + i) ny + j; boundary on any of the six faces
        const int nxy = P.nx * P.ny;
        const int k = c / nxy, rr = c - k * nxy;
        const int i = rr / P.ny, j = rr - i * P.ny;
        return k == 0 || k == P.nz - 1 || i == 0 || j == 0 || i == P.nx - 1 || j == P.ny - 1;
    } else {
        int i = c / P.ny, j = c - (c / P.ny) * P.ny;
        return i == 0 || j == 0 || i == P.nx - 1 || j == P.ny - 1;
    }
}

__device__ __forceinline__ bool wsync(WCtx& x) {
    ProfScope ps(x.prof, PF_BARRIER);
    prof_count(x.prof, PF_BARRIERS, 1ull);
    return team_sync(x.st.bar, x.st.status, x.G, x.b, x.gen, x.st.diag, x.P.spin_limit, x.P.fault_barrier);
}

__device__ __forceinline__ double* wpart(const WCtx& x, int g) {
    return x.st.part + ((size_t)x.parity * x.G + g) * PMAXW;
}

// Publish `cnt` partial entries of this CTA starting at `off` from the shared
// accumulator (chunked Gram passes publish several pieces before one reduce).
__device__ __forceinline__ void wpublish_chunk(WCtx& x, const double* acc, int off, int cnt) {
    double* dst = wpart(x, x.b) + off;
    for (int e = threadIdx.x; e < cnt; e += NT) dst[e] = acc[e];
}

// Two-stage team sum of entries [0, count) of the partials into the reduced
// buffer of the same parity (x.redp afterwards). Before the call every CTA
// published its partial with wpublish_chunk. The hook runs between the two
// barriers (used to zero X rows that other CTAs stop reading at the first
// barrier). A reduced buffer stays valid until the second reduction after it.
template <class Hook>
__device__ inline bool wreduce(WCtx& x, int count, Hook hook) {
    if (!wsync(x)) return false;
    hook();
    if (x.G == 1) {
        // one CTA: its partial is the sum; read it in place (the partial of
        // this parity is next written two reductions later, like `red`)
        x.redp = wpart(x, 0);
        x.parity ^= 1;
        return wsync(x);
    }
    {
        ProfScope ps(x.prof, PF_REDUCE);
        // CTA b sums the slice [e0, e1) over the G partials. Blocks of RCH
        // elements x RSPL partial-splits keep RSPL independent L2 loads in
        // flight per element (adjacent threads read adjacent elements); a warp
        // folds its two splits, the rest are combined in a fixed order, so the
        // sum is deterministic.
        constexpr int RCH = 16, RSPL = NT / RCH;
        __shared__ double s_part[NT / 2];
        const int per = (count + x.G - 1) / x.G;
        const int e0 = x.b * per, e1 = min(count, e0 + per);
        const double* base = x.st.part + (size_t)x.parity * x.G * PMAXW;
        double* red = x.st.red + (size_t)x.parity * PMAXW;
        const int el = threadIdx.x % RCH, sp = threadIdx.x / RCH;
        for (int eb = e0; eb < e1; eb += RCH) {
            const int e = eb + el;
            double a = 0.0;
            if (e < e1)
                for (int g = sp; g < x.G; g += RSPL) a += ldcg(base + (size_t)g * PMAXW + e);
            a += __shfl_xor_sync(0xffffffffu, a, RCH);
            if ((threadIdx.x & 31) < RCH) s_part[threadIdx.x / 32 * RCH + el] = a;
            __syncthreads();
            if (threadIdx.x < RCH && eb + threadIdx.x < e1) {
                double t = 0.0;
                for (int q = 0; q < RSPL / 2; ++q) t += s_part[q * RCH + threadIdx.x];
                red[eb + threadIdx.x] = t;
            }
            __syncthreads();
        }
    }
    x.redp = x.st.red + (size_t)x.parity * PMAXW;
    x.parity ^= 1;
    return wsync(x);
}
__device__ inline bool wreduce(WCtx& x, int count) {
    return wreduce(x, count, [] {});
}

// red[off + i*n + j] -> D[i*ld + j]  (m x n)
__device__ inline void load_red(const WCtx& x, int off, int m, int n, double* D, int ld) {
    for (int e = threadIdx.x; e < m * n; e += NT) D[(e / n) * ld + e % n] = ldcg(x.redp + off + e);
    __syncthreads();
}

// ---------------------------------------------------------------- algebra ---
// C (m x n) = alpha op(A) op(B) + beta C; op(A) = A^T when ta (A stored k x m),
// op(B) = B^T when tb (B stored n x k). C must not alias A or B.
__device__ inline void g_mm(double* C, int ldc, const double* A, int lda, bool ta, const double* B, int ldb, bool tb,
                            int m, int k, int n, double alpha = 1.0, double beta = 0.0) {
    for (int e = threadIdx.x; e < m * n; e += NT) {
        const int i = e / n, j = e - (e / n) * n;
        double s = 0.0;
#pragma unroll 8
        for (int l = 0; l < k; ++l) {
            const double a = ta ? A[l * lda + i] : A[i * lda + l];
            const double bb = tb ? B[j * ldb + l] : B[l * ldb + j];
            s = fma(a, bb, s);
        }
        double v = alpha * s;
        if (beta != 0.0) v = fma(beta, C[i * ldc + j], v);
        C[i * ldc + j] = v;
    }
    __syncthreads();
}
__device__ inline void g_copy(double* D, int ldd, const double* A, int lda, int m, int n) {
    for (int e = threadIdx.x; e < m * n; e += NT) D[(e / n) * ldd + e % n] = A[(e / n) * lda + e % n];
    __syncthreads();
}
__device__ inline void g_zero(double* D, int ldd, int m, int n) {
    for (int e = threadIdx.x; e < m * n; e += NT) D[(e / n) * ldd + e % n] = 0.0;
    __syncthreads();
}

// ----------------------------------------------------------- row helpers ---
// Tile moves between global memory and shared memory. Loads are asynchronous
// copies (cp.async): a thread issues every copy of its share of the tile before
// waiting once, so a tile costs about one memory latency instead of one per
// element, and the data never passes through registers. Pairs of doubles move
// as 16-byte copies that bypass L1 (.cg); single doubles use 8-byte copies
// through L1 (.ca), which is safe because a CTA only loads rows that it wrote
// itself in this launch (L1 holds no other SM's data for them).
__device__ __forceinline__ double2 ldcg2(const double* p) { return __ldcg(reinterpret_cast<const double2*>(p)); }
__device__ __forceinline__ bool pairs_ok(const double* t, const double* A, int k, int c0, int lda, int ldt, int tc) {
    return ((k | c0 | lda | ldt | tc) & 1) == 0 &&
           ((reinterpret_cast<uintptr_t>(t) | reinterpret_cast<uintptr_t>(A)) & 15) == 0;
}
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async8(void* smem, const void* gmem) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// This thread's elements of a nr x w tile in row order, NT apart: one division
// at the start instead of one per element.
struct RowWalk {
    int r, j, w, dr, dj;
    __device__ __forceinline__ explicit RowWalk(int w_) : w(w_) {
        r = threadIdx.x / w;
        j = threadIdx.x - r * w;
        dr = NT / w;
        dj = NT - dr * w;
    }
    __device__ __forceinline__ void next() {
        r += dr;
        j += dj;
        if (j >= w) {
            j -= w;
            ++r;
        }
    }
};

// rows [r0, r0+nr) x cols [c0, c0+k) of A (ld lda) -> t (ld ldt) at column tc.
// On return this thread's copies have landed; the caller's __syncthreads makes
// the whole tile visible to the CTA.
__device__ __forceinline__ void wload(double* t, int ldt, int tc, const double* A, int lda, int c0, int r0, int nr,
                                      int k) {
    if (k <= 0) return;
    if (pairs_ok(t, A, k, c0, lda, ldt, tc)) {
#pragma unroll 1
        for (RowWalk x(k >> 1); x.r < nr; x.next())
            cp_async16(t + x.r * ldt + tc + 2 * x.j, A + (size_t)(r0 + x.r) * lda + c0 + 2 * x.j);
    } else {
#pragma unroll 1
        for (RowWalk x(k); x.r < nr; x.next())
            cp_async8(t + x.r * ldt + tc + x.j, A + (size_t)(r0 + x.r) * lda + c0 + x.j);
    }
    cp_async_wait_all();
}
__device__ __forceinline__ void wstore(double* A, int lda, int c0, const double* t, int ldt, int tc, int r0, int nr,
                                       int k) {
    if (k <= 0) return;
    if (pairs_ok(t, A, k, c0, lda, ldt, tc)) {
#pragma unroll 1
        for (RowWalk x(k >> 1); x.r < nr; x.next())
            *reinterpret_cast<double2*>(A + (size_t)(r0 + x.r) * lda + c0 + 2 * x.j) =
                *reinterpret_cast<const double2*>(t + x.r * ldt + tc + 2 * x.j);
        return;
    }
#pragma unroll 1
    for (RowWalk x(k); x.r < nr; x.next()) A[(size_t)(r0 + x.r) * lda + c0 + x.j] = t[x.r * ldt + tc + x.j];
}

// Row products of a shared-memory tile: for rows r < nr and columns j < w,
//   epi(r, j, sum_{l < kd} A[r * lda + l] * mget(l, j)).
// A warp takes 16 rows x 8 columns and walks l in steps of four on the FP64
// tensor pipe: per step two loads of A and one of M for 512 products, where a
// thread's 4 x 2 micro-tile took six loads for eight. Entries with l >= kd are
// replaced by zeros (the tile's other columns are not read); rows and columns
// beyond the tile repeat its last ones and are dropped. The map from (r, j) to
// threads depends on nr and w only, so a second call may update what the first
// one's epi wrote.
template <class MGet, class Epi>
__device__ __forceinline__ void row_mm(int nr, int kd, int w, const double* A, int lda, MGet mget, Epi epi) {
    if (w <= 0) return;
    const int lane = threadIdx.x & 31, kr = lane & 3, ci = lane >> 2;
    const int jt = (w + 7) >> 3, total = jt * ((nr + 15) >> 4);
#pragma unroll 1
    for (int it = threadIdx.x >> 5; it < total; it += NT / 32) {
        const int rp = it / jt, j0 = 8 * (it - rp * jt), r0 = 16 * rp;
        const double* a0 = A + min(r0 + ci, nr - 1) * lda;
        const double* a1 = A + min(r0 + 8 + ci, nr - 1) * lda;
        const int jb = min(j0 + ci, w - 1);
        double d[2][2] = {};
#pragma unroll 2
        for (int l0 = 0; l0 < kd; l0 += 4) {
            const int l = l0 + kr;
            const bool in = l < kd;
            const double b = in ? mget(l, jb) : 0.0;
            const double x0 = in ? a0[l] : 0.0, x1 = in ? a1[l] : 0.0;
            w_mma(d[0], x0, b);
            w_mma(d[1], x1, b);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int r = r0 + 8 * h + ci, j = j0 + 2 * kr;
            if (r < nr) {
                if (j < w) epi(r, j, d[h][0]);
                if (j + 1 < w) epi(r, j + 1, d[h][1]);
            }
        }
    }
}

// One Gram block of a feature tile: acc[off + i*wb + j] += sum_r F[r][ca+i] F[r][cb+j].
struct GBlock {
    int ca, wa, cb, wb, off;
};
// Accumulate a list of blocks over a tile of nr rows on the FP64 tensor pipe. An
// item is 8 columns i x 16 columns j of one block; the items of all blocks are
// dealt to the warps in list order, and where they leave warps over, 2 or 4
// warps share an item's rows and add their sums one after the other, so the
// result depends only on (blocks, nr), not on timing. Two accumulator sets per
// tile (alternate row quads) keep dependent products apart. Columns beyond a
// block are read (the tile's next ones, still inside the shared work area) into
// entries that are not stored. Against a 2 x 2 register tile per thread, four
// loads for four products, a step loads three values for 512.
__device__ inline void gram_blocks(double* acc, const double* F, int ldf, int nr, const GBlock* bl, int nb) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, kr = lane & 3, ci = lane >> 2;
    constexpr int WARPS = NT / 32;
    int total = 0;
#pragma unroll 1
    for (int q = 0; q < nb; ++q) total += ((bl[q].wa + 7) >> 3) * ((bl[q].wb + 15) >> 4);
    const int parts = total * 4 <= WARPS ? 4 : total * 2 <= WARPS ? 2 : 1;
#pragma unroll 1
    for (int base = 0; base < total; base += WARPS / parts) {
        int off = base + warp / parts;
        const int part = warp & (parts - 1);
        const bool valid = off < total;
        GBlock g{0, 0, 0, 0, 0};
        int tj = 1;
        if (valid) {
#pragma unroll 1
            for (int q = 0; q < nb; ++q) {
                g = bl[q];
                tj = (g.wb + 15) >> 4;
                const int cnt = ((g.wa + 7) >> 3) * tj;
                if (off < cnt) break;
                off -= cnt;
            }
        }
        const int i0 = 8 * (off / tj), j0 = 16 * (off - (off / tj) * tj);
        const bool two = j0 + 8 < g.wb;
        double d[2][2][2] = {};   // [row quad parity][column tile]
        if (valid) {
            const double* pa = F + kr * ldf + g.ca + i0 + ci;
            const double* pb = F + kr * ldf + g.cb + j0 + ci;
            const int step = 4 * parts * ldf;
            int r = 4 * part;
            pa += r * ldf;
            pb += r * ldf;
#pragma unroll 1
            for (; r + 4 * parts + 4 <= nr; r += 8 * parts) {
                const double x0 = pa[0], x1 = pa[step];
                const double y0 = pb[0], y1 = pb[step];
                w_mma(d[0][0], x0, y0);
                w_mma(d[1][0], x1, y1);
                if (two) {
                    w_mma(d[0][1], x0, pb[8]);
                    w_mma(d[1][1], x1, pb[step + 8]);
                }
                pa += 2 * step;
                pb += 2 * step;
            }
#pragma unroll 1
            for (; r < nr; r += 4 * parts) {
                const bool in = r + kr < nr;
                const double x0 = in ? pa[0] : 0.0, y0 = in ? pb[0] : 0.0, z0 = in && two ? pb[8] : 0.0;
                w_mma(d[0][0], x0, y0);
                if (two) w_mma(d[0][1], x0, z0);
                pa += step;
                pb += step;
            }
        }
#pragma unroll 1
        for (int p = 0; p < parts; ++p) {
            if (p > 0) __syncthreads();
            if (valid && part == p) {
                const int i = i0 + ci;
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const int j = j0 + 8 * h + 2 * kr + u;
                        if (i < g.wa && j < g.wb) acc[g.off + i * g.wb + j] += d[0][h][u] + d[1][h][u];
                    }
            }
        }
    }
}

}  // namespace TITUS_WIDE_NS
}  // namespace titus
