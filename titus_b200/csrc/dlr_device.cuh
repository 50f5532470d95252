// Device building blocks of the persistent DLR energy-step kernel (sm_100a, FP64).
//
// One "team" of G CTAs advances one solve. Rows of the spatial factors
// (cells, row i*ny+j) and of the angular factors (moments) are partitioned over
// the team's CTAs; every reduction over rows goes through per-CTA partial
// buffers in global memory (L2 resident) and is summed by every CTA in the
// same order, so all CTAs of a team hold bit-identical small matrices and take
// identical control-flow decisions without a broadcast step.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace titus {

constexpr int NT = 512;        // threads per CTA
constexpr int NW = NT / 32;    // warps per CTA
constexpr int KM = 24;         // max basis width handled by this build
constexpr int QM = 32;         // row length of the reduced ordinates in memory
constexpr int QMAX = QM < KM ? QM : KM;   // most reduced ordinates a problem may have: the fixed-rank kernel's row
                                          // loads and products take at most KM columns
constexpr int TR = 40;         // rows per staged tile: one pair of columns per thread
constexpr int NOPS = 4;        // Ax, Az, |Ax|, |Az|
constexpr int KK = KM * KM;
constexpr int PMAX = 8 * KK;  // partial-reduction capacity (doubles); >= 2KK + 2 KM QM
constexpr int NCAND = 3 * KM;  // max W completion candidates examined

// status codes written by the device
constexpr int ST_OK = 0;
constexpr int ST_BARRIER_TIMEOUT = 1;
constexpr int ST_CHOL_BREAKDOWN = 2;
constexpr int ST_COMPLETION = 3;
constexpr int ST_JACOBI = 4;

struct Csr {
    const int32_t* rowptr;
    const int32_t* col;
    const double* val;
};

// Problem data resident on the device (shared by all teams).
struct DevProblem {
    int nx, ny, n, N, npn, q, nE, r;
    double dx, dy, dE, theta, theta_index, c_eta, rank_tol;
    const double* rinv;       // n: 1/density
    const double* stopping;   // nE
    const double* bc_energy;  // nE
    const double* sigma;      // nE x (npn+1)
    const double* bc_space;   // n
    const double* bc_angle;   // q
    const double* omega;      // q x 3
    const double* mred;       // N x q
    const int32_t* lof;       // N: Legendre order l of moment m
    Csr op[6];                // Ax, Az, |Ax|, |Az|; 3D problems also Ay, |Ay| (z streaming)
    const int32_t* xcomp; int nxcomp;
    const int32_t* wcomp; int nwcomp;
    const uint8_t* restore;   // n: 1 if ordinate-0 value is restored after the sweep
    unsigned long long* prof; // optional phase timers (SM cycles), recorded by CTA 0 of team 0
    int zero_smem;            // 1: clear the dynamic shared memory at kernel start
    long long spin_limit;     // polls before a team barrier gives up (0 = default, about a second)
    int fault_barrier;        // test hook: CTA 1 does not arrive at this barrier generation (<= 0: off)
    int precision;            // 0: FP64; 1: MIXED (tensor-core operator Grams, adaptive integrators)
    int nz;                   // 3D problems: z layers (cell (i, j, k) at row (k nx + i) ny + j); 0 in 2D
    double dz;                // 3D problems: z spacing
};

// Phase-timer categories (titus_profile reports them in this order).
enum ProfCat { PF_BARRIER = 0, PF_REDUCE, PF_JACOBI, PF_CHOL, PF_COMPLETE, PF_ROWS_STREAM, PF_ROWS_SCATTER,
               PF_RF_PASSES, PF_SMALL, PF_TOTAL, PF_PROLOGUE, PF_COUNT };
// event counters in the timer buffer (profiled CTA only; the buffer has PF_SLOTS entries)
constexpr int PF_SVD_SWEEPS = 12, PF_SVD_CALLS = 13;
constexpr int PF_EIG_CALLS = 16, PF_EIG_SWEEPS = 17, PF_CHOL_CALLS = 18, PF_RF_SLOW = 19, PF_RF_FAST = 20,
              PF_BARRIERS = 21;
constexpr int PF_SLOTS = 32;
__device__ __forceinline__ void prof_count(unsigned long long* p, int slot, unsigned long long v) {
    if (p && threadIdx.x == 0) p[slot] += v;
}

// Exclusive phase timers (SM cycles): time is charged to the innermost open
// scope. Slot PF_COUNT collects unscoped time (not reported), slots PF_CUR /
// PF_T hold the open category and the last timestamp; only thread 0 of the
// profiled CTA touches them.
constexpr int PF_CUR = 14, PF_T = 15;
struct ProfScope {
    unsigned long long* p;
    int cat;
    int prev;
    __device__ ProfScope(unsigned long long* p_, int c) : p(p_), cat(c), prev(PF_COUNT) {
        if (p && threadIdx.x == 0) {
            const unsigned long long now = clock64();
            prev = (int)p[PF_CUR];
            p[prev] += now - p[PF_T];
            p[PF_CUR] = (unsigned long long)c;
            p[PF_T] = now;
        }
    }
    __device__ ~ProfScope() {
        if (p && threadIdx.x == 0) {
            const unsigned long long now = clock64();
            p[cat] += now - p[PF_T];
            p[PF_CUR] = (unsigned long long)prev;
            p[PF_T] = now;
        }
    }
};
__device__ __forceinline__ void prof_begin(unsigned long long* p) {
    if (p && threadIdx.x == 0) {
        p[PF_CUR] = PF_COUNT;   // unclassified slot, not reported
        p[PF_T] = clock64();
    }
}

// Per-team device state.
struct TeamState {
    double* X;      // n x KM
    double* K;      // n x KM   (K, then C of the range finder)
    double* W;      // N x KM
    double* L;      // N x KM
    double* psi0;   // n x QM
    double* psi1;   // n x QM
    double* dose;   // n
    double* S;      // KM x KM (final S written back)
    double* part;   // 2 x G x PMAX partial reductions (double-buffered)
    double* red;    // PMAX: second-stage reduced entries (large teams)
    unsigned* bar;  // [0, G): arrival generation per CTA; [G]: release generation
    int* status;    // device error flag
    int* info;      // [0]=rank, [1]=steps done, [2]=psi buffer index, [3]=next n
    double* diag;   // 16: breakdown diagnostics (see record_breakdown)
    int* rank_hist; // nE
    double* eta_hist;
    double* bound_hist;
    double* time_hist;
    double* Y;      // 3 x n x KM: RK4 integrator stage buffers of the K-step (KUP, two stage inputs)
    double* Z;      // 3 x N x KM: the same for the L-step
};

__device__ __forceinline__ double ldcg(const double* p) { return __ldcg(p); }
__device__ __forceinline__ int ldcg(const int* p) { return __ldcg(p); }
__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}


// Team barrier, one hop through L2: after the CTA's writes, thread 0 fences and
// adds 1 to the team's arrival counter flags[G], then waits (acquire loads)
// until the counter reaches gen * G, i.e. every CTA of the team has arrived at
// this generation. The counter runs modulo 2^32; the signed difference compares
// correctly while fewer than 2^31 arrivals separate the two values. flags[0, G)
// are not used. Every spin is bounded (`spin_limit` polls, default 2^21 with
// 200 ns sleeps: about a second); on expiry the status flag is set, the
// diagnostics record the CTA, the counter it saw and the one it waited for, and
// all CTAs leave. `fault_gen` >= 1 is a test hook: CTA 1 skips its arrival at
// that generation, so the wait runs out (the host reads the status; nothing
// faults). Returns false if the team's status flag is set.
__device__ inline bool team_sync(unsigned* flags, int* status, int G, int b, unsigned& gen, double* diag = nullptr,
                                 long long spin_limit = 0, int fault_gen = -1) {
    __shared__ int s_ok;
    const long long limit = spin_limit > 0 ? spin_limit : (1ll << 21);
    __syncthreads();
    ++gen;
    if (G == 1) {
        // a one-CTA team: __syncthreads already orders the block's global
        // writes before its later reads; only the status flag is shared
        if (threadIdx.x == 0) s_ok = (ldcg(status) == 0);
        __syncthreads();
        return s_ok;
    }
    if (threadIdx.x == 0) {
        __threadfence();
        const unsigned target = gen * (unsigned)G;
        const bool skip = (b == 1 && (int)gen == fault_gen);
        unsigned seen = skip ? ld_acquire(flags + G) : atomicAdd(flags + G, 1u) + 1u;
        long long it = 0;
        while ((int)(seen - target) < 0) {
            if (++it > limit) {
                if (atomicCAS(status, 0, ST_BARRIER_TIMEOUT) == 0 && diag) {
                    diag[8] = b;
                    diag[9] = seen;
                    diag[10] = target;
                    diag[14] = gen;
                }
                break;
            }
            if (it > 32) __nanosleep(200);
            if ((it & 255) == 0 && ldcg(status) != 0) break;
            seen = ld_acquire(flags + G);
        }
        __threadfence();
        s_ok = (ldcg(status) == 0);
    }
    __syncthreads();
    return s_ok;
}

__device__ __forceinline__ void set_status(int* status, int code) {
    atomicCAS(status, 0, code);
}

// ---------------------------------------------------------------------------
// Small dense helpers on one CTA. Matrices are row-major with leading dim KM.
// ---------------------------------------------------------------------------

// D += A B on an 8 x 8 tile, four columns of A at a time (FP64 tensor pipe): a
// lane holds A[lane / 4][lane % 4], B[lane % 4][lane / 4] and
// D[lane / 4][2 (lane % 4) + {0, 1}].
__device__ __forceinline__ void w_mma(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}

// The 8 x 8 blocks of an m x n result over the CTA's warps: f(r, j, o) with the
// lane's row r of A, its column j of B (each possibly past the end, but inside
// the padded tiles) and o, the first of the two columns of row r that its
// accumulators hold. `rot` shifts the first block to another warp, so that
// several small products in a row fill the warps.
template <class F>
__device__ __forceinline__ void for_blocks(int m, int n, int rot, F f) {
    const int lane = threadIdx.x & 31, nb = (n + 7) >> 3, total = ((m + 7) >> 3) * nb;
#pragma unroll 1
    for (int b = ((int)(threadIdx.x >> 5) + NW - rot % NW) % NW; b < total; b += NW) {
        const int rb = b / nb, jb = b - rb * nb;
        f(8 * rb + (lane >> 2), 8 * jb + (lane >> 2), 8 * jb + 2 * (lane & 3));
    }
}

// d += sum_{l < kd} a[l * sa] * b[l * sb], kd <= KM: `a` is the lane's row of A
// and `b` its column of B. All operands are fetched before the first product:
// the chain of products is what a block waits for, and a loop over l of unknown
// length costs more than its six steps. Columns past kd count as zero.
__device__ __forceinline__ void mma_dot(double (&d)[2], int kd, const double* a, int sa, const double* b, int sb) {
    static_assert(QMAX <= KM && KM % 8 == 0, "kd may be the number of ordinates; two steps of four at a time");
    const int kr = threadIdx.x & 3;
    double av[KM / 4], bv[KM / 4];
#pragma unroll
    for (int s = 0; s < KM / 4; ++s) {
        const int l = 4 * s + kr;
        av[s] = l < kd ? a[l * sa] : 0.0;
        bv[s] = l < kd ? b[l * sb] : 0.0;
    }
#pragma unroll
    for (int s = 0; s < KM / 4; s += 2)
        if (4 * s < kd) {
            w_mma(d, av[s], bv[s]);
            w_mma(d, av[s + 1], bv[s + 1]);
        }
}

// C = A(m x k) * B(k x n); C must not alias A or B.
__device__ inline void sm_mm(double* C, const double* A, const double* B, int m, int k, int n) {
    for_blocks(m, n, 0, [&](int r, int j, int o) {
        double d[2] = {0.0, 0.0};
        mma_dot(d, k, A + r * KM, 1, B + j, KM);
        C[r * KM + o] = d[0];
        C[r * KM + o + 1] = d[1];
    });
    __syncthreads();
}
// C = A(m x k) * B^T (B is n x k)
__device__ inline void sm_mmt(double* C, const double* A, const double* B, int m, int k, int n) {
    for_blocks(m, n, 0, [&](int r, int j, int o) {
        double d[2] = {0.0, 0.0};
        mma_dot(d, k, A + r * KM, 1, B + j * KM, 1);
        C[r * KM + o] = d[0];
        C[r * KM + o + 1] = d[1];
    });
    __syncthreads();
}
__device__ inline void sm_copy(double* D, const double* A, int m, int n) {
    for (int e = threadIdx.x; e < m * n; e += NT) D[(e / n) * KM + e % n] = A[(e / n) * KM + e % n];
    __syncthreads();
}
__device__ inline void sm_zero(double* D, int m, int n) {
    for (int e = threadIdx.x; e < m * n; e += NT) D[(e / n) * KM + e % n] = 0.0;
    __syncthreads();
}

// Round-robin (tournament) pairing for the parallel cyclic Jacobi method:
// round t, slot s -> pair (p, q), p < q; returns false for the dummy slot.
__device__ __forceinline__ bool rr_pair(int m, int t, int s, int k, int& p, int& q) {
    // positions 0..m-1; position 0 fixed, others rotate by t. For pos >= 1 and
    // 0 <= t <= m-2 the rotated index lies in [1, 2m-3]: one conditional
    // subtraction replaces the modulo.
    auto at = [&](int pos) -> int {
        if (pos == 0) return 0;
        int v = pos - 1 + (m - 1) - t;
        if (v >= m - 1) v -= m - 1;
        return 1 + v;
    };
    int a = at(s), b = at(m - 1 - s);
    p = min(a, b);
    q = max(a, b);
    return q < k;
}

// Symmetric eigendecomposition by parallel cyclic Jacobi.
// In: A (k x k symmetric, in smem work array Aw). Out: lam[k] descending,
// V (k x k, columns eigenvectors, same order). Aw and V are smem arrays.
static __device__ __noinline__ void jacobi_eig(double* Aw, double* V, double* lam, int k, int* status) {
    __shared__ double rc[KM / 2 + 1], rs[KM / 2 + 1];
    __shared__ int rp[KM / 2 + 1], rq[KM / 2 + 1];
    __shared__ int s_rot[2];  // per-sweep-parity flag: a reset never races a late reader
    __shared__ double s_lam[KM];
    __shared__ int s_perm[KM];
    for (int e = threadIdx.x; e < k * k; e += NT) V[(e / k) * KM + e % k] = ((e / k) == (e % k)) ? 1.0 : 0.0;
    __syncthreads();
    if (k <= 1) {
        if (threadIdx.x == 0 && k == 1) lam[0] = Aw[0];
        __syncthreads();
        return;
    }
    const int m = k + (k & 1);
    const int npairs = m / 2;
    int sweep = 0;
    for (; sweep < 40; ++sweep) {
        const int par = sweep & 1;
        if (threadIdx.x == 0) s_rot[par] = 0;
        __syncthreads();
        for (int t = 0; t < m - 1; ++t) {
            if (threadIdx.x < npairs) {
                int p, q;
                double c = 1.0, s = 0.0;
                bool valid = rr_pair(m, t, threadIdx.x, k, p, q);
                if (valid) {
                    double apq = Aw[p * KM + q];
                    double app = Aw[p * KM + p], aqq = Aw[q * KM + q];
                    if (apq != 0.0 && fabs(apq) > 1e-15 * sqrt(fabs(app * aqq))) {
                        double theta = (aqq - app) / (2.0 * apq);
                        double t_;
                        if (fabs(theta) > 1e150) t_ = 0.5 / theta;
                        else t_ = copysign(1.0, theta) / (fabs(theta) + sqrt(theta * theta + 1.0));
                        c = 1.0 / sqrt(t_ * t_ + 1.0);
                        s = t_ * c;
                        s_rot[par] = 1;
                    }
                } else {
                    p = q = -1;
                }
                rc[threadIdx.x] = c;
                rs[threadIdx.x] = s;
                rp[threadIdx.x] = p;
                rq[threadIdx.x] = q;
            }
            __syncthreads();
            // rows: A <- J^T A
            for (int e = threadIdx.x; e < npairs * k; e += NT) {
                int pi = e / k, j = e % k;
                int p = rp[pi], q = rq[pi];
                if (p < 0) continue;
                double c = rc[pi], s = rs[pi];
                if (s == 0.0) continue;
                double ap = Aw[p * KM + j], aq = Aw[q * KM + j];
                Aw[p * KM + j] = c * ap - s * aq;
                Aw[q * KM + j] = s * ap + c * aq;
            }
            __syncthreads();
            // columns: A <- A J, V <- V J
            for (int e = threadIdx.x; e < npairs * k; e += NT) {
                int pi = e / k, i = e % k;
                int p = rp[pi], q = rq[pi];
                if (p < 0) continue;
                double c = rc[pi], s = rs[pi];
                if (s == 0.0) continue;
                double ap = Aw[i * KM + p], aq = Aw[i * KM + q];
                Aw[i * KM + p] = c * ap - s * aq;
                Aw[i * KM + q] = s * ap + c * aq;
                double vp = V[i * KM + p], vq = V[i * KM + q];
                V[i * KM + p] = c * vp - s * vq;
                V[i * KM + q] = s * vp + c * vq;
            }
            __syncthreads();
        }
        if (!s_rot[par]) break;
    }
    (void)status;
    // sort descending (stable): rank of each eigenvalue
    for (int i = threadIdx.x; i < k; i += NT) s_lam[i] = Aw[i * KM + i];
    __syncthreads();
    for (int i = threadIdx.x; i < k; i += NT) {
        double li = s_lam[i];
        int rank = 0;
        for (int j = 0; j < k; ++j) {
            double lj = s_lam[j];
            if (lj > li || (lj == li && j < i)) ++rank;
        }
        s_perm[rank] = i;
    }
    __syncthreads();
    // permute V columns into Aw as scratch, then copy back
    for (int e = threadIdx.x; e < k * k; e += NT) {
        int i = e / k, j = e % k;
        Aw[i * KM + j] = V[i * KM + s_perm[j]];
    }
    __syncthreads();
    for (int e = threadIdx.x; e < k * k; e += NT) V[(e / k) * KM + e % k] = Aw[(e / k) * KM + e % k];
    for (int j = threadIdx.x; j < k; j += NT) lam[j] = s_lam[s_perm[j]];
    __syncthreads();
}

// On breakdown with `flag`, the first CTA to fail records in diag:
// [0] stage tag, [1] side (0 = X, 1 = W), [2] k, [3] first bad pivot index,
// [4] its value, [5] G[0][0], [6] min diagonal of G, [7] energy index.
__device__ inline void record_breakdown(double* diag, int* status, int tag, int side, int k, int bj, double bd,
                                 const double* G, int n) {
    if (atomicCAS(status, 0, ST_CHOL_BREAKDOWN) == 0 && diag) {
        double mn = INFINITY;
        for (int a = 0; a < k; ++a) mn = fmin(mn, G[a * KM + a]);
        diag[0] = tag;
        diag[1] = side;
        diag[2] = k;
        diag[3] = bj;
        diag[4] = bd;
        diag[5] = k > 0 ? G[0] : 0.0;
        diag[6] = mn;
        diag[7] = n;
    }
}

// Two upper Cholesky factorisations R^T R = G with R^{-1} side by side (either
// may be skipped): the lower half of the CTA's warps takes X's, the upper half
// W's. Elimination without square roots: the row operations that make
// G = L D L^T upper triangular are applied to the identity as well (its rows grow
// in the part of R below the diagonal), so that L^{-1} is there when the last
// pivot is; R = D^{1/2} L^T and R^{-1} = L^{-T} D^{-1/2} are scaled at the end. The
// chain of one step (pivot load, reciprocal, product, update, barrier) is what
// bounds it. One warp per matrix, columns in registers and the inverse by back
// substitution, took 25 us a pair at k = 20; this takes 8 us.
// Writes the condition estimates ||R||_F ||R^{-1}||_F (+inf on a non-positive
// pivot); `flag` makes a breakdown a device status.
static __device__ __noinline__ void dual_chol(bool dx, const double* GX, double* RX, double* RiX, int kx, double* condX,
                                              bool dw, const double* GW, double* RW, double* RiW, int kw, double* condW,
                                              int* status, bool flag, double* diag = nullptr, int tag = 0, int n = 0) {
    constexpr int HW = NW / 2, ROWS = (KM + HW - 1) / HW;
    static_assert(KM <= 32, "one column of the matrix per lane");
    __shared__ double s_nr[NW], s_ni[NW], s_d[2];
    __shared__ int s_bad[2];
    const int lane = threadIdx.x & 31, side = threadIdx.x >= NT / 2, warp = (threadIdx.x >> 5) - side * HW;
    const bool on = side ? dw : dx;
    const double* G = side ? GW : GX;
    double* R = side ? RW : RX;
    double* Ri = side ? RiW : RiX;
    __builtin_assume(__isShared(G));
    __builtin_assume(__isShared(R));
    __builtin_assume(__isShared(Ri));
    const int k = on ? (side ? kw : kx) : 0;
    const int steps = max(dx ? kx : 0, dw ? kw : 0) - 1;
    if (threadIdx.x < 2) s_bad[threadIdx.x] = -1;
#pragma unroll
    for (int u = 0; u < ROWS; ++u) {
        const int i = warp + u * HW;
        if (i < k && lane < k) R[i * KM + lane] = lane >= i ? G[i * KM + lane] : 0.0;
    }
    __syncthreads();
    bool ok = true;
    const auto pivot = [&](int j) {
        const double d = R[j * KM + j];
        if (ok && !(d > 0.0)) {
            ok = false;
            if (warp == 0 && lane == 0) {
                s_bad[side] = j;
                s_d[side] = d;
            }
        }
        return d;
    };
#pragma unroll 1
    for (int j = 0; j < steps; ++j) {
        if (j < k - 1) {
            const double d = pivot(j);
            const double inv = -1.0 / (d > 0.0 ? d : 1.0);
            const double rj = R[j * KM + min(lane, k - 1)];
#pragma unroll
            for (int u = 0; u < ROWS; ++u) {
                const int i = j + 1 + warp + u * HW;
                if (i < k) {
                    const double f = R[j * KM + i] * inv;
                    // columns l >= i: U; l < j: the identity's rows, whose entry j is f itself
                    if (lane < k && (lane >= i || lane <= j))
                        R[i * KM + lane] = lane == j ? f : fma(f, rj, R[i * KM + lane]);
                }
            }
        }
        __syncthreads();
    }
    if (k > 0) pivot(k - 1);
    __syncthreads();
    double nr = 0.0, ni = 0.0;
#pragma unroll
    for (int u = 0; u < ROWS; ++u) {
        const int i = warp + u * HW;
        if (i < k) {
            const double di = R[i * KM + i];
            const double piv = di > 0.0 ? sqrt(di) : 1.0;
            __syncwarp();
            if (lane < k) {
                const double v = lane == i ? piv : R[i * KM + lane] / piv;
                const double w = lane == i ? 1.0 / piv : v;
                R[i * KM + lane] = lane >= i ? v : 0.0;
                Ri[lane * KM + i] = lane <= i ? w : 0.0;
                nr = lane >= i ? fma(v, v, nr) : nr;
                ni = lane <= i ? fma(w, w, ni) : ni;
            }
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        nr += __shfl_xor_sync(0xffffffffu, nr, o);
        ni += __shfl_xor_sync(0xffffffffu, ni, o);
    }
    if (lane == 0) {
        s_nr[side * HW + warp] = nr;
        s_ni[side * HW + warp] = ni;
    }
    __syncthreads();
    const auto cond = [&](int sd) -> double {
        double tr = 0.0, ti = 0.0;
#pragma unroll
        for (int w = 0; w < HW; ++w) {
            tr += s_nr[sd * HW + w];
            ti += s_ni[sd * HW + w];
        }
        const double c = sqrt(tr) * sqrt(ti);
        return s_bad[sd] < 0 && c < INFINITY ? c : INFINITY;
    };
    const double cx = dx ? cond(0) : 0.0, cw = dw ? cond(1) : 0.0;
    if (flag && threadIdx.x == 0) {
        if (!(cx < INFINITY)) record_breakdown(diag, status, tag, 0, kx, s_bad[0], s_bad[0] < 0 ? 0.0 : s_d[0], GX, n);
        if (!(cw < INFINITY)) record_breakdown(diag, status, tag, 1, kw, s_bad[1], s_bad[1] < 0 ? 0.0 : s_d[1], GW, n);
    }
    __syncthreads();
    if (condX) *condX = cx;
    if (condW) *condW = cw;
}

}  // namespace titus
