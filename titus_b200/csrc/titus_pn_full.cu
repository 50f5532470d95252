// Full-rank P_N first-collision solver (SolveFirstCollisionSource,
// code/SolverCSD.jl:465-586) on the GPU.
//
// State: the collided flux u (n x ldu, one row per cell i*ny + j, the moments in
// the column order of pn_tiles.cuh), the reduced ordinates psi (n x QM, ordinate
// fastest) and the dose. One energy step n is one kernel (pt_step_kernel): the
// beam inflow at energy[n] (csd.S[n-1]) formed where it is read, the upwind
// sweep of the interior cells, psi <- (psi - dE flux) / (1 + dE sigma_0)
// (:517-545), uTilde = u - dE (L2x u Ax + L2y u Az + L1x u |Ax| + L1y u |Az|) with
// the matrix-free density-weighted stencils (stencils.jl:12-130), collision
// (1 + dE D)^{-1}, in-scattering dE Dvec (MReduced psi), and the dose with
// csd.SMid (:548-575). Boundary rows of u are zero throughout. The whole sweep
// is captured once into a CUDA graph and launched as one unit.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "pn_tiles.cuh"
#include "titus_handle.h"

using namespace titus;
using titus_host::fail;
using titus_pn::PtArgs;

namespace {

constexpr int PN_NT = 256;    // threads per CTA of the cell-wise kernels
// Largest moment counts taken: P59 forward, P39 adjoint. They are the interface's; the
// kernels need no more shared memory for more moments (pt_patches leaves the small
// kernel where its images would not fit), only longer tables.
constexpr int PN_MAX_MOMENTS = 3632, ADJ_MAX_MOMENTS = 1600;

// 8 x 8 cells, 96 operator tiles a stage, two CTAs a SM: as many tiles as fit beside
// the stencil coefficients in shared memory (200 x 200, P29: 1255 us a step with 80
// tiles, 1132 with 112 and the coefficients in registers, 1086 so).
using Shape2D = titus_pn::PtShape<2, 1, 1, 8, 96, 2>;

}  // namespace

struct titus_pn_state {
    double *u[2] = {nullptr, nullptr}, *psi[2] = {nullptr, nullptr}, *dose = nullptr;
    PtArgs args{};              // forward tables
    PtArgs adj{};               // with the transposed tables, built by the first adjoint
    bool have_adj = false;
    titus_pn::PtLayout layout;
    int32_t* col_of = nullptr;
    int cur_u = 0, cur_psi = 0;
    int steps_done = 0;
    bool have_result = false;
    cudaStream_t cap = nullptr;   // capture stream (graphs are recorded here, launched on the caller's)
    cudaGraphExec_t exec = nullptr;   // the last sweep's graph, reused while n_end is the same
    int exec_n_end = -1;
    std::vector<void*> allocs;
    // adjoint workspace (titus_dose_adjoint), sized for (checkpoints, segment length)
    double *ck_u = nullptr, *ck_psi = nullptr, *seg = nullptr, *mu[2] = {nullptr, nullptr},
           *psib[2] = {nullptr, nullptr}, *pw = nullptr, *g = nullptr, *grad = nullptr, *gprof = nullptr,
           *dose_scr = nullptr, *wt = nullptr, *tg = nullptr, *gpart = nullptr;
    int adj_nck = -1, adj_k = -1;
    std::vector<void*> adj_allocs;
    void adj_release() {
        for (void* p : adj_allocs) cudaFree(p);
        adj_allocs.clear();
        adj_nck = adj_k = -1;
    }
    ~titus_pn_state() {
        if (exec) cudaGraphExecDestroy(exec);
        adj_release();
        for (void* p : allocs) cudaFree(p);
        if (cap) cudaStreamDestroy(cap);
    }
};

namespace {

struct PnAlloc {
    titus_pn_state* st;
    template <class T>
    int operator()(T** p, size_t count, const T* host = nullptr) const {
        int rc = titus_host::upload(p, host, count);
        if (rc == TITUS_OK && *p) st->allocs.push_back((void*)*p);
        return rc;
    }
};

int pn_operators(const titus_solver* s, std::vector<titus_pn::HostCsr>& ops) {
    ops.resize(4);
    for (int d = 0; d < 4; ++d) {
        int rc = titus_pn::download_csr(s->P.op[d], s->N, ops[d]);
        if (rc) return rc;
    }
    return TITUS_OK;
}

int pn_build(titus_solver* s, titus_pn_state* st) {
    const PnAlloc alloc{st};
    std::vector<titus_pn::HostCsr> ops;
    std::vector<double> mred;
    int rc;
    if ((rc = pn_operators(s, ops)) || (rc = titus_pn::download_mred(s, mred))) return rc;
    st->layout = titus_pn::pt_layout(ops, {false, false, true, true}, s->N, Shape2D::NT);
    if ((rc = titus_pn::pt_common(s, st->layout, st->args, st->col_of, alloc))) return rc;
    titus_pn::pt_patches<Shape2D>(ops, s->num_sms, st->args);
    if ((rc = titus_pn::pt_operator_tables<Shape2D>(ops, false, s->N, st->layout, mred, s->q, st->args, alloc))) return rc;
    const size_t nL = (size_t)s->n * st->layout.ldu;
    if ((rc = alloc(&st->u[0], nL)) || (rc = alloc(&st->u[1], nL)) || (rc = alloc(&st->psi[0], (size_t)s->n * QM)) ||
        (rc = alloc(&st->psi[1], (size_t)s->n * QM)) || (rc = alloc(&st->dose, (size_t)s->n)) ||
        (rc = titus_pn::pt_prepare<Shape2D, 0>()) || (rc = titus_pn::pt_prepare<Shape2D, 1>()))
        return rc;
    CK(cudaStreamCreateWithFlags(&st->cap, cudaStreamNonBlocking));
    return TITUS_OK;
}

// Device state and operator tables, built on first use from the uploaded CSR of the A_d.
int pn_ensure(titus_solver* s) {
    if (s->pn) return TITUS_OK;
    if (!s->smid) return fail(TITUS_ERR_ARG, "the full-rank P_N solver needs problem->stopping_mid (csd.SMid)");
    if (s->N > PN_MAX_MOMENTS)
        return fail(TITUS_ERR_CUDA, "full-rank solver set-up: N = %d moments exceed the supported N <= %d", s->N,
                    PN_MAX_MOMENTS);
    auto* st = new titus_pn_state();
    const int rc = pn_build(s, st);
    if (rc) {
        delete st;
        return rc;
    }
    s->pn = st;
    return TITUS_OK;
}

// The state the sweep starts from: u, psi and dose zero (SetupIC is zero for the
// beam problems). Both u buffers: the steps write interior rows only.
int pn_reset(titus_solver* s, titus_pn_state* st, cudaStream_t stream) {
    const size_t nL = (size_t)s->n * st->layout.ldu;
    CK(cudaMemsetAsync(st->u[0], 0, nL * sizeof(double), stream));
    CK(cudaMemsetAsync(st->u[1], 0, nL * sizeof(double), stream));
    CK(cudaMemsetAsync(st->psi[0], 0, (size_t)s->n * QM * sizeof(double), stream));
    CK(cudaMemsetAsync(st->dose, 0, (size_t)s->n * sizeof(double), stream));
    return TITUS_OK;
}

}  // namespace

void titus_host::pn_free(titus_solver* s) {
    delete s->pn;
    s->pn = nullptr;
}

extern "C" int titus_pn_full_solve_device(titus_solver_t* s, const titus_options_t* opt, void* stream_) {
    if (!s) return fail(TITUS_ERR_ARG, "solver is NULL");
    if (opt && opt->precision != TITUS_PRECISION_FP64)
        return fail(TITUS_ERR_ARG, "the full-rank P_N solver runs in FP64 only (precision %d)", opt->precision);
    if (s->nz) return titus_host::pn3_solve_device(s, opt, (cudaStream_t)stream_);
    int rc = pn_ensure(s);
    if (rc) return rc;
    titus_pn_state* st = s->pn;
    cudaStream_t stream = (cudaStream_t)stream_;
    int n_end = s->nE;
    if (opt && opt->max_steps > 0) n_end = std::min(n_end, 1 + opt->max_steps);
    if ((rc = pn_reset(s, st, stream))) return rc;
    // record the sweep into a graph on the capture stream (once per n_end), then
    // launch it on `stream`
    if (!st->exec || st->exec_n_end != n_end) {
        if (st->exec) {
            CK(cudaStreamSynchronize(stream));   // the old graph may still be running
            cudaGraphExecDestroy(st->exec);
            st->exec = nullptr;
            st->exec_n_end = -1;
        }
        CK(cudaStreamBeginCapture(st->cap, cudaStreamCaptureModeThreadLocal));
        int cu = 0;
        for (int n = 2; n <= n_end; ++n) {
            titus_pn::pt_step<Shape2D, 0>(st->args, n, st->u[cu], nullptr, st->psi[cu], st->psi[cu ^ 1],
                                          st->u[cu ^ 1], st->dose, nullptr, st->cap);
            cu ^= 1;
        }
        if (n_end >= 2)
            titus_pn::pt_psi_boundary_kernel<2><<<(int)(((size_t)s->n * s->q + PN_NT - 1) / PN_NT), PN_NT, 0, st->cap>>>(
                st->args, n_end, st->psi[cu]);
        cudaGraph_t graph = nullptr;
        cudaError_t e = cudaStreamEndCapture(st->cap, &graph);
        if (e != cudaSuccess) return fail(TITUS_ERR_CUDA, "graph capture: %s", cudaGetErrorString(e));
        cudaGraphExec_t exec = nullptr;
        e = cudaGraphInstantiate(&exec, graph, 0);
        cudaGraphDestroy(graph);
        if (e != cudaSuccess) return fail(TITUS_ERR_CUDA, "graph instantiation: %s", cudaGetErrorString(e));
        st->exec = exec;
        st->exec_n_end = n_end;
    }
    CK(cudaGraphLaunch(st->exec, stream));
    st->cur_u = st->cur_psi = (n_end - 1) & 1;
    st->steps_done = n_end - 1;
    st->have_result = true;
    return TITUS_OK;
}

extern "C" int titus_pn_full_fetch(titus_solver_t* s, double* u_out, double* dose_out, double* psi_out) {
    if (!s) return fail(TITUS_ERR_ARG, "solver is NULL");
    if (s->nz) return titus_host::pn3_fetch(s, u_out, dose_out, psi_out);
    if (!s->pn || !s->pn->have_result) return fail(TITUS_ERR_ARG, "no full-rank solve has run on this handle");
    titus_pn_state* st = s->pn;
    CK(cudaDeviceSynchronize());
    CK(cudaGetLastError());
    if (u_out) {
        // moment order in the buffer that the last step read (n x ldu >= n x N)
        double* tmp = st->u[st->cur_u ^ 1];
        titus_pn::pt_unpack_kernel<<<s->num_sms * 8, PN_NT>>>(s->n, s->N, st->layout.ldu, st->col_of,
                                                              st->u[st->cur_u], tmp);
        CK(cudaGetLastError());
        CK(cudaDeviceSynchronize());
        const size_t row = (size_t)s->N * sizeof(double);
        CK(s->host_copy.copy2d(u_out, row, tmp, row, row, s->n));
    }
    if (dose_out) CK(cudaMemcpy(dose_out, st->dose, (size_t)s->n * sizeof(double), cudaMemcpyDeviceToHost));
    if (psi_out)
        CK(cudaMemcpy2D(psi_out, s->q * sizeof(double), st->psi[st->cur_psi], QM * sizeof(double),
                        s->q * sizeof(double), s->n, cudaMemcpyDeviceToHost));
    return TITUS_OK;
}

extern "C" int titus_pn_full_solve(titus_solver_t* s, const titus_options_t* opt, double* u_out, double* dose_out,
                                   double* psi_out) {
    int rc = titus_pn_full_solve_device(s, opt, nullptr);
    if (rc) return rc;
    return titus_pn_full_fetch(s, u_out, dose_out, psi_out);
}

// ---------------------------------------------------------------------------
// Adjoint of the full-rank sweep (titus_dose_adjoint): gradients of a dose
// objective J with respect to the cell densities and to PsiBeam's spatial
// profile, by the exact transpose of the explicit step above, run from the
// last energy step back to the first. The stored adjoint state is mu = P_int
// lambda / (1 + dE D) with g c_n / rho added to moment 0 before the division
// (c_n the dose weight). Per backward step n:
//   pn_adj_psi_w_kernel  w = (psibar + P_int (dE (mu Dvec) MReduced + g c_n / rho
//                      MReduced[0,:])) / (1 + dE sigma_0), the adjoint of psi';
//   pt_step_kernel<.., 1>  lambda' = mu - dE sum_d (L_d^T mu) A_d^T and, in the same
//                      pass, dJ/drho_c += dE / rho_c sum_d (L_d^T mu A_d^T)[c] . u_{n-1}[c]
//                      (every entry of L_d carries 1/rho of its column cell; moving
//                      A_d to the adjoint side leaves no product u A_d to form),
//                      written as mu of step n - 1;
//   pn_adj_psi_bc_kernel  psibar_bc = w - dE F^T w, the transposed upwind sweep;
//                      on boundary cells it is the inflow's sensitivity
//                      (dJ/dprofile += psibar_bc . inflow factor), elsewhere it
//                      carries to the previous step.
// Checkpoints: (u, psi) entering every k-th step are kept from one forward
// pass; each segment of k steps is recomputed from its checkpoint into a
// k-slot buffer of u states and then run backward.
// ---------------------------------------------------------------------------
namespace {

// dose weight dE SMid[n-1] / (1 + (n == 2 or n == nE)) of step n
__device__ __forceinline__ double dose_weight(const PtArgs& a, int n) {
    const double half = (n == 2 || n == a.nE) ? 2.0 : 1.0;
    return a.dE * a.smid[n - 2] / half;
}

// mu of the last step: lambda = 0, so only the dose term of moment 0 (whose D is 0)
__global__ void pn_adj_start_kernel(PtArgs a, int n, const double* __restrict__ g, double* __restrict__ mu) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= a.n || titus_pn::pt_bnd<2>(a, c)) return;
    mu[(size_t)c * a.ldu + a.col_m0] = g[c] * dose_weight(a, n) * a.rinv[c];
}

// A CTA forms w for 8 cells: its warps split the columns, each multiplies its
// share of mu with Dvec MReduced (mma.m8n8k4.f64, up to QM / 8 ordinate tiles), and
// the partial sums meet in shared memory in warp order. mu is read once.
constexpr int PW_WARPS = 4;
__global__ void __launch_bounds__(32 * PW_WARPS) pn_adj_psi_w_kernel(PtArgs a, int n, const double* __restrict__ mu,
                                                                     const double* __restrict__ g,
                                                                     const double* __restrict__ psib,
                                                                     double* __restrict__ w) {
    __shared__ double part[PW_WARPS][8][QM];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int c0 = blockIdx.x * 8, c = min(c0 + (lane >> 2), a.n - 1);
    const double* sg = a.sigma + (size_t)(n - 1) * (a.npn + 1);
    double acc[QM / 8][2] = {};
    for (int k0 = warp * 4; k0 < a.ldu; k0 += 4 * PW_WARPS) {
        const int col = k0 + (lane & 3), mom = __ldg(a.momp + col);
        const double m = __ldg(mu + (size_t)c * a.ldu + col) * __ldg(sg + __ldg(a.lofp + col));
#pragma unroll
        for (int t = 0; t < QM / 8; ++t) {
            if (8 * t >= a.q) break;
            const int k = 8 * t + (lane >> 2);
            const double b = k < a.q && mom >= 0 ? __ldg(a.mred + (size_t)mom * a.q + k) : 0.0;
            titus_pn::pt_mma(acc[t], m, b);
        }
    }
#pragma unroll
    for (int t = 0; t < QM / 8; ++t) {
        part[warp][lane >> 2][8 * t + 2 * (lane & 3)] = acc[t][0];
        part[warp][lane >> 2][8 * t + 2 * (lane & 3) + 1] = acc[t][1];
    }
    __syncthreads();
    const double cn = dose_weight(a, n);
    for (int e = threadIdx.x; e < 8 * a.q; e += blockDim.x) {
        const int r = e / a.q, k = e - r * a.q, cc = c0 + r;
        if (cc >= a.n) break;
        double v = psib[(size_t)cc * QM + k];
        if (!titus_pn::pt_bnd<2>(a, cc)) {
            double sum = 0.0;
#pragma unroll
            for (int q = 0; q < PW_WARPS; ++q) sum += part[q][r][k];
            v += a.dE * sum + g[cc] * cn * a.rinv[cc] * a.mred[k];
        }
        w[(size_t)cc * QM + k] = v / (1.0 + a.dE * sg[0]);
    }
}

__global__ void __launch_bounds__(PN_NT) pn_adj_psi_bc_kernel(PtArgs a, int n, const double* __restrict__ w,
                                                              double* __restrict__ psib_out,
                                                              double* __restrict__ gprof) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= a.n) return;
    const bool bnd = titus_pn::pt_bnd<2>(a, c);
    const double bcf = a.inflow[n - 1];
    auto W = [&](int cc, int kk) -> double { return (cc >= 0 && cc < a.n) ? w[(size_t)cc * QM + kk] : 0.0; };
    double acc = 0.0;
    for (int kk = 0; kk < a.q; ++kk) {
        const double ox = a.omega[kk * 3 + 0], oz = a.omega[kk * 3 + 2];
        const double ax = ox / a.dx, az = oz / a.dy;
        const double wc = W(c, kk);
        // transpose of the upwind differences: the cell's own row and the rows
        // of the downwind neighbours that difference against it
        double ft = (ox >= 0.0 ? ax : -ax) * wc + (oz >= 0.0 ? az : -az) * wc;
        ft += ox >= 0.0 ? -ax * W(c + a.ny, kk) : ax * W(c - a.ny, kk);
        ft += oz >= 0.0 ? -az * W(c + 1, kk) : az * W(c - 1, kk);
        const double pbc = wc - a.dE * ft;
        if (bnd) {
            acc = fma(pbc, bcf * a.bc_angle[kk], acc);
            psib_out[(size_t)c * QM + kk] = 0.0;
        } else {
            psib_out[(size_t)c * QM + kk] = pbc;
        }
    }
    if (bnd) gprof[c] += acc;
}

__global__ void pn_adj_objective_kernel(int n, const double* __restrict__ dose, const double* __restrict__ wt,
                                        const double* __restrict__ tg, double* __restrict__ g) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    const double wc = wt ? wt[c] : 1.0;
    const double tc = tg ? tg[c] : 0.0;
    g[c] = 2.0 * wc * (dose[c] - tc);
}

// the column groups' shares of dJ/drho in group order, and the explicit 1/rho of
// the dose: dJ/drho_c -= g_c dose_c / rho_c
__global__ void pn_adj_final_kernel(int n, int ngroups, const double* __restrict__ rinv,
                                    const double* __restrict__ dose, const double* __restrict__ g,
                                    const double* __restrict__ gpart, double* __restrict__ grad) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    double s = 0.0;
    for (int k = 0; k < ngroups; ++k) s += gpart[(size_t)k * n + c];
    grad[c] = s - g[c] * dose[c] * rinv[c];
}

int adj_ensure(titus_solver* s, titus_pn_state* st, int nck, int k) {
    if (!st->have_adj) {
        std::vector<titus_pn::HostCsr> ops;
        int rc = pn_operators(s, ops);
        if (rc) return rc;
        st->adj = st->args;
        if ((rc = titus_pn::pt_operator_tables<Shape2D>(ops, true, s->N, st->layout, {}, s->q, st->adj, PnAlloc{st})))
            return rc;
        st->have_adj = true;
    }
    if (st->adj_nck == nck && st->adj_k == k) return TITUS_OK;
    st->adj_release();
    const size_t nL = (size_t)s->n * st->layout.ldu, nQ = (size_t)s->n * QM, n = (size_t)s->n;
    auto al = [&](double** p, size_t count) {
        int rc = titus_host::upload(p, (const double*)nullptr, count);
        if (rc == TITUS_OK && *p) st->adj_allocs.push_back((void*)*p);
        return rc;
    };
    int rc;
    if ((rc = al(&st->ck_u, (size_t)nck * nL)) || (rc = al(&st->ck_psi, (size_t)nck * nQ)) ||
        (rc = al(&st->seg, (size_t)k * nL)) || (rc = al(&st->mu[0], nL)) || (rc = al(&st->mu[1], nL)) ||
        (rc = al(&st->psib[0], nQ)) || (rc = al(&st->psib[1], nQ)) ||
        (rc = al(&st->pw, nQ)) || (rc = al(&st->g, n)) || (rc = al(&st->grad, n)) || (rc = al(&st->gprof, n)) ||
        (rc = al(&st->dose_scr, n)) || (rc = al(&st->wt, n)) || (rc = al(&st->tg, n)) ||
        (rc = al(&st->gpart, (size_t)st->adj.t.ngroups * n))) {
        st->adj_release();
        return rc;
    }
    st->adj_nck = nck;
    st->adj_k = k;
    return TITUS_OK;
}

}  // namespace

extern "C" int titus_dose_adjoint(titus_solver_t* s, int32_t method, const titus_options_t* opt, const double* weight,
                                  const double* target, const double* dj_ddose, int32_t checkpoint_every,
                                  double* objective_out, double* dose_out, double* grad_density,
                                  double* grad_profile) {
    if (!s) return fail(TITUS_ERR_ARG, "solver is NULL");
    if (s->nz) return fail(TITUS_ERR_ARG, "titus_dose_adjoint: the adjoint runs the reference's 2D problems");
    if (method != TITUS_PN_FULL)
        return fail(TITUS_ERR_ARG, "titus_dose_adjoint: method %d has no adjoint (TITUS_PN_FULL = %d)", method,
                    TITUS_PN_FULL);
    if (opt && opt->precision != TITUS_PRECISION_FP64)
        return fail(TITUS_ERR_ARG, "the adjoint runs in FP64 only (precision %d)", opt->precision);
    if (checkpoint_every < 0) return fail(TITUS_ERR_ARG, "checkpoint_every must be >= 0 (0 = about sqrt(steps))");
    int rc = pn_ensure(s);
    if (rc) return rc;
    titus_pn_state* st = s->pn;
    const size_t n = (size_t)s->n, nL = n * st->layout.ldu, nQ = n * QM;
    int n_end = s->nE;
    if (opt && opt->max_steps > 0) n_end = std::min(n_end, 1 + opt->max_steps);
    const int steps = n_end - 1;
    if (steps < 1) return fail(TITUS_ERR_ARG, "the energy grid has no step");
    int k = checkpoint_every > 0 ? checkpoint_every : (int)std::ceil(std::sqrt((double)steps));
    k = std::max(1, std::min(k, steps));
    const int nck = (steps + k - 1) / k;
    if (s->N > ADJ_MAX_MOMENTS)
        return fail(TITUS_ERR_LIMIT, "titus_dose_adjoint: N = %d moments exceed the supported N <= %d", s->N,
                    ADJ_MAX_MOMENTS);
    if ((rc = adj_ensure(s, st, nck, k))) return rc;
    // objective weights / target or a given dJ/d(dose)
    if (dj_ddose) {
        CK(cudaMemcpy(st->g, dj_ddose, n * sizeof(double), cudaMemcpyHostToDevice));
    } else {
        if (weight) CK(cudaMemcpy(st->wt, weight, n * sizeof(double), cudaMemcpyHostToDevice));
        if (target) CK(cudaMemcpy(st->tg, target, n * sizeof(double), cudaMemcpyHostToDevice));
    }
    const PtArgs& a = st->args;
    const PtArgs& at = st->adj;
    cudaStream_t strm = nullptr;
    const int gcell = (int)((n + PN_NT - 1) / PN_NT);
    const int gw = (s->n + 7) / 8;
    auto forward = [&](int nn, const double* u, const double* psi, double* psi_new, double* u_new, double* dose) {
        titus_pn::pt_step<Shape2D, 0>(a, nn, u, nullptr, psi, psi_new, u_new, dose, nullptr, strm);
    };
    // forward pass with checkpoints of (u, psi) entering steps 2, 2 + k, ...
    if ((rc = pn_reset(s, st, strm))) return rc;
    int cu = 0;
    for (int nn = 2; nn <= n_end; ++nn) {
        if ((nn - 2) % k == 0) {
            const size_t i = (size_t)(nn - 2) / k;
            CK(cudaMemcpyAsync(st->ck_u + i * nL, st->u[cu], nL * sizeof(double), cudaMemcpyDeviceToDevice, strm));
            CK(cudaMemcpyAsync(st->ck_psi + i * nQ, st->psi[cu], nQ * sizeof(double), cudaMemcpyDeviceToDevice, strm));
        }
        forward(nn, st->u[cu], st->psi[cu], st->psi[cu ^ 1], st->u[cu ^ 1], st->dose);
        cu ^= 1;
    }
    CK(cudaGetLastError());
    // dJ/d(dose)
    if (!dj_ddose)
        pn_adj_objective_kernel<<<gcell, PN_NT, 0, strm>>>(s->n, st->dose, weight ? st->wt : nullptr,
                                                           target ? st->tg : nullptr, st->g);
    // boundary rows of the adjoint states and of the recomputed u stay zero: the steps write interior rows only
    CK(cudaMemsetAsync(st->mu[0], 0, nL * sizeof(double), strm));
    CK(cudaMemsetAsync(st->mu[1], 0, nL * sizeof(double), strm));
    CK(cudaMemsetAsync(st->seg, 0, (size_t)k * nL * sizeof(double), strm));
    CK(cudaMemsetAsync(st->psib[0], 0, nQ * sizeof(double), strm));
    CK(cudaMemsetAsync(st->gpart, 0, (size_t)at.t.ngroups * n * sizeof(double), strm));
    CK(cudaMemsetAsync(st->gprof, 0, n * sizeof(double), strm));
    pn_adj_start_kernel<<<gcell, PN_NT, 0, strm>>>(a, n_end, st->g, st->mu[0]);
    int cl = 0;
    for (int i = nck - 1; i >= 0; --i) {
        const int a0 = 2 + i * k, b0 = std::min(a0 + k - 1, n_end);
        auto useg = [&](int j) { return j == 0 ? st->ck_u + (size_t)i * nL : st->seg + (size_t)j * nL; };
        // recompute u entering steps a0 + 1 .. b0 (the dose goes to scratch)
        CK(cudaMemcpyAsync(st->psi[0], st->ck_psi + (size_t)i * nQ, nQ * sizeof(double), cudaMemcpyDeviceToDevice,
                           strm));
        int rp = 0;
        for (int j = 0; j + a0 < b0; ++j) {
            forward(a0 + j, useg(j), st->psi[rp], st->psi[rp ^ 1], useg(j + 1), st->dose_scr);
            rp ^= 1;
        }
        // backward through the segment
        for (int nn = b0; nn >= a0; --nn) {
            pn_adj_psi_w_kernel<<<gw, 32 * PW_WARPS, 0, strm>>>(a, nn, st->mu[cl], st->g, st->psib[cl], st->pw);
            titus_pn::pt_step<Shape2D, 1>(at, nn, st->mu[cl], useg(nn - a0), nullptr, nullptr, st->mu[cl ^ 1],
                                          st->gpart, st->g, strm);
            pn_adj_psi_bc_kernel<<<gcell, PN_NT, 0, strm>>>(a, nn, st->pw, st->psib[cl ^ 1], st->gprof);
            cl ^= 1;
        }
        CK(cudaGetLastError());
    }
    pn_adj_final_kernel<<<gcell, PN_NT, 0, strm>>>(s->n, at.t.ngroups, a.rinv, st->dose, st->g, st->gpart, st->grad);
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(strm));
    std::vector<double> dose(n), gvec(n);
    CK(cudaMemcpy(dose.data(), st->dose, n * sizeof(double), cudaMemcpyDeviceToHost));
    if (dose_out) std::copy(dose.begin(), dose.end(), dose_out);
    if (grad_density) CK(cudaMemcpy(grad_density, st->grad, n * sizeof(double), cudaMemcpyDeviceToHost));
    if (grad_profile) CK(cudaMemcpy(grad_profile, st->gprof, n * sizeof(double), cudaMemcpyDeviceToHost));
    if (objective_out) {
        double J = 0.0;
        if (dj_ddose) {
            J = std::nan("");
        } else {
            for (size_t c = 0; c < n; ++c) {
                const double wc = weight ? weight[c] : 1.0, tc = target ? target[c] : 0.0;
                J += wc * (dose[c] - tc) * (dose[c] - tc);
            }
        }
        *objective_out = J;
    }
    // the forward state buffers now hold the last recomputation, not a solve's result
    st->have_result = false;
    return TITUS_OK;
}
