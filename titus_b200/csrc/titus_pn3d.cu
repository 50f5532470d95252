// Full-rank P_N first-collision solver on a 3D grid: the z extension of
// SolveFirstCollisionSource (code/SolverCSD.jl:465-586; the reference itself
// is 2D only). Cell (i, j, k) has row (k*nx + i)*ny + j; the boundary (ghost)
// cells are those on any face. Six streaming pairs, summed in this order:
//   (L2x, Ax), (L2y, Az), (L1x, |Ax|), (L1y, |Az|), (L2z, Ay), (L1z, |Ay|)
// -- the 2D list with the z pair appended; spatial z streams with Ay and the
// sweep's z term uses Omega_y.
//
// One energy step n is one kernel (pt_step_kernel of pn_tiles.cuh): the beam
// inflow at energy[n] (csd.S[n-1]) formed where it is read, the upwind sweep of
// the interior cells in x, y and z, psi <- (psi - dE flux) / (1 + dE sigma_0),
// uTilde = u - dE sum_d (L_d u) A_d, collision (1 + dE D)^{-1}, in-scattering dE
// Dvec (MReduced psi), boundary rows zero, and the dose with csd.SMid. The
// whole sweep is captured once into a CUDA graph and launched as one unit.
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

constexpr int P3_NT = 256;
constexpr int P3_NOP = 6;
// Largest moment count taken: P64. It is the interface's, not the kernels' (titus_pn_full.cu).
constexpr int P3_MAX_MOMENTS = 4266;

// 4 x 2 x 8 cells, 56 operator tiles a stage, two CTAs a SM: as many tiles as fit beside
// the stencil coefficients and the larger halo in shared memory (64^3, P13: 1667 us a
// step with 48 tiles, 1584 with 64 and the coefficients in registers, 1538 so).
using Shape3D = titus_pn::PtShape<3, 1, 4, 2, 56, 2>;

}  // namespace

struct titus_pn3_state {
    double *u[2] = {nullptr, nullptr}, *psi[2] = {nullptr, nullptr}, *dose = nullptr;
    PtArgs args{};
    titus_pn::PtLayout layout;
    int32_t* col_of = nullptr;
    int cur_u = 0, cur_psi = 0;
    int steps_done = 0;
    bool have_result = false;
    cudaStream_t cap = nullptr;
    cudaGraphExec_t exec = nullptr;
    int exec_n_end = -1;
    std::vector<void*> allocs;
    ~titus_pn3_state() {
        if (exec) cudaGraphExecDestroy(exec);
        for (void* p : allocs) cudaFree(p);
        if (cap) cudaStreamDestroy(cap);
    }
};

namespace {

struct P3Alloc {
    titus_pn3_state* st;
    template <class T>
    int operator()(T** p, size_t count, const T* host = nullptr) const {
        int rc = titus_host::upload(p, host, count);
        if (rc == TITUS_OK && *p) st->allocs.push_back((void*)*p);
        return rc;
    }
};

int pn3_build(titus_solver* s, titus_pn3_state* st) {
    const P3Alloc alloc{st};
    const Csr dev[P3_NOP] = {s->P.op[0], s->P.op[1], s->P.op[2], s->P.op[3], s->op3[0], s->op3[1]};
    std::vector<titus_pn::HostCsr> ops(P3_NOP);
    int rc;
    for (int d = 0; d < P3_NOP; ++d)
        if ((rc = titus_pn::download_csr(dev[d], s->N, ops[d]))) return rc;
    std::vector<double> mred;
    if ((rc = titus_pn::download_mred(s, mred))) return rc;
    st->layout = titus_pn::pt_layout(ops, {false, false, true, true, false, true}, s->N, Shape3D::NT);
    if ((rc = titus_pn::pt_common(s, st->layout, st->args, st->col_of, alloc))) return rc;
    titus_pn::pt_patches<Shape3D>(ops, s->num_sms, st->args);
    if ((rc = titus_pn::pt_operator_tables<Shape3D>(ops, false, s->N, st->layout, mred, s->q, st->args, alloc))) return rc;
    const size_t nL = (size_t)s->n * st->layout.ldu;
    if ((rc = alloc(&st->u[0], nL)) || (rc = alloc(&st->u[1], nL)) || (rc = alloc(&st->psi[0], (size_t)s->n * QM)) ||
        (rc = alloc(&st->psi[1], (size_t)s->n * QM)) || (rc = alloc(&st->dose, (size_t)s->n)) ||
        (rc = titus_pn::pt_prepare<Shape3D, 0>()))
        return rc;
    CK(cudaStreamCreateWithFlags(&st->cap, cudaStreamNonBlocking));
    return TITUS_OK;
}

int pn3_ensure(titus_solver* s) {
    if (s->pn3) return TITUS_OK;
    if (!s->smid) return fail(TITUS_ERR_ARG, "the full-rank P_N solver needs problem->stopping_mid (csd.SMid)");
    if ((long long)s->n * s->q >= (1LL << 31)) return fail(TITUS_ERR_LIMIT, "n * q >= 2^31");
    if (s->N > P3_MAX_MOMENTS)
        return fail(TITUS_ERR_LIMIT, "N = %d moments exceed the 3D solver's limit of %d", s->N, P3_MAX_MOMENTS);
    auto* st = new titus_pn3_state();
    const int rc = pn3_build(s, st);
    if (rc) {
        delete st;
        return rc;
    }
    s->pn3 = st;
    return TITUS_OK;
}

}  // namespace

void titus_host::pn3_free(titus_solver* s) {
    delete s->pn3;
    s->pn3 = nullptr;
}

int titus_host::pn3_solve_device(titus_solver* s, const titus_options_t* opt, cudaStream_t stream) {
    int rc = pn3_ensure(s);
    if (rc) return rc;
    titus_pn3_state* st = s->pn3;
    const size_t nL = (size_t)s->n * st->layout.ldu;
    int n_end = s->nE;
    if (opt && opt->max_steps > 0) n_end = std::min(n_end, 1 + opt->max_steps);
    // both u buffers: the steps write interior rows only
    CK(cudaMemsetAsync(st->u[0], 0, nL * sizeof(double), stream));
    CK(cudaMemsetAsync(st->u[1], 0, nL * sizeof(double), stream));
    CK(cudaMemsetAsync(st->psi[0], 0, (size_t)s->n * QM * sizeof(double), stream));
    CK(cudaMemsetAsync(st->dose, 0, (size_t)s->n * sizeof(double), stream));
    const int par_end = (n_end - 1) & 1;
    if (st->exec && st->exec_n_end == n_end) {
        CK(cudaGraphLaunch(st->exec, stream));
    } else {
        if (st->exec) {
            CK(cudaStreamSynchronize(stream));   // the old graph may still be running
            cudaGraphExecDestroy(st->exec);
            st->exec = nullptr;
            st->exec_n_end = -1;
        }
        CK(cudaStreamBeginCapture(st->cap, cudaStreamCaptureModeThreadLocal));
        int cu = 0;
        for (int n = 2; n <= n_end; ++n) {
            titus_pn::pt_step<Shape3D, 0>(st->args, n, st->u[cu], nullptr, st->psi[cu], st->psi[cu ^ 1],
                                          st->u[cu ^ 1], st->dose, nullptr, st->cap);
            cu ^= 1;
        }
        if (n_end >= 2)
            titus_pn::pt_psi_boundary_kernel<3><<<(int)(((size_t)s->n * s->q + P3_NT - 1) / P3_NT), P3_NT, 0, st->cap>>>(
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
        CK(cudaGraphLaunch(exec, stream));
    }
    st->cur_u = par_end;
    st->cur_psi = par_end;
    st->steps_done = n_end - 1;
    st->have_result = true;
    return TITUS_OK;
}

int titus_host::pn3_fetch(titus_solver* s, double* u_out, double* dose_out, double* psi_out) {
    if (!s->pn3 || !s->pn3->have_result) return fail(TITUS_ERR_ARG, "no full-rank solve has run on this handle");
    titus_pn3_state* st = s->pn3;
    CK(cudaDeviceSynchronize());
    CK(cudaGetLastError());
    if (u_out) {
        // moment order in the buffer that the last step read (n x ldu >= n x N)
        double* tmp = st->u[st->cur_u ^ 1];
        titus_pn::pt_unpack_kernel<<<s->num_sms * 8, P3_NT>>>(s->n, s->N, st->layout.ldu, st->col_of,
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
