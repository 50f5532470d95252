// One explicit step of the full-rank P_N solvers (2D: titus_pn_full.cu, 3D:
// titus_pn3d.cu) as a block-sparse FP64 matrix product:
//
//   u'[c, :] = collide( u[c, :] + sum_d (L_d u)[c, :] A_d )
//
// The stencils L_d act on cells and the P_N matrices A_d on moments, so the
// step is one contraction over (operator, moment) whose left operand is formed
// from neighbouring rows of u where it is read and whose right operand is the
// same for every cell.
//
// Moment order. The Roe matrices |A_d| are dense inside the eight parity
// classes of the spherical harmonics (109 of 900 entries per row at P29) and
// zero between them, and A_d maps a class to one other. The columns of u are
// stored class by class (the connected components of the |A_d|, found from
// their CSR), inside a class by (|k|, l); an 8-column output tile then meets few
// 4-row input tiles that hold anything: 41 of 232 per operator at P29, 25 of 56
// at P13 in 3D (all operators together). Only those tiles are stored and
// multiplied. Any other sparsity pattern gives a longer list, not a different
// result.
//
// Work split. A CTA owns a patch of 64 interior cells (8 consecutive j times 8
// neighbouring lines) and one group of up to NT output tiles; a warp keeps the
// accumulators of its line in registers over the whole contraction. The CTA
// walks chunks of 16 input columns: the patch's rows and the faces of its halo,
// the chunk's operator tiles and its program arrive by cp.async in a two-stage
// ring. Axis by axis a warp forms the two stencil images of its line in shared
// memory (private to the warp) and executes the program's runs: one run is a
// slice of the accumulators (a quad or half of one) and the four-column steps
// whose tiles hold anything there, so no test is made per tile. Nothing n x N
// besides u and u' goes through memory, and there is no second pass: the
// ordinates psi' of the patch, the in-scattering (the same runs with psi' for
// images and MReduced for tiles, first), the collision and the dose are formed
// in the same kernel.
//
// What bounds it: the FP64 tensor pipe at 47 % busy (200 x 200, P29), the rest the
// latency of image and tile loads between the products with 16 warps a SM; memory
// takes a tenth of the time. Two tiles per warp in m (fewer instructions, 8 warps)
// was slower, as was a mask test per tile. Device time a step, CSR walks before ->
// now: 200 x 200 P29 7399 -> 1086 us, 64^3 P13 5149 -> 1538 us.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <numeric>
#include <utility>
#include <vector>

#include "titus_handle.h"

namespace titus_pn {

constexpr int PT_KC = 16;                 // input columns per chunk
constexpr int PT_LD = PT_KC + 4;          // row stride of a staged chunk (doubles): the 4 x 8 bytes of
                                          // four neighbouring rows fall in different banks
constexpr int PT_STAGES = 2;
constexpr int PT_MAXQ = 4;                // accumulator quads of a group

// Program of a chunk: per image (2 * axis + 0: central, + 1: second difference;
// 6: ordinates) one word with a four-bit k-mask per accumulator quad; bit k
// stands for the image columns 4 k .. 4 k + 3. Tiles follow in the order image,
// quad, k.
struct PtProgram {
    uint16_t runs[8];
};
constexpr int PT_PROG = 16;   // bytes of a program

struct PtChunk {
    int col0;       // first input column, -1: in-scattering
    int n16;        // 16-byte pieces of its tiles; the chunks of a group follow one another
};
constexpr int PT_PSI = 256;   // program word 7: 0 or PT_PSI + s, the ordinates 16 s .. 16 s + 15
struct PtGroup {
    int slot_tile[PT_MAXQ];    // first 8-column output tile of each accumulator quad
    int slot_width[PT_MAXQ];   // tiles of the quad (0: unused)
    int chunk0, nchunks;
    int tile0;                 // first packed operator tile
    int npsi;                  // the first npsi chunks form the in-scattering
    int m0;                    // accumulator tile of moment 0 (4 * quad + tile), -1: in another group
};

// Device tables of one direction (forward: A_d, adjoint: A_d^T).
struct PtTables {
    const PtGroup* group;
    const PtChunk* chunk;
    const PtProgram* prog;   // one per chunk
    const double* tile;   // packed tiles, 32 doubles in B-fragment lane order
    int ngroups;
};

struct PtArgs {
    int nx, ny, nz, nxy, n, ldu, q, npn, nE;
    int px, py, pz;           // patches per axis
    double dx, dy, dz, dE;
    double h[3], h2[3];       // -1 / (2 d), 1 / d along x, y, z
    const double* rinv;       // n
    const double* smid;       // nE - 1
    const double* bc_space;   // n
    const double* bc_angle;   // q
    const double* omega;      // q x 3
    const double* ordw;       // 3 x q: Omega_x / dx, Omega_z / dy, Omega_y / dz (2D: 0)
    const double* inflow;     // nE: PsiBeam's energy factor of step n at [n - 1]
    const double* sigma;      // nE x (npn+1)
    const double* mred;       // N x q
    const int32_t* lofp;      // ldu: Legendre order of the column's moment (0 for padding)
    const int32_t* momp;      // ldu: moment of the column (-1 for padding)
    int col_m0;               // column of moment 0
    PtTables t;
    // small problems: the operators as one merged list per output column
    int small;                // > 0: pt_small_kernel with that many fours of cells per CTA
    const int32_t* sp;        // ldu + 1
    const int32_t* si;        // image * ldu + input column
    const double* sv;
};

template <int DIM>
__device__ __forceinline__ bool pt_bnd(const PtArgs& a, int c) {
    const int k = DIM == 3 ? c / a.nxy : 0, r = DIM == 3 ? c - k * a.nxy : c;
    const int i = r / a.ny, j = r - i * a.ny;
    if (DIM == 3 && (k == 0 || k == a.nz - 1)) return true;
    return i == 0 || i == a.nx - 1 || j == 0 || j == a.ny - 1;
}

// psi' of the boundary cells, which only the final result needs: the inflow, without flux.
template <int DIM>
__global__ void pt_psi_boundary_kernel(PtArgs a, int n, double* __restrict__ psi_out) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= a.n * a.q) return;
    const int c = e / a.q, k = e - c * a.q;
    if (!pt_bnd<DIM>(a, c)) return;
    const double sig0 = a.sigma[(size_t)(n - 1) * (a.npn + 1)];
    psi_out[(size_t)c * titus::QM + k] = a.inflow[n - 1] * a.bc_space[c] * a.bc_angle[k] / (1.0 + a.dE * sig0);
}

// u (n x N, moment order) from the stored columns.
static __global__ void pt_unpack_kernel(int n, int N, int ldu, const int32_t* __restrict__ col_of,
                                        const double* __restrict__ u, double* __restrict__ out) {
    const size_t total = (size_t)n * N;
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
        const size_t c = e / N;
        out[e] = u[c * ldu + __ldg(col_of + (e - c * N))];
    }
}

__device__ __forceinline__ void pt_cp16(void* smem, const void* gmem) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void pt_mma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

// Shape of a CTA: eight warps, each one line of 8 cells along j, the lines
// arranged LZ x LX (3D) or 1 x LX (2D); TMAX operator tiles a stage.
template <int DIM_, int MT_, int LZ_, int LX_, int TMAX_, int CTAS_>
struct PtShape {
    static constexpr int DIM = DIM_, MT = MT_, LZ = LZ_, LX = LX_, TMAX = TMAX_, CTAS = CTAS_;
    static constexpr int LINES = LZ * LX, WARPS = LINES / MT, NTHR = 32 * WARPS, NT = 4 * PT_MAXQ;
    // staged rows: the patch, then the two x, y and z faces
    static constexpr int XF = 8 * LINES, YF = XF + 2 * LZ * 8, ZF = YF + 2 * LINES;
    static constexpr int ROWS = ZF + (DIM == 3 ? 2 * LX * 8 : 0);
    static constexpr int STAGE = ROWS * PT_LD + TMAX * 32 + PT_PROG / 8;   // doubles
    static constexpr int IMG = MT * 8 * PT_LD;                             // one image of a warp
    static constexpr int COEF = 3 * DIM * 8 * LINES;                       // stencil coefficients of the patch
    static constexpr int COLS = 3 * 8 * NT + NT / 2 + COEF;                // column, tile and cell constants
    static constexpr size_t SMEM = (PT_STAGES * (size_t)STAGE + WARPS * 2 * IMG + COLS) * sizeof(double);
    static constexpr int RSLOTS = (ROWS * (PT_KC / 2) + NTHR - 1) / NTHR;
    static constexpr int TSLOTS = (TMAX * 16 + NTHR - 1) / NTHR;
    static_assert(CTAS * (SMEM + 1024) <= 228 * 1024, "shared memory of an SM");
};

// The products of one run: a quad of the accumulators. Two neighbouring tiles
// are stored interleaved, so that one 16-byte load serves both.
template <int MT>
__device__ __forceinline__ void pt_run(double (&acc)[MT][4][2], unsigned mask, const double2*& bs,
                                       const double* img) {
    auto step = [&](int k) {
        double af[MT];
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) af[mt] = img[mt * 8 * PT_LD + 4 * k];
        const double2 b0 = bs[0], b1 = bs[32];
        bs += 64;
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
            pt_mma(acc[mt][0], af[mt], b0.x);
            pt_mma(acc[mt][1], af[mt], b0.y);
            pt_mma(acc[mt][2], af[mt], b1.x);
            pt_mma(acc[mt][3], af[mt], b1.y);
        }
    };
    if (mask == 15) {
#pragma unroll
        for (int k = 0; k < 4; ++k) step(k);
    } else {
        for (; mask; mask &= mask - 1) step(__ffs((int)mask) - 1);
    }
}
// The runs of one image: word w holds the k-masks of quads 0..3, four bits each.
template <int MT>
__device__ __forceinline__ void pt_runs(double (&acc)[PT_MAXQ][MT][4][2], unsigned w, const double2*& bs,
                                        const double* img) {
#pragma unroll
    for (int q = 0; q < PT_MAXQ; ++q)
        if (w >> 4 * q & 15) pt_run(acc[q], w >> 4 * q & 15, bs, img);
}

// psi' = (psi - dE flux) / (1 + dE sigma_0) of ordinate k in the interior cell c =
// (i, j(, kz)): the upwind sweep (SolverCSD.jl:541-545); boundary neighbours hold the inflow.
template <int DIM>
__device__ __forceinline__ double pt_psi_new(const PtArgs& a, int n, double den, const double* __restrict__ psi_in,
                                             int c, int i, int j, int kz, int k) {
    const double bc = __ldg(a.inflow + n - 1), ang = __ldg(a.bc_angle + k);
    auto val = [&](int off, bool bnd) {
        return bnd ? bc * __ldg(a.bc_space + c + off) * ang : __ldg(psi_in + (size_t)(c + off) * titus::QM + k);
    };
    const double pc = __ldg(psi_in + (size_t)c * titus::QM + k);
    const double wx = __ldg(a.ordw + k), wy = __ldg(a.ordw + a.q + k);
    double flux = wx * (wx >= 0.0 ? pc - val(-a.ny, i == 1) : val(a.ny, i == a.nx - 2) - pc) +
                  wy * (wy >= 0.0 ? pc - val(-1, j == 1) : val(1, j == a.ny - 2) - pc);
    if (DIM == 3) {
        const double wz = __ldg(a.ordw + 2 * a.q + k);
        flux += wz * (wz >= 0.0 ? pc - val(-a.nxy, kz == 1) : val(a.nxy, kz == a.nz - 2) - pc);
    }
    return (pc - a.dE * flux) / den;
}

// ADJ = 0: u_out = the step above from u = src. dose[c] += its increment.
// ADJ = 1: src = mu, the adjoint state divided by the collision factor; with the
//   transposed operators and stencils this forms lambda' = mu - dE sum_d (L_d^T mu) A_d^T,
//   accumulates dJ/drho_c = dE / rho_c sum_d (L_d^T mu A_d^T)[c] . u[c] (the
//   operator sum of lambda' against the forward state `fwd`, one partial per column
//   group in acc_out[g * n + c]) and writes mu of step n - 1 to u_out.
template <class S, int ADJ>
__global__ void __launch_bounds__(S::NTHR, S::CTAS)
    pt_step_kernel(PtArgs a, int n, const double* __restrict__ src, const double* __restrict__ fwd,
                   const double* __restrict__ psi_in, double* __restrict__ psi_out, double* __restrict__ u_out,
                   double* __restrict__ acc_out, const double* __restrict__ g) {
    constexpr int DIM = S::DIM, NT = S::NT, MT = S::MT;
    extern __shared__ __align__(16) double pt_smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double* img = pt_smem + PT_STAGES * S::STAGE + warp * 2 * S::IMG;
    double* fac = pt_smem + PT_STAGES * S::STAGE + S::WARPS * 2 * S::IMG;   // per output column
    double* coef = fac + 3 * 8 * NT;   // [axis][minus, centre, plus][cell], -dE folded in
    int* tcol = reinterpret_cast<int*>(coef + S::COEF);   // first column of a tile, -1: unused
    const int ngr = a.t.ngroups;
    const int gi = blockIdx.x % ngr, patch = blockIdx.x / ngr;
    const PtGroup* grp = a.t.group + gi;
    const int chunk0 = __ldg(&grp->chunk0), nchunks = __ldg(&grp->nchunks);
    // patch origin (interior cells start at index 1 on every axis)
    const int pj = patch % a.py, pr = patch / a.py;
    const int pi = DIM == 3 ? pr % a.px : pr, pk = DIM == 3 ? pr / a.px : 0;
    const int j0 = 1 + pj * 8, i0 = 1 + pi * S::LX, k0 = DIM == 3 ? 1 + pk * S::LZ : 0;

    // staged rows of this thread: each 16-byte column pair it copies (NULL: none)
    const double* rowp[S::RSLOTS];
#pragma unroll
    for (int s = 0; s < S::RSLOTS; ++s) {
        const int row = (tid + s * S::NTHR) >> 3;
        int lj, lx, lz = 0;
        if (row < S::XF) {
            lj = row & 7;
            lx = (row >> 3) % S::LX;
            lz = (row >> 3) / S::LX;
        } else if (row < S::YF) {
            const int f = row - S::XF;
            lx = f < S::LZ * 8 ? -1 : S::LX;
            lj = f & 7;
            lz = (f >> 3) % S::LZ;
        } else if (row < S::ZF) {
            const int f = row - S::YF;
            lj = f < S::LINES ? -1 : 8;
            lx = f % S::LINES % S::LX;
            lz = f % S::LINES / S::LX;
        } else {
            const int f = row - S::ZF;
            lz = f < S::LX * 8 ? -1 : S::LZ;
            lj = f & 7;
            lx = (f >> 3) % S::LX;
        }
        const int j = j0 + lj, i = i0 + lx, k = DIM == 3 ? k0 + lz : 0;
        // a row outside the grid is read by no interior cell
        const bool in = row < S::ROWS && j < a.ny && i < a.nx && (DIM == 2 || k < a.nz);
        rowp[s] = in ? src + (size_t)((k * a.nx + i) * a.ny + j) * a.ldu + (tid & 7) * 2 : nullptr;
    }
    const int2* chunk = reinterpret_cast<const int2*>(a.t.chunk) + chunk0;
    const double* tilep = a.t.tile + (size_t)__ldg(&grp->tile0) * 32 + tid * 2;
    auto issue = [&](int ci, int2 cd) {
        double* us = pt_smem + (ci % PT_STAGES) * S::STAGE;
        double* bs = us + S::ROWS * PT_LD + tid * 2;
        if (cd.x >= 0) {
            double* dp = us + (tid >> 3) * PT_LD + (tid & 7) * 2;
#pragma unroll
            for (int s = 0; s < S::RSLOTS; ++s)
                if (rowp[s]) pt_cp16(dp + s * (S::NTHR / 8) * PT_LD, rowp[s] + cd.x);
        }
#pragma unroll
        for (int s = 0; s < S::TSLOTS; ++s)
            if (tid + s * S::NTHR < cd.y) pt_cp16(bs + s * S::NTHR * 2, tilep + s * S::NTHR * 2);
        tilep += cd.y * 2;
        if (tid == 0) pt_cp16(us + S::ROWS * PT_LD + S::TMAX * 32, a.t.prog + chunk0 + ci);
    };
    const int2 none{-1, 0};
    if (nchunks > 0) issue(0, __ldg(chunk));
    asm volatile("cp.async.commit_group;" ::: "memory");
    int2 next = nchunks > 1 ? __ldg(chunk + 1) : none;   // read a chunk ahead of its copies

    const double* sg = a.sigma + (size_t)(n - 1) * (a.npn + 1);
    const double sig0 = __ldg(sg);
    const double dE = a.dE;
    // column constants: the in-scattering factor dE Dvec and 1 / (1 + dE D) (adjoint: of step n - 1) as the sum
    // of two doubles, since the rounding of one would add up in the same direction step after step (6e-16
    // against 2.9e-16 after 40 steps at P29)
    for (int e = tid; e < 8 * NT; e += S::NTHR) {
        const int q = e >> 5, t = (e >> 3) & 3;
        double f = 0.0, r = 0.0, rl = 0.0;
        if (t < __ldg(&grp->slot_width[q])) {
            const int l = __ldg(a.lofp + (__ldg(&grp->slot_tile[q]) + t) * 8 + (e & 7));
            const double* s1 = ADJ ? sg - (n > 2 ? a.npn + 1 : 0) : sg;
            f = dE * __ldg(s1 + l);
            const double den = 1.0 + dE * (__ldg(s1) - __ldg(s1 + l));
            r = 1.0 / den;
            rl = r * fma(-r, den, 1.0);
        }
        fac[e] = f;
        fac[8 * NT + e] = r;
        fac[16 * NT + e] = rl;
    }
    if (tid < NT) tcol[tid] = tid % 4 < __ldg(&grp->slot_width[tid / 4]) ? (__ldg(&grp->slot_tile[tid / 4]) + tid % 4) * 8 : -1;
    for (int e = tid; e < 8 * S::LINES; e += S::NTHR) {
        const int line = e >> 3, j = j0 + (e & 7), i = i0 + line % S::LX, k = DIM == 3 ? k0 + line / S::LX : 0;
        const bool in = j < a.ny - 1 && i < a.nx - 1 && (DIM == 2 || k < a.nz - 1);
        const double* rc = a.rinv + (in ? (k * a.nx + i) * a.ny + j : 0);
        const int off[3] = {in && !ADJ ? a.ny : 0, in && !ADJ ? 1 : 0, in && !ADJ ? a.nxy : 0};
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            coef[(3 * d) * 8 * S::LINES + e] = -dE * (a.h[d] * __ldg(rc - off[d]));
            coef[(3 * d + 1) * 8 * S::LINES + e] = -dE * (a.h2[d] * __ldg(rc));
            coef[(3 * d + 2) * 8 * S::LINES + e] = -dE * (a.h[d] * __ldg(rc + off[d]));
        }
    }
    // this lane's cells, their rows in the stage and the rows of their neighbours
    const int lj = lane >> 2, kl = lane & 3, cj = j0 + lj;
    bool live[MT];
    int cell[MT], oc[MT], oxm[MT], oxp[MT], oym[MT], oyp[MT], ozm[MT], ozp[MT];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
        const int line = warp * MT + mt, lx = line % S::LX, lz = line / S::LX;
        const int ci = i0 + lx, ck = DIM == 3 ? k0 + lz : 0, r0 = line * 8 + lj;
        live[mt] = cj < a.ny - 1 && ci < a.nx - 1 && (DIM == 2 || ck < a.nz - 1);
        cell[mt] = live[mt] ? (ck * a.nx + ci) * a.ny + cj : 0;
        oc[mt] = r0 * PT_LD + kl;
        oxm[mt] = (lx > 0 ? r0 - 8 : S::XF + lz * 8 + lj) * PT_LD + kl;
        oxp[mt] = (lx < S::LX - 1 ? r0 + 8 : S::XF + (S::LZ + lz) * 8 + lj) * PT_LD + kl;
        oym[mt] = (lj > 0 ? r0 - 1 : S::YF + line) * PT_LD + kl;
        oyp[mt] = (lj < 7 ? r0 + 1 : S::YF + S::LINES + line) * PT_LD + kl;
        ozm[mt] = ozp[mt] = 0;
        if (DIM == 3) {
            ozm[mt] = (lz > 0 ? r0 - 8 * S::LX : S::ZF + lx * 8 + lj) * PT_LD + kl;
            ozp[mt] = (lz < S::LZ - 1 ? r0 + 8 * S::LX : S::ZF + (S::LX + lx) * 8 + lj) * PT_LD + kl;
        }
    }
    const int npsi = ADJ ? 0 : __ldg(&grp->npsi);
    const int m0t = __ldg(&grp->m0);
    const bool m0lane = (a.col_m0 & 7) >> 1 == kl, m0odd = a.col_m0 & 1;
    double unc[MT];   // MReduced[0,:] psi' on the lane that holds moment 0
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) unc[mt] = 0.0;

    double acc[NT / 4][MT][4][2];
#pragma unroll
    for (int q = 0; q < NT / 4; ++q)
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int t = 0; t < 4; ++t) acc[q][mt][t][0] = acc[q][mt][t][1] = 0.0;

    double* im = img + lj * PT_LD + kl;   // this lane's element of an 8-row, 4-column fragment
    for (int ci = 0; ci < nchunks; ++ci) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();   // chunk ci is here, and no warp reads the stage of chunk ci - 1 any more
        if (ci + 1 < nchunks) issue(ci + 1, next);
        asm volatile("cp.async.commit_group;" ::: "memory");
        next = ci + 2 < nchunks ? __ldg(chunk + ci + 2) : none;
        const double* us = pt_smem + (ci % PT_STAGES) * S::STAGE;
        const double2* bs = reinterpret_cast<const double2*>(us + S::ROWS * PT_LD) + lane;
        const uint4 prg = *reinterpret_cast<const uint4*>(us + S::ROWS * PT_LD + S::TMAX * 32);
        const int kind = __shfl_sync(0xffffffffu, prg.w >> 16, 0);
        const unsigned px = __shfl_sync(0xffffffffu, prg.x, 0), py = __shfl_sync(0xffffffffu, prg.y, 0),
                       pz = __shfl_sync(0xffffffffu, prg.z, 0), pw = __shfl_sync(0xffffffffu, prg.w, 0) & 0xffff;
        if (ADJ || kind < PT_PSI) {
            // the adjoint's central differences change sign, the second differences are symmetric
            auto axis = [&](unsigned nc, unsigned ns, int d, const int(&om)[MT], const int(&op)[MT]) {
                if ((nc | ns) == 0) return;
#pragma unroll
                for (int mt = 0; mt < MT; ++mt) {
                    const double* cf = coef + 3 * d * 8 * S::LINES + (warp * MT + mt) * 8 + lj;
                    const double cm = cf[0], cc = cf[8 * S::LINES], cp = cf[16 * S::LINES];
                    double* dst = im + mt * 8 * PT_LD;
                    if (ns == 0) {
#pragma unroll
                        for (int k = 0; k < PT_KC / 4; ++k) {
                            const double lo = cm * us[om[mt] + 4 * k], hi = cp * us[op[mt] + 4 * k];
                            dst[4 * k] = ADJ ? hi - lo : lo - hi;
                        }
                    } else {
#pragma unroll
                        for (int k = 0; k < PT_KC / 4; ++k) {
                            const double lo = cm * us[om[mt] + 4 * k], hi = cp * us[op[mt] + 4 * k];
                            dst[4 * k] = ADJ ? hi - lo : lo - hi;
                            dst[S::IMG + 4 * k] = fma(cc, us[oc[mt] + 4 * k], lo + hi);
                        }
                    }
                }
                __syncwarp();
                pt_runs(acc, nc, bs, im);
                pt_runs(acc, ns, bs, im + S::IMG);
                __syncwarp();   // the next images overwrite these
            };
            axis(px & 0xffff, px >> 16, 0, oxm, oxp);
            axis(py & 0xffff, py >> 16, 1, oym, oyp);
            if (DIM == 3) axis(pz & 0xffff, pz >> 16, 2, ozm, ozp);
        } else {
            const double den = 1.0 + dE * sig0;
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) {
                const int line = warp * MT + mt, ix = i0 + line % S::LX, iz = k0 + line / S::LX, c = cell[mt];
#pragma unroll 1
                for (int k4 = 0; k4 < PT_KC / 4; ++k4) {
                    const int k = (kind - PT_PSI) * PT_KC + 4 * k4 + kl;
                    double v = 0.0;
                    if (k < a.q && live[mt]) {
                        v = pt_psi_new<DIM>(a, n, den, psi_in, c, ix, cj, iz, k);
                        if (gi == 0) psi_out[(size_t)c * titus::QM + k] = v;
                    }
                    im[mt * 8 * PT_LD + 4 * k4] = v;
                }
            }
            __syncwarp();
            pt_runs(acc, pw, bs, im);
            __syncwarp();
            if (ci == npsi - 1) {
                // dE Dvec (MReduced psi')
#pragma unroll
                for (int t = 0; t < NT; ++t) {
                    const double2 f = *reinterpret_cast<const double2*>(fac + t * 8 + 2 * kl);
#pragma unroll
                    for (int mt = 0; mt < MT; ++mt) {
                        double(&x)[2] = acc[t / 4][mt][t % 4];
                        if (t == m0t) unc[mt] = m0odd ? x[1] : x[0];
                        x[0] *= f.x;
                        x[1] *= f.y;
                    }
                }
            }
        }
    }

    // the column constants come from other threads: the chunk loop's barriers order them, unless no operator
    // has an entry in these columns (an adjoint group without chunks)
    if (nchunks == 0) __syncthreads();
    // epilogue: lane holds columns 2 kl + {0, 1} of every tile for its cells
    double dcell[MT];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) dcell[mt] = 0.0;
#pragma unroll
    for (int t = 0; t < NT; ++t) {
        if (tcol[t] >= 0) {
            const int col = tcol[t] + 2 * kl;
            const double2 r = *reinterpret_cast<const double2*>(fac + 8 * NT + t * 8 + 2 * kl),
                          rl = *reinterpret_cast<const double2*>(fac + 16 * NT + t * 8 + 2 * kl);
            const bool m0 = t == m0t && m0lane;
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) {
                if (!live[mt]) continue;
                const size_t ix = (size_t)cell[mt] * a.ldu + col;
                const double2 uc = __ldg(reinterpret_cast<const double2*>(src + ix));
                const double(&x)[2] = acc[t / 4][mt][t % 4];
                double2 out{uc.x + x[0], uc.y + x[1]};
                if (ADJ) {
                    const double2 f = __ldg(reinterpret_cast<const double2*>(fwd + ix));
                    dcell[mt] = fma(x[0], f.x, dcell[mt]);
                    dcell[mt] = fma(x[1], f.y, dcell[mt]);
                    if (m0 && n > 2) {   // mu of step n - 1: its dose term
                        const double half = n - 1 == 2 ? 2.0 : 1.0;
                        const double add = g[cell[mt]] * (dE * a.smid[n - 3] / half) * a.rinv[cell[mt]];
                        (m0odd ? out.y : out.x) += add;
                    }
                }
                out.x = fma(out.x, r.x, out.x * rl.x);
                out.y = fma(out.y, r.y, out.y * rl.y);
                if (!ADJ && m0) {
                    const double half = (n == 2 || n == a.nE) ? 2.0 : 1.0;
                    acc_out[cell[mt]] += dE * ((m0odd ? out.y : out.x) + unc[mt]) * a.smid[n - 2] *
                                         a.rinv[cell[mt]] / half;
                }
                *reinterpret_cast<double2*>(u_out + ix) = out;
            }
        }
    }
    if (ADJ) {
        // the four lanes of a cell hold disjoint columns; acc carries -dE of the sum
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
            double v = dcell[mt];
            v += __shfl_xor_sync(0xffffffffu, v, 1);
            v += __shfl_xor_sync(0xffffffffu, v, 2);
            if (live[mt] && kl == 0) acc_out[(size_t)gi * a.n + cell[mt]] -= __ldg(a.rinv + cell[mt]) * v;
        }
    }
}

// The same step for problems that leave most of the chip idle: with a patch per
// CTA they give tens of CTAs, each with a chain of ten and more chunks. Here a
// CTA forms all images of four cells (of several fours where the columns leave
// threads over) in shared memory, and a thread walks the merged nonzeros of one
// column for four cells. A step at 50 x 50 takes 10.0 us at P7 (19.3 tiled), 15.4
// at P9 (28.3). The work is one shared load per nonzero and two cells, so the
// tiled kernel is ahead from about PS_WORK nonzeros over all cells on (100 x 100,
// P7: 27 us and 26; 80 x 80, P9: 36 and 28; 120 x 120, P7: 34 and 27; 24^3, P5: 31
// and 28; 100 x 100, P13: 166 and 73).
constexpr int PS_CELLS = 4, PS_NT = 128, PS_MAXG = 8;
constexpr int PS_SMEM_MAX = 96 * 1024;          // images of a CTA
constexpr long long PS_WORK = 10 * 1000 * 1000;
template <int DIM, int ADJ>
__global__ void __launch_bounds__(PS_NT)
    pt_small_kernel(PtArgs a, int n, const double* __restrict__ src, const double* __restrict__ fwd,
                    const double* __restrict__ psi_in, double* __restrict__ psi_out, double* __restrict__ u_out,
                    double* __restrict__ acc_out, const double* __restrict__ g) {
    extern __shared__ __align__(16) double pt_smem[];   // [four][image][column][cell]
    __shared__ double psis[PS_MAXG * PS_CELLS][titus::QM];
    __shared__ double red[PS_NT][PS_CELLS];
    __shared__ double coef[PS_MAXG * PS_CELLS][3 * DIM];
    __shared__ int cells[PS_MAXG * PS_CELLS], ijk[PS_MAXG * PS_CELLS][3];
    const int tid = threadIdx.x, ldu = a.ldu, nf = a.small;
    const int iy = a.ny - 2, ix = a.nx - 2, total = iy * ix * (DIM == 3 ? a.nz - 2 : 1);
    const int first = blockIdx.x * PS_CELLS * nf, nc = min(PS_CELLS * nf, total - first);
    const double* sg = a.sigma + (size_t)(n - 1) * (a.npn + 1);
    const double dE = a.dE;
    // this thread's four cells, first column and list, read ahead of their use
    const int f = nf > 1 ? tid / ldu : 0, colf = nf > 1 ? tid - f * ldu : tid;
    int e0 = 0, e1 = 0, m = -1;
    double sl = 0.0, s0 = 0.0;
    const double* s1 = ADJ ? sg - (n > 2 ? a.npn + 1 : 0) : sg;
    auto column = [&](int col) {
        e0 = __ldg(a.sp + col);
        e1 = __ldg(a.sp + col + 1);
        m = __ldg(a.momp + col);
        sl = __ldg(s1 + __ldg(a.lofp + col));
        s0 = __ldg(s1);
    };
    if (f < nf && colf < ldu) column(colf);
    if (tid < nc) {
        const int e = first + tid, r = e / iy;
        const int j = 1 + e - r * iy, i = 1 + (DIM == 3 ? r % ix : r), k = DIM == 3 ? 1 + r / ix : 0;
        const int c = (k * a.nx + i) * a.ny + j;
        cells[tid] = c;
        ijk[tid][0] = i;
        ijk[tid][1] = j;
        ijk[tid][2] = k;
        const double r0 = __ldg(a.rinv + c);
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            const int off = ADJ ? 0 : d == 0 ? a.ny : d == 1 ? 1 : a.nxy;
            coef[tid][3 * d] = -dE * (a.h[d] * __ldg(a.rinv + c - off));
            coef[tid][3 * d + 1] = -dE * (a.h2[d] * r0);
            coef[tid][3 * d + 2] = -dE * (a.h[d] * __ldg(a.rinv + c + off));
        }
    }
    __syncthreads();
    // images, the cells of a column side by side (cells beyond the grid stay unused)
    for (int e = tid; e < nc * ldu; e += PS_NT) {
        const int cl = e / ldu, col = e - cl * ldu;
        const double* row = src + (size_t)cells[cl] * ldu + col;
        double* dst = pt_smem + ((size_t)(cl / PS_CELLS) * 2 * DIM * ldu + col) * PS_CELLS + cl % PS_CELLS;
        const double u0 = __ldg(row);
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            const ptrdiff_t off = (ptrdiff_t)(d == 0 ? a.ny : d == 1 ? 1 : a.nxy) * ldu;
            const double lo = coef[cl][3 * d] * __ldg(row - off), hi = coef[cl][3 * d + 2] * __ldg(row + off);
            dst[(size_t)(2 * d) * ldu * PS_CELLS] = ADJ ? hi - lo : lo - hi;
            dst[(size_t)(2 * d + 1) * ldu * PS_CELLS] = fma(coef[cl][3 * d + 1], u0, lo + hi);
        }
    }
    if (!ADJ)
        for (int e = tid; e < nc * a.q; e += PS_NT) {
            const int cl = e / a.q, k = e - cl * a.q;
            const double v = pt_psi_new<DIM>(a, n, 1.0 + dE * __ldg(sg), psi_in, cells[cl], ijk[cl][0], ijk[cl][1],
                                             ijk[cl][2], k);
            psi_out[(size_t)cells[cl] * titus::QM + k] = v;
            psis[cl][k] = v;
        }
    __syncthreads();
    double dcell[PS_CELLS];
#pragma unroll
    for (int cl = 0; cl < PS_CELLS; ++cl) dcell[cl] = 0.0;
    if (f < nf) {
        const int base = f * PS_CELLS;
        const double2* img = reinterpret_cast<const double2*>(pt_smem) + (size_t)f * 2 * DIM * ldu * (PS_CELLS / 2);
        for (int col = colf; col < ldu; col += nf > 1 ? ldu : PS_NT) {
            if (col != colf) column(col);
            double acc[PS_CELLS], sc[PS_CELLS];
#pragma unroll
            for (int cl = 0; cl < PS_CELLS; ++cl) acc[cl] = sc[cl] = 0.0;
#pragma unroll 8
            for (int e = e0; e < e1; ++e) {
                const double v = __ldg(a.sv + e);
                const double2* im = img + (size_t)__ldg(a.si + e) * (PS_CELLS / 2);
#pragma unroll
                for (int h = 0; h < PS_CELLS / 2; ++h) {
                    const double2 x = im[h];
                    acc[2 * h] = fma(v, x.x, acc[2 * h]);
                    acc[2 * h + 1] = fma(v, x.y, acc[2 * h + 1]);
                }
            }
            if (!ADJ && m >= 0)
#pragma unroll 4
                for (int k = 0; k < a.q; ++k) {
                    const double w = __ldg(a.mred + (size_t)m * a.q + k);
#pragma unroll
                    for (int cl = 0; cl < PS_CELLS; ++cl) sc[cl] = fma(w, psis[base + cl][k], sc[cl]);
                }
            const double dv = dE * sl, den = 1.0 + dE * (s0 - sl);
#pragma unroll
            for (int cl = 0; cl < PS_CELLS; ++cl) {
                if (base + cl >= nc) break;
                const int c = cells[base + cl];
                const size_t at = (size_t)c * ldu + col;
                double out = __ldg(src + at) + acc[cl];
                if (ADJ) {
                    dcell[cl] = fma(acc[cl], __ldg(fwd + at), dcell[cl]);
                    if (col == a.col_m0 && n > 2) {
                        const double half = n - 1 == 2 ? 2.0 : 1.0;
                        out += g[c] * (dE * a.smid[n - 3] / half) * a.rinv[c];
                    }
                } else {
                    out += dv * sc[cl];
                }
                out /= den;
                u_out[at] = out;
                if (!ADJ && col == a.col_m0) {
                    const double half = (n == 2 || n == a.nE) ? 2.0 : 1.0;
                    acc_out[c] += dE * (out + sc[cl]) * a.smid[n - 2] * a.rinv[c] / half;
                }
            }
        }
    }
    if (ADJ) {
        // the threads' column sums, in thread order
#pragma unroll
        for (int cl = 0; cl < PS_CELLS; ++cl) red[tid][cl] = dcell[cl];
        __syncthreads();
        if (tid < nc) {
            const int t0 = nf > 1 ? tid / PS_CELLS * ldu : 0, t1 = nf > 1 ? t0 + ldu : PS_NT;
            double t = 0.0;
            for (int w = t0; w < t1; ++w) t += red[w][tid % PS_CELLS];
            acc_out[cells[tid]] -= __ldg(a.rinv + cells[tid]) * t;
        }
    }
}

// ------------------------------------------------------------------ host ---

// CSR of one operator on the host (row p, column m).
struct HostCsr {
    std::vector<int32_t> rp, ci;
    std::vector<double> v;
};

inline int download_csr(const titus::Csr& op, int N, HostCsr& h) {
    h.rp.resize(N + 1);
    CK(cudaMemcpy(h.rp.data(), op.rowptr, (N + 1) * sizeof(int32_t), cudaMemcpyDeviceToHost));
    const int nnz = h.rp[N];
    h.ci.resize(nnz);
    h.v.resize(nnz);
    if (nnz) {
        CK(cudaMemcpy(h.ci.data(), op.col, nnz * sizeof(int32_t), cudaMemcpyDeviceToHost));
        CK(cudaMemcpy(h.v.data(), op.val, nnz * sizeof(double), cudaMemcpyDeviceToHost));
    }
    return TITUS_OK;
}

// Column order of the stored moments.
struct PtLayout {
    int ldu = 0;
    std::vector<int32_t> col_of;      // N: column of a moment
    std::vector<int32_t> moment_of;   // ldu: moment of a column, -1 for padding
    std::vector<PtGroup> groups;      // chunk fields unset
};

// Classes = connected components of the |A| patterns (`roe` marks them in ops);
// each padded to whole 8-column tiles while that costs at most a fifth, packed
// first-fit by decreasing size into groups of up to `nt` tiles.
inline PtLayout pt_layout(const std::vector<HostCsr>& ops, const std::vector<bool>& roe, int N, int nt) {
    std::vector<int> root(N);
    std::iota(root.begin(), root.end(), 0);
    auto find = [&](int x) {
        while (root[x] != x) x = root[x] = root[root[x]];
        return x;
    };
    for (size_t d = 0; d < ops.size(); ++d)
        if (roe[d])
            for (int p = 0; p < N; ++p)
                for (int e = ops[d].rp[p]; e < ops[d].rp[p + 1]; ++e) root[find(p)] = find(ops[d].ci[e]);
    std::vector<std::vector<int>> cls;
    std::vector<int> id(N, -1);
    for (int m = 0; m < N; ++m) {
        const int f = find(m);
        if (id[f] < 0) {
            id[f] = (int)cls.size();
            cls.emplace_back();
        }
        cls[id[f]].push_back(m);
    }
    for (auto& c : cls)
        std::sort(c.begin(), c.end(), [](int x, int y) {
            const int lx = (int)std::sqrt((double)x), ly = (int)std::sqrt((double)y);
            const int kx = std::abs(x - lx * lx - lx), ky = std::abs(y - ly * ly - ly);
            return kx != ky ? kx < ky : x < y;
        });
    PtLayout L;
    L.col_of.assign(N, 0);
    const int nq = nt / 4;
    // groups over the tile range [t0, t0 + n): evenly split, quads side by side
    auto quads = [&](int t0, int n) {
        const int parts = (n + nt - 1) / nt;
        for (int s = 0; s < parts; ++s) {
            const int b0 = t0 + n * s / parts, b1 = t0 + n * (s + 1) / parts;
            PtGroup g{};
            for (int t = b0, q = 0; t < b1; t += 4, ++q) {
                g.slot_tile[q] = t;
                g.slot_width[q] = std::min(4, b1 - t);
            }
            L.groups.push_back(g);
        }
    };
    long long padded = 0;
    for (auto& c : cls) padded += (c.size() + 7) / 8 * 8;
    if (padded * 5 <= (long long)N * 6) {
        std::vector<int> order(cls.size());
        std::iota(order.begin(), order.end(), 0);
        std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return cls[x].size() > cls[y].size(); });
        std::vector<std::vector<int>> bins;
        std::vector<int> fill;
        for (int o : order) {
            const int tiles = (int)(cls[o].size() + 7) / 8;
            size_t b = 0;
            while (b < bins.size() && fill[b] + tiles > nt) ++b;
            if (b == bins.size()) {
                bins.emplace_back();
                fill.push_back(0);
            }
            bins[b].push_back(o);
            fill[b] += tiles;
        }
        for (size_t b = 0; b < bins.size(); ++b) {
            const int tile0 = (int)L.moment_of.size() / 8;
            int need = 0;
            for (int o : bins[b]) {
                for (int m : cls[o]) L.moment_of.push_back(m);
                while (L.moment_of.size() % 8) L.moment_of.push_back(-1);
                need += ((int)(cls[o].size() + 7) / 8 + 3) / 4;
            }
            if (need <= nq) {   // every class starts a quad of its own
                PtGroup g{};
                int t = tile0, q = 0;
                for (int o : bins[b])
                    for (int left = (int)(cls[o].size() + 7) / 8; left > 0; left -= 4, ++q) {
                        g.slot_tile[q] = t;
                        g.slot_width[q] = std::min(4, left);
                        t += g.slot_width[q];
                    }
                L.groups.push_back(g);
            } else {
                quads(tile0, fill[b]);
            }
        }
    } else {
        for (auto& c : cls)
            for (int m : c) L.moment_of.push_back(m);
        while (L.moment_of.size() % 8) L.moment_of.push_back(-1);
        quads(0, (int)L.moment_of.size() / 8);
    }
    // whole 16-column chunks
    while (L.moment_of.size() % PT_KC) L.moment_of.push_back(-1);
    L.ldu = (int)L.moment_of.size();
    for (int c = 0; c < L.ldu; ++c)
        if (L.moment_of[c] >= 0) L.col_of[L.moment_of[c]] = c;
    return L;
}

struct PtHostTables {
    std::vector<PtGroup> group;
    std::vector<PtChunk> chunk;
    std::vector<PtProgram> prog;
    std::vector<double> tile;
};

// Chunks, programs and packed tiles of out = sum_d img_d A_d (or A_d^T) in the
// layout's column order; `tmax` tiles fit a stage. Operators in the order L2x,
// L2y, L1x, L1y(, L2z, L1z). The forward tables start with the in-scattering
// (`mred`: N x q_ord).
inline PtHostTables pt_tables(const std::vector<HostCsr>& ops, bool transpose, int N, const PtLayout& L, int tmax,
                              const std::vector<double>& mred, int q_ord) {
    PtHostTables T;
    const int nk4 = L.ldu / 4, nn8 = L.ldu / 8, nops = (int)ops.size();
    // image (2 * axis + form of difference) of an operator
    const int image_of[6] = {0, 2, 1, 3, 4, 5};
    // (op, k4, n8) -> packed values
    std::vector<std::vector<int>> slot(nops, std::vector<int>((size_t)nk4 * nn8, -1));
    std::vector<double> vals;
    for (int d = 0; d < nops; ++d)
        for (int p = 0; p < N; ++p)
            for (int e = ops[d].rp[p]; e < ops[d].rp[p + 1]; ++e) {
                if (ops[d].v[e] == 0.0) continue;
                const int k = L.col_of[transpose ? ops[d].ci[e] : p], m = L.col_of[transpose ? p : ops[d].ci[e]];
                int& s = slot[d][(size_t)(k / 4) * nn8 + m / 8];
                if (s < 0) {
                    s = (int)(vals.size() / 32);
                    vals.resize(vals.size() + 32, 0.0);
                }
                // B fragment of mma.m8n8k4: lane 4 * column + row
                vals[(size_t)s * 32 + (m % 8) * 4 + k % 4] += ops[d].v[e];
            }
    // two tiles, interleaved lane by lane; get(t, lane) gives an element of tile t = 0, 1
    auto store_pair = [&](auto get) {
        for (int lane = 0; lane < 32; ++lane)
            for (int t = 0; t < 2; ++t) T.tile.push_back(get(t, lane));
    };
    struct Run {
        int image, op, q;
        unsigned kmask;
    };
    for (PtGroup g : L.groups) {
        g.chunk0 = (int)T.chunk.size();
        g.tile0 = (int)(T.tile.size() / 32);
        g.m0 = -1;
        for (int q = 0; q < PT_MAXQ; ++q)
            for (int t = 0; t < g.slot_width[q]; ++t)
                if (L.col_of[0] / 8 == g.slot_tile[q] + t) g.m0 = 4 * q + t;
        int nq = 0;
        while (nq < PT_MAXQ && g.slot_width[nq] > 0) ++nq;
        for (int k0 = 0; !transpose && k0 < q_ord;) {
            // as many four-ordinate steps a chunk as its stage holds
            const int kend = std::min({q_ord, k0 / PT_KC * PT_KC + PT_KC, k0 + tmax / (4 * nq) * 4});
            PtProgram pr{};
            const int tile0 = (int)(T.tile.size() / 32);
            unsigned kmask = 0;
            for (int k = k0; k < kend; k += 4) kmask |= 1u << (k % PT_KC / 4);
            for (int q = 0; q < nq; ++q) {
                pr.runs[6] |= (uint16_t)(kmask << 4 * q);
                for (int k = k0; k < kend; k += 4)
                    for (int h = 0; h < 4; h += 2)
                        store_pair([&](int t, int lane) {
                            const bool in = h + t < g.slot_width[q];
                            const int m = in ? L.moment_of[(g.slot_tile[q] + h + t) * 8 + lane / 4] : -1;
                            const int kk = k + lane % 4;
                            return m >= 0 && kk < q_ord ? mred[(size_t)m * q_ord + kk] : 0.0;
                        });
            }
            pr.runs[7] = (uint16_t)(PT_PSI + k0 / PT_KC);
            T.chunk.push_back(PtChunk{-1, 16 * ((int)(T.tile.size() / 32) - tile0)});
            T.prog.push_back(pr);
            ++g.npsi;
            k0 = kend;
        }
        for (int col0 = 0; col0 < L.ldu; col0 += PT_KC) {
            std::vector<Run> todo;
            for (int d = 0; d < nops; ++d)
                for (int q = 0; q < nq; ++q) {
                    unsigned kmask = 0;
                    for (int k = 0; k < PT_KC / 4; ++k)
                        for (int t = 0; t < g.slot_width[q]; ++t)
                            if (slot[d][(size_t)(col0 / 4 + k) * nn8 + g.slot_tile[q] + t] >= 0) kmask |= 1u << k;
                    if (kmask) todo.push_back(Run{image_of[d], d, q, kmask});
                }
            std::stable_sort(todo.begin(), todo.end(), [](const Run& x, const Run& y) { return x.image < y.image; });
            // as many runs a chunk as its stage holds tiles for (the columns come again for the rest)
            for (size_t b = 0; b < todo.size();) {
                PtProgram pr{};
                const int tile0 = (int)(T.tile.size() / 32);
                int tiles = 0;
                for (; b < todo.size() && tiles + 4 * __builtin_popcount(todo[b].kmask) <= tmax; ++b) {
                    const Run& x = todo[b];
                    pr.runs[x.image] |= (uint16_t)(x.kmask << 4 * x.q);
                    for (int k = 0; k < PT_KC / 4; ++k)
                        if (x.kmask >> k & 1)
                            for (int h = 0; h < 4; h += 2)
                                store_pair([&](int t, int lane) {
                                    const int sl = h + t < g.slot_width[x.q]
                                                       ? slot[x.op][(size_t)(col0 / 4 + k) * nn8 + g.slot_tile[x.q] + h + t]
                                                       : -1;
                                    return sl >= 0 ? vals[(size_t)sl * 32 + lane] : 0.0;
                                });
                    tiles = (int)(T.tile.size() / 32) - tile0;
                }
                T.chunk.push_back(PtChunk{col0, 16 * tiles});
                T.prog.push_back(pr);
            }
        }
        g.nchunks = (int)T.chunk.size() - g.chunk0;
        T.group.push_back(g);
    }
    return T;
}

// Uploads a table set; `alloc(ptr, count, host)` returns a status and owns the memory.
template <class Alloc>
int pt_upload(const PtHostTables& T, PtTables& t, Alloc alloc) {
    PtGroup* gr = nullptr;
    PtChunk* ch = nullptr;
    PtProgram* pg = nullptr;
    double* tl = nullptr;
    int rc;
    if ((rc = alloc(&gr, T.group.size(), T.group.data())) || (rc = alloc(&ch, T.chunk.size(), T.chunk.data())) ||
        (rc = alloc(&pg, T.prog.size(), T.prog.data())) || (rc = alloc(&tl, T.tile.size(), T.tile.data())))
        return rc;
    t = PtTables{gr, ch, pg, tl, (int)T.group.size()};
    return TITUS_OK;
}

// Kernel arguments shared by the 2D and 3D solvers, with the column-ordered copy
// of the Legendre orders.
template <class Alloc>
int pt_common(const titus_solver* s, const PtLayout& L, PtArgs& a, int32_t*& d_col_of, Alloc alloc) {
    const titus::DevProblem& P = s->P;
    a = PtArgs{};
    a.nx = P.nx;
    a.ny = P.ny;
    a.nz = s->nz;
    a.nxy = P.nx * P.ny;
    a.n = P.n;
    a.ldu = L.ldu;
    a.q = P.q;
    a.npn = P.npn;
    a.nE = P.nE;
    a.dx = P.dx;
    a.dy = P.dy;
    a.dz = s->dz;
    a.dE = P.dE;
    a.rinv = P.rinv;
    a.smid = s->smid;
    a.bc_space = P.bc_space;
    a.bc_angle = P.bc_angle;
    a.omega = P.omega;
    a.sigma = P.sigma;
    a.mred = P.mred;
    a.col_m0 = L.col_of[0];
    std::vector<int32_t> lof(P.N), lofp(L.ldu, 0);
    CK(cudaMemcpy(lof.data(), P.lof, lof.size() * sizeof(int32_t), cudaMemcpyDeviceToHost));
    for (int m = 0; m < P.N; ++m) lofp[L.col_of[m]] = lof[m];
    const double d[3] = {P.dx, P.dy, s->nz ? s->dz : 1.0};
    for (int k = 0; k < 3; ++k) {
        a.h[k] = -1.0 / 2.0 / d[k];
        a.h2[k] = 2.0 / 2.0 / d[k];
    }
    std::vector<double> omega(3 * P.q), ordw(3 * P.q, 0.0), bce(P.nE), stop(P.nE), inflow(P.nE, 0.0);
    CK(cudaMemcpy(omega.data(), P.omega, omega.size() * sizeof(double), cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(bce.data(), P.bc_energy, bce.size() * sizeof(double), cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(stop.data(), P.stopping, stop.size() * sizeof(double), cudaMemcpyDeviceToHost));
    for (int k = 0; k < P.q; ++k) {
        ordw[k] = omega[3 * k] / P.dx;
        ordw[P.q + k] = omega[3 * k + 2] / P.dy;
        if (s->nz) ordw[2 * P.q + k] = omega[3 * k + 1] / s->dz;
    }
    // energy[n] with csd.S[n-1]; bc_energy holds scale exp(-sE (E0-E_k)^2) S_k rho_min
    for (int n = 2; n <= P.nE; ++n) inflow[n - 1] = bce[n - 1] / stop[n - 1] * stop[n - 2];
    int32_t *dl = nullptr, *dmo = nullptr;
    double *dow = nullptr, *din = nullptr;
    int rc;
    if ((rc = alloc(&dow, ordw.size(), ordw.data())) || (rc = alloc(&din, inflow.size(), inflow.data())) ||
        (rc = alloc(&dl, lofp.size(), lofp.data())) || (rc = alloc(&dmo, L.moment_of.size(), L.moment_of.data())) ||
        (rc = alloc(&d_col_of, L.col_of.size(), L.col_of.data())))
        return rc;
    a.lofp = dl;
    a.ordw = dow;
    a.inflow = din;
    a.momp = dmo;
    return TITUS_OK;
}

// MReduced (N x q) on the host.
inline int download_mred(const titus_solver* s, std::vector<double>& mred) {
    mred.resize((size_t)s->P.N * s->P.q);
    CK(cudaMemcpy(mred.data(), s->P.mred, mred.size() * sizeof(double), cudaMemcpyDeviceToHost));
    return TITUS_OK;
}

// The small kernel's merged lists (images in operator order within a column).
template <class Alloc>
int pt_small_tables(const std::vector<HostCsr>& ops, bool transpose, int N, const PtLayout& L, PtArgs& a, Alloc alloc) {
    const int image_of[6] = {0, 2, 1, 3, 4, 5};
    std::vector<std::vector<std::pair<int32_t, double>>> rows(L.ldu);
    for (size_t d = 0; d < ops.size(); ++d)
        for (int p = 0; p < N; ++p)
            for (int e = ops[d].rp[p]; e < ops[d].rp[p + 1]; ++e) {
                const int k = L.col_of[transpose ? ops[d].ci[e] : p], m = L.col_of[transpose ? p : ops[d].ci[e]];
                rows[m].emplace_back(image_of[d] * L.ldu + k, ops[d].v[e]);
            }
    std::vector<int32_t> sp(1, 0), si;
    std::vector<double> sv;
    for (auto& r : rows) {
        for (auto& e : r) {
            si.push_back(e.first);
            sv.push_back(e.second);
        }
        sp.push_back((int32_t)si.size());
    }
    int32_t *dp = nullptr, *di = nullptr;
    double* dv = nullptr;
    int rc;
    if ((rc = alloc(&dp, sp.size(), sp.data())) || (rc = alloc(&di, si.size(), si.data())) ||
        (rc = alloc(&dv, sv.size(), sv.data())))
        return rc;
    a.sp = dp;
    a.si = di;
    a.sv = dv;
    return TITUS_OK;
}

template <int DIM>
size_t pt_small_smem(int ldu, int fours) {
    return (size_t)fours * 2 * DIM * ldu * PS_CELLS * sizeof(double);
}

// Patches of the grid, and which kernel takes its steps.
template <class S>
void pt_patches(const std::vector<HostCsr>& ops, int num_sms, PtArgs& a) {
    auto cnt = [](int interior, int w) { return interior > 0 ? (interior + w - 1) / w : 0; };
    a.py = cnt(a.ny - 2, 8);
    a.px = cnt(a.nx - 2, S::LX);
    a.pz = S::DIM == 3 ? cnt(a.nz - 2, S::LZ) : 1;
    long long nnz = 0;
    for (const HostCsr& h : ops) nnz += (long long)h.v.size();
    const long long cells = (long long)std::max(0, a.ny - 2) * std::max(0, a.nx - 2) *
                            (S::DIM == 3 ? std::max(0, a.nz - 2) : 1);
    // fours of cells per CTA: as the columns leave threads over, but at least two CTAs per SM
    int fours = std::max(1, std::min(PS_MAXG, PS_NT / a.ldu));
    while (fours > 1 && cells < (long long)2 * num_sms * PS_CELLS * fours) --fours;
    a.small = cells * nnz <= PS_WORK && pt_small_smem<S::DIM>(a.ldu, fours) <= (size_t)PS_SMEM_MAX ? fours : 0;
}

// The tables of the kernel that takes the steps.
template <class S, class Alloc>
int pt_operator_tables(const std::vector<HostCsr>& ops, bool transpose, int N, const PtLayout& L,
                       const std::vector<double>& mred, int q, PtArgs& a, Alloc alloc) {
    if (a.small) {
        a.t = PtTables{};
        a.t.ngroups = 1;
        return pt_small_tables(ops, transpose, N, L, a, alloc);
    }
    return pt_upload(pt_tables(ops, transpose, N, L, S::TMAX, mred, q), a.t, alloc);
}

template <class S, int ADJ>
int pt_prepare() {
    CK(cudaFuncSetAttribute(pt_step_kernel<S, ADJ>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM));
    CK(cudaFuncSetAttribute(pt_small_kernel<S::DIM, ADJ>, cudaFuncAttributeMaxDynamicSharedMemorySize, PS_SMEM_MAX));
    return TITUS_OK;
}

template <class S, int ADJ>
void pt_step(const PtArgs& a, int n, const double* src, const double* fwd, const double* psi_in, double* psi_out,
             double* u_out, double* acc, const double* g, cudaStream_t st) {
    if (a.small) {
        const int cells = std::max(0, a.nx - 2) * std::max(0, a.ny - 2) * (S::DIM == 3 ? std::max(0, a.nz - 2) : 1);
        if (cells > 0)
            pt_small_kernel<S::DIM, ADJ><<<(cells + PS_CELLS * a.small - 1) / (PS_CELLS * a.small), PS_NT,
                                           pt_small_smem<S::DIM>(a.ldu, a.small), st>>>(a, n, src, fwd, psi_in, psi_out,
                                                                                       u_out, acc, g);
        return;
    }
    const int grid = a.px * a.py * a.pz * a.t.ngroups;
    if (grid > 0)
        pt_step_kernel<S, ADJ><<<grid, S::NTHR, S::SMEM, st>>>(a, n, src, fwd, psi_in, psi_out, u_out, acc, g);
}

}  // namespace titus_pn
