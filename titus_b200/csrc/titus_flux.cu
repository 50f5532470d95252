// Second-order limited upwind transport flux of the uncollided ordinates:
// solveFlux! (code/SolverCSD.jl:295-386) with its limiter helpers minmod and
// slopefit (:288-293), as the standalone C-ABI operator titus_limited_flux.
//
// Layout: phi and flux hold nx*ny*q doubles, cell (i, j) ordinate l at
// (i*ny + j)*q + l (the library's psi layout; i runs over x, j over y). The
// reference writes interior cells 2 <= i < nx-2, 2 <= j < ny-2 (1-based 3:N-2)
// and leaves the others as they were; so does this kernel.
//
// Each (cell, ordinate) needs the centre value and four neighbours per axis:
// offsets -2..+1 where the ordinate's component is >= 0, -1..+2 where it is
// negative. With the window shifted by one for negative components the two cases
// are one formula, so the lanes of a warp do not part. A thread owns kCells
// consecutive j of one ordinate and walks rows along x: each x face is formed
// once, each y face 1 + 1/kCells times, and the differences that neighbouring
// faces share are formed once. A warp reads 256 contiguous bytes per operand
// where q >= 32 and q * 8 byte pieces otherwise; DRAM sees phi once and flux
// once. The limiter arithmetic (limiter.cuh) keeps the reference's values, so the
// result is the same IEEE double as the FP64 restatement of the loop body.
#include <cuda_runtime.h>

#include <climits>
#include <cstdint>

#include "../../include/titus.h"
#include "limiter.cuh"

namespace titus_host {
int fail(int code, const char* fmt, ...);
}

namespace {

constexpr int kFluxThreads = 128;

// A thread's j cells, the rows of the x window in flight ahead of their use and
// the unrolling of the row loop. Without rows ahead the loop waited for one load
// from memory a row (468 us at 2048 x 2048 x 16, 65 % of the stalls); measured
// there with (cells, ahead, unroll): (2,1,1) 323, (2,3,2) 293, (4,1,1) 310,
// (4,2,1) 317, (4,3,1) 287, (4,3,2) 271, (4,4,2) 321 us of kernel; at 1024 x 1024 80 us.
// A call from Python among others takes 281 to 296 us at 2048 x 2048.
constexpr int kCells = 4, kAhead = 3, kUnroll = 2;

// Rows a thread walks: 32 where that leaves 150 000 threads, else as many fewer
// as it takes, down to 2. A row costs a chain of dependent loads and limiters of
// about a microsecond, so a small grid (100 x 100 x 12: 33 us with 32 rows) wants
// short walks; a long walk saves the two rows that start it.
constexpr long long kThreadsWanted = 150000;
int rows_per_thread(int nx, long long per_row) {
    const long long rows = (nx - 4) * per_row / kThreadsWanted;
    return rows >= 32 ? 32 : rows < 2 ? 2 : (int)rows;
}

// grid: x covers the (j group, ordinate) pairs of a row; y chunks of `rows`
// interior rows starting at row0 + rows * blockIdx.y.
__global__ void __launch_bounds__(kFluxThreads) limited_flux_kernel(int nx, int ny, int q, int row0, int rows,
                                                                    double dx, double dy,
                                                                    const double* __restrict__ ox,
                                                                    const double* __restrict__ oz,
                                                                    const double* __restrict__ phi,
                                                                    double* __restrict__ flux) {
    const int t = blockIdx.x * kFluxThreads + threadIdx.x;
    const int grp = t / q, l = t - grp * q;
    const int j0 = 2 + kCells * grp;
    if (j0 >= ny - 2) return;
    const int i0 = row0 + rows * (int)blockIdx.y;
    const int i1 = min(i0 + rows, nx - 2);
    if (i0 >= i1) return;
    const double wx = __ldg(ox + l), wz = __ldg(oz + l);
    // qReduced[q,1] / dx and qReduced[q,3] / dy, as the reference divides
    const double cx = __ddiv_rn(wx, dx), cz = __ddiv_rn(wz, dy);
    const bool px = wx >= 0.0, pz = wz >= 0.0;
    const size_t sx = (size_t)ny * q;
    // column offsets of the cells and of the y window (clamped: a group may reach past the grid)
    int jc[kCells], jw[kCells + 3];
#pragma unroll
    for (int c = 0; c < kCells; ++c) jc[c] = min(j0 + c, ny - 1) * q + l;
#pragma unroll
    for (int c = 0; c < kCells + 3; ++c) jw[c] = min(j0 + c - (pz ? 2 : 1), ny - 1) * q + l;
    // x window: rows r - 1, r of each cell with r = i (component >= 0) or i + 1, the doubled
    // difference across them and the face before
    const double* xr = phi + (size_t)(i0 + (px ? 0 : 1)) * sx;
    double e0[kCells], e1[kCells], d0[kCells], H[kCells];
#pragma unroll
    for (int c = 0; c < kCells; ++c) {
        const double em = __ldg(xr - 2 * sx + jc[c]);
        e0[c] = __ldg(xr - sx + jc[c]);
        e1[c] = __ldg(xr + jc[c]);
        d0[c] = titus_lim::twice_diff(e0[c], e1[c]);
        H[c] = titus_lim::face(em, e0[c], e1[c], titus_lim::twice_diff(em, e0[c]), d0[c], px);
    }
    const double* yr = phi + (size_t)i0 * sx;
    double* f = flux + (size_t)i0 * sx;
    // rows r + 1 .. r + kAhead of the x window, in flight while the rows before them are used; the walk's
    // last row r + 1 is the last one read
    double ahead[kAhead][kCells];
    const int last = i1 - i0;   // rows r + 1 that the walk needs
#pragma unroll
    for (int d = 0; d < kAhead; ++d)
#pragma unroll
        for (int c = 0; c < kCells; ++c) ahead[d][c] = d < last ? __ldg(xr + (size_t)(d + 1) * sx + jc[c]) : 0.0;
#pragma unroll kUnroll
    for (int i = i0; i < i1; ++i) {
        double e2[kCells], y[kCells + 3];
#pragma unroll
        for (int c = 0; c < kCells + 3; ++c) y[c] = __ldg(yr + jw[c]);
#pragma unroll
        for (int c = 0; c < kCells; ++c) {
            e2[c] = ahead[0][c];
#pragma unroll
            for (int d = 0; d + 1 < kAhead; ++d) ahead[d][c] = ahead[d + 1][c];
            ahead[kAhead - 1][c] = i + kAhead < i1 ? __ldg(xr + (size_t)(kAhead + 1) * sx + jc[c]) : 0.0;
        }
        double dp = titus_lim::twice_diff(y[0], y[1]), dn = titus_lim::twice_diff(y[1], y[2]);
        double below = titus_lim::face(y[0], y[1], y[2], dp, dn, pz);
#pragma unroll
        for (int c = 0; c < kCells; ++c) {
            dp = dn;
            dn = titus_lim::twice_diff(y[c + 2], y[c + 3]);
            const double above = titus_lim::face(y[c + 1], y[c + 2], y[c + 3], dp, dn, pz);
            const double ns = __dsub_rn(above, below);
            below = above;
            const double d1 = titus_lim::twice_diff(e1[c], e2[c]);
            const double Hn = titus_lim::face(e0[c], e1[c], e2[c], d0[c], d1, px);
            const double ew = __dsub_rn(Hn, H[c]);
            H[c] = Hn;
            d0[c] = d1;
            e0[c] = e1[c];
            e1[c] = e2[c];
            // qReduced[q,1] / dx * (east - west) + qReduced[q,3] / dy * (north - south)
            if (j0 + c < ny - 2) f[jc[c]] = __dadd_rn(__dmul_rn(cx, ew), __dmul_rn(cz, ns));
        }
        xr += sx;
        yr += sx;
        f += sx;
    }
}

}  // namespace

extern "C" int titus_limited_flux(int32_t nx, int32_t ny, int32_t q, double dx, double dy, const double* omega_x,
                                  const double* omega_z, const double* phi, double* flux, void* stream) {
    using titus_host::fail;
    if (nx < 0 || ny < 0 || q < 1) return fail(TITUS_ERR_ARG, "titus_limited_flux: nx=%d ny=%d q=%d", nx, ny, q);
    if (!(dx > 0.0) || !(dy > 0.0)) return fail(TITUS_ERR_ARG, "titus_limited_flux: dx, dy must be > 0");
    if (!omega_x || !omega_z || !phi || !flux) return fail(TITUS_ERR_ARG, "titus_limited_flux: NULL pointer");
    if (nx < 5 || ny < 5) return TITUS_OK;   // no interior cell
    const long long row = (long long)ny * q;
    if (row > INT_MAX - kFluxThreads) return fail(TITUS_ERR_LIMIT, "titus_limited_flux: ny*q = %lld too large", row);
    const double* pb = phi;
    const double* fb = flux;
    const size_t total = (size_t)nx * (size_t)row;
    if (pb < fb + total && fb < pb + total)
        return fail(TITUS_ERR_ARG, "titus_limited_flux: phi and flux overlap");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const long long per_row = (long long)((ny - 4 + kCells - 1) / kCells) * q;
    const unsigned gx = (unsigned)((per_row + kFluxThreads - 1) / kFluxThreads);
    const int rows = rows_per_thread(nx, per_row);
    const long long chunks = (nx - 4 + rows - 1) / rows;
    // at most 65535 row chunks per launch (grid y limit)
    for (long long c0 = 0; c0 < chunks; c0 += 65535) {
        const unsigned gy = (unsigned)((chunks - c0) < 65535 ? (chunks - c0) : 65535);
        limited_flux_kernel<<<dim3(gx, gy), kFluxThreads, 0, st>>>(nx, ny, q, 2 + (int)(c0 * rows), rows, dx, dy,
                                                                   omega_x, omega_z, phi, flux);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return fail(TITUS_ERR_CUDA, "titus_limited_flux: %s", cudaGetErrorString(e));
    }
    return TITUS_OK;
}
