// kmc_laplace.cu -- Laplace basis fields on the device.
//
// The potential of a network is a superposition of unit-voltage solutions
// of the Laplace problem on its mesh (init_V / update_V,
// kmc_dopant_networks.py:706-822, solve P1 elements with Dirichlet data on
// the whole boundary).  On the uniform right-triangle mesh the P1 system is
// the anisotropic 5-point stencil
//     (2cx + 2cy) u_ij - cx (u_i,j-1 + u_i,j+1) - cy (u_i-1,j + u_i+1,j) = 0,
// cx = hy/hx, cy = hx/hy, whose matrix cx (I ⊗ T_x) + cy (T_y ⊗ I), with
// T = tridiag(-1, 2, -1), is diagonalised by discrete sine transforms:
//     T_n = Q_n diag(lambda) Q_n,  Q_n[a][b] = sqrt(2/n) sin(pi (a+1)(b+1)/n),
//     lambda_b = 2 - 2 cos(pi (b+1)/n)   (n = cells, size n-1).
// So U = Q_y ((Q_y F Q_x) ./ (cx lambda_x + cy lambda_y)) Q_x, F the
// right-hand side carrying the boundary data: exact up to rounding (no
// iteration, no tolerance).  All fields of one mesh are solved in one batch;
// P1 sampling at the acceptors follows.  This replaces the per-geometry CPU
// solve when geometries churn (serving).
//
// F is zero but for the nodes beside the boundary, so its transform is four
// matrix-vector products a field (the sides' data) and four outer products.
// The inverse transform is the work: two products with Q a field, FP64, whose
// unit takes 64 cycles a warp instruction and SM quarter, spread over
// more blocks than the SMs hold at once.  Q itself is never stored: its entries are the 2n values
// sin(pi q/n), q = (k+1)(j+1) mod 2n, in shared memory.  (Half the products
// could be had from Q's mirror symmetry Q[k][m-1-j] = (-1)^k Q[k][j]; that
// moved the result by 7e-15, where this is within 1e-15 of the plain products.
// Against 113-bit arithmetic, 99 x 99 cells: rms error 1.60e-14 and 1.48e-14
// on two layouts, the plain products in FP64 1.60e-14 and 1.48e-14.)
// Four launches; 9 fields of 99 x 99 cells: 74 us (141 us in nine launches
// with Q and dense products in 16 x 16 tiles).
#include <cmath>
#include <cstdint>
#include <cuda_runtime.h>

#include "kmc_internal.h"

namespace kmc {
namespace {

constexpr int kSides = 4;              // left, right (along y), bottom, top (along x)
constexpr int kThreads = 128;
// Rows of a field per block of a product.  Few, so that even small meshes give
// blocks to every SM several times over, but a block's copy of the sine table
// (2n entries) is shared by its rows.  Kernels of 9 fields, us, at 3 / 4 / 6 /
// 8 / 12 rows: 30 cells a side 30 / 30 / 35 / 34 / 39, 99: 74 / 86 / 89 / 104
// / 137, 150: 142 / 183 / 180 / 237 / 242, 99 x 300: 252 / 296 / 329 / 382 /
// 518, 300: 934 / 981 / 903 / 1161 / 1190, 1000: 30 / 32 / 34 / 32 / 36 ms,
// 2000: 237 / 237 / 344 / 343 / 238 ms.
constexpr int kRows = 3;

// Per direction: sqrt(2/n) sin(pi q/n), q = 0 .. 2n-1, and the eigenvalues
// 2 - 2 cos(pi (k+1)/n).
struct Tables {
    double *sx, *sy, *lx, *ly;
};

__global__ void table_kernel(int nx, int ny, Tables t)
{
    const double pi = 3.14159265358979323846;
    const int total = 2 * nx + 2 * ny + (nx - 1) + (ny - 1);
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < total; k += gridDim.x * blockDim.x) {
        int q = k;
        if (q < 2 * nx) { t.sx[q] = sqrt(2.0 / nx) * sin(pi * static_cast<double>(q) / nx); continue; }
        q -= 2 * nx;
        if (q < 2 * ny) { t.sy[q] = sqrt(2.0 / ny) * sin(pi * static_cast<double>(q) / ny); continue; }
        q -= 2 * ny;
        if (q < nx - 1) { t.lx[q] = 2.0 - 2.0 * cos(pi * (q + 1) / nx); continue; }
        q -= nx - 1;
        t.ly[q] = 2.0 - 2.0 * cos(pi * (q + 1) / ny);
    }
}

// The table of n cells in shared memory, or (no room: very fine meshes) where
// it is.
__device__ __forceinline__ const double *staged(const double *tab, int n, double *sh)
{
    if (!sh) return tab;
    for (int q = threadIdx.x; q < 2 * n; q += blockDim.x) sh[q] = tab[q];
    return sh;
}

// (a * b) mod m for a, b < m
__device__ __forceinline__ int mulmod(int a, int b, int m)
{
    return static_cast<int>((static_cast<long long>(a) * b) % m);
}

// The transforms of the boundary data beside each side: G[f][side][l] =
// sum_i Q[l][i] g_i, a warp a value.
__global__ void __launch_bounds__(kThreads) side_kernel(int nx, int ny, int nf, Tables t, const double *grid,
                                                        double *G, int in_smem)
{
    extern __shared__ double sh[];
    const int f = blockIdx.z, side = blockIdx.y;
    const int n = side < 2 ? ny : nx, m = n - 1, stride = max(nx, ny) - 1;
    const double *g = grid + static_cast<long long>(f) * (ny + 1) * (nx + 1);
    const double *tab = staged(side < 2 ? t.sy : t.sx, n, in_smem ? sh : nullptr);
    // the side's interior nodes: data[i * step]
    const long long step = side < 2 ? nx + 1 : 1;
    const double *data = side == 0 ? g + nx + 1 : side == 1 ? g + nx + 1 + nx : side == 2 ? g + 1
                                                          : g + static_cast<long long>(ny) * (nx + 1) + 1;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    for (int l = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5); l < m; l += gridDim.x * (kThreads / 32)) {
        double acc = 0.0;
        int q = mulmod(l + 1, lane + 1, 2 * n);
        const int dq = mulmod(l + 1, 32, 2 * n);
        for (int i = lane; i < m; i += 32) {
            acc = fma(tab[q], data[i * step], acc);
            q += dq;
            if (q >= 2 * n) q -= 2 * n;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) G[(static_cast<long long>(f) * kSides + side) * stride + l] = acc;
    }
}

// kRows rows of in (a row of m values each) times Q of n = m + 1 cells: a
// thread a value.
template <typename Store>
__device__ __forceinline__ void rows_times_q(const double *in, int rows, int m, const double *tab, Store store)
{
    const int n2 = 2 * (m + 1);
    for (int it = threadIdx.x; it < rows * m; it += blockDim.x) {
        const int r = it / m, j = it - (it / m) * m;
        const double *v = in + r * m;
        double acc = 0.0;
        int q = j + 1;                      // (k+1)(j+1) mod 2n
#pragma unroll 4
        for (int k = 0; k < m; ++k) {
            acc = fma(v[k], tab[q], acc);
            q += j + 1;
            if (q >= n2) q -= n2;
        }
        store(r, j, acc);
    }
}

// Y = W Qx, W[l][k] the transformed right-hand side over the eigenvalues.
__global__ void __launch_bounds__(kThreads) x_kernel(int nx, int ny, double cx, double cy, Tables t, const double *G,
                                                     double *Y, double *W, int in_smem)
{
    extern __shared__ double sh[];
    const int f = blockIdx.y, mj = nx - 1, mi = ny - 1, stride = max(nx, ny) - 1;
    const int l0 = blockIdx.x * kRows, rows = min(kRows, mi - l0);
    const long long at = static_cast<long long>(f) * mi * mj;
    double *w = in_smem ? sh + 2 * nx : W + at + static_cast<long long>(l0) * mj;
    const double *tab = staged(t.sx, nx, in_smem ? sh : nullptr);
    const double *g = G + static_cast<long long>(f) * kSides * stride;
    for (int it = threadIdx.x; it < rows * mj; it += blockDim.x) {
        const int r = it / mj, k = it - (it / mj) * mj, l = l0 + r;
        // Qx[0][k], Qx[mj-1][k], Qy[l][0], Qy[l][mi-1]
        const double x0 = t.sx[k + 1], x1 = t.sx[mulmod(mj, k + 1, 2 * nx)];
        const double y0 = t.sy[l + 1], y1 = t.sy[mulmod(mi, l + 1, 2 * ny)];
        const double num = cx * (g[l] * x0 + g[stride + l] * x1) + cy * (g[2 * stride + k] * y0 + g[3 * stride + k] * y1);
        w[it] = num / (cx * t.lx[k] + cy * t.ly[l]);
    }
    __syncthreads();
    // transposed (j, l): the next product reads its rows
    double *out = Y + at;
    rows_times_q(w, rows, mj, tab, [&](int r, int j, double v) { out[static_cast<long long>(j) * mi + l0 + r] = v; });
}

// U = Qy Y into the interior of the nodal grids: columns of U are rows of the
// transposed Y times Qy (symmetric).
__global__ void __launch_bounds__(kThreads) y_kernel(int nx, int ny, Tables t, const double *Y, double *grid,
                                                     int in_smem)
{
    extern __shared__ double sh[];
    const int f = blockIdx.y, mj = nx - 1, mi = ny - 1;
    const int j0 = blockIdx.x * kRows, rows = min(kRows, mj - j0);
    const double *tab = staged(t.sy, ny, in_smem ? sh : nullptr);
    const double *w = Y + static_cast<long long>(f) * mi * mj + static_cast<long long>(j0) * mi;
    if (in_smem) {
        double *copy = sh + 2 * ny;
        for (int it = threadIdx.x; it < rows * mi; it += blockDim.x) copy[it] = w[it];
        w = copy;
        __syncthreads();
    }
    double *g = grid + static_cast<long long>(f) * (ny + 1) * (nx + 1);
    rows_times_q(w, rows, mi, tab,
                 [&](int r, int i, double v) { g[static_cast<long long>(i + 1) * (nx + 1) + j0 + r + 1] = v; });
}

// Boundary data of every basis field: field e < P is 1 on electrode e's
// nodes, field P on the rest of the boundary.  The node coordinates and
// comparisons are the host's (boundary_owner in laplace.py), operation for
// operation; interior nodes are set to 0.
__global__ void boundary_kernel(int nx, int ny, double hx, double hy, double xdim, double surplus, int P,
                                const double *xy, double *grid)
{
    const int nodes = (nx + 1) * (ny + 1);
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nodes; k += gridDim.x * blockDim.x) {
        const int i = k / (nx + 1), j = k - i * (nx + 1);
        const bool edge = i == 0 || j == 0 || i == ny || j == nx;
        int owner = P;
        if (edge) {
            const double x = __dmul_rn(static_cast<double>(j), hx), y = __dmul_rn(static_cast<double>(i), hy);
            for (int e = 0; e < P; ++e) {
                const double ex = xy[2 * e], ey = xy[2 * e + 1];
                const bool mine = (ex == 0 || ex == xdim)
                                      ? (x == ex && y >= __dsub_rn(ey, surplus) && y <= __dadd_rn(ey, surplus))
                                      : (x >= __dsub_rn(ex, surplus) && x <= __dadd_rn(ex, surplus) && y == ey);
                if (mine) { owner = e; break; }      // the first match wins
            }
        }
        for (int f = 0; f <= P; ++f) grid[static_cast<long long>(f) * nodes + k] = edge && owner == f ? 1.0 : 0.0;
    }
}

// P1 interpolation on the "right" diagonal triangulation (ix,iy)-(ix+1,iy+1).
__global__ void p1_sample_kernel(int nx, int ny, double hx, double hy, int nf, const double *grid,
                                 int np, const double *xy, double *out)
{
    for (long long k = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
         k < static_cast<long long>(np) * nf; k += static_cast<long long>(gridDim.x) * blockDim.x) {
        const int f = static_cast<int>(k / np), p = static_cast<int>(k - static_cast<long long>(f) * np);
        const double sx = xy[2 * p] / hx, sy = xy[2 * p + 1] / hy;
        int ix = static_cast<int>(floor(sx)), iy = static_cast<int>(floor(sy));
        ix = ix < 0 ? 0 : (ix > nx - 1 ? nx - 1 : ix);
        iy = iy < 0 ? 0 : (iy > ny - 1 ? ny - 1 : iy);
        const double xi = sx - ix, eta = sy - iy;
        const double *g = grid + static_cast<long long>(f) * (ny + 1) * (nx + 1);
        const double f00 = g[iy * (nx + 1) + ix], f10 = g[iy * (nx + 1) + ix + 1];
        const double f01 = g[(iy + 1) * (nx + 1) + ix], f11 = g[(iy + 1) * (nx + 1) + ix + 1];
        out[k] = (xi >= eta) ? f00 + xi * (f10 - f00) + eta * (f11 - f10)
                             : f00 + eta * (f01 - f00) + xi * (f11 - f01);
    }
}

template <typename K>
int allow_smem(K *kernel, size_t smem)
{
    if (smem <= 48 * 1024) return KMC_OK;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               static_cast<int>(smem));
    return e == cudaSuccess ? KMC_OK : fail_cuda(e, "laplace_basis: shared memory");
}

int grid_for(long long n)
{
    const long long b = (n + 255) / 256;
    return static_cast<int>(b < 1 ? 1 : (b > 4096 ? 4096 : b));
}

// Doubles of workspace: Y, the sides' transforms, the transformed right-hand
// side where a block's rows do not fit its shared memory (0: they do), tables.
struct LaplaceSpace {
    size_t fields, sides, copy, tables;
};
LaplaceSpace laplace_space(int nx, int ny, int nf)
{
    const size_t mi = ny - 1, mj = nx - 1, longest = nx > ny ? nx : ny;
    LaplaceSpace s;
    s.fields = mi * mj * nf;
    s.sides = kSides * (longest - 1) * nf;
    s.copy = sizeof(double) * (kRows + 2) * longest > 200 * 1024 ? s.fields : 0;
    s.tables = 2 * (static_cast<size_t>(nx) + ny) + mi + mj;
    return s;
}

}  // namespace
}  // namespace kmc

using namespace kmc;

extern "C" size_t kmc_laplace_workspace_size(int32_t nx, int32_t ny, int32_t n_fields)
{
    if (nx < 2 || ny < 2 || n_fields < 1) return 0;
    const LaplaceSpace s = laplace_space(nx, ny, n_fields);
    return sizeof(double) * (s.fields + s.sides + s.copy + s.tables);
}

extern "C" int kmc_laplace_basis(int32_t nx, int32_t ny, double hx, double hy, int32_t n_fields,
                                 double *grid, void *workspace, size_t workspace_bytes, void *stream)
{
    if (nx < 2 || ny < 2 || n_fields < 1 || !(hx > 0) || !(hy > 0))
        return fail(KMC_ERR_INVALID, "laplace_basis: bad mesh (nx %d, ny %d, fields %d)", nx, ny, n_fields);
    if (!grid || !workspace) return fail(KMC_ERR_INVALID, "laplace_basis: NULL pointer");
    if (workspace_bytes < kmc_laplace_workspace_size(nx, ny, n_fields))
        return fail(KMC_ERR_INVALID, "laplace_basis: workspace too small");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int mi = ny - 1, mj = nx - 1;
    const LaplaceSpace sp = laplace_space(nx, ny, n_fields);
    double *ws = static_cast<double *>(workspace);
    double *Y = ws, *G = Y + sp.fields, *W = G + sp.sides, *tab = W + sp.copy;
    const Tables t{tab, tab + 2 * nx, tab + 2 * nx + 2 * ny, tab + 2 * nx + 2 * ny + mj};
    const double cx = hy / hx, cy = hx / hy;
    const int longest = nx > ny ? nx : ny, in_smem = sp.copy == 0;
    const size_t smem_side = in_smem ? sizeof(double) * 2 * longest : 0;
    const size_t smem_x = in_smem ? sizeof(double) * (2 * static_cast<size_t>(nx) + static_cast<size_t>(kRows) * mj) : 0;
    const size_t smem_y = in_smem ? sizeof(double) * (2 * static_cast<size_t>(ny) + static_cast<size_t>(kRows) * mi) : 0;
    int rc;
    if ((rc = allow_smem(side_kernel, smem_side)) != KMC_OK || (rc = allow_smem(x_kernel, smem_x)) != KMC_OK ||
        (rc = allow_smem(y_kernel, smem_y)) != KMC_OK)
        return rc;
    table_kernel<<<grid_for(3LL * (nx + ny)), 128, 0, st>>>(nx, ny, t);
    side_kernel<<<dim3((longest + 7) / 8, kSides, n_fields), kThreads, smem_side, st>>>(nx, ny, n_fields, t, grid, G, in_smem);
    x_kernel<<<dim3((mi + kRows - 1) / kRows, n_fields), kThreads, smem_x, st>>>(nx, ny, cx, cy, t, G, Y, W, in_smem);
    y_kernel<<<dim3((mj + kRows - 1) / kRows, n_fields), kThreads, smem_y, st>>>(nx, ny, t, Y, grid, in_smem);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? KMC_OK : fail_cuda(e, "laplace_basis launch");
}

extern "C" int kmc_laplace_boundary(int32_t nx, int32_t ny, double xdim, double ydim, double surplus,
                                    int32_t n_electrodes, const double *xy, double *grid, void *stream)
{
    if (nx < 1 || ny < 1 || n_electrodes < 0 || !(xdim > 0) || !(ydim > 0))
        return fail(KMC_ERR_INVALID, "laplace_boundary: bad mesh (nx %d, ny %d, electrodes %d)", nx, ny, n_electrodes);
    if (!grid || (!xy && n_electrodes > 0)) return fail(KMC_ERR_INVALID, "laplace_boundary: NULL pointer");
    const long long nodes = static_cast<long long>(nx + 1) * (ny + 1);
    if (nodes > (1LL << 30)) return fail(KMC_ERR_INVALID, "laplace_boundary: mesh too large");
    boundary_kernel<<<grid_for(nodes), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        nx, ny, xdim / nx, ydim / ny, xdim, surplus, n_electrodes, xy, grid);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? KMC_OK : fail_cuda(e, "laplace_boundary launch");
}

extern "C" int kmc_p1_sample(int32_t nx, int32_t ny, double hx, double hy, int32_t n_fields,
                             const double *grid, int32_t n_points, const double *xy, double *out,
                             void *stream)
{
    if (nx < 1 || ny < 1 || n_fields < 1 || n_points < 0 || !(hx > 0) || !(hy > 0))
        return fail(KMC_ERR_INVALID, "p1_sample: bad sizes");
    if (n_points == 0) return KMC_OK;
    if (!grid || !xy || !out) return fail(KMC_ERR_INVALID, "p1_sample: NULL pointer");
    const long long tot = static_cast<long long>(n_points) * n_fields;
    p1_sample_kernel<<<grid_for(tot), 256, 0, static_cast<cudaStream_t>(stream)>>>(nx, ny, hx, hy, n_fields,
                                                                                 grid, n_points, xy, out);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? KMC_OK : fail_cuda(e, "p1_sample launch");
}

namespace kmc {

int preload_laplace()
{
    int rc;
    if ((rc = touch_kernel(table_kernel)) != KMC_OK) return rc;
    if ((rc = touch_kernel(side_kernel)) != KMC_OK) return rc;
    if ((rc = touch_kernel(x_kernel)) != KMC_OK) return rc;
    if ((rc = touch_kernel(y_kernel)) != KMC_OK) return rc;
    if ((rc = touch_kernel(boundary_kernel)) != KMC_OK) return rc;
    return touch_kernel(p1_sample_kernel);
}

}  // namespace kmc
