/*
 * Cell-averaged topography on the device: setaux's bathymetry for every
 * cell of a raster (a level of a forest, or any uniform grid).
 *
 * One thread per cell. The cell's integral follows cellgridintegrate
 * (src/fc2d_geoclaw/geolib_source/cellgridintegrate2.f:1-90): the finest
 * grid overlapping the cell alone if it holds the whole cell, else the
 * inclusion-exclusion over the ranked grids of rectintegral
 * (geolib_source/topo_module.f90:1460-1548), I(R, m) = I(R, m+1) -
 * I(R n G_m, m+1) + T(G_m, R n G_m), evaluated here with an explicit stack
 * instead of recursion; T is topointegral (geolib_source/topointegral.f):
 * the exact integral of the bilinear interpolant over each node cell of G
 * the rectangle touches (bilinearintegral.f). Then the cell average is the
 * integral over dx * dy (fortran_source/geoclaw_setaux_fort.f90:107-168),
 * and cells outside the domain copy the nearest cell inside (:178-215).
 * Compiled without FMA contraction, in the Fortran expressions' order.
 */
#include <cuda_runtime.h>

#include "gf_internal.h"

namespace gf {

namespace {

struct Rect {
    double x1, x2, y1, y2;
};

__device__ __forceinline__ bool cut(const Rect& r, const gf_topo_grid& g, Rect* o, double* area)
{
    o->x1 = fmax(r.x1, g.xlow);
    o->x2 = fmin(r.x2, g.xhi);
    o->y1 = fmax(r.y1, g.ylow);
    o->y2 = fmin(r.y2, g.yhi);
    if (o->x2 > o->x1 && o->y2 > o->y1) {
        *area = (o->x2 - o->x1) * (o->y2 - o->y1);
        return true;
    }
    *area = 0.0;
    return false;
}

/* integral of the bilinear interpolant of g over r (r within g's extent up
 * to rounding, which the clamp absorbs) */
__device__ double grid_integral(Rect r, const gf_topo_grid& g)
{
    double s = 0.0;
    const double xxhi = g.xlow + (g.mx - 1) * g.dx, yyhi = g.ylow + (g.my - 1) * g.dy;
    if ((r.x1 - g.xlow) < 0.0 || (r.x2 - xxhi) > 0.0) {
        r.x1 = fmax(g.xlow, r.x1);
        r.x2 = fmin(xxhi, r.x2);
    }
    if ((r.y1 - g.ylow) < 0.0 || (r.y2 - yyhi) > 0.0) {
        r.y1 = fmax(g.ylow, r.y1);
        r.y2 = fmin(yyhi, r.y2);
    }
    const int j0 = max((int)((r.y1 - g.ylow) / g.dy) + 1, 1);
    const int i0 = max((int)((r.x1 - g.xlow) / g.dx) + 1, 1);
    const int i1 = min((int)ceil((r.x2 - g.xlow) / g.dx) + 1, g.mx);
    const int j1 = min((int)ceil((r.y2 - g.ylow) / g.dy) + 1, g.my);
    for (int jj = j0; jj < j1; ++jj) {
        const double y1 = g.ylow + (jj - 1.0) * g.dy, y2 = g.ylow + jj * g.dy;
        /* nodes are stored north to south: row (my - jj) holds y1 */
        const double* row1 = g.z + (long)(g.my - jj) * g.mx;
        const double* row2 = row1 - g.mx;
        const double ylo = fmax(r.y1, y1), yhi = fmin(r.y2, y2);
        const double sumeta = (yhi + ylo - 2.0 * y1) / g.dy;
        for (int ii = i0; ii < i1; ++ii) {
            const double x1 = g.xlow + (ii - 1.0) * g.dx, x2 = g.xlow + ii * g.dx;
            const double z11 = row1[ii - 1], z21 = row1[ii], z12 = row2[ii - 1], z22 = row2[ii];
            const double xlo = fmax(r.x1, x1), xhi = fmin(r.x2, x2);
            const double area = (yhi - ylo) * (xhi - xlo);
            const double sumxi = (xhi + xlo - 2.0 * x1) / g.dx;
            const double a = z21 - z11, b = z12 - z11, c = z22 - z21 - z12 + z11;
            s = s + (0.5 * (a * sumxi + b * sumeta) + 0.25 * c * sumxi * sumeta + z11) * area;
        }
    }
    return s;
}

/* inclusion-exclusion over ranks m..n-1 without recursion: frames hold the
 * rectangle, the rank, the stage and the partial sums */
__device__ double ranked_integral(Rect r0, int m0, const gf_topo_grid* grids, const int* order, int n)
{
    struct Frame {
        Rect r, cut;
        double a;
        int m, stage;
    };
    Frame st[GF_TOPO_MAX_FILES];
    int sp = 0;
    double ret = 0.0;
    st[0].r = r0;
    st[0].m = m0;
    st[0].stage = 0;
    while (sp >= 0) {
        Frame& F = st[sp];
        const gf_topo_grid& G = grids[order[F.m]];
        if (F.m == n - 1) {
            Rect c;
            double area;
            ret = cut(F.r, G, &c, &area) ? grid_integral(c, G) : 0.0;
            --sp;
            continue;
        }
        if (F.stage == 0) {
            F.stage = 1;
            st[sp + 1].r = F.r;
            st[sp + 1].m = F.m + 1;
            st[sp + 1].stage = 0;
            ++sp;
            continue;
        }
        if (F.stage == 1) {
            F.a = ret;
            double area;
            cut(F.r, G, &F.cut, &area);
            if (area > 0) {
                F.stage = 2;
                st[sp + 1].r = F.cut;
                st[sp + 1].m = F.m + 1;
                st[sp + 1].stage = 0;
                ++sp;
                continue;
            }
            ret = F.a;
            --sp;
            continue;
        }
        /* stage 2: ret holds the coarser ranks' integral over the cut */
        ret = F.a - ret + grid_integral(F.cut, G);
        --sp;
    }
    return ret;
}

__device__ bool cell_integral(const Rect& cell, const gf_topo_grid* grids, const int* order, int n,
                              double* out)
{
    for (int m = 0; m < n; ++m) {
        const gf_topo_grid& G = grids[order[m]];
        const double cellarea = (cell.x2 - cell.x1) * (cell.y2 - cell.y1);
        Rect c;
        double area;
        if (cut(cell, G, &c, &area)) {
            if (area == cellarea) *out = 0.0 + grid_integral(c, G);
            else *out = ranked_integral(cell, m, grids, order, n);
            return true;
        }
    }
    *out = 0.0;
    return false;
}

/* Tile of raster cells of a CTA, and the most node cells of a column (row) of
 * cells that its tables hold: coarser cells take the general path. */
constexpr int kTX = 32, kTY = 8, kNodes = 40;

/* One axis of the integral of a column (row) of cells [lo, hi] over a grid:
 * the node cells i0 .. i1 - 1 it touches, and for each the width of the
 * overlap and the sum of its two ends in units of the spacing, as
 * grid_integral forms them. */
struct AxisNode {
    double width, sum;
};
__device__ __forceinline__ void axis_range(double& lo, double& hi, double low, double d, int n, int* i0, int* i1)
{
    const double top = low + (n - 1) * d;
    if ((lo - low) < 0.0 || (hi - top) > 0.0) {
        lo = fmax(low, lo);
        hi = fmin(top, hi);
    }
    *i0 = max((int)((lo - low) / d) + 1, 1);
    *i1 = min((int)ceil((hi - low) / d) + 1, n);
}
__device__ __forceinline__ AxisNode axis_node(double lo, double hi, double low, double d, int ii)
{
    const double x1 = low + (ii - 1.0) * d, x2 = low + ii * d;
    const double a = fmax(lo, x1), b = fmin(hi, x2);
    return {b - a, (b + a - 2.0 * x1) / d};
}

/* One thread per cell. The kernel is bound by FP64 issue (two lanes a clock),
 * and most of it went into quotients that depend on the cell's column or row
 * alone: a tile now forms them once per column and row of cells, in shared
 * memory, for the cells that lie whole in the finest grid they touch (the
 * same operations in the same order, so the same bits); the others (cells that
 * a grid's edge cuts, cells over more node cells than the tables hold) take
 * cell_integral. */
__global__ void __launch_bounds__(kTX* kTY)
    topo_raster_kernel(const gf_topo_grid* __restrict__ grids, const int* __restrict__ order, int n, int nx, int ny,
                       int halo, double xlower, double ylower, double dx, double dy, double xupper, double yupper,
                       double* __restrict__ out, int* __restrict__ err)
{
    __shared__ AxisNode xt[kNodes][kTX], yt[kTY][kNodes];
    __shared__ double cx[kTX][2], cy[kTY][2];
    __shared__ int xr[kTX][2], yr[kTY][2];
    __shared__ unsigned char outx[kTX], outy[kTY];
    const int tx = threadIdx.x, ty = threadIdx.y, t = ty * kTX + tx;
    const long p = nx + 2 * halo;
    const int tiles = (int)((p + kTX - 1) / kTX), by = blockIdx.x / tiles, bx = blockIdx.x - by * tiles;
    const int i = bx * kTX + tx, j = by * kTY + ty;
    if (t < kTX) {
        const int gi = i - halo;
        const double x1 = xlower + (double)gi * dx, x2 = xlower + (double)(gi + 1) * dx, x = 0.5 * (x1 + x2);
        cx[tx][0] = x1;
        cx[tx][1] = x2;
        outx[tx] = x > xupper || x < xlower;
    } else if (t < kTX + kTY) {
        const int k = t - kTX, gj = by * kTY + k - halo;
        const double y1 = ylower + (double)gj * dy, y2 = ylower + (double)(gj + 1) * dy, y = 0.5 * (y1 + y2);
        cy[k][0] = y1;
        cy[k][1] = y2;
        outy[k] = y > yupper || y < ylower;
    }
    __syncthreads();
    const Rect cell = {cx[tx][0], cx[tx][1], cy[ty][0], cy[ty][1]};
    const bool live = i < p && j < ny + 2 * halo && !outx[tx] && !outy[ty];
    /* 0 no grid yet, 1 done, 2 general path */
    int state = live ? 0 : 1;
    double v = 0.0;
    for (int m = 0; m < n; ++m) {
        const gf_topo_grid& G = grids[order[m]];
        const bool meets = state == 0 && fmin(cell.x2, G.xhi) > fmax(cell.x1, G.xlow) &&
                           fmin(cell.y2, G.yhi) > fmax(cell.y1, G.ylow);
        const bool whole = meets && cell.x1 >= G.xlow && cell.x2 <= G.xhi && cell.y1 >= G.ylow && cell.y2 <= G.yhi;
        if (meets && !whole) state = 2;
        if (!__syncthreads_or(whole)) {
            if (!__syncthreads_or(state == 0)) break;
            continue;
        }
        if (t < kTX) {
            double lo = cx[tx][0], hi = cx[tx][1];
            axis_range(lo, hi, G.xlow, G.dx, G.mx, &xr[tx][0], &xr[tx][1]);
        } else if (t < kTX + kTY) {
            const int k = t - kTX;
            double lo = cy[k][0], hi = cy[k][1];
            axis_range(lo, hi, G.ylow, G.dy, G.my, &yr[k][0], &yr[k][1]);
        }
        __syncthreads();
        {
            double lo = cx[tx][0], hi = cx[tx][1];
            const double top = G.xlow + (G.mx - 1) * G.dx;
            if ((lo - G.xlow) < 0.0 || (hi - top) > 0.0) {
                lo = fmax(G.xlow, lo);
                hi = fmin(top, hi);
            }
            const int i0 = xr[tx][0], c = min(xr[tx][1] - i0, kNodes);
            for (int e = ty; e < c; e += kTY) xt[e][tx] = axis_node(lo, hi, G.xlow, G.dx, i0 + e);
        }
        {
            double lo = cy[ty][0], hi = cy[ty][1];
            const double top = G.ylow + (G.my - 1) * G.dy;
            if ((lo - G.ylow) < 0.0 || (hi - top) > 0.0) {
                lo = fmax(G.ylow, lo);
                hi = fmin(top, hi);
            }
            const int j0 = yr[ty][0], c = min(yr[ty][1] - j0, kNodes);
            for (int e = tx; e < c; e += kTX) yt[ty][e] = axis_node(lo, hi, G.ylow, G.dy, j0 + e);
        }
        __syncthreads();
        if (whole) {
            const int i0 = xr[tx][0], nc = xr[tx][1] - i0, j0 = yr[ty][0], nr = yr[ty][1] - j0;
            if (nc > kNodes || nr > kNodes) {
                state = 2;
            } else {
                double s = 0.0;
                for (int r = 0; r < nr; ++r) {
                    /* nodes are stored north to south: row (my - jj) holds the lower ones */
                    const double* row1 = G.z + (long)(G.my - (j0 + r)) * G.mx + (i0 - 1);
                    const double* row2 = row1 - G.mx;
                    const AxisNode Y = yt[ty][r];
                    double z11 = nc > 0 ? row1[0] : 0.0, z12 = nc > 0 ? row2[0] : 0.0;
                    for (int c = 0; c < nc; ++c) {
                        const AxisNode X = xt[c][tx];
                        const double z21 = row1[c + 1], z22 = row2[c + 1];
                        const double area = Y.width * X.width;
                        const double a = z21 - z11, b = z12 - z11, d = z22 - z21 - z12 + z11;
                        s = s + (0.5 * (a * X.sum + b * Y.sum) + 0.25 * d * X.sum * Y.sum + z11) * area;
                        z11 = z21;
                        z12 = z22;
                    }
                }
                v = 0.0 + s;
                state = 1;
            }
        }
        if (!__syncthreads_or(state == 0)) break;
    }
    if (!live) return;
    if (state == 2) cell_integral(cell, grids, order, n, &v);
    if (state == 0) *err = 1; /* no grid under the cell */
    out[(long)j * p + i] = v / (dx * dy);
}

/* cells outside the domain take the cell inside that setaux's index shift
 * names: i + max(0, ceil((xlower - x)/dx)) - max(0, ceil((x - xupper)/dx)). A
 * column's and a row's part of the test are formed once per tile. */
__global__ void __launch_bounds__(kTX* kTY)
    topo_outside_kernel(double* __restrict__ out, int nx, int ny, int halo, double xlower, double ylower, double dx,
                        double dy, double xupper, double yupper)
{
    __shared__ unsigned char outx[kTX], outy[kTY];
    const int tx = threadIdx.x, ty = threadIdx.y, t = ty * kTX + tx;
    const long p = nx + 2 * halo;
    const int tiles = (int)((p + kTX - 1) / kTX), by = blockIdx.x / tiles, bx = blockIdx.x - by * tiles;
    const int i = bx * kTX + tx, j0 = by * kTY, j = j0 + ty;
    if (t < kTX) {
        const double x = xlower + ((i - halo) + 0.5) * dx;
        outx[tx] = x < xlower || x > xupper;
    } else if (t < kTX + kTY) {
        const double y = ylower + ((j0 + (t - kTX) - halo) + 0.5) * dy;
        outy[t - kTX] = y < ylower || y > yupper;
    }
    __syncthreads();
    if (i >= p || j >= ny + 2 * halo || !(outx[tx] || outy[ty])) return;
    const double x = xlower + ((i - halo) + 0.5) * dx, y = ylower + ((j - halo) + 0.5) * dy;
    const int ii = i + (int)fmax(0.0, ceil((xlower - x) / dx)) - (int)fmax(0.0, ceil((x - xupper) / dx));
    const int jj = j + (int)fmax(0.0, ceil((ylower - y) / dy)) - (int)fmax(0.0, ceil((y - yupper) / dy));
    out[(long)j * p + i] = out[(long)jj * p + ii];
}

} // namespace

cudaError_t launch_topo_raster(const gf_topo_grid* grids, const int* order, int n, int nx, int ny, int halo,
                               double xlower, double ylower, double dx, double dy, double xupper,
                               double yupper, double* out, int* err, cudaStream_t st)
{
    if (n < 1 || n > GF_TOPO_MAX_FILES) return cudaErrorInvalidValue;
    const long tiles = (long)((nx + 2 * halo + kTX - 1) / kTX) * ((ny + 2 * halo + kTY - 1) / kTY);
    if (tiles > 0x7fffffffL) return cudaErrorInvalidValue; /* 5e11 cells */
    const dim3 block(kTX, kTY), grid((unsigned)tiles);
    topo_raster_kernel<<<grid, block, 0, st>>>(grids, order, n, nx, ny, halo, xlower, ylower, dx, dy, xupper, yupper,
                                               out, err);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess || halo == 0) return e;
    topo_outside_kernel<<<grid, block, 0, st>>>(out, nx, ny, halo, xlower, ylower, dx, dy, xupper, yupper);
    return cudaGetLastError();
}

} // namespace gf
