/*
 * Cell-averaged topography on the device: setaux's bathymetry for every
 * cell of a raster (a level of a forest, or any uniform grid).
 *
 * The cell's integral follows cellgridintegrate
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

__device__ __forceinline__ bool cell_integral_inline(const Rect& cell, const gf_topo_grid* grids, const int* order,
                                                     int n, double* out)
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

__device__ __noinline__ bool cell_integral(const Rect& cell, const gf_topo_grid* grids, const int* order, int n,
                                           double* out)
{
    return cell_integral_inline(cell, grids, order, n, out);
}

/* raster index g along an axis, a cell outside the domain taken as the
 * cell inside that setaux's index shift names:
 * i + max(0, ceil((xlower - x)/dx)) - max(0, ceil((x - xupper)/dx)) */
__device__ __forceinline__ int inside_index(int g, double low, double d, double up)
{
    const double x = low + (g + 0.5) * d;
    if (x < low || x > up) g += (int)fmax(0.0, ceil((low - x) / d)) - (int)fmax(0.0, ceil((x - up) / d));
    return g;
}

/* Cells over more nodes of the finest grid than the tiles' tables hold: one
 * thread per cell, a chain of thousands of node cells each. */
__global__ void __launch_bounds__(128)
    topo_coarse_kernel(const gf_topo_grid* __restrict__ grids, const int* __restrict__ order, int n, int nx, int ny,
                       int halo, double xlower, double ylower, double dx, double dy, double xupper, double yupper,
                       double* __restrict__ out, int* __restrict__ err)
{
    const long p = nx + 2 * halo, e = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (e >= p * (ny + 2 * halo)) return;
    const int gi = inside_index((int)(e % p) - halo, xlower, dx, xupper);
    const int gj = inside_index((int)(e / p) - halo, ylower, dy, yupper);
    const Rect cell = {xlower + (double)gi * dx, xlower + (double)(gi + 1) * dx, ylower + (double)gj * dy,
                       ylower + (double)(gj + 1) * dy};
    double v;
    if (!cell_integral_inline(cell, grids, order, n, &v)) *err = 1;
    out[e] = v / (dx * dy);
}

/* Tile of raster cells of a CTA of kTX x kTY threads: kRows rows, some for each
 * thread. kNodes: the most node cells of a column (row) of cells that its tables
 * hold; coarser cells take the general path. */
constexpr int kTX = 32, kNodes = 40;

/* One axis of the integral of a column (row) of cells [lo, hi] over a grid:
 * the node cells i0 .. i1 - 1 it touches, and for each the width of the
 * overlap and half the sum of its two ends in units of the spacing. */
struct AxisNode {
    double width, half;
};
struct AxisCell {
    double lo, hi;   /* the cell's sides                          */
    double clo, chi; /* clamped to the grid                       */
    int i0, i1;      /* its node cells                            */
    int meets;       /* bit 0: overlaps the grid, bit 1: inside it */
};
__device__ __forceinline__ void axis_range(AxisCell& A, double low, double d, int n)
{
    const double top = low + (n - 1) * d;
    double lo = A.lo, hi = A.hi;
    if ((lo - low) < 0.0 || (hi - top) > 0.0) {
        lo = fmax(low, lo);
        hi = fmin(top, hi);
    }
    A.clo = lo;
    A.chi = hi;
    A.i0 = max((int)((lo - low) / d) + 1, 1);
    A.i1 = min((int)ceil((hi - low) / d) + 1, n);
}
__device__ __forceinline__ AxisNode axis_node(double lo, double hi, double low, double d, int ii)
{
    const double x1 = low + (ii - 1.0) * d, x2 = low + ii * d;
    const double a = fmax(lo, x1), b = fmin(hi, x2);
    return {b - a, 0.5 * ((b + a - 2.0 * x1) / d)};
}

/* v / area, correctly rounded, from the rounded reciprocal of area (Markstein,
 * "Computation of elementary functions on the IBM RISC System/6000 processor",
 * 1990): the first step makes the quotient faithful, the second exact. Five FP64
 * operations; the general quotient takes about twice as many. Out of the range
 * where no step can over- or underflow, or without a reciprocal (0): the
 * quotient itself. */
__device__ __forceinline__ double over_area(double v, double area, double rarea)
{
    const unsigned e = (unsigned)(__double_as_longlong(v) >> 52) & 0x7ff;
    if (e - 512u > 1024u || rarea == 0.0) return v / area;
    double q = v * rarea;
    q = fma(fma(-area, q, v), rarea, q);
    return fma(fma(-area, q, v), rarea, q);
}

/* The kernel is bound by FP64 issue (two lanes a clock), and most of it would go
 * into tests and quotients that depend on a cell's column or row alone. A tile of
 * 32 columns and kRows rows forms them once per column and row, one warp an axis, in shared
 * memory, for the cells that lie whole in the finest grid they touch; what is
 * left for a cell are the 14 operations of each node cell under it and the last
 * quotient. Halves of the axis sums stand for the factors 1/2 and 1/4 of the
 * bilinear form (powers of two, which no rounding sees), and the difference of a
 * node column serves both cells beside it: the same bits. The other cells (cells
 * that a grid's edge cuts, cells over more node cells than the tables hold) are
 * gathered from 8 rows on, so that the column under an edge fills one warp, and
 * take cell_integral. 1535^2 cells over a 1025^2 grid with a 513^2 inset, ncu: 625 us
 * with a warp for each row of them, 422 us gathered (82 % FP64 pipe, 89 FP64
 * instructions for 32 cells; tiles of 32 rows). Cells outside the domain are cells inside to this
 * kernel (a pass of its own over the raster took 31 us). */
template <int kTY, int kRows>
__global__ void __launch_bounds__(kTX* kTY)
    topo_raster_kernel(const gf_topo_grid* __restrict__ grids, const int* __restrict__ order, int n, int nx, int ny,
                       int halo, double xlower, double ylower, double dx, double dy, double xupper, double yupper,
                       double area, double rarea, double* __restrict__ out, int* __restrict__ err)
{
    constexpr int kPer = kRows / kTY;
    constexpr bool kGather = kRows > 4;
    __shared__ AxisNode xt[kNodes][kTX], yt[kNodes][kTX];
    __shared__ AxisCell ax[kTX], ay[kTX];
    __shared__ unsigned short rest[kTX * kRows]; /* cells of the general path */
    __shared__ int nrest;
    const int tx = threadIdx.x, ty = threadIdx.y;
    const long p = nx + 2 * halo;
    const int tiles = (int)((p + kTX - 1) / kTX), by = blockIdx.x / tiles, bx = blockIdx.x - by * tiles;
    const int i = bx * kTX + tx, jb = by * kRows;
    if (ty == 2 && tx == 0) nrest = 0;
    if (ty < 2) { /* warp 0 the columns, warp 1 the rows */
        const double low = ty ? ylower : xlower, d = ty ? dy : dx, up = ty ? yupper : xupper;
        const int g = inside_index((ty ? jb + tx : i) - halo, low, d, up);
        AxisCell& A = ty ? ay[tx] : ax[tx];
        A.lo = low + (double)g * d;
        A.hi = low + (double)(g + 1) * d;
    }
    __syncthreads();
    /* of this thread's cells, bit q for row ty + q kTY: still without a grid, to
     * take the general path */
    unsigned open = 0, general = 0, live;
    for (int q = 0; q < kPer; ++q) {
        const int k = ty + q * kTY;
        if (i < p && jb + k < ny + 2 * halo) open |= 1u << q;
    }
    live = open;
    double v[kPer] = {};
    for (int m = 0; m < n; ++m) {
        const gf_topo_grid& G = grids[order[m]];
        if (ty < 2) {
            AxisCell& A = ty ? ay[tx] : ax[tx];
            const double low = ty ? G.ylow : G.xlow, high = ty ? G.yhi : G.xhi;
            A.meets = (fmin(A.hi, high) > fmax(A.lo, low) ? 1 : 0) | (A.lo >= low && A.hi <= high ? 2 : 0);
        }
        __syncthreads();
        unsigned whole = 0;
        for (int q = 0; q < kPer; ++q) {
            const int both = ax[tx].meets & ay[ty + q * kTY].meets;
            if ((both & 1) && (open >> q & 1)) {
                open &= ~(1u << q);
                if (both & 2) whole |= 1u << q;
                else general |= 1u << q;
            }
        }
        if (__syncthreads_or(whole != 0)) {
            if (ty == 0) axis_range(ax[tx], G.xlow, G.dx, G.mx);
            else if (ty == 1) axis_range(ay[tx], G.ylow, G.dy, G.my);
            __syncthreads();
            {
                const AxisCell& A = ax[tx];
                const int c = A.i1 - A.i0 <= kNodes ? A.i1 - A.i0 : 0;
                for (int e = ty; e < c; e += kTY) xt[e][tx] = axis_node(A.clo, A.chi, G.xlow, G.dx, A.i0 + e);
            }
            {
                const AxisCell& A = ay[tx];
                const int c = A.i1 - A.i0 <= kNodes ? A.i1 - A.i0 : 0;
                for (int e = kTY - 1 - ty; e < c; e += kTY) yt[e][tx] = axis_node(A.clo, A.chi, G.ylow, G.dy, A.i0 + e);
            }
            __syncthreads();
            const int i0 = ax[tx].i0, nc = ax[tx].i1 - i0;
#pragma unroll
            for (int q = 0; q < kPer; ++q) {
                if (!(whole >> q & 1)) continue;
                const int k = ty + q * kTY, j0 = ay[k].i0, nr = ay[k].i1 - j0;
                if (nc > kNodes || nr > kNodes) {
                    general |= 1u << q;
                    continue;
                }
                double s = 0.0;
                for (int r = 0; r < nr; ++r) {
                    /* nodes are stored north to south: row (my - jj) holds the lower ones */
                    const double* row1 = G.z + (long)(G.my - (j0 + r)) * G.mx + (i0 - 1);
                    const double* row2 = row1 - G.mx;
                    const AxisNode Y = yt[r][k];
                    double z11 = nc > 0 ? row1[0] : 0.0, z12 = nc > 0 ? row2[0] : 0.0;
                    double b = z12 - z11;
                    for (int c = 0; c < nc; ++c) {
                        const AxisNode X = xt[c][tx];
                        const double z21 = row1[c + 1], z22 = row2[c + 1];
                        const double area = Y.width * X.width;
                        const double a = z21 - z11, bn = z22 - z21, d = bn - z12 + z11;
                        s = s + ((a * X.half + b * Y.half) + d * X.half * Y.half + z11) * area;
                        z11 = z21;
                        z12 = z22;
                        b = bn;
                    }
                }
                v[q] = 0.0 + s;
            }
        }
        if (!__syncthreads_or(open != 0)) break;
    }
    if (open) *err = 1; /* no grid under a cell */
    for (int q = 0; q < kPer; ++q) {
        const int k = ty + q * kTY;
        __syncwarp();
        const bool cutc = general >> q & 1;
        const int ncut = __popc(__ballot_sync(0xffffffffu, cutc));
        if (kGather && cutc && ncut < kTX / 4) {
            rest[atomicAdd(&nrest, 1)] = (unsigned short)(k * kTX + tx);
            continue;
        }
        if (cutc) {
            const Rect cell = {ax[tx].lo, ax[tx].hi, ay[k].lo, ay[k].hi};
            cell_integral(cell, grids, order, n, &v[q]);
        }
        if (live >> q & 1) out[(long)(jb + k) * p + i] = over_area(v[q], area, rarea);
    }
    if (!kGather) return;
    __syncthreads();
    for (int e = ty * kTX + tx; e < nrest; e += kTX * kTY) {
        const int k = rest[e] / kTX, c = rest[e] % kTX;
        const Rect cell = {ax[c].lo, ax[c].hi, ay[k].lo, ay[k].hi};
        double w = 0.0;
        cell_integral(cell, grids, order, n, &w);
        out[(long)(jb + k) * p + bx * kTX + c] = over_area(w, area, rarea);
    }
}

} // namespace

cudaError_t launch_topo_raster(const gf_topo_grid* grids, const int* order, int n, int nx, int ny, int halo,
                               double xlower, double ylower, double dx, double dy, double xupper,
                               double yupper, double finest, double* out, int* err, cudaStream_t st)
{
    if (n < 1 || n > GF_TOPO_MAX_FILES) return cudaErrorInvalidValue;
    const long cols = (nx + 2 * halo + kTX - 1) / kTX;
    const double area = dx * dy;
    const double rarea = area > 1e-150 && area < 1e150 ? 1.0 / area : 0.0;
    const long cells = (long)(nx + 2 * halo) * (ny + 2 * halo);
    /* cells beyond the tables gain nothing from tiles (64^2 and 128^2 cells of 64
     * and 32 m over a 0.5 m inset 35.0 and 10.2 ms so, 37.8 and 11.0 in tiles;
     * 256^2 of 16 m 2.84 and 2.16) */
    if (fmax(dx, dy) > (kNodes - 2) * finest) {
        if (cells > 128L * 0x7fffffffL) return cudaErrorInvalidValue;
        topo_coarse_kernel<<<(unsigned)((cells + 127) / 128), 128, 0, st>>>(grids, order, n, nx, ny, halo, xlower,
                                                                            ylower, dx, dy, xupper, yupper, out, err);
        return cudaGetLastError();
    }
    /* 32 rows a CTA share most of what belongs to a column, but leave SMs idle on
     * small rasters, and so do 8 on smaller ones, where a gathered warp of cut
     * cells is a longer chain than each cell in its place: us for 64^2 / 512^2 /
     * 2048^2 cells with 4 rows 1650 / 460 / -, 8 rows 1775 / 350 / 2410, 32 rows
     * 3314 / 369 / 2275 */
    auto run = [&](auto* kern, int ty, int rows) -> cudaError_t {
        const long tiles = cols * ((ny + 2 * halo + rows - 1) / rows);
        if (tiles > 0x7fffffffL) return cudaErrorInvalidValue; /* 3e11 cells */
        kern<<<(unsigned)tiles, dim3(kTX, ty), 0, st>>>(grids, order, n, nx, ny, halo, xlower, ylower, dx, dy, xupper,
                                                        yupper, area, rarea, out, err);
        return cudaGetLastError();
    };
    if (cells >= 8L * sm_count() * kTX * 32) return run(topo_raster_kernel<8, 32>, 8, 32);
    if (cells >= 2L * sm_count() * kTX * 8) return run(topo_raster_kernel<8, 8>, 8, 8);
    return run(topo_raster_kernel<4, 4>, 4, 4);
}

} // namespace gf
