/*
 * Ghost-cell fill of a same-level patch batch on the device.
 *
 * Step 1 copies face and corner ghost cells from aligned same-level
 * neighbours (fclaw2d_source/fc2d_geoclaw_copy_fort.f:11-107). Step 2 applies
 * the physical boundary rule of every side with no neighbour, in the
 * reference's order left, right, bottom, top over the full ghost extent
 * (fortran_source/geoflood_bc2_fort.f90:7-409), including the hydrograph
 * inflow state (hydrograph/hydrograh_module.f90:224-331). Step 1 reads only
 * neighbours' interior cells and step 2 only its own patch, so one CTA per
 * patch needs no grid-wide barrier.
 */
#include <cuda_runtime.h>

#include "gf_cmp.cuh"
#include "gf_internal.h"

namespace gf {

namespace {

__device__ __forceinline__ double* plane(double* base, long patch, int field, int S, int nf)
{
    return base + (patch * nf + field) * (long)S;
}

/* x to the double 2.0 / 3.0, as the reference's power: for positive x in the
 * single-precision range t = x y0 from the single-precision y0 of x^(-1/3) and
 * one third-order step of the binomial series, x y0 (1 - e)^(-1/3) with
 * e = 1 - x y0^3; pow otherwise. As the start of an iteration that is enough
 * (within 5 units of the last place). LAST: the error stays at the last rounding
 * (0.5; pow 1.3) with three small terms: the product's rounding tl, which e and
 * the sum take up, and ln(x) times what the double lies below two thirds,
 * 2/3 2^-54. y0 y0 is exact (24 bits each). */
template <bool LAST>
__device__ __forceinline__ double pow23(double x)
{
    if (!(x > 1.0e-30 && x < 1.0e30)) return pow(x, 2.0 / 3.0);
    const float xf = gf_f32(x);
    const double y0 = gf_f64_pos(rcbrtf(xf)), y2 = y0 * y0;
    const double t = x * y0;
    if (!LAST) {
        const double e = fma(-t, y2, 1.0);
        return fma(t * e, fma(2.0 / 9.0, e, 1.0 / 3.0), t);
    }
    const double tl = fma(x, y0, -t);
    const double e = fma(-tl, y2, fma(-t, y2, 1.0));
    const double below = static_cast<double>(logf(xf)) * (-2.0 / 3.0 * 5.5511151231257827e-17);
    return t + fma(t, fma(e, fma(2.0 / 9.0, e, 1.0 / 3.0), below), tl);
}

__device__ __forceinline__ double root(double a)
{
    return gf_pos_normal(a) ? gf_sqrt_n(a) : sqrt(a);
}

/* Riemann_invariants / two_shock (hydrograh_module.f90:224-331), discharge
 * form; tol is the single-precision literal 1.0e-6 of the Fortran. The whole
 * iteration is one chain of FP64 instructions of 64 clocks each, and a ghost
 * fill lasts as long as it does: quotients share one refined reciprocal, roots
 * are refined likewise, what does not change stays outside (a served round's
 * ghost fill with an inflow side 42-49 us with pow and IEEE quotients). */
__device__ void inflow_riemann(double g, double rsg, double q0hu, double h1, double u1, double& h0, bool two)
{
    const double tol = (double)1.0e-6f;
    const double x = q0hu * rsg;
    h0 = pow23<false>(two ? x : 0.5 * x);
    if (!two) {
        const double fixed = fma(2.0, root(g * h1), -u1);
        for (int i = 1; i <= 100; ++i) {
            /* fxn = q0/h0 - 2 sqrt(g h0) - u1 + 2 sqrt(g h1), dfxn = -q0/h0^2 - sqrt(g/h0) */
            const double r = gf_rcp(h0), s = root(g * h0), q = q0hu * r;
            const double fxn = fma(-2.0, s, q) + fixed;
            if (fabs(fxn) < tol) return;
            const double dfxn = -(q + s) * r;
            h0 = fma(-fxn, gf_rcp(dfxn), h0);
        }
        return;
    }
    const double r1 = gf_rcp(h1);
    for (int i = 1; i <= 100; ++i) {
        /* a = g (1/h0 + 1/h1) / 2, n = sqrt(a): fxn = q0/h0 - u1 - (h0 - h1) n,
         * dfxn = -q0/h0^2 - n + g (h0 - h1) / (4 h0^2 n). The depth is as far off
         * as fxn is: n comes from its own series, not as a product with 1 / n, and
         * q takes its residual up (it is ready before n). 33000 states against
         * long double, mean and largest error in ulps: 0.44 and 7.7 (0.49 without
         * either); IEEE quotients and roots 0.44 and 9.5. */
        const double r = gf_rcp(h0), d = h0 - h1, a = (0.5 * g) * (r + r1);
        double q = q0hu * r;
        q = fma(fma(-h0, q, q0hu), r, q);
        double n, rn;
        if (gf_pos_normal(a)) {
            const double y = gf_rsqrt_seed(a), t = a * y, e = fma(-t, y, 1.0), c = fma(0.375, e, 0.5);
            n = fma(t * e, c, t);
            rn = fma(y * e, c, y);
        } else {
            rn = rsqrt(a);
            n = a * rn;
        }
        const double fxn = fma(-d, n, q - u1);
        if (fabs(fxn) < tol) return;
        const double dfxn = fma((0.25 * g) * (d * rn), r * r, -fma(q, r, n));
        h0 = fma(-fxn, gf_rcp(dfxn), h0);
    }
}

/* Inflow ghost state inside the channel window; false = mirror (wall) case. */
__device__ bool inflow_state(const gf_phys& P, double q0hu, double h1, double hu1, double& h,
                             double& hu)
{
    const double g = P.grav;
    if (h1 < P.dry_tolerance) {
        const double hh = pow23<true>(q0hu / sqrt(g));
        h = hh > 0.001 ? hh : 0.001;
        hu = q0hu;
        return true;
    }
    if (q0hu != 0.0) {
        const double rsg = rsqrt(g), u1 = hu1 / h1;
        double h0;
        inflow_riemann(g, rsg, q0hu, h1, u1, h0, false);
        if (h0 > h1) inflow_riemann(g, rsg, q0hu, h1, u1, h0, true);
        /* Where the iteration steps to a negative depth its root is not a
         * number (the reference's too). It keeps the sign of an invalid root:
         * the update's integer comparisons then take the ghost cell as dry. */
        h = h0 == h0 ? h0 : __longlong_as_double(static_cast<long long>(0xfff8000000000000ull));
        hu = q0hu;
        return true;
    }
    return false;
}

/* Threads of a patch: every ghost cell in at most two rounds, every cell of
 * the x or the y sides in one (32^2: 272 and 144 cells, 16^2: 144 and 80, 8^2:
 * 80 and 48). */
template <int M>
constexpr int kGhostThreads = M == 32 ? 160 : M == 16 ? 96 : 96;

template <int M>
__global__ void __launch_bounds__(kGhostThreads<M>) ghost_fill_kernel(const gf_ghost_block* __restrict__ blocks,
                                                         const gf_ghost_ref* __restrict__ list,
                                                         int nlist,
                                                         const gf_phys* __restrict__ phys_table)
{
    constexpr int N = M + 4, S = N * N, MBC = 2;
    if ((int)blockIdx.x >= nlist) return;
    /* list == nullptr: one block, patch = blockIdx.x */
    const gf_ghost_ref ref = list ? list[blockIdx.x] : gf_ghost_ref{0, (int)blockIdx.x};
    const gf_ghost_block& blk = blocks[ref.block];
    if (blk.skip) return;
    const long p = ref.local;
    double* __restrict__ q = blk.q;
    const gf_bc_spec bc = blk.bc;
    const int* __restrict__ nbr = blk.nbr;
    int nb[8];
#pragma unroll
    for (int s = 0; s < 8; ++s) nb[s] = nbr[8 * p + s];

    /* dry-patch culling: the patch's last update was an identity, no
     * neighbour holds water and no side takes inflow, so this step's update
     * would be the identity again; mark it skipped and leave its ghosts */
    if (blk.fl) {
        bool skip = blk.fl[p].ident != 0;
#pragma unroll
        for (int s = 0; s < 8; ++s) {
            if (nb[s] >= 0) skip = skip && blk.fl[nb[s]].wet == 0;
            else if (nb[s] != -1) skip = false;               /* filled by another route */
            else if (s < 4 && bc.mthbc[s] == 0) skip = false; /* hydrograph side */
        }
        __syncthreads(); /* every thread has read the flags before thread 0 writes */
        if (threadIdx.x == 0) blk.fl[p].skip = skip ? 1 : 0;
        if (skip) return;
    }

    /* ---- step 1: same-level face and corner copies: the ghost cells by
     * number (two rows below, two above, then the sides row by row), all loads
     * of a thread ahead of its stores ---- */
    constexpr int NG = S - M * M, NT = kGhostThreads<M>, IT = (NG + NT - 1) / NT;
    double val[IT][3];
    int dst[IT];
#pragma unroll
    for (int it = 0; it < IT; ++it) {
        const int e = threadIdx.x + it * NT;
        dst[it] = -1;
        if (e >= NG) continue;
        int ii, jj; /* array column and row */
        if (e < 4 * N) {
            const int r = e / N;
            ii = e - r * N;
            jj = r < 2 ? r : M + r;
        } else {
            const int r = (e - 4 * N) / 4, c = (e - 4 * N) % 4;
            ii = c < 2 ? c : M + c;
            jj = 2 + r;
        }
        const bool L = ii < 2, R = ii >= M + 2, B = jj < 2, T = jj >= M + 2;
        int src = L ? nb[0] : nb[1];
        if (B || T) src = L ? (B ? nb[4] : nb[6]) : R ? (B ? nb[5] : nb[7]) : (B ? nb[2] : nb[3]);
        if (src < 0) continue;
        const int k2 = (jj + (B ? M : T ? -M : 0)) * N + ii + (L ? M : R ? -M : 0);
        dst[it] = jj * N + ii;
        const double* from = plane(q, src, 0, S, 3) + k2;
#pragma unroll
        for (int f = 0; f < 3; ++f) val[it][f] = from[f * S];
    }
    double* own = plane(q, p, 0, S, 3);
#pragma unroll
    for (int it = 0; it < IT; ++it)
        if (dst[it] >= 0) {
#pragma unroll
            for (int f = 0; f < 3; ++f) own[f * S + dst[it]] = val[it][f];
        }
    const bool phys_side[4] = {nb[0] == -1, nb[1] == -1, nb[2] == -1, nb[3] == -1};
    if (!(phys_side[0] || phys_side[1] || phys_side[2] || phys_side[3])) return;
    __syncthreads();

    const gf_phys& P = phys_table[blk.phys_of ? blk.phys_of[p] : blk.phys];
    const gf_patch_geom G = blk.geom[p];
    double* qh = plane(q, p, 0, S, 3);
    double* qu = plane(q, p, 1, S, 3);
    double* qv = plane(q, p, 2, S, 3);
    double* b = plane(blk.aux, p, 0, S, blk.maux);
    auto at = [](int i, int j) { return (j + 1) * N + (i + 1); };

    /* ---- step 2a: x sides (left then right are disjoint), all rows ---- */
    for (int e = threadIdx.x; e < 2 * N * MBC; e += blockDim.x) {
        const int side = e / (N * MBC); /* 0 left, 1 right */
        const int r = e % (N * MBC);
        const int j = r / MBC + 1 - MBC, ibc = r % MBC + 1;
        if (!phys_side[side]) continue;
        const int rule = bc.mthbc[side];
        const int ig = side == 0 ? 1 - ibc : M + ibc;        /* ghost          */
        const int im = side == 0 ? ibc : M + 1 - ibc;        /* mirror source  */
        const int ie = side == 0 ? 1 : M;                    /* boundary cell  */
        const int kg = at(ig, j);
        bool mirror = false;
        if (rule == 0 && bc.hydro_side[side]) {
            const double y = G.ylower + (j - 0.5) * G.dy;
            bool inflow = false;
            if (fabs(y - bc.y0) <= bc.width / 2.0) {
                double h, hu;
                inflow = inflow_state(P, bc.q0hu, qh[at(ie, j)], qu[at(ie, j)], h, hu);
                if (inflow) { qh[kg] = h; qu[kg] = hu; qv[kg] = 0.0; }
            }
            mirror = !inflow;
        } else if (rule == 1) {
            const int ks = at(ie, j);
            b[kg] = b[ks];
            qh[kg] = qh[ks]; qu[kg] = qu[ks]; qv[kg] = qv[ks];
        } else if (rule == 3) {
            mirror = true;
        }
        if (mirror) {
            const int ks = at(im, j);
            b[kg] = b[ks];
            qh[kg] = qh[ks]; qu[kg] = -qu[ks]; qv[kg] = qv[ks];
        }
    }
    __syncthreads();

    /* ---- step 2b: y sides (bottom then top are disjoint), all columns ---- */
    for (int e = threadIdx.x; e < 2 * N * MBC; e += blockDim.x) {
        const int side = 2 + e / (N * MBC); /* 2 bottom, 3 top */
        const int r = e % (N * MBC);
        const int i = r / MBC + 1 - MBC, jbc = r % MBC + 1;
        if (!phys_side[side]) continue;
        const int rule = bc.mthbc[side];
        const int jg = side == 2 ? 1 - jbc : M + jbc;
        const int jm = side == 2 ? jbc : M + 1 - jbc;
        const int je = side == 2 ? 1 : M;
        const int kg = at(i, jg);
        bool mirror = false;
        if (rule == 0 && bc.hydro_side[side]) {
            const double x = G.xlower + (i - 0.5) * G.dx;
            bool inflow = false;
            if (fabs(x - bc.x0) <= bc.width / 2.0) {
                double h, hu;
                /* the reference feeds q(2) (x momentum) on the y sides too */
                inflow = inflow_state(P, bc.q0hu, qh[at(i, je)], qu[at(i, je)], h, hu);
                if (inflow) { qh[kg] = h; qu[kg] = hu; qv[kg] = 0.0; }
            }
            mirror = !inflow;
        } else if (rule == 1) {
            const int ks = at(i, je);
            b[kg] = b[ks];
            qh[kg] = qh[ks]; qu[kg] = qu[ks]; qv[kg] = qv[ks];
        } else if (rule == 3) {
            mirror = true;
        }
        if (mirror) {
            const int ks = at(i, jm);
            b[kg] = b[ks];
            qh[kg] = qh[ks]; qu[kg] = qu[ks]; qv[kg] = -qv[ks];
        }
    }
}

} // namespace

cudaError_t launch_ghost_fill(int m, const gf_ghost_block* blocks, const gf_ghost_ref* list,
                              int nlist, const gf_phys* phys, cudaStream_t st)
{
    if (nlist <= 0) return cudaSuccess;
    switch (m) {
    case 32: ghost_fill_kernel<32><<<nlist, kGhostThreads<32>, 0, st>>>(blocks, list, nlist, phys); break;
    case 16: ghost_fill_kernel<16><<<nlist, kGhostThreads<16>, 0, st>>>(blocks, list, nlist, phys); break;
    case 8: ghost_fill_kernel<8><<<nlist, kGhostThreads<8>, 0, st>>>(blocks, list, nlist, phys); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

} // namespace gf
