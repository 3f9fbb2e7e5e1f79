/*
 * The patch update of gf_patch_update.cuh, streamed over the rows of a patch
 * (contracted build, whole patches).
 *
 * patch_update_kernel sweeps x, then y, over a patch that lies whole in shared
 * memory, with flux accumulators for every cell: 200 KB for 32^2, one CTA on
 * an SM, and its FP64 pipes idle while that CTA stages, prepares, lists,
 * writes or waits at a barrier (measured 61 % busy on wet 32^2 patches). Here a
 * band of R rows moves up the patch: the x faces of the band's rows and the y
 * faces below them are solved together, limited, split per cell, and a row of
 * cells is finished and written once the rows around it are done, two rows
 * behind. Shared memory holds rings of rows instead of planes and no
 * accumulators (a cell's sums are formed at once, in registers): about half, so
 * two CTAs share an SM and fill each other's gaps.
 *
 * Band b covers the x slices and the y faces of the array rows a0 = 1 + b R ..
 * a0 + R - 1 (y face f lies between array rows f - 1 and f). With A the normal
 * solves, B1 the limiter, B2 the cells' records and G the finished rows:
 *   x: A, B1, B2 of the rows a0 .. a0 + R - 1;
 *   y: A of the faces a0 .., B1 of a0 - 1 .. a0 + R - 2 (a face needs both
 *      neighbours), B2 of the cell rows a0 - 2 .. a0 + R - 3, G of the same.
 * Two barriers a band, as in the sweeps:
 *   [A of b | B2 of b - 1 | dry list of b | staging of b + 1 made ready]
 *   [B1 of b | class list of b + 1 | G of b - 1].
 * Every value is formed by the same operations and summed in the same order as
 * by the sweeps: the results are the same bits.
 *
 * The window kernel splits a patch over a cluster of K CTAs, each with the rows
 * of one window, all staged at its start. x and y faces side by side fill the
 * warps of an SM that holds one window (14 chunks of normal solves for four
 * rows of 32^2): a lone 32^2 patch 42 us over K = 8 (the sweeps split over the
 * same cluster 50), 24 patches 55 us over K = 4 (76), 72 90 us over K = 2 (107).
 * What is left is the chain of FP64 instructions of one face and one cell, 64
 * cycles each.
 *
 * Before a band is staged the item's depths are read once. A patch without
 * water is written at once; else the bands start and end with its wet rows (the
 * records before them are zero), and the rows beyond are written like a dry
 * patch.
 */
#ifndef GF_PATCH_STREAM_CUH
#define GF_PATCH_STREAM_CUH

#include "gf_patch_update.cuh"

namespace GF_KNS {

template <int M, int R, int K = 1>
struct StreamSmem {
    static constexpr int N = M + 2 * GF_MBC;
    static constexpr int RW = M / K;             /* cell rows that the CTA finishes       */
    static constexpr int FA = M + 3, FB = M + 1; /* x faces of a slice: solved, limited  */
    static constexpr int NC = M + 2;             /* y faces of a row (columns 1 .. M + 2) */
    static constexpr int NB = (RW + 3 + R - 1) / R;
    static constexpr bool ONE = NB == 1;
    /* rows in use at once: G of b - 1 reads from a0 - R - 2, staging of b + 1
     * writes to a0 + 2 R - 1; a window stages all its rows at its start */
    static constexpr int ROWS = K == 1 && 3 * R + 2 < N ? 3 * R + 2 : RW + 4;
    /* one row more of the wet flags: B2 looks below its first row */
    static constexpr int WROWS = K == 1 && 3 * R + 3 < N ? 3 * R + 3 : RW + 4;
    static constexpr int PL = ROWS * N;
    static constexpr int WS = 11, OS = 9, CS = 9; /* record strides, as in Smem */
    static constexpr int OFF_H = 0, OFF_HU = PL, OFF_HV = 2 * PL, OFF_B = 3 * PL, OFF_U = 4 * PL, OFF_V = 5 * PL,
                         OFF_C = 6 * PL, OFF_RC = 7 * PL;
    /* rings of rows; with one band, its rows */
    static constexpr int RX = ONE ? RW + 2 : R, RWY = ONE ? RW + 3 : R + 2, ROY = ONE ? RW + 1 : R + 1,
                         RCX = ONE ? RW + 2 : R + 3, RCY = ONE ? RW : R;
    static constexpr int OFF_WX = 8 * PL;
    static constexpr int OFF_WY = OFF_WX + RX * FA * WS;
    static constexpr int OFF_OX = OFF_WY + RWY * NC * WS;
    static constexpr int OFF_OY = OFF_OX + RX * FB * OS;
    static constexpr int OFF_CX = OFF_OY + ROY * NC * OS;
    static constexpr int OFF_CY = OFF_CX + RCX * M * CS;
    static constexpr int OFF_SC = OFF_CY + RCY * NC * CS;
    static constexpr int OFF_BAR = OFF_SC + 16;
    static constexpr int OFF_INT = OFF_BAR + 2;
    /* [parity][smooth, edge, full, dry], [parity][wet, dry], wet rows, cursors */
    static constexpr int CNT_B = 8, CNT_ROWS = 12, CNT_CUR = 14, CNT_INTS = CNT_CUR + 2 * (NB + 1);
    static constexpr int LIST_A = R * (FA + NC), LIST_B = R * (FB + NC);
    static constexpr size_t OFF_LIST = (size_t)OFF_INT * 8 + CNT_INTS * 4;
    static constexpr size_t OFF_WET = (OFF_LIST + (2 * LIST_A + LIST_B) * 2 + 15) / 16 * 16;
    static constexpr size_t BYTES = (OFF_WET + WROWS * N + 15) / 16 * 16;
    static __device__ __forceinline__ int slot(int row) { return ROWS == N ? row : row % ROWS; }
    /* wet flag of (row, column) */
    static __device__ __forceinline__ int wi(int row, int col) { return (WROWS == N ? row : row % WROWS) * N + col; }
};

/* Rows of band b of the RW rows above array row o + 1: x slices and y faces
 * from a0 (x1, y1 past their ends), y limited faces l0 .. l1 - 1, finished cell
 * rows c0 .. c1 - 1. */
template <int RW, int R>
struct StreamBand {
    int a0, nx, ny, l0, nl, c0, nc;
    __device__ __forceinline__ StreamBand(int b, int o)
    {
        a0 = 1 + o + b * R;
        const int y1 = min(a0 + R, o + RW + 4);
        nx = min(a0 + R, o + RW + 3) - a0;
        ny = y1 - a0;
        l0 = max(a0 - 1, o + 2);
        nl = max(min(y1 - 1, o + RW + 3) - l0, 0);
        c0 = max(a0 - 2, o + 2);
        nc = max(min(y1 - 2, o + RW + 2) - c0, 0);
    }
};

template <class L>
__device__ __forceinline__ gf_cell stream_cell(const double* sm, bool wet, int k, bool y)
{
    gf_cell c;
    c.h = sm[L::OFF_H + k];
    c.b = sm[L::OFF_B + k];
    c.c = sm[L::OFF_C + k];
    c.rc = sm[L::OFF_RC + k];
    c.wet = wet;
    c.hun = sm[(y ? L::OFF_HV : L::OFF_HU) + k];
    c.hut = sm[(y ? L::OFF_HU : L::OFF_HV) + k];
    c.un = sm[(y ? L::OFF_V : L::OFF_U) + k];
    c.ut = sm[(y ? L::OFF_U : L::OFF_V) + k];
    return c;
}

/* One work item; as patch_item. K > 1: window win of the K windows of rows
 * whose CTAs form a cluster; its largest speed goes to *part. */
template <int M, int NT, int R, int K = 1>
__device__ __forceinline__ bool stream_item(double* sm, uint64_t* bar, uint32_t& phase, gf_patch_work wk, int wi,
                                            const gf_phys* __restrict__ phys_table, double dt_uniform,
                                            const double* __restrict__ group_dt, const int* __restrict__ group_par,
                                            int maux, double* __restrict__ cfl_out,
                                            unsigned long long* __restrict__ group_max, int* __restrict__ err,
                                            int win = 0, double* part = nullptr)
{
    using L = StreamSmem<M, R, K>;
    using Band = StreamBand<L::RW, R>;
    constexpr int N = L::N, S = N * N, NB = L::NB, RW = L::RW;
    const int o = K > 1 ? win * RW : 0; /* first row that the item reads */
    const int top = o + RW + 4;         /* past the last */
    int* cnt = reinterpret_cast<int*>(sm + L::OFF_INT);
    uint16_t* la = reinterpret_cast<uint16_t*>(reinterpret_cast<char*>(sm) + L::OFF_LIST);
    uint16_t *lm = la + L::LIST_A, *lb = lm + L::LIST_A;
    unsigned char* wet = reinterpret_cast<unsigned char*>(sm) + L::OFF_WET;
    double* sc = sm + L::OFF_SC;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;

    const double dt = group_dt ? group_dt[wk.group] : dt_uniform;
    if (group_dt && !(dt > 0.0)) return true;
    if (group_par && group_par[wk.group]) {
        double* t = wk.q;
        wk.q = wk.qout;
        wk.qout = t;
    }
    if (wk.fl && wk.fl->skip) return true;
    const gf_phys P = phys_table[wk.phys];
    const double g = P.grav, drytol = P.dry_tolerance;
    if (__syncthreads_or(threadIdx.x == 0 && err && *reinterpret_cast<volatile int*>(err) != 0)) {
        if (K > 1) {
            cluster_arrive();
            cluster_wait();
        }
        return false;
    }

    auto stage = [&](int r0, int r1) { /* one thread */
        mbar_expect_tx(bar, (uint32_t)(4 * (r1 - r0) * N * sizeof(double)));
        for (int r = r0; r < r1;) { /* runs of rows that do not wrap in the ring */
            const int s = L::slot(r), n = min(r1 - r, L::ROWS - s);
            const uint32_t bytes = (uint32_t)(n * N * sizeof(double));
#pragma unroll
            for (int p = 0; p < 3; ++p) bulk_g2s(sm + L::OFF_H + p * L::PL + s * N, wk.q + p * S + r * N, bytes, bar);
            bulk_g2s(sm + L::OFF_B + s * N, wk.aux + r * N, bytes, bar);
            r += n;
        }
    };
    int any_wet = 0, changed = 0;
    unsigned kept = 0; /* K > 1: bit r - o, row r holds a cell b4step2 leaves alone */
    /* b4step2 and the quotients of the cells e0, e0 + step, .. of rows r0 .. */
    auto prepare = [&](int r0, int e0, int e1, int step) {
        for (int e = e0; e < e1; e += step) {
            const int rr = e / N, col = e - rr * N, k = L::slot(r0 + rr) * N + col;
            double h = sm[L::OFF_H + k];
            if (d_lt<true>(h, drytol)) {
                h = d_max<true>(h, 0.0);
                sm[L::OFF_H + k] = h;
                sm[L::OFF_HU + k] = 0.0;
                sm[L::OFF_HV + k] = 0.0;
            } else if (K > 1) {
                kept |= 1u << (r0 + rr - o);
            }
            const bool w = d_gt<true>(h, drytol);
            wet[L::wi(r0 + rr, col)] = w ? 1 : 0;
            any_wet |= w;
            double u = 0.0, v = 0.0, c = 0.0, rc = 0.0;
            if (w) {
                const double gh = gf_mul(g, h);
                rc = gf_pos_normal(gh) ? gf_rsqrt_n(gh) : rsqrt(gh);
                c = gf_mul(gh, rc);
                const double rh = gf_mul(g, gf_mul(rc, rc));
                u = gf_mul(sm[L::OFF_HU + k], rh);
                v = gf_mul(sm[L::OFF_HV + k], rh);
            }
            sm[L::OFF_U + k] = u;
            sm[L::OFF_V + k] = v;
            sm[L::OFF_C + k] = c;
            sm[L::OFF_RC + k] = rc;
        }
    };
    uint32_t staged = phase; /* parity of the staging in flight */
    auto wait_staged = [&]() -> bool { return mbar_wait(bar, staged, kWaitPolls); };
    auto fail = [&]() -> bool {
        if (threadIdx.x == 0) atomicExch(err, 1);
        mbar_wait(bar, staged, kWaitPolls); /* let any copy in flight land */
        return false;
    };

    unsigned* rows = reinterpret_cast<unsigned*>(cnt + L::CNT_ROWS);
    auto constants = [&]() { /* the last warp: the item's constants, one lane each */
        const double q = (lane < 2 ? dt : 1.0) / (lane == 0 ? wk.dx : lane == 1 ? wk.dy : 16.0 * g);
        if (lane < 3) sc[SC_DTDX + lane] = q;
        if (lane == 3) sc[SC_RSG] = rsqrt(g);
        if (lane == 4) {
            const double crit = fmax(drytol * g, 1e-6);
            sc[SC_CRIT] = crit;
            sc[SC_CRIT2] = sqrt(crit);
        }
        if (lane >= 8 && lane < 8 + GF_MAX_MANNING) {
            const double n = P.manning_coefficient[lane - 8];
            sc[SC_KF + lane - 8] = gf_mul(gf_mul(dt, g), gf_mul(n, n));
        }
        if (lane == 16) sc[SC_CFL] = 0.0;
    };
    for (int k = threadIdx.x; k < L::CNT_INTS; k += NT) cnt[k] = 0;
    __syncthreads();
    if (K > 1) {
        if (threadIdx.x == 0) stage(o, top);
        if (warp == NT / 32 - 1) constants();
    } else {
        /* the rows that hold a cell b4step2 would leave alone (h >= dry_tolerance) */
        constexpr int IT = (S + NT - 1) / NT;
        double h[IT];
#pragma unroll
        for (int it = 0; it < IT; ++it) {
            const int k = threadIdx.x + it * NT;
            h[it] = k < S ? wk.q[k] : -1.0;
        }
        unsigned lo = 0, hi = 0;
#pragma unroll
        for (int it = 0; it < IT; ++it) {
            const int k = threadIdx.x + it * NT, row = k / N;
            if (k < S && !d_lt<true>(h[it], drytol)) {
                if (row < 32) lo |= 1u << row;
                else hi |= 1u << (row - 32);
            }
        }
        lo = __reduce_or_sync(0xffffffffu, lo);
        hi = __reduce_or_sync(0xffffffffu, hi);
        if (lane == 0 && (lo | hi)) {
            atomicOr(&rows[0], lo);
            atomicOr(&rows[1], hi);
        }
        __syncthreads();
    }
    double* gq = wk.qout ? wk.qout : wk.q;
    /* interior rows r0 .. r1 - 1 without water: b4step2 alone changes them */
    auto write_dry = [&](int r0, int r1) {
        for (int e = threadIdx.x; e < (r1 - r0) * M; e += NT) {
            const int rr = e / M, k = (r0 + rr) * N + 2 + (e - rr * M);
            gq[k] = d_max<true>(wk.q[k], 0.0);
            gq[S + k] = 0.0;
            gq[2 * S + k] = 0.0;
        }
    };
    if (wk.fl && win == 0) { /* b4step2 changes a cell's bits unless h >= 0 and both momenta are +0 */
        int water = 0;
        for (int k = threadIdx.x; k < S; k += NT) {
            const double h = wk.q[k];
            if (d_lt<true>(h, drytol))
                changed |= (__double_as_longlong(h) < 0) | (__double_as_longlong(wk.q[S + k]) != 0) |
                           (__double_as_longlong(wk.q[2 * S + k]) != 0);
            else if (K > 1) water |= d_gt<true>(h, drytol);
        }
        changed = __syncthreads_or(changed);
        if (K > 1) {
            water = __syncthreads_or(water);
            if (threadIdx.x == 0) {
                wk.fl->ident = (!water && !changed) ? 1 : 0;
                wk.fl->wet = water ? 1 : 0;
            }
        }
    }
    if (K > 1) {
        const bool ok = __syncthreads_and(wait_staged());
        if (!ok) fail();
        /* the windows are written in place: none before all are staged */
        cluster_arrive();
        if (!ok) {
            cluster_wait();
            return false;
        }
        staged ^= 1u;
        prepare(o, threadIdx.x, (RW + 4) * N, NT);
        kept = __reduce_or_sync(0xffffffffu, kept);
        if (lane == 0 && kept) atomicOr(&rows[0], kept);
        __syncthreads();
    }
    const unsigned long long wrows = (unsigned long long)rows[1] << 32 | rows[0]; /* from row o */
    if (wrows == 0) {
        if (K > 1) cluster_wait();
        write_dry(o + 2, o + RW + 2);
        if (K == 1 && threadIdx.x == 0) {
            if (wk.fl) {
                wk.fl->ident = !changed ? 1 : 0;
                wk.fl->wet = 0;
            }
            if (cfl_out) cfl_out[wi] = 0.0;
            if (group_max) atomicMax(group_max + wk.group, dkey(0.0));
        }
        __syncthreads();
        return true;
    }
    /* bands b0 .. b1: the solves of the first wet row, up to the finish of the
     * row above the last */
    const int w0 = __ffsll((long long)wrows) - 1, w1 = 63 - __clzll((long long)wrows);
    const int b0 = max(w0 - 1, 0) / R, b1 = min(NB - 1, (min(w1 + 1, RW + 1) + 2 + R - 1) / R - 1);
    const int first = o + 1 + b0 * R; /* its array row */
    if (K == 1 && threadIdx.x == 0) stage(max(first - 3, 0), min(first + R, N));
    if (b0 > 0) /* the records below the first band */
        for (int k = L::OFF_WX + (int)threadIdx.x; k < L::OFF_SC; k += NT) sm[k] = 0.0;
    if (K == 1) {
        if (warp == NT / 32 - 1) constants();
        if (!__syncthreads_and(wait_staged())) return fail();
        prepare(max(first - 3, 0), threadIdx.x, (min(first + R, N) - max(first - 3, 0)) * N, NT);
        staged ^= 1u;
    }
    if (K == 1 || b0 > 0) __syncthreads();

    const double dtdx = sc[SC_DTDX], dtdy = sc[SC_DTDY], crit = sc[SC_CRIT], crit2 = sc[SC_CRIT2];
    const double hx = gf_mul(0.5, dtdx), hy = gf_mul(0.5, dtdy);
    const int fidx = P.friction_index - 1;
    double smax_x = 0.0, smax_y = 0.0;

    /* one place in the list of class k (k < 0: none) for every lane */
    auto place = [&](int* base_of, int k) -> int {
        const unsigned m = __match_any_sync(0xffffffffu, k);
        const int lead = __ffs(m) - 1;
        int base = 0;
        if (lane == lead && k >= 0) base = atomicAdd(&base_of[k], __popc(m));
        return __shfl_sync(0xffffffffu, base, lead) + __popc(m & ((1u << lane) - 1u));
    };
    /* the normal-solve faces of band b by class, as list_chunk: entries number
     * the x faces by row, then the y faces by row */
    auto list_a = [&](const Band& B, int par, int c) {
        const int na = B.nx * L::FA + B.ny * L::NC;
        const bool act = 32 * c + lane < na;
        const int i = act ? 32 * c + lane : 0;
        const bool y = i >= B.nx * L::FA;
        int kl, kr;
        bool wl, wr;
        if (!y) {
            const int ts = i / L::FA, row = B.a0 + ts, col = i - ts * L::FA;
            kl = L::slot(row) * N + col;
            kr = kl + 1;
            wl = wet[L::wi(row, col)] != 0;
            wr = wet[L::wi(row, col) + 1] != 0;
        } else {
            const int j = i - B.nx * L::FA, ts = j / L::NC, col = 1 + (j - ts * L::NC), f = B.a0 + ts;
            kl = L::slot(f - 1) * N + col;
            kr = L::slot(f) * N + col;
            wl = wet[L::wi(f - 1, col)] != 0;
            wr = wet[L::wi(f, col)] != 0;
        }
        const double* U = sm + (y ? L::OFF_V : L::OFF_U);
        int cls = 3;
        bool flag = false;
        if (wl | wr) {
            const int k = gf_face_class(gf_f32(sm[L::OFF_H + kl]), gf_f32(sm[L::OFF_H + kr]), gf_f32(U[kl]),
                                        gf_f32(U[kr]), gf_f32(sm[L::OFF_C + kl]), gf_f32(sm[L::OFF_C + kr]),
                                        gf_f32(sm[L::OFF_B + kl]), gf_f32(sm[L::OFF_B + kr]), wl, wr, gf_f32(g),
                                        gf_f32(crit), gf_f32(crit2));
            cls = k == 0 ? 0 : k == 3 ? 2 : 1;
            flag = k == 2;
        }
        const int pos = place(cnt + 4 * par, act ? cls : -1);
        if (act) {
            uint16_t* to = (cls == 1 || cls == 2) ? lm : la;
            to[cls >= 2 ? na - 1 - pos : pos] = (uint16_t)(i | (flag ? 0x8000 : 0));
        }
    };
    auto chunk_a = [&](const Band& B, int par, int c) {
        const int ns = cnt[4 * par], ne = cnt[4 * par + 1], nh = cnt[4 * par + 2], nd = cnt[4 * par + 3];
        const int nA = ns + ne + nh + nd, idx = 32 * c + lane;
        if (idx >= nA) return;
        const int v = idx < nh ? lm[nA - 1 - idx] : idx < nh + ne ? lm[idx - nh] : idx < nA - nd ? la[idx - nh - ne] : la[idx];
        const int i = v & 0x7fff;
        const bool y = i >= B.nx * L::FA;
        int kl, kr;
        bool wl, wr;
        double* w;
        if (!y) {
            const int ts = i / L::FA, row = B.a0 + ts, col = i - ts * L::FA;
            kl = L::slot(row) * N + col;
            kr = kl + 1;
            wl = wet[L::wi(row, col)] != 0;
            wr = wet[L::wi(row, col) + 1] != 0;
            w = sm + L::OFF_WX + i * L::WS;
        } else {
            const int j = i - B.nx * L::FA, ts = j / L::NC, col = 1 + (j - ts * L::NC), f = B.a0 + ts;
            kl = L::slot(f - 1) * N + col;
            kr = L::slot(f) * N + col;
            wl = wet[L::wi(f - 1, col)] != 0;
            wr = wet[L::wi(f, col)] != 0;
            w = sm + L::OFF_WY + ((f % L::RWY) * L::NC + col - 1) * L::WS;
        }
        if (idx >= nA - nd) { /* both cells dry: no waves */
#pragma unroll
            for (int q = 0; q < L::WS; ++q) w[q] = 0.0;
            return;
        }
        const gf_cell cl = stream_cell<L>(sm, wl, kl, y), cr = stream_cell<L>(sm, wr, kr, y);
        double s[3], fw[3][3];
        if (idx < nh) {
            full_solve(cl, cr, g, drytol, sc, w);
            s[0] = w[0]; s[1] = w[1]; s[2] = w[2];
        } else {
            if (32 * c < nh + ne) gf_rpn2_edge(cl, cr, (v & 0x8000) != 0, g, crit, crit2, s, fw);
            else gf_rpn2_smooth(cl, cr, g, s, fw);
            w[0] = s[0]; w[1] = s[1]; w[2] = s[2];
            w[3] = fw[0][0]; w[4] = fw[0][1]; w[5] = fw[0][2];
            w[6] = fw[1][1];
            w[7] = fw[2][0]; w[8] = fw[2][1]; w[9] = fw[2][2];
        }
        const double m = d_max_abs<true>(d_max_abs<true>(d_max_abs<true>(y ? smax_y : smax_x, s[0]), s[1]), s[2]);
        if (y) smax_y = m;
        else smax_x = m;
    };
    /* limited face i of band b: its records and its cells' wet flags */
    auto limited = [&](const Band& B, int i, int& w, int& wl, int& wr, int& o, int& kl, int& kr) -> bool {
        const bool y = i >= B.nx * L::FB;
        if (!y) {
            const int ts = i / L::FB, n = 1 + (i - ts * L::FB);
            w = L::OFF_WX + (ts * L::FA + n) * L::WS;
            wl = w - L::WS;
            wr = w + L::WS;
            o = L::OFF_OX + i * L::OS;
            kl = L::wi(B.a0 + ts, n);
            kr = kl + 1;
        } else {
            const int j = i - B.nx * L::FB, ts = j / L::NC, c = j - ts * L::NC, f = B.l0 + ts;
            w = L::OFF_WY + ((f % L::RWY) * L::NC + c) * L::WS;
            wl = L::OFF_WY + (((f - 1) % L::RWY) * L::NC + c) * L::WS;
            wr = L::OFF_WY + (((f + 1) % L::RWY) * L::NC + c) * L::WS;
            o = L::OFF_OY + ((f % L::ROY) * L::NC + c) * L::OS;
            kl = L::wi(f - 1, c + 1);
            kr = L::wi(f, c + 1);
        }
        return y;
    };
    auto list_b = [&](const Band& B, int par, int c) {
        const int nb = B.nx * L::FB + B.nl * L::NC, i = 32 * c + lane;
        const bool act = i < nb;
        bool dry = false;
        if (act) {
            int w, wl, wr, o, kl, kr;
            limited(B, i, w, wl, wr, o, kl, kr);
            dry = !(wet[kl] | wet[kr]);
        }
        const int pos = place(cnt + L::CNT_B + 2 * par, act ? (dry ? 1 : 0) : -1);
        if (act) lb[dry ? nb - 1 - pos : pos] = (uint16_t)i;
    };
    auto chunk_b1 = [&](const Band& B, int par, int c) {
        const int nw = cnt[L::CNT_B + 2 * par], idx = 32 * c + lane;
        if (idx >= nw + cnt[L::CNT_B + 2 * par + 1]) return;
        int w, wl, wr, o, kl, kr;
        const bool y = limited(B, lb[idx], w, wl, wr, o, kl, kr);
        double* op = sm + o;
        if (idx >= nw) {
#pragma unroll
            for (int q = 0; q < L::OS; ++q) op[q] = 0.0;
            return;
        }
        double amdq[3], apdq[3], cq[3];
        face_terms_fast(sm + w, sm + wl, sm + wr, P, y ? dtdy : dtdx, amdq, apdq, cq);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            op[k] = amdq[k];
            op[3 + k] = apdq[k];
            op[6 + k] = cq[k];
        }
    };
    auto chunk_b2 = [&](const Band& B, int c) {
        const int i = 32 * c + lane;
        if (i >= B.nx * M + B.nc * L::NC) return;
        const bool y = i >= B.nx * M;
        int k, w, wl, wr, k_lo, k_hi; /* the cell, wet flags along the sweep, neighbours across it */
        const double *ol, *orr;
        double* r;
        if (!y) {
            const int ts = i / M, n = i - ts * M, row = B.a0 + ts; /* array column n + 2 */
            k = L::slot(row) * N + n + 2;
            w = L::wi(row, n + 2);
            wl = w - 1;
            wr = w + 1;
            k_lo = L::slot(row - 1) * N + n + 2;
            k_hi = L::slot(row + 1) * N + n + 2;
            ol = sm + L::OFF_OX + (ts * L::FB + n) * L::OS;
            orr = ol + L::OS;
            r = sm + L::OFF_CX + ((row % L::RCX) * M + n) * L::CS;
        } else {
            const int j = i - B.nx * M, ts = j / L::NC, n = j - ts * L::NC, row = B.c0 + ts; /* array column n + 1 */
            k = L::slot(row) * N + n + 1;
            w = L::wi(row, n + 1);
            wl = L::wi(row - 1, n + 1);
            wr = L::wi(row + 1, n + 1);
            k_lo = k - 1;
            k_hi = k + 1;
            ol = sm + L::OFF_OY + ((row % L::ROY) * L::NC + n) * L::OS;
            orr = sm + L::OFF_OY + (((row + 1) % L::ROY) * L::NC + n) * L::OS;
            r = sm + L::OFF_CY + ((row % L::RCY) * L::NC + n) * L::CS;
        }
        if (!(wet[wl] | wet[w] | wet[wr])) { /* both faces between dry cells: no waves */
#pragma unroll
            for (int q = 0; q < L::CS; ++q) r[q] = 0.0;
            return;
        }
        double Nv[3], bm[3], bp[3];
        cell_terms(ol, orr, stream_cell<L>(sm, wet[w] != 0, k, y), sm[L::OFF_B + k_lo], sm[L::OFF_B + k_hi], P.transverse, Nv,
                   bm, bp);
        /* global component order (h, hu, hv) */
        const int g1 = y ? 2 : 1, g2 = y ? 1 : 2;
        r[0] = Nv[0]; r[g1] = Nv[1]; r[g2] = Nv[2];
        r[3] = bp[0]; r[3 + g1] = bp[1]; r[3 + g2] = bp[2];
        r[6] = bm[0]; r[6 + g1] = bm[1]; r[6 + g2] = bm[2];
    };
    /* finished cells: the sums of the sweeps in their order, the update and the
     * friction term */
    auto chunk_g = [&](const Band& B, int c) {
        const int i = 32 * c + lane;
        if (i >= B.nc * M) return;
        const int ts = i / M, n = i - ts * M, row = B.c0 + ts;
        const double* xb = sm + L::OFF_CX + (((row - 1) % L::RCX) * M + n) * L::CS;
        const double* xo = sm + L::OFF_CX + ((row % L::RCX) * M + n) * L::CS;
        const double* xa = sm + L::OFF_CX + (((row + 1) % L::RCX) * M + n) * L::CS;
        const double* yo = sm + L::OFF_CY + ((row % L::RCY) * L::NC + n + 1) * L::CS; /* columns i - 1, i, i + 1 */
        const double *yb = yo - L::CS, *ya = yo + L::CS;
        const int k = L::slot(row) * N + n + 2;
        double q[3] = {sm[L::OFF_H + k], sm[L::OFF_HU + k], sm[L::OFF_HV + k]};
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            double DY = gf_mul(hx, xb[3 + m]);
            DY = fma(hx, gf_sub(xo[6 + m], xo[3 + m]), DY);
            DY = fma(-hx, xa[6 + m], DY);
            double DX = fma(hy, yb[3 + m], xo[m]);
            DX = fma(hy, gf_sub(yo[6 + m], yo[3 + m]), DX);
            DX = fma(-hy, ya[6 + m], DX);
            DY = gf_add(DY, yo[m]);
            q[m] = fma(-dtdy, DY, fma(-dtdx, DX, q[m]));
        }
        const int e = row * N + n + 2;
        if (P.src_term > 0) {
            const double nvar = (P.variable_friction && fidx >= 0 && fidx < maux) ? wk.aux[(size_t)fidx * S + e] : 0.0;
            src2_cell<true>(P, dt, sc + SC_KF, sm[L::OFF_B + k], nvar, q[0], q[1], q[2]);
        }
        gq[e] = q[0];
        gq[S + e] = q[1];
        gq[2 * S + e] = q[2];
    };

    {
        const Band B0(b0, o);
        for (int c = warp; 32 * c < B0.nx * L::FA + B0.ny * L::NC; c += NT / 32) list_a(B0, b0 & 1, c);
    }
    __syncthreads();
    int* cur = cnt + L::CNT_CUR;
    auto next = [&](int ph) -> int {
        int c = 0;
        if (lane == 0) c = atomicAdd(&cur[ph], 1);
        return __shfl_sync(0xffffffffu, c, 0);
    };
    auto chunks = [](int n) { return (n + 31) / 32; };
    for (int b = b0;; ++b) {
        /* more: rows above the band still to come (the last band's records need
         * the bathymetry above it); mlist: a next band to list */
        const bool have = b <= b1, more = K == 1 && have && b + 1 < NB, mlist = b < b1;
        const Band B(b, o), Bp(b - 1, o);
        const int par = b & 1;
        /* ---- A | B2 of the band before | dry list | next rows ---- */
        const int r0 = 1 + (b + 1) * R, r1 = more ? min(r0 + R, N) : r0;
        if (more && threadIdx.x == 0) stage(r0, r1);
        const int ca = have ? chunks(B.nx * L::FA + B.ny * L::NC) : 0, c2 = b > b0 ? chunks(Bp.nx * M + Bp.nc * L::NC) : 0;
        const int cl = have ? chunks(B.nx * L::FB + B.nl * L::NC) : 0;
        const int cp = chunks((r1 - r0) * N);
        bool ok = true;
        for (int c; (c = next(2 * b)) < ca + c2 + cl + cp;) {
            if (c < ca) {
                chunk_a(B, par, c);
            } else if ((c -= ca) < c2) {
                chunk_b2(Bp, c);
            } else if ((c -= c2) < cl) {
                list_b(B, par, c);
            } else {
                c -= cl;
                ok = ok && wait_staged();
                if (ok) prepare(r0, 32 * c + lane, min((r1 - r0) * N, 32 * c + 32), 32);
            }
        }
        if (!__syncthreads_and(ok)) return fail();
        /* the counts of the next lists start at zero; nobody reads them now */
        if (threadIdx.x < 2) cnt[L::CNT_B + 2 * (par ^ 1) + threadIdx.x] = 0;
        /* ---- B1 | class list of the next band | finished rows ---- */
        if (more) staged ^= 1u;
        const Band Bn(b + 1, o);
        if (K > 1 && b == b0 + 1) cluster_wait(); /* the first rows to be written */
        const int c1 = cl, cn = mlist ? chunks(Bn.nx * L::FA + Bn.ny * L::NC) : 0, cg = b > b0 ? chunks(Bp.nc * M) : 0;
        for (int c; (c = next(2 * b + 1)) < c1 + cn + cg;) {
            if (c < c1) chunk_b1(B, par, c);
            else if ((c -= c1) < cn) list_a(Bn, par ^ 1, c);
            else chunk_g(Bp, c - cn);
        }
        /* the next staging overwrites rows read here */
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (threadIdx.x < 4) cnt[4 * par + threadIdx.x] = 0;
        if (!have) break;
    }
    phase = staged;
    {
        const Band B0(b0, o), B1(b1, o);
        write_dry(o + 2, B0.c0);
        write_dry(B1.c0 + B1.nc, o + RW + 2);
    }

    if (K == 1 && wk.fl) {
        any_wet = __syncthreads_or(any_wet);
        if (threadIdx.x == 0) {
            wk.fl->ident = (!any_wet && !changed) ? 1 : 0;
            wk.fl->wet = any_wet ? 1 : 0;
        }
    }
    {
        unsigned long long v = dkey(d_max_nn<true>(dtdx * smax_x, dtdy * smax_y));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long w = __shfl_xor_sync(0xffffffffu, v, o);
            v = w > v ? w : v;
        }
        if (lane == 0) atomicMax(reinterpret_cast<unsigned long long*>(sc + SC_CFL), v);
    }
    __syncthreads();
    if (K > 1) { /* the cluster forms the patch CFL */
        if (threadIdx.x == 0) *part = sc[SC_CFL];
    } else if (threadIdx.x == 0) {
        double cfl = sc[SC_CFL];
        if (cfl > P.maxcfl_cap) cfl = 0.0;
        if (cfl_out) cfl_out[wi] = cfl;
        if (group_max) atomicMax(group_max + wk.group, dkey(cfl));
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    return true;
}

template <int M, int NT, int R, int MINB>
__global__ void __launch_bounds__(NT, MINB)
    patch_update_stream_kernel(const gf_patch_work* __restrict__ work, int nwork,
                               const gf_phys* __restrict__ phys_table, double dt_uniform,
                               const double* __restrict__ group_dt, const int* __restrict__ group_par,
                               int maux, double* __restrict__ cfl_out,
                               unsigned long long* __restrict__ group_max, int* __restrict__ err)
{
    using L = StreamSmem<M, R>;
    extern __shared__ __align__(128) double sm[];
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm + L::OFF_BAR);
    if (threadIdx.x == 0) mbar_init(bar, 1);
    __syncthreads();
    uint32_t phase = 0;
    for (int wi = blockIdx.x; wi < nwork; wi += gridDim.x)
        if (!stream_item<M, NT, R>(sm, bar, phase, work[wi], wi, phys_table, dt_uniform, group_dt, group_par, maux,
                                   cfl_out, group_max, err))
            return;
}

/* A patch over a cluster of K CTAs on K SMs: CTA r finishes the rows r M / K ..
 * of the interior and solves the faces that these read, the ones at its edges
 * once more than its neighbour does, so nothing but the speeds passes between
 * the CTAs. The patch CFL is the largest of theirs, read by CTA 0 through
 * distributed shared memory; the last barrier keeps every CTA until then. */
template <int M, int NT, int R, int K, int MINB>
__global__ void __cluster_dims__(K, 1, 1) __launch_bounds__(NT, MINB)
    patch_update_window_kernel(const gf_patch_work* __restrict__ work, int nwork,
                               const gf_phys* __restrict__ phys_table, double dt_uniform,
                               const double* __restrict__ group_dt, const int* __restrict__ group_par,
                               int maux, double* __restrict__ cfl_out,
                               unsigned long long* __restrict__ group_max, int* __restrict__ err)
{
    static_assert(M % K == 0 && M / K + 4 <= 32, "rows split evenly, their flags in one word");
    namespace cg = cooperative_groups;
    using L = StreamSmem<M, R, K>;
    extern __shared__ __align__(128) double sm[];
    cg::cluster_group cluster = cg::this_cluster();
    const int r = (int)cluster.block_rank();
    const int wi = blockIdx.x / K;
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm + L::OFF_BAR);
    double* part = sm + L::OFF_SC + SC_PART;
    if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        *part = 0.0;
    }
    __syncthreads();
    /* these tests are the same on every CTA of the cluster: it leaves whole */
    if (wi >= nwork) return;
    const gf_patch_work wk = work[wi];
    if (group_dt && !(group_dt[wk.group] > 0.0)) return;
    if (wk.fl && wk.fl->skip) return;
    uint32_t phase = 0;
    stream_item<M, NT, R, K>(sm, bar, phase, wk, wi, phys_table, dt_uniform, group_dt, group_par, maux, cfl_out,
                             group_max, err, r, part);
    cluster.sync();
    if (r == 0 && threadIdx.x == 0) {
        double cfl = 0.0;
        for (int q = 0; q < K; ++q) cfl = d_max_nn<true>(cfl, *cluster.map_shared_rank(part, q));
        if (cfl > phys_table[wk.phys].maxcfl_cap) cfl = 0.0;
        if (cfl_out) cfl_out[wi] = cfl;
        if (group_max) atomicMax(group_max + wk.group, dkey(cfl));
    }
    cluster.sync();
}

/* Every patch size in one persistent launch, as patch_update_mixed_kernel,
 * two CTAs an SM. */
template <int R8, int R16, int R32>
struct MixedStreamSmem {
    static constexpr size_t B8 = StreamSmem<8, R8>::BYTES, B16 = StreamSmem<16, R16>::BYTES,
                            B32 = StreamSmem<32, R32>::BYTES;
    static constexpr size_t MAXB = B8 > B16 ? (B8 > B32 ? B8 : B32) : (B16 > B32 ? B16 : B32);
    static constexpr size_t OFF_CTL = (MAXB + 15) / 16 * 16; /* mbarrier, two cursor slots */
    static constexpr size_t BYTES = OFF_CTL + 32;
};

template <int NT, int R8, int R16, int R32>
__global__ void __launch_bounds__(NT, 2)
    patch_update_mixed_stream_kernel(const gf_patch_work* __restrict__ work, int n32, int n16, int n8,
                                     const gf_phys* __restrict__ phys_table, double dt_uniform,
                                     const double* __restrict__ group_dt, const int* __restrict__ group_par,
                                     int maux, double* __restrict__ cfl_out,
                                     unsigned long long* __restrict__ group_max, int* __restrict__ err,
                                     unsigned int* __restrict__ sched)
{
    using X = MixedStreamSmem<R8, R16, R32>;
    extern __shared__ __align__(128) double sm[];
    uint64_t* bar = reinterpret_cast<uint64_t*>(reinterpret_cast<char*>(sm) + X::OFF_CTL);
    volatile int* slot = reinterpret_cast<volatile int*>(reinterpret_cast<char*>(sm) + X::OFF_CTL + 8);
    if (threadIdx.x == 0) mbar_init(bar, 1);
    __syncthreads();
    const int nwork = n32 + n16 + n8;
    uint32_t phase = 0;
    /* cursor and its two slots: see patch_update_mixed_kernel */
    for (int it = 0;; ++it) {
        if (threadIdx.x == 0) slot[it & 1] = (int)atomicAdd(sched, 1u);
        __syncthreads();
        const int wi = slot[it & 1];
        if (wi >= nwork) break;
        bool ok;
        if (wi < n32)
            ok = stream_item<32, NT, R32>(sm, bar, phase, work[wi], wi, phys_table, dt_uniform, group_dt, group_par,
                                          maux, cfl_out, group_max, err);
        else if (wi < n32 + n16)
            ok = stream_item<16, NT, R16>(sm, bar, phase, work[wi], wi, phys_table, dt_uniform, group_dt, group_par,
                                          maux, cfl_out, group_max, err);
        else
            ok = stream_item<8, NT, R8>(sm, bar, phase, work[wi], wi, phys_table, dt_uniform, group_dt, group_par,
                                        maux, cfl_out, group_max, err);
        if (!ok) break;
    }
    if (threadIdx.x == 0) {
        if (atomicAdd(sched + 1, 1u) == gridDim.x - 1) {
            atomicExch(sched, 0u);
            atomicExch(sched + 1, 0u);
        }
    }
}

} // namespace GF_KNS

#endif
