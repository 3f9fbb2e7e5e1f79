/*
 * Fused GeoClaw patch update for sm_103a: b4step2 + step2 + CFL + src2 on a
 * batch of patches, one CTA per patch.
 *
 * Reference behaviour (paths relative to the GeoFlood source tree):
 *   geoclaw_update              src/fc2d_geoclaw/fc2d_geoclaw.cpp:352-387
 *   b4step2                     fortran_source/geoclaw_b4step2_fort.f90:183-186
 *   step2 sweeps                fortran_source/geoclaw_step2_fort.f90:80-250
 *   flux2 (f-wave form)         fortran_source/geoclaw_flux2fw_fort.f:113-267
 *   limiter / philim            fortran_source/geoclaw_limiter_fort.f:34-58, philim.f
 *   flux-difference update      fortran_source/geoclaw_step2_wrap_fort.f:95-115
 *   src2 (Manning friction)     fortran_source/geoclaw_src2_fort.f90:41-71
 *
 * The kernel computes exactly the faces the interior update depends on:
 * normal solves on faces 0..m+2 of slices 0..m+1, limiting / transverse
 * splitting on faces 1..m+1 (the Fortran's own ranges), and writes the
 * interior cells only. Ghost cells are refilled by the ghost-fill step
 * before they are read again, so their post-step values are not part of
 * the state.
 *
 * The update is FP64-issue bound on GB300 (the FP64 pipe, not HBM, is the
 * ceiling), so the layout of the work aims at few FP64 instructions and
 * uniform warps:
 *   - per-cell quotients computed once (hu/h, hv/h, sqrt(g h), and in the
 *     contracted build 1/sqrt(g h));
 *   - the faces of each band are listed by class (both cells wet, with the
 *     short solve or the full one; one wet; both dry) so a warp runs one
 *     code path; dry faces only store zeros;
 *   - the per-face outputs of a band go to shared memory and each interior
 *     cell gathers its six contributing faces in slice order, so every cell
 *     is written by one thread per band, in a fixed order: deterministic and
 *     independent of launch shape (no atomics on the data).
 *
 * EXACT = true is the parity build: the reference's four flux accumulators
 * fm, fp, gm, gp summed in its order and every division as written; compiled
 * with floating-point contraction off it reproduces the Fortran's rounding.
 */
#ifndef GF_PATCH_UPDATE_CUH
#define GF_PATCH_UPDATE_CUH

#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "gf_riemann.cuh"
#include "gf_types.h"

#ifndef GF_KNS
#define GF_KNS gf
#endif

namespace GF_KNS {

/* ---- bulk-async (TMA) copy + mbarrier helpers (inline PTX, sm_90+) ---- */
__device__ __forceinline__ uint32_t smem_u32(const void* p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
                 : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar)
{
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}
/* Polls of a wait before it gives up: a poll of a phase that does not
 * complete suspends about 3.8 us on GB300 (gf_probe_bounded_wait), so the
 * limit is about half a second, far above any staging copy. */
constexpr uint32_t kWaitPolls = 1u << 17;

/* Bounded wait on phase `parity`; returns false if the limit ran out. */
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, uint32_t max_iter)
{
    for (uint32_t it = 0; it < max_iter; ++it) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

/* Barrier of the CTAs of a cluster, in two halves. */
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.aligned;" ::: "memory"); }

/* sign(s) * x for the limiter's factor: x with its sign bit flipped when s
 * is negative (-0 included), on the integer pipe instead of a product */
__device__ __forceinline__ double with_sign_of(double x, double s)
{
    const unsigned long long ux = static_cast<unsigned long long>(__double_as_longlong(x));
    const unsigned long long us = static_cast<unsigned long long>(__double_as_longlong(s));
    return __longlong_as_double(static_cast<long long>(ux ^ (us & 0x8000000000000000ull)));
}

/* Order-preserving key of a non-negative double (for atomicMax). */
__device__ __forceinline__ unsigned long long dkey(double v)
{
    return static_cast<unsigned long long>(__double_as_longlong(v));
}

template <int M>
struct Geo {
    static constexpr int N = M + 2 * GF_MBC; /* cells per row incl. halo */
    static constexpr int S = N * N;          /* cells per plane          */
    static constexpr int FA = M + 3;         /* normal-solve faces/slice */
    static constexpr int FB = M + 1;         /* limited faces / slice    */
    static constexpr int NSLICE = M + 2;     /* slices 0..m+1            */
};

/* Shared-memory layout (doubles unless noted). NACC flux accumulators of 3
 * components per interior cell: 2 (DX, DY) in the contracted build, 4 (fm,
 * fp, gm, gp) in the exact build. The contracted build also keeps a
 * 1/sqrt(g h) plane. */
template <int M, int RB, bool EXACT = false>
struct Smem {
    using G = Geo<M>;
    static constexpr int NACC = EXACT ? 4 : 2;
    static constexpr int NBAND = (G::NSLICE + RB - 1) / RB;
    /* Odd strides (in doubles) spread a warp's accesses to face records and
     * accumulator rows over the shared-memory banks. Face record: s[3] +
     * fw[3][3] (1 pad) in the exact build; the contracted build leaves out the
     * middle f-wave's two zero components: s[3], fw0[3], fw1[1], fw2[3], 1 pad */
    static constexpr int W_STRIDE = EXACT ? 13 : 11;
    /* limited-face records: exact build faddm faddp A B C D (3 comps each, 1
     * pad); contracted build amdq apdq cq (local order) */
    static constexpr int O_STRIDE = EXACT ? 19 : 9;
    /* per-cell records of the contracted build: N (flux difference), U (up-going
     * and Dn (down-going transverse parts), global order, one slot per face slot */
    static constexpr int C_STRIDE = 9;
    static constexpr int MS = M + 1;    /* accumulator row stride            */
    static constexpr int PLANE = M * MS; /* one accumulator component        */
    static constexpr int OFF_H = 0;
    static constexpr int OFF_HU = OFF_H + G::S;
    static constexpr int OFF_HV = OFF_HU + G::S;
    static constexpr int OFF_B = OFF_HV + G::S;
    static constexpr int OFF_U = OFF_B + G::S;
    static constexpr int OFF_V = OFF_U + G::S;
    static constexpr int OFF_C = OFF_V + G::S;
    static constexpr int OFF_RC = OFF_C + G::S;                     /* contracted only */
    static constexpr int OFF_ACC = OFF_RC + (EXACT ? 0 : G::S);     /* NACC x [3][M*M] */
    static constexpr int OFF_W = OFF_ACC + NACC * 3 * PLANE;
    static constexpr int OFF_O = OFF_W + RB * G::FA * W_STRIDE;
    static constexpr int OFF_C2 = OFF_O + RB * G::FB * O_STRIDE;   /* contracted only */
    /* per item: dt/dx, dt/dy, 1/(16 g), 1/sqrt(g), the sonic tolerances, the
     * friction factors, the CFL maximum (SC_*) */
    static constexpr int OFF_SC = OFF_C2 + (EXACT ? 0 : RB * G::FB * C_STRIDE);
    static constexpr int OFF_BAR = OFF_SC + 16;                     /* 1 x u64     */
    /* integer region: class counts per band and face lists (u16) */
    static constexpr int OFF_INT = OFF_BAR + 2;
    static constexpr int NCLS = 5;                                  /* face classes, see build_lists */
    /* exact: [band][A|B][class][count|pos]; contracted: [sweep][band][A classes
     * smooth, edge, full, dry | B classes wet, dry], then a chunk cursor per
     * phase of each sweep */
    static constexpr int CNT_SWEEP = NBAND * 6, CNT_CUR = 2 * CNT_SWEEP, CUR_SWEEP = 2 * (NBAND + 1);
    static constexpr int CNT_INTS = EXACT ? NBAND * 2 * NCLS * 2 : CNT_CUR + 2 * CUR_SWEEP;
    static constexpr int LIST_A = G::NSLICE * G::FA;
    static constexpr int LIST_B = G::NSLICE * G::FB;
    /* contracted: also a list of edge and full-solve faces, and all three for
     * either sweep (the y sweep's are made during the x sweep) */
    static constexpr int LIST_SWEEP = 2 * LIST_A + LIST_B;
    static constexpr int LISTS = EXACT ? LIST_A + LIST_B : 2 * LIST_SWEEP;
    static constexpr size_t INT_BYTES = ((CNT_INTS * 4 + LISTS * 2) + 15) / 16 * 16;
    static constexpr size_t OFF_WET_BYTES = (size_t)OFF_INT * 8 + INT_BYTES;
    /* exact: class of each normal-solve face of the sweep (u8), kept between
     * the count and place passes */
    static constexpr size_t OFF_FCLS_BYTES = OFF_WET_BYTES + ((G::S + 15) / 16) * 16;
    static constexpr size_t BYTES = OFF_FCLS_BYTES + (EXACT ? ((LIST_A + 15) / 16) * 16 : 0);
};

enum { SC_DTDX, SC_DTDY, SC_C16G, SC_RSG, SC_CRIT, SC_CRIT2, SC_KF, SC_CFL = SC_KF + GF_MAX_MANNING, SC_PART };

/* Load the cell view for a face sweep in direction DIR (0 = x, 1 = y). */
template <int DIR, bool EXACT, class L>
__device__ __forceinline__ gf_cell load_cell(const double* sm, const unsigned char* wet, int k)
{
    gf_cell c;
    c.h = sm[L::OFF_H + k];
    c.b = sm[L::OFF_B + k];
    c.c = sm[L::OFF_C + k];
    c.wet = wet[k] != 0;
    if (DIR == 0) {
        c.hun = sm[L::OFF_HU + k]; c.hut = sm[L::OFF_HV + k];
        c.un = sm[L::OFF_U + k];   c.ut = sm[L::OFF_V + k];
    } else {
        c.hun = sm[L::OFF_HV + k]; c.hut = sm[L::OFF_HU + k];
        c.un = sm[L::OFF_V + k];   c.ut = sm[L::OFF_U + k];
    }
    c.rc = EXACT ? 0.0 : sm[L::OFF_RC + k];
    return c;
}

/* The faces one sweep computes. The x sweep takes the slices (rows) 0..M + 1,
 * the y sweep the columns; records of a band are packed by the faces of a slice
 * (fa, fb). */
template <int M, int RB>
struct SweepWin {
    static constexpr int ts_lo = 0, nsl = M + 2; /* slices ts_lo .. ts_lo + nsl - 1           */
    static constexpr int na_lo = 0, fa = M + 3;  /* normal-solve faces na_lo .. na_lo + fa - 1 */
    static constexpr int nb_lo = 1, fb = M + 1;  /* limited faces nb_lo .. nb_lo + fb - 1      */
    static constexpr int rb = RB;                /* slices per band                            */
};

/* The full solve into a face record (contracted build). Not inlined: faces
 * that need it are few, its registers stay its own, and the kernels share one
 * body of it and so its bits. */
static __device__ __noinline__ void full_solve(const gf_cell& cl, const gf_cell& cr, double g, double drytol,
                                               const double* sc, double* w)
{
    double s[3], fw[3][3];
    gf_rpn2_face<true>(cl, cr, g, drytol, sc[SC_C16G], sc[SC_RSG], sc[SC_CRIT], sc[SC_CRIT2], s, fw);
    w[0] = s[0]; w[1] = s[1]; w[2] = s[2];
    w[3] = fw[0][0]; w[4] = fw[0][1]; w[5] = fw[0][2];
    w[6] = fw[1][1];
    w[7] = fw[2][0]; w[8] = fw[2][1]; w[9] = fw[2][2];
}

/* A sweep's face lists in shared memory: class counts, cursors, lists. */
struct SweepLists {
    int* cnt;
    int* cur;
    uint16_t *la, *lb, *lm;
};

/* Contracted build: the faces 32 c .. 32 c + 31 of one band of a sweep into
 * the band's lists by class (gf_face_class), so that a warp of the solves runs
 * one code path. Normal solves: edge faces (lm from the front, their flag in
 * bit 15), faces for the full solve (lm from the back), smooth faces (la from
 * the front), both cells dry (la from the back); limited faces: some water (lb
 * from the front), none (from the back). Lists filled from both ends need no
 * counts beforehand, and a warp's faces of one class take their places with
 * one atomic. */
template <int M, int RB, int DIR>
__device__ __forceinline__ void list_chunk(const double* sm, const unsigned char* wet, const SweepLists& ls, double g,
                                           double crit, double crit2, int band, int c)
{
    constexpr SweepWin<M, RB> w{};
    using L = Smem<M, RB, false>;
    constexpr int N = Geo<M>::N;
    const double* U = sm + (DIR == 0 ? L::OFF_U : L::OFF_V);
    const int lane = threadIdx.x & 31;
    const int ns = min(w.rb, w.nsl - band * w.rb), na = ns * w.fa;
    if (32 * c >= na) return; /* the whole warp */
    const bool act = 32 * c + lane < na;
    const int i = act ? 32 * c + lane : 0;
    const int ts = i / w.fa, n = w.na_lo + (i - ts * w.fa), t = w.ts_lo + band * w.rb + ts;
    const int kl = DIR == 0 ? (t + 1) * N + n : n * N + (t + 1), kr = kl + (DIR == 0 ? 1 : N);
    const bool wl = wet[kl] != 0, wr = wet[kr] != 0;
    int cls = 3; /* 0 smooth, 1 edge, 2 full, 3 dry */
    bool flag = false;
    if (wl | wr) {
        const int k = gf_face_class(gf_f32(sm[L::OFF_H + kl]), gf_f32(sm[L::OFF_H + kr]), gf_f32(U[kl]), gf_f32(U[kr]),
                                    gf_f32(sm[L::OFF_C + kl]), gf_f32(sm[L::OFF_C + kr]), gf_f32(sm[L::OFF_B + kl]),
                                    gf_f32(sm[L::OFF_B + kr]), wl, wr, gf_f32(g), gf_f32(crit), gf_f32(crit2));
        cls = k == 0 ? 0 : k == 3 ? 2 : 1;
        flag = k == 2;
    }
    /* one place in the list of class k (k < 0: none) for every lane */
    auto place = [&](int k) -> int {
        const unsigned m = __match_any_sync(0xffffffffu, k);
        const int lead = __ffs(m) - 1;
        int base = 0;
        if (lane == lead && k >= 0) base = atomicAdd(&ls.cnt[band * 6 + k], __popc(m));
        return __shfl_sync(0xffffffffu, base, lead) + __popc(m & ((1u << lane) - 1u));
    };
    const int pa = place(act ? cls : -1);
    if (act) {
        uint16_t* to = ((cls == 1 || cls == 2) ? ls.lm : ls.la) + band * w.rb * w.fa;
        to[cls >= 2 ? na - 1 - pa : pa] = (uint16_t)(i | (flag ? 0x8000 : 0));
    }
    const bool limited = act && n >= w.nb_lo && n < w.nb_lo + w.fb, dry = cls == 3;
    const int pb = place(limited ? (dry ? 5 : 4) : -1);
    if (limited)
        ls.lb[band * w.rb * w.fb + (dry ? ns * w.fb - 1 - pb : pb)] = (uint16_t)(ts * w.fb + (n - w.nb_lo));
}

/* Exact build: for every band of one sweep direction, the normal-solve faces
 * (list A) and the limited faces (list B) ordered by class. Classes: 0..2
 * both cells wet, by the wave structure riemanntype will find (0 two shocks,
 * the costly branch, first so that one class boundary at most splits its
 * warps; 1 two rarefactions; 2 a shock and a rarefaction; list B puts all wet
 * pairs in class 0); 3 one cell wet; 4 both dry. The wave structure is
 * estimated without a square root (F_max <= 0 as delu <= 0 and
 * delu^2 hmin hmax >= (hmax - hmin)^2 g (hmin + hmax) / 2); it only orders the
 * list. Two passes (count, then place) over all faces. */
template <int M, int NT, int RB, int DIR>
__device__ __forceinline__ void build_lists_exact(const double* sm, const unsigned char* wet, int* cnt, uint16_t* la,
                                                  uint16_t* lb, double g)
{
    constexpr SweepWin<M, RB> w{};
    using G = Geo<M>;
    using L = Smem<M, RB, true>;
    constexpr int N = G::N;
    constexpr int NC = L::NCLS;
    unsigned char* fcls = const_cast<unsigned char*>(reinterpret_cast<const unsigned char*>(sm)) + L::OFF_FCLS_BYTES;
    auto cidx = [](int n, int t) -> int {
        return DIR == 0 ? (t + 1) * N + (n + 1) : (n + 1) * N + (t + 1);
    };
    /* cnt layout: [band][list 0|1][class 0..4][0 = count, 1 = position] */
    auto C = [&](int band, int list, int cls, int w2) -> int& {
        return cnt[((band * 2 + list) * NC + cls) * 2 + w2];
    };
    for (int k = threadIdx.x; k < L::CNT_INTS; k += NT) cnt[k] = 0;
    __syncthreads();
    for (int f = threadIdx.x; f < w.nsl * w.fa; f += NT) {
        const int ts = f / w.fa, n = w.na_lo + f % w.fa;
        const int t = w.ts_lo + ts;
        const int kl = cidx(n - 1, t), kr = cidx(n, t);
        const int nw = wet[kl] + wet[kr];
        int cls = nw == 0 ? 4 : nw == 1 ? 3 : 0;
        if (nw == 2) {
            const double hL = sm[L::OFF_H + kl], hR = sm[L::OFF_H + kr];
            const double uL = sm[(DIR == 0 ? L::OFF_U : L::OFF_V) + kl];
            const double uR = sm[(DIR == 0 ? L::OFF_U : L::OFF_V) + kr];
            const double cL = sm[L::OFF_C + kl], cR = sm[L::OFF_C + kr];
            const double delu = uR - uL;
            const double hmin = fmin(hL, hR), hmax = fmax(hL, hR);
            const double dh = hmax - hmin;
            if (delu + 2.0 * (fmin(cL, cR) - fmax(cL, cR)) > 0.0) cls = 1;
            else if (delu <= 0.0 && delu * delu * (hmin * hmax) >= dh * dh * (0.5 * g) * (hmin + hmax)) cls = 0;
            else cls = 2;
        }
        fcls[f] = (unsigned char)cls;
        atomicAdd(&C(ts / w.rb, 0, cls, 0), 1);
    }
    for (int f = threadIdx.x; f < w.nsl * w.fb; f += NT) {
        const int ts = f / w.fb, n = w.nb_lo + f % w.fb;
        const int t = w.ts_lo + ts;
        const int nw = wet[cidx(n - 1, t)] + wet[cidx(n, t)];
        atomicAdd(&C(ts / w.rb, 1, nw == 0 ? 4 : nw == 1 ? 3 : 0, 0), 1);
    }
    __syncthreads();
    for (int e = threadIdx.x; e < L::NBAND * 2; e += NT) {
        const int band = e >> 1, list = e & 1;
        int acc = 0;
        for (int cls = 0; cls < NC; ++cls) {
            C(band, list, cls, 1) = acc;
            acc += C(band, list, cls, 0);
        }
    }
    __syncthreads();
    for (int f = threadIdx.x; f < w.nsl * w.fa; f += NT) {
        const int band = (f / w.fa) / w.rb;
        const int pos = atomicAdd(&C(band, 0, fcls[f], 1), 1);
        la[band * w.rb * w.fa + pos] = (uint16_t)(f - band * w.rb * w.fa);
    }
    for (int f = threadIdx.x; f < w.nsl * w.fb; f += NT) {
        const int ts = f / w.fb, n = w.nb_lo + f % w.fb;
        const int t = w.ts_lo + ts;
        const int nw = wet[cidx(n - 1, t)] + wet[cidx(n, t)];
        const int band = ts / w.rb;
        const int pos = atomicAdd(&C(band, 1, nw == 0 ? 4 : nw == 1 ? 3 : 0, 1), 1);
        lb[band * w.rb * w.fb + pos] = (uint16_t)(f - band * w.rb * w.fb);
    }
    __syncthreads();
}

/* Fluctuations and limited second-order term of one face in the contracted
 * build, from its record wc and its neighbours' wl, wr along the sweep (the
 * middle f-wave is (0, beta2, 0) in local order). Only the upwind neighbour's
 * projection is formed; the middle wave's ratio of projection and norm is
 * the quotient of the two beta2. */
__device__ __forceinline__ void face_terms_fast(const double* wc, const double* wl, const double* wr, const gf_phys& P,
                                                double dtdn, double amdq[3], double apdq[3], double cq[3])
{
    constexpr bool F = true;
    const double s0 = wc[0], s1 = wc[1], s2 = wc[2];
    const double f0[3] = {wc[3], wc[4], wc[5]}, f1 = wc[6], f2[3] = {wc[7], wc[8], wc[9]};
    if (d_ltz<F>(s0) && d_gtz<F>(s2)) { /* one outer wave each way: no sums */
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            amdq[c] = f0[c];
            apdq[c] = f2[c];
        }
    } else {
        const double w0m = d_ltz<F>(s0) ? 1.0 : d_gtz<F>(s0) ? 0.0 : 0.5;
        const double w2m = d_ltz<F>(s2) ? 1.0 : d_gtz<F>(s2) ? 0.0 : 0.5;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            amdq[c] = fma(w0m, f0[c], gf_mul(w2m, f2[c]));
            apdq[c] = fma(1.0 - w0m, f0[c], gf_mul(1.0 - w2m, f2[c]));
        }
    }
    if (d_eqz<F>(s1)) {
        amdq[1] = fma(0.5, f1, amdq[1]);
        apdq[1] = fma(0.5, f1, apdq[1]);
    } else {
        const bool l = d_ltz<F>(s1);
        const double v = gf_add(l ? amdq[1] : apdq[1], f1);
        amdq[1] = l ? v : amdq[1];
        apdq[1] = l ? apdq[1] : v;
    }
    cq[0] = cq[1] = cq[2] = 0.0;
    if (P.order == 1) return;
    auto outer = [&](double s, const double* fa, int at, int meth) -> double { /* waves 0 and 2 */
        double lim = 1.0;
        if (meth != 0) {
            const double* pw = (d_gtz<F>(s) ? wl : wr) + at;
            const double wnorm2 = fma(fa[2], fa[2], fma(fa[1], fa[1], gf_mul(fa[0], fa[0])));
            if (gf_pos_normal(wnorm2))
                lim = gf_philim<F>(wnorm2, fma(pw[2], fa[2], fma(pw[1], fa[1], gf_mul(pw[0], fa[0]))), meth);
        }
        return gf_mul(with_sign_of(fma(-fabs(s), dtdn, 1.0), s), lim);
    };
    {
        const double fl = outer(s0, f0, 3, P.mthlim[0]);
        cq[0] = gf_mul(fl, f0[0]); cq[1] = gf_mul(fl, f0[1]); cq[2] = gf_mul(fl, f0[2]);
    }
    {
        double lim = 1.0;
        if (P.mthlim[1] != 0 && gf_pos_normal(fabs(f1))) {
            const double up = (d_gtz<F>(s1) ? wl : wr)[6];
            /* MC: opposite signs, or no upwind wave, give zero without the quotient */
            lim = P.mthlim[1] == 4 && (d_eqz<F>(up) || opposite_signs(up, f1))
                      ? 0.0
                      : gf_philim_r<F>(d_div<F>(up, f1), P.mthlim[1]);
        }
        cq[1] = fma(gf_mul(with_sign_of(fma(-fabs(s1), dtdn, 1.0), s1), lim), f1, cq[1]);
    }
    {
        const double fl = outer(s2, f2, 7, P.mthlim[2]);
        cq[0] = fma(fl, f2[0], cq[0]); cq[1] = fma(fl, f2[1], cq[1]); cq[2] = fma(fl, f2[2], cq[2]);
    }
}

/* Per cell of a slice in the contracted build, from the terms of its left and
 * right face (ol, or): the flux difference N = faddm(right) - faddp(left) =
 * P + Q/2 with P = amdq(right) + apdq(left), Q = cq(right) - cq(left), and the
 * transverse split of the fluctuations that enter the cell. rpt2 is linear in
 * its input and the cell alone decides its branches, so the splits of
 * amdq(right) and apdq(left) (with the second-order terms for transverse = 2)
 * are one split of their sum P + Q (P for transverse = 1): bm is the down-going
 * part, bp the up-going part, equal to the sum of the reference's two splits up
 * to rounding. Local component order. */
__device__ __forceinline__ void cell_terms(const double* ol, const double* orr, const gf_cell& cc, double b_lo,
                                           double b_hi, int transverse, double N[3], double bm[3], double bp[3])
{
    double Pv[3], Qv[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        Pv[q] = gf_add(orr[q], ol[3 + q]);
        Qv[q] = gf_sub(orr[6 + q], ol[6 + q]);
        N[q] = fma(0.5, Qv[q], Pv[q]);
        bm[q] = bp[q] = 0.0;
    }
    if (transverse != 0 && cc.wet) {
        double x[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) x[q] = transverse == 2 ? gf_add(Pv[q], Qv[q]) : Pv[q];
        gf_rpt2_fast(cc, b_lo, b_hi, x, bm, bp);
    }
}

/* One sweep direction over all slices, banded. Accumulates into the flux
 * accumulators (contracted build: the x sweep starts them); returns this
 * thread's max |s| over normal faces. side: further work of 32 items a chunk
 * that its phases take along (contracted build; the face lists still to be
 * made). */
template <int M, int NT, int RB, int DIR, bool EXACT, class Side>
__device__ __forceinline__ double sweep(double* sm, const unsigned char* wet, const SweepLists& ls, const gf_phys& P,
                                        const Side& side)
{
    using G = Geo<M>;
    using L = Smem<M, RB, EXACT>;
    constexpr int N = G::N;
    constexpr bool FAST = !EXACT;
    double* W = sm + L::OFF_W;
    double* O = sm + L::OFF_O;
    const double g = P.grav, drytol = P.dry_tolerance;
    const double* sc = sm + L::OFF_SC;
    const double dtdn = sc[DIR == 0 ? SC_DTDX : SC_DTDY], c16g = sc[SC_C16G], rsg = sc[SC_RSG];
    const double crit = sc[SC_CRIT], crit2 = sc[SC_CRIT2];
    const double half_dtdn = 0.5 * dtdn;
    int* cnt = ls.cnt;
    uint16_t *la = ls.la, *lb = ls.lb;
    const uint16_t* lm = ls.lm; /* contracted build */
    /* local component l -> global component (h, hu, hv) */
    constexpr int G1 = (DIR == 0) ? 1 : 2; /* normal momentum     */
    constexpr int G2 = (DIR == 0) ? 2 : 1; /* transverse momentum */
    constexpr int MM = L::PLANE; /* component stride of the accumulators */
    double smax = 0.0;

    auto cidx = [](int n, int t) -> int {
        return DIR == 0 ? (t + 1) * N + (n + 1) : (n + 1) * N + (t + 1);
    };
    auto aidx = [](int n, int t) -> int {
        return DIR == 0 ? (n - 1) + L::MS * (t - 1) : (t - 1) + L::MS * (n - 1);
    };
    auto C = [&](int band, int list, int cls) -> int {
        return cnt[((band * 2 + list) * L::NCLS + cls) * 2 + 0];
    };

    constexpr SweepWin<M, RB> win{};
    constexpr int fa = win.fa, fb = win.fb;
    if constexpr (EXACT) build_lists_exact<M, NT, RB, DIR>(sm, wet, cnt, la, lb, g);
    /* record of limited face `face` (nb_lo..) of band slice ts */
    auto orec = [&](int ts, int face) -> const double* {
        return O + (ts * fb + (face - win.nb_lo)) * L::O_STRIDE;
    };
    /* per-cell record of cell `cell` of band slice ts (contracted build) */
    double* C2 = sm + L::OFF_C2;
    auto crec = [&](int ts, int cell) -> double* {
        return C2 + (ts * fb + (cell - win.nb_lo)) * L::C_STRIDE;
    };

    /* Contracted build: DX, DY. Exact build: fm(i+1,j), fp(i,j), gm(i,j+1),
     * gp(i,j) of the reference, in sweep coordinates N_M, N_P (normal) and
     * T_M, T_P (transverse), each summed in the reference's order (slices in
     * increasing order, x sweeps before y sweeps). */
    double* ACCN = sm + L::OFF_ACC + (DIR == 0 ? 0 : 3 * MM);
    double* ACCT = sm + L::OFF_ACC + (DIR == 0 ? 3 * MM : 0);
    double* NM = sm + L::OFF_ACC + (DIR == 0 ? 0 : 6 * MM);
    double* NP = NM + 3 * MM;
    double* TM = sm + L::OFF_ACC + (DIR == 0 ? 6 * MM : 0);
    double* TP = TM + 3 * MM;

    /* cells [e0, e0 + step, ..) of those the slices t0..t1 feed: n in [1, M],
     * t in [t0-1, t1+1] (interior) */
    auto gather_cells = [&](int t0, int t1) -> int {
        return (min(M, t1 + 1) - max(1, t0 - 1) + 1) * M;
    };
    auto gather = [&](int t0, int t1, int e0, int e1, int step) {
        const int ta = max(1, t0 - 1);
        constexpr int nn = M;
        for (int e = e0; e < e1; e += step) {
            const int ts = e / nn;
            const int t = ta + ts;
            const int n = 1 + (e - ts * nn);
            const int a = aidx(n, t);
            if (EXACT) {
                if (t - 1 >= t0 && t - 1 <= t1) { /* slice below: up-going parts */
                    const double* fr = orec(t - 1 - t0, n + 1);
                    const double* fl = orec(t - 1 - t0, n);
#pragma unroll
                    for (int c = 0; c < 3; ++c) TP[a + c * MM] += (0.0 - fr[9 + c]) - fl[15 + c];
                }
                if (t >= t0 && t <= t1) {
                    const double* fr = orec(t - t0, n + 1);
                    const double* fl = orec(t - t0, n);
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        NM[a + c * MM] += fr[c];
                        NP[a + c * MM] += fl[3 + c];
                        TM[a + c * MM] += (0.0 - fr[9 + c]) - fl[15 + c];
                        TP[a + c * MM] += (0.0 - fr[6 + c]) - fl[12 + c];
                    }
                }
                if (t + 1 >= t0 && t + 1 <= t1) { /* slice above: down-going parts */
                    const double* fr = orec(t + 1 - t0, n + 1);
                    const double* fl = orec(t + 1 - t0, n);
#pragma unroll
                    for (int c = 0; c < 3; ++c) TM[a + c * MM] += (0.0 - fr[6 + c]) - fl[12 + c];
                }
            } else {
                /* each slice's part enters the accumulators on its own, slices in
                 * increasing order, so the sums do not depend on where the band
                 * boundaries fall: every tile shape gives the same bits. A
                 * slice's per-cell record holds its flux difference N and the
                 * up-going (U) and down-going (Dn) transverse parts. The slice
                 * below comes first: in the x sweep it starts the sums. */
                double T[3];
                if (t - 1 >= t0 && t - 1 <= t1) { /* slice below: up-going parts */
                    const double* r = crec(t - 1 - t0, n);
#pragma unroll
                    for (int c = 0; c < 3; ++c)
                        T[c] = DIR == 0 ? gf_mul(half_dtdn, r[3 + c]) : fma(half_dtdn, r[3 + c], ACCT[a + c * MM]);
                } else {
#pragma unroll
                    for (int c = 0; c < 3; ++c) T[c] = ACCT[a + c * MM];
                }
                if (t >= t0 && t <= t1) {
                    const double* r = crec(t - t0, n);
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        ACCN[a + c * MM] = DIR == 0 ? r[c] : gf_add(ACCN[a + c * MM], r[c]);
                        T[c] = fma(half_dtdn, gf_sub(r[6 + c], r[3 + c]), T[c]);
                    }
                }
                if (t + 1 >= t0 && t + 1 <= t1) { /* slice above: down-going parts */
                    const double* r = crec(t + 1 - t0, n);
#pragma unroll
                    for (int c = 0; c < 3; ++c) T[c] = fma(-half_dtdn, r[6 + c], T[c]);
                }
#pragma unroll
                for (int c = 0; c < 3; ++c) ACCT[a + c * MM] = T[c];
            }
        }
    };

    /* exact build: a2 / b2 both cells wet, a1 / b1 one wet, a0 / b0 both dry */
    auto counts_a = [&](int band, int& a2, int& a1, int& a0) {
        a2 = C(band, 0, 0) + C(band, 0, 1) + C(band, 0, 2);
        a1 = C(band, 0, 3);
        a0 = C(band, 0, 4);
    };
    auto counts_b = [&](int band, int& b2, int& b1, int& b0) {
        b2 = C(band, 1, 0);
        b1 = C(band, 1, 3);
        b0 = C(band, 1, 4);
    };

    /* ---- stage A: normal Riemann solves, faces 0..M+2, by class ---- */
    auto stage_a_exact = [&](int t0, int band) {
        const uint16_t* lA = la + band * win.rb * fa;
        int a2, a1, a0;
        counts_a(band, a2, a1, a0);
        for (int idx = threadIdx.x; idx < a2 + a1 + a0; idx += NT) {
            const int f = lA[idx];
            double* w = W + f * L::W_STRIDE;
            if (idx >= a2 + a1) { /* both cells dry: no waves */
#pragma unroll
                for (int q = 0; q < L::W_STRIDE; ++q) w[q] = 0.0;
                continue;
            }
            const int t = t0 + f / fa;
            const int n = win.na_lo + f % fa;
            const gf_cell cl = load_cell<DIR, EXACT, L>(sm, wet, cidx(n - 1, t));
            const gf_cell cr = load_cell<DIR, EXACT, L>(sm, wet, cidx(n, t));
            double s[3], fw[3][3];
            gf_rpn2_face<false>(cl, cr, g, drytol, c16g, rsg, crit, crit2, s, fw);
#pragma unroll
            for (int mw = 0; mw < 3; ++mw) {
                w[mw] = s[mw];
                w[3 + 3 * mw + 0] = fw[mw][0];
                w[3 + 3 * mw + 1] = fw[mw][1];
                w[3 + 3 * mw + 2] = fw[mw][2];
                smax = d_max_abs<FAST>(smax, s[mw]);
            }
        }
    };
    /* contracted build: faces 32 c .. 32 c + 31 of the band's list, in the
     * order full solve, edge, smooth, dry: the longest first. A chunk with an
     * edge face solves its smooth faces as edge faces too, not both ways. */
    auto chunk_a = [&](int t0, int band, int c) {
        const int ns = cnt[band * 6], ne = cnt[band * 6 + 1], nh = cnt[band * 6 + 2], nd = cnt[band * 6 + 3];
        const int nA = ns + ne + nh + nd, idx = 32 * c + (int)(threadIdx.x & 31);
        if (idx >= nA) return;
        const uint16_t* lA = la + band * win.rb * fa;
        const uint16_t* lM = lm + band * win.rb * fa;
        const int v = idx < nh ? lM[nA - 1 - idx] : idx < nh + ne ? lM[idx - nh] : idx < nA - nd ? lA[idx - nh - ne] : lA[idx];
        const int f = v & 0x7fff;
        double* w = W + f * L::W_STRIDE;
        if (idx >= nA - nd) { /* both cells dry: no waves */
#pragma unroll
            for (int q = 0; q < L::W_STRIDE; ++q) w[q] = 0.0;
            return;
        }
        const int ts = f / fa;
        const int t = t0 + ts;
        const int n = win.na_lo + (f - ts * fa);
        const gf_cell cl = load_cell<DIR, EXACT, L>(sm, wet, cidx(n - 1, t));
        const gf_cell cr = load_cell<DIR, EXACT, L>(sm, wet, cidx(n, t));
        if (idx < nh) {
            full_solve(cl, cr, g, drytol, sc, w);
#pragma unroll
            for (int mw = 0; mw < 3; ++mw) smax = d_max_abs<FAST>(smax, w[mw]);
            return;
        }
        double s[3], fw[3][3];
        if (32 * c < nh + ne) gf_rpn2_edge(cl, cr, (v & 0x8000) != 0, g, crit, crit2, s, fw);
        else gf_rpn2_smooth(cl, cr, g, s, fw);
#pragma unroll
        for (int mw = 0; mw < 3; ++mw) {
            w[mw] = s[mw];
            smax = d_max_abs<FAST>(smax, s[mw]);
        }
        w[3] = fw[0][0]; w[4] = fw[0][1]; w[5] = fw[0][2];
        w[6] = fw[1][1];
        w[7] = fw[2][0]; w[8] = fw[2][1]; w[9] = fw[2][2];
    };

    /* Fluctuations from the unlimited f-waves (rpn2_geoclaw.f:359-376) and
     * the limited second-order term cqxx of one face (flux2: limiter.f /
     * philim.f and the correction loop), exact build. */
    auto face_terms_exact = [&](const double* wc, double amdq[3], double apdq[3], double cq[3]) {
        double s[3], fw[3][3];
#pragma unroll
        for (int mw = 0; mw < 3; ++mw) {
            s[mw] = wc[mw];
            fw[mw][0] = wc[3 + 3 * mw]; fw[mw][1] = wc[4 + 3 * mw]; fw[mw][2] = wc[5 + 3 * mw];
        }
        amdq[0] = amdq[1] = amdq[2] = 0.0;
        apdq[0] = apdq[1] = apdq[2] = 0.0;
        cq[0] = cq[1] = cq[2] = 0.0;
#pragma unroll
        for (int mw = 0; mw < 3; ++mw) {
            if (s[mw] < 0.0) {
                amdq[0] += fw[mw][0]; amdq[1] += fw[mw][1]; amdq[2] += fw[mw][2];
            } else if (s[mw] > 0.0) {
                apdq[0] += fw[mw][0]; apdq[1] += fw[mw][1]; apdq[2] += fw[mw][2];
            } else {
                amdq[0] += 0.5 * fw[mw][0]; amdq[1] += 0.5 * fw[mw][1]; amdq[2] += 0.5 * fw[mw][2];
                apdq[0] += 0.5 * fw[mw][0]; apdq[1] += 0.5 * fw[mw][1]; apdq[2] += 0.5 * fw[mw][2];
            }
        }
        if (P.order == 1) return;
        const double* wl = wc - L::W_STRIDE; /* face n-1 */
        const double* wr = wc + L::W_STRIDE; /* face n+1 */
#pragma unroll
        for (int mw = 0; mw < 3; ++mw) {
            const double* fa = fw[mw];
            double lim = 1.0;
            if (P.mthlim[mw] != 0) {
                /* dot products in the global (h, hu, hv) order */
                const double a0 = fa[0], a1 = (DIR == 0) ? fa[1] : fa[2], a2 = (DIR == 0) ? fa[2] : fa[1];
                const double* ql = wl + 3 + 3 * mw;
                const double* qr = wr + 3 + 3 * mw;
                const double l0 = ql[0], l1 = (DIR == 0) ? ql[1] : ql[2], l2 = (DIR == 0) ? ql[2] : ql[1];
                const double r0 = qr[0], r1 = (DIR == 0) ? qr[1] : qr[2], r2 = (DIR == 0) ? qr[2] : qr[1];
                const double wnorm2 = a0 * a0 + a1 * a1 + a2 * a2;
                if (wnorm2 != 0.0) {
                    /* the upwind neighbour's projection only (the same
                     * products in the same order) */
                    const bool up = s[mw] > 0.0;
                    const double p0 = up ? l0 : r0, p1 = up ? l1 : r1, p2 = up ? l2 : r2;
                    const double dot = p0 * a0 + p1 * a1 + p2 * a2;
                    lim = gf_philim<false>(wnorm2, dot, P.mthlim[mw]);
                }
            }
            const double fac = copysign(1.0, s[mw]) * (1.0 - fabs(s[mw]) * dtdn);
            cq[0] += fac * (lim * fa[0]);
            cq[1] += fac * (lim * fa[1]);
            cq[2] += fac * (lim * fa[2]);
        }
    };

    /* ---- exact build, stage B: limiter, 2nd-order terms, both transverse
     * splits of every face (flux2's per-face order) ---- */
    auto stage_b_exact = [&](int t0, int band) {
        const uint16_t* lB = lb + band * win.rb * fb;
        int b2, b1, b0;
        counts_b(band, b2, b1, b0);
        for (int idx = threadIdx.x; idx < b2 + b1 + b0; idx += NT) {
            const int f = lB[idx];
            double* o = O + f * L::O_STRIDE;
            if (idx >= b2 + b1) {
#pragma unroll
                for (int q = 0; q < L::O_STRIDE; ++q) o[q] = 0.0;
                continue;
            }
            const int t = t0 + f / fb;
            const int n = win.nb_lo + f % fb;
            const int kl = cidx(n - 1, t), kr = cidx(n, t);
            const double* wc = W + ((t - t0) * fa + (n - win.na_lo)) * L::W_STRIDE;
            double amdq[3], apdq[3], cq[3];
            face_terms_exact(wc, amdq, apdq, cq);
            double faddm[3] = {amdq[0], amdq[1], amdq[2]};
            double faddp[3] = {-apdq[0], -apdq[1], -apdq[2]};
            if (P.order != 1) {
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    faddm[c] += 0.5 * cq[c];
                    faddp[c] += 0.5 * cq[c];
                }
                if (P.transverse == 2) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        amdq[c] += cq[c];
                        apdq[c] -= cq[c];
                    }
                }
            }
            double A[3] = {0, 0, 0}, B[3] = {0, 0, 0}, Cc[3] = {0, 0, 0}, D[3] = {0, 0, 0};
            if (P.transverse != 0) {
                double bm[3], bp[3];
                if (wet[kl]) { /* rpt2 imp=1: left-going part into cell n-1 */
                    const gf_cell cl = load_cell<DIR, EXACT, L>(sm, wet, kl);
                    gf_rpt2_face(cl, sm[L::OFF_B + cidx(n - 1, t - 1)],
                                       sm[L::OFF_B + cidx(n - 1, t + 1)], drytol, amdq, bm, bp);
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        A[c] = half_dtdn * bm[c];
                        B[c] = half_dtdn * bp[c];
                    }
                }
                if (wet[kr]) { /* rpt2 imp=2: right-going part into cell n */
                    const gf_cell cr = load_cell<DIR, EXACT, L>(sm, wet, kr);
                    gf_rpt2_face(cr, sm[L::OFF_B + cidx(n, t - 1)],
                                       sm[L::OFF_B + cidx(n, t + 1)], drytol, apdq, bm, bp);
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        Cc[c] = half_dtdn * bm[c];
                        D[c] = half_dtdn * bp[c];
                    }
                }
            }
            /* write in global component order (h, hu, hv) */
            o[0] = faddm[0]; o[G1] = faddm[1]; o[G2] = faddm[2];
            o[3] = faddp[0]; o[3 + G1] = faddp[1]; o[3 + G2] = faddp[2];
            o[6] = A[0]; o[6 + G1] = A[1]; o[6 + G2] = A[2];
            o[9] = B[0]; o[9 + G1] = B[1]; o[9 + G2] = B[2];
            o[12] = Cc[0]; o[12 + G1] = Cc[1]; o[12 + G2] = Cc[2];
            o[15] = D[0]; o[15 + G1] = D[1]; o[15 + G2] = D[2];
        }
    };

    /* ---- contracted build, stage B1: per limited face, the fluctuations
     * amdq, apdq and the limited second-order term cq (local order) ---- */
    auto chunk_b1 = [&](int band, int c) {
        const uint16_t* lB = lb + band * win.rb * fb;
        const int nw = cnt[band * 6 + 4], nB = nw + cnt[band * 6 + 5];
        const int idx = 32 * c + (int)(threadIdx.x & 31);
        if (idx >= nB) return;
        const int f = lB[idx];
        double* o = O + f * L::O_STRIDE;
        if (idx >= nw) {
#pragma unroll
            for (int q = 0; q < L::O_STRIDE; ++q) o[q] = 0.0;
            return;
        }
        const int ts = f / fb;
        const int n = win.nb_lo + (f - ts * fb);
        const double* wc = W + (ts * fa + (n - win.na_lo)) * L::W_STRIDE;
        double amdq[3], apdq[3], cq[3];
        face_terms_fast(wc, wc - L::W_STRIDE, wc + L::W_STRIDE, P, dtdn, amdq, apdq, cq);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            o[k] = amdq[k];
            o[3 + k] = apdq[k];
            o[6 + k] = cq[k];
        }
    };

    /* ---- contracted build, stage B2: per cell n of each band slice, its
     * record from its faces n and n+1 (cell_terms) ---- */
    auto chunk_b2 = [&](int t0, int t1, int c) {
        const int ncell = fb - 1;
        const int e = 32 * c + (int)(threadIdx.x & 31);
        if (e < (t1 - t0 + 1) * ncell) {
            const int ts = e / ncell;
            const int n = win.nb_lo + (e - ts * ncell);
            const int t = t0 + ts;
            const int k = cidx(n, t);
            double* r = crec(ts, n);
            if (!(wet[cidx(n - 1, t)] | wet[k] | wet[cidx(n + 1, t)])) {
                /* faces n and n+1 both between dry cells: no waves */
#pragma unroll
                for (int q = 0; q < L::C_STRIDE; ++q) r[q] = 0.0;
                return;
            }
            const double* orr = O + (ts * fb + (n + 1 - win.nb_lo)) * L::O_STRIDE; /* face n+1 */
            const double* orl = O + (ts * fb + (n - win.nb_lo)) * L::O_STRIDE;     /* face n   */
            double Nv[3], bm[3], bp[3];
            cell_terms(orl, orr, load_cell<DIR, EXACT, L>(sm, wet, k), sm[L::OFF_B + cidx(n, t - 1)],
                       sm[L::OFF_B + cidx(n, t + 1)], P.transverse, Nv, bm, bp);
            /* global component order (h, hu, hv) */
            r[0] = Nv[0]; r[G1] = Nv[1]; r[G2] = Nv[2];
            r[3] = bp[0]; r[3 + G1] = bp[1]; r[3 + G2] = bp[2];
            r[6] = bm[0]; r[6 + G1] = bm[1]; r[6 + G2] = bm[2];
        }
    };

    const int ts_end = win.ts_lo + win.nsl;
    int prev_t0 = -1, prev_t1 = -1;
    if constexpr (EXACT) {
        auto gather_all = [&](int ta, int tb) { gather(ta, tb, threadIdx.x, gather_cells(ta, tb), NT); };
        for (int t0 = win.ts_lo, band = 0; t0 < ts_end; t0 += win.rb, ++band) {
            const int t1 = min(t0 + win.rb, ts_end) - 1; /* last slice of band */
            stage_a_exact(t0, band);
            if (prev_t0 >= 0) gather_all(prev_t0, prev_t1);
            __syncthreads();
            stage_b_exact(t0, band);
            __syncthreads();
            prev_t0 = t0;
            prev_t1 = t1;
        }
        gather_all(prev_t0, prev_t1);
        __syncthreads();
    } else {
        /* Contracted build, pipelined over bands with two barriers per band:
         * [stage A of band b | B2 of band b-1], [B1 of band b | gather of band
         * b-1]. Each stage reads what the phase before the last barrier wrote.
         * A warp takes the next 32 items of a phase from its cursor, the
         * costly stage first: warps (and the four schedulers, each with an
         * FP64 pipe of its own) that got short items take more of them. The
         * lists' chunks run beside the solves, off the FP64 pipe. */
        int* cur = ls.cur;
        auto next = [&](int phase) -> int {
            int c = 0;
            if ((threadIdx.x & 31) == 0) c = atomicAdd(&cur[phase], 1);
            return __shfl_sync(0xffffffffu, c, 0);
        };
        for (int t0 = win.ts_lo, band = 0;; t0 += win.rb, ++band) {
            const bool have = t0 < ts_end;
            const int t1 = have ? min(t0 + win.rb, ts_end) - 1 : -1;
            const int nsl = t1 - t0 + 1, psl = prev_t0 >= 0 ? prev_t1 - prev_t0 + 1 : 0;
            const int ca = have ? (nsl * fa + 31) / 32 : 0, c2 = (psl * (fb - 1) + 31) / 32;
            const int sa = side.count(2 * band);
            for (int c; (c = next(2 * band)) < ca + sa + c2;) {
                if (c < ca) chunk_a(t0, band, c);
                else if (c < ca + sa) side.run(2 * band, c - ca);
                else chunk_b2(prev_t0, prev_t1, c - ca - sa);
            }
            __syncthreads();
            const int c1 = have ? (nsl * fb + 31) / 32 : 0;
            const int ng = psl ? gather_cells(prev_t0, prev_t1) : 0, cg = (ng + 31) / 32;
            const int sb = side.count(2 * band + 1);
            for (int c; (c = next(2 * band + 1)) < c1 + sb + cg;) {
                if (c < c1) {
                    chunk_b1(band, c);
                } else if (c < c1 + sb) {
                    side.run(2 * band + 1, c - c1);
                } else {
                    const int e0 = 32 * (c - c1 - sb);
                    gather(prev_t0, prev_t1, e0 + (int)(threadIdx.x & 31), min(ng, e0 + 32), 32);
                }
            }
            __syncthreads();
            if (!have) break;
            prev_t0 = t0;
            prev_t1 = t1;
        }
    }
    return smax;
}

/* Manning friction source term on one interior cell (geoclaw_src2_fort.f90:41-71).
 * The contracted build forms h^(-7/3) and one reciprocal of 1 + dt gamma
 * instead of pow and three divisions: from the single-precision y0 of
 * h^(-1/3), one third-order step of the binomial series,
 * y0^7 (1 - e)^(-7/3) = y0^7 (1 + 7 e/3 + 35 e^2/9 + ...), e = 1 - h y0^3
 * (23 bits -> past the FP64 rounding): no FP64 division, cube root or
 * conversion is taken. */
template <bool FAST>
__device__ __forceinline__ void src2_cell(const gf_phys& P, double dt, const double* kf, double bathy, double nvar,
                                          double& h, double& hu, double& hv)
{
    if (!P.friction_forcing) return;
    if (h < 1.0e-30) {
        hu = 0.0;
        hv = 0.0;
    } else if (h <= P.friction_depth) {
        /* coefficient, or in the contracted build dt g coefficient^2 (kf: of
         * the Manning table) */
        double coeff = 0.0;
        if (!P.variable_friction) {
            for (int nman = P.num_manning; nman >= 1; --nman)
                if (bathy < P.manning_break[nman - 1]) coeff = FAST ? kf[nman - 1] : P.manning_coefficient[nman - 1];
        } else {
            coeff = FAST ? gf_mul(gf_mul(dt, P.grav), gf_mul(nvar, nvar)) : nvar;
        }
        if (FAST) {
            /* 1e-30 <= h here: a normal single-precision number */
            const double y0 = gf_f64_pos(rcbrtf(gf_f32(h)));
            const double y3 = gf_mul(gf_mul(y0, y0), y0);
            const double e = fma(-h, y3, 1.0);
            const double y7 = gf_mul(gf_mul(y3, y3), y0);
            const double hm73 = fma(gf_mul(y7, e), fma(35.0 / 9.0, e, 7.0 / 3.0), y7); /* h^(-7/3) */
            const double mom = d_sqrt<FAST>(fma(hu, hu, gf_mul(hv, hv)));
            const double rdg = gf_rcp(fma(gf_mul(mom, coeff), hm73, 1.0));
            hu = gf_mul(hu, rdg);
            hv = gf_mul(hv, rdg);
        } else {
            const double gamma =
                sqrt(hu * hu + hv * hv) * P.grav * (coeff * coeff) / pow(h, 7.0 / 3.0);
            const double dgamma = 1.0 + dt * gamma;
            hu = hu / dgamma;
            hv = hv / dgamma;
        }
    }
}

/* One work item of the fused update: stage the patch, b4step2, both face
 * sweeps, flux differencing + src2, CFL. All threads of the CTA take part;
 * returns false (on every thread) when the staging copy's wait timed out,
 * after the error flag is set and the copy has landed or been waited for. */
template <int M, int NT, int RB, bool EXACT>
__device__ __forceinline__ bool patch_item(double* sm, uint64_t* bar, uint32_t& phase, gf_patch_work wk,
                                           int wi, const gf_phys* __restrict__ phys_table,
                                           double dt_uniform, const double* __restrict__ group_dt,
                                           const int* __restrict__ group_par, int maux,
                                           double* __restrict__ cfl_out,
                                           unsigned long long* __restrict__ group_max, int* __restrict__ err)
{
    using G = Geo<M>;
    using L = Smem<M, RB, EXACT>;
    constexpr int N = G::N;
    constexpr int S = G::S;
    constexpr bool FAST = !EXACT;
    int* cnt = reinterpret_cast<int*>(sm + L::OFF_INT);
    uint16_t* lists = reinterpret_cast<uint16_t*>(cnt + L::CNT_INTS);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned char* wet = reinterpret_cast<unsigned char*>(sm) + L::OFF_WET_BYTES;
    double* sc = sm + L::OFF_SC;

    const double dt = group_dt ? group_dt[wk.group] : dt_uniform;
    /* a group with no step this round (dt <= 0) is skipped as a whole */
    if (group_dt && !(dt > 0.0)) return true;
    if (group_par && group_par[wk.group]) {
        /* the group's state lives in the second buffer: read there, write back */
        double* t = wk.q;
        wk.q = wk.qout;
        wk.qout = t;
    }
    /* culled: this update would be an exact identity (the ghost fill decided) */
    if (wk.fl && wk.fl->skip) return true;
    const gf_phys P = phys_table[wk.phys];
    const double g = P.grav, drytol = P.dry_tolerance;

    /* after a wait of this launch (or an earlier one of the same step) gave
     * up, the step has failed: later items leave at once */
    const bool failed = __syncthreads_or(threadIdx.x == 0 && err && *reinterpret_cast<volatile int*>(err) != 0);
    if (failed) return false;

    /* ---- stage the patch (h, hu, hv planes and b) with bulk copies ---- */
    if (threadIdx.x == 0) {
        mbar_expect_tx(bar, (uint32_t)(4 * S * sizeof(double)));
        bulk_g2s(sm + L::OFF_H, wk.q, (uint32_t)(3 * S * sizeof(double)), bar);
        bulk_g2s(sm + L::OFF_B, wk.aux, (uint32_t)(S * sizeof(double)), bar);
    }
    const uint32_t ph = phase;
    phase ^= 1u;
    const bool staged = __syncthreads_and(mbar_wait(bar, ph, kWaitPolls));
    if (!staged) {
        if (threadIdx.x == 0) atomicExch(err, 1);
        mbar_wait(bar, ph, kWaitPolls); /* let any copy in flight land */
        return false;
    }

    /* ---- b4step2 on all cells + per-cell quotients ---- */
    int any_wet = 0, changed = 0;
    if (warp == NT / 32 - 1) {
        /* the item's constants, one lane each: formed by every thread they
         * would cost as much FP64 time as a band's limiter */
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
            sc[SC_KF + lane - 8] = (dt * g) * (n * n);
        }
        if (lane == 16) sc[SC_CFL] = 0.0;
    }
    for (int k = threadIdx.x; k < S; k += NT) {
        double h = sm[L::OFF_H + k];
        if (d_lt<FAST>(h, drytol)) {
            /* b4step2 changes this cell's bits unless h >= 0 and both momenta are +0 */
            changed |= (__double_as_longlong(h) < 0) | (__double_as_longlong(sm[L::OFF_HU + k]) != 0) |
                       (__double_as_longlong(sm[L::OFF_HV + k]) != 0);
            h = d_max<FAST>(h, 0.0);
            sm[L::OFF_H + k] = h;
            sm[L::OFF_HU + k] = 0.0;
            sm[L::OFF_HV + k] = 0.0;
        }
        const bool w = d_gt<FAST>(h, drytol);
        wet[k] = w ? 1 : 0;
        any_wet |= w;
        double u = 0.0, v = 0.0, c = 0.0, rc = 0.0;
        if (w) {
            if (FAST) {
                /* rc^2 = 1 / (g h), so 1 / h = g rc^2 within a few ulps:
                 * two products instead of a reciprocal */
                const double gh = g * h;
                rc = gf_pos_normal(gh) ? gf_rsqrt_n(gh) : rsqrt(gh);
                c = gh * rc;
                const double rh = g * (rc * rc);
                u = sm[L::OFF_HU + k] * rh;
                v = sm[L::OFF_HV + k] * rh;
            } else {
                u = sm[L::OFF_HU + k] / h;
                v = sm[L::OFF_HV + k] / h;
                c = sqrt(g * h);
            }
        }
        sm[L::OFF_U + k] = u;
        sm[L::OFF_V + k] = v;
        sm[L::OFF_C + k] = c;
        if (FAST) sm[L::OFF_RC + k] = rc;
    }
    if (EXACT)
        for (int k = threadIdx.x; k < L::NACC * 3 * L::PLANE; k += NT) sm[L::OFF_ACC + k] = 0.0;
    else
        for (int k = threadIdx.x; k < L::CNT_INTS; k += NT) cnt[k] = 0;
    any_wet = __syncthreads_or(any_wet);
    if (wk.fl) changed = __syncthreads_or(changed);

    const double dtdx = sc[SC_DTDX], dtdy = sc[SC_DTDY];
    double smax_x = 0.0, smax_y = 0.0;
    if (any_wet) {
        if constexpr (EXACT) {
            struct {
                __device__ int count(int) const { return 0; }
                __device__ void run(int, int) const {}
            } none;
            const SweepLists ls = {cnt, nullptr, lists, lists + L::LIST_A, nullptr};
            smax_x = sweep<M, NT, RB, 0, EXACT>(sm, wet, ls, P, none);
            smax_y = sweep<M, NT, RB, 1, EXACT>(sm, wet, ls, P, none);
        } else {
            /* The x sweep's first band is listed before it, every next band's
             * faces during the band before, and the y sweep's spread over all
             * phases of the x sweep. */
            struct Side {
                const double* sm;
                const unsigned char* wet;
                SweepLists x, y;
                double g, crit, crit2;
                int nbx, ncx, ncy, ny; /* x bands, chunks of a band of x and y, chunks of y */
                __device__ __forceinline__ int xs(int p) const
                {
                    return (p >> 1) + 1 < nbx ? ((p & 1) ? ncx - ncx / 2 : ncx / 2) : 0;
                }
                __device__ __forceinline__ int y0(int p) const { return min(p, 2 * nbx) * ny / (2 * nbx); }
                __device__ __forceinline__ int count(int p) const { return xs(p) + y0(p + 1) - y0(p); }
                __device__ __forceinline__ void run(int p, int c) const
                {
                    const int nx = xs(p);
                    if (c < nx) {
                        list_chunk<M, RB, 0>(sm, wet, x, g, crit, crit2, (p >> 1) + 1, (p & 1) ? ncx / 2 + c : c);
                    } else {
                        const int e = y0(p) + c - nx, band = e / ncy;
                        list_chunk<M, RB, 1>(sm, wet, y, g, crit, crit2, band, e - band * ncy);
                    }
                }
            };
            struct None {
                __device__ __forceinline__ int count(int) const { return 0; }
                __device__ __forceinline__ void run(int, int) const {}
            };
            auto lists_of = [&](int d) -> SweepLists {
                uint16_t* p = lists + d * L::LIST_SWEEP;
                return {cnt + d * L::CNT_SWEEP, cnt + L::CNT_CUR + d * L::CUR_SWEEP, p, p + L::LIST_A,
                        p + L::LIST_A + L::LIST_B};
            };
            constexpr int NBAND = (M + 2 + RB - 1) / RB, NCH = (RB * (M + 3) + 31) / 32;
            Side side = {sm, wet, lists_of(0), lists_of(1), g, sc[SC_CRIT], sc[SC_CRIT2], NBAND, NCH, NCH, NBAND * NCH};
            for (int c = warp; c < side.ncx; c += NT / 32)
                list_chunk<M, RB, 0>(sm, wet, side.x, g, side.crit, side.crit2, 0, c);
            __syncthreads();
            smax_x = sweep<M, NT, RB, 0, EXACT>(sm, wet, side.x, P, side);
            smax_y = sweep<M, NT, RB, 1, EXACT>(sm, wet, side.y, P, None());
        }
    }

    /* ---- flux-difference update, src2, write interior ---- */
    double* gq = wk.qout ? wk.qout : wk.q;
    const double* gaux = wk.aux;
    const int fidx = P.friction_index - 1;
    for (int e = threadIdx.x; e < M * M; e += NT) {
        const int i = 1 + e % M, j = 1 + e / M;
        const int k = (j + 1) * N + (i + 1);
        double h = sm[L::OFF_H + k], hu = sm[L::OFF_HU + k], hv = sm[L::OFF_HV + k];
        constexpr int PL = L::PLANE;
        const int a = (i - 1) + L::MS * (j - 1); /* accumulator index of the cell */
        if (EXACT) {
            /* q - dtdx*(fm(i+1,j) - fp(i,j)) - dtdy*(gm(i,j+1) - gp(i,j)) */
            const double* FM = sm + L::OFF_ACC;
            const double* FP = FM + 3 * PL;
            const double* GM = FP + 3 * PL;
            const double* GP = GM + 3 * PL;
            h = h - dtdx * (FM[a] - FP[a]) - dtdy * (GM[a] - GP[a]);
            hu = hu - dtdx * (FM[a + PL] - FP[a + PL]) - dtdy * (GM[a + PL] - GP[a + PL]);
            hv = hv - dtdx * (FM[a + 2 * PL] - FP[a + 2 * PL]) - dtdy * (GM[a + 2 * PL] - GP[a + 2 * PL]);
        } else if (any_wet) {
            const double* DX = sm + L::OFF_ACC;
            const double* DY = sm + L::OFF_ACC + 3 * PL;
            h = fma(-dtdy, DY[a], fma(-dtdx, DX[a], h));
            hu = fma(-dtdy, DY[a + PL], fma(-dtdx, DX[a + PL], hu));
            hv = fma(-dtdy, DY[a + 2 * PL], fma(-dtdx, DX[a + 2 * PL], hv));
        }
        if (P.src_term > 0) {
            const double nvar = (P.variable_friction && fidx >= 0 && fidx < maux)
                                    ? gaux[(size_t)fidx * S + k]
                                    : 0.0;
            src2_cell<FAST>(P, dt, sc + SC_KF, sm[L::OFF_B + k], nvar, h, hu, hv);
        }
        gq[k] = h;
        gq[S + k] = hu;
        gq[2 * S + k] = hv;
    }

    if (wk.fl && threadIdx.x == 0) {
        wk.fl->ident = (!any_wet && !changed) ? 1 : 0;
        wk.fl->wet = any_wet ? 1 : 0;
    }

    /* ---- CFL: the largest of dt/dx |s| and dt/dy |s|, over the warp, then over
     * the CTA, on the integer pipe (non-negative doubles order as integers);
     * NaN speeds were left out face by face ---- */
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
    if (threadIdx.x == 0) {
        double cfl = sc[SC_CFL];
        if (cfl > P.maxcfl_cap) cfl = 0.0;
        if (cfl_out) cfl_out[wi] = cfl;
        if (group_max) atomicMax(group_max + wk.group, dkey(cfl));
    }
    /* shared memory is restaged by the bulk (async-proxy) copies of the next
     * work item: order this item's generic-proxy accesses before them */
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    return true;
}

/* The fused kernel for one patch size: one CTA per work item, or a
 * persistent grid striding over the work list. */
template <int M, int NT, int RB, int MINB, bool EXACT>
__global__ void __launch_bounds__(NT, MINB)
    patch_update_kernel(const gf_patch_work* __restrict__ work, int nwork,
                        const gf_phys* __restrict__ phys_table, double dt_uniform,
                        const double* __restrict__ group_dt, const int* __restrict__ group_par,
                        int maux, double* __restrict__ cfl_out,
                        unsigned long long* __restrict__ group_max, int* __restrict__ err)
{
    using L = Smem<M, RB, EXACT>;
    extern __shared__ __align__(128) double sm[];
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm + L::OFF_BAR);
    if (threadIdx.x == 0) mbar_init(bar, 1);
    __syncthreads();
    uint32_t phase = 0;
    for (int wi = blockIdx.x; wi < nwork; wi += gridDim.x)
        if (!patch_item<M, NT, RB, EXACT>(sm, bar, phase, work[wi], wi, phys_table, dt_uniform, group_dt,
                                          group_par, maux, cfl_out, group_max, err))
            return;
}

/* Shared-memory bytes of the mixed kernel: the largest class layout, then
 * the mbarrier and the two work-cursor slots. */
template <int RB8, int RB16, int RB32, bool EXACT>
struct MixedSmem {
    static constexpr size_t B8 = Smem<8, RB8, EXACT>::BYTES, B16 = Smem<16, RB16, EXACT>::BYTES,
                            B32 = Smem<32, RB32, EXACT>::BYTES;
    static constexpr size_t MAXB = B8 > B16 ? (B8 > B32 ? B8 : B32) : (B16 > B32 ? B16 : B32);
    static constexpr size_t OFF_CTL = (MAXB + 15) / 16 * 16;
    static constexpr size_t BYTES = OFF_CTL + 32;
};

/* All patch sizes in one persistent launch. The work list holds the mx = 32
 * items, then the mx = 16 items, then the mx = 8 items; CTAs take items in
 * that order from a device cursor (sched[0]) so that the long items start
 * first and the short ones fill the tail. sched[1] counts CTAs that found
 * the list empty; the last of them resets both counters for the next launch
 * (both start at zero). */
template <int NT, int RB8, int RB16, int RB32, bool EXACT>
__global__ void __launch_bounds__(NT, 1)
    patch_update_mixed_kernel(const gf_patch_work* __restrict__ work, int n32, int n16, int n8,
                              const gf_phys* __restrict__ phys_table, double dt_uniform,
                              const double* __restrict__ group_dt, const int* __restrict__ group_par,
                              int maux, double* __restrict__ cfl_out,
                              unsigned long long* __restrict__ group_max, int* __restrict__ err,
                              unsigned int* __restrict__ sched)
{
    using X = MixedSmem<RB8, RB16, RB32, EXACT>;
    extern __shared__ __align__(128) double sm[];
    uint64_t* bar = reinterpret_cast<uint64_t*>(reinterpret_cast<char*>(sm) + X::OFF_CTL);
    volatile int* slot = reinterpret_cast<volatile int*>(reinterpret_cast<char*>(sm) + X::OFF_CTL + 8);
    if (threadIdx.x == 0) mbar_init(bar, 1);
    __syncthreads();
    const int nwork = n32 + n16 + n8;
    uint32_t phase = 0;
    /* the cursor value goes through one of two slots by iteration parity: a
     * skipped item has no barrier after its read, and the next write goes to
     * the other slot */
    for (int it = 0;; ++it) {
        if (threadIdx.x == 0) slot[it & 1] = (int)atomicAdd(sched, 1u);
        __syncthreads();
        const int wi = slot[it & 1];
        if (wi >= nwork) break;
        bool ok;
        if (wi < n32)
            ok = patch_item<32, NT, RB32, EXACT>(sm, bar, phase, work[wi], wi, phys_table, dt_uniform, group_dt,
                                                 group_par, maux, cfl_out, group_max, err);
        else if (wi < n32 + n16)
            ok = patch_item<16, NT, RB16, EXACT>(sm, bar, phase, work[wi], wi, phys_table, dt_uniform, group_dt,
                                                 group_par, maux, cfl_out, group_max, err);
        else
            ok = patch_item<8, NT, RB8, EXACT>(sm, bar, phase, work[wi], wi, phys_table, dt_uniform, group_dt,
                                               group_par, maux, cfl_out, group_max, err);
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
