/*
 * Kernel instantiations and launchers for the patch update and the
 * host-layout conversions used at the drop-in boundary.
 *
 * The tile shapes per patch size and the choice among them stand at kTiles8 ..
 * kTiles32 and pick_tile.
 */
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>

#include "gf_internal.h"
#include "gf_patch_update.cuh"
#include "gf_patch_stream.cuh"

namespace gf {

template <int M, int NT, int RB, int MINB>
static cudaError_t launch_update(const gf_patch_work* work, int nwork, const gf_phys* phys,
                                 double dt, const double* gdt, const int* gpar, int maux, double* cfl,
                                 unsigned long long* gmax, int* err, int max_ctas, cudaStream_t st)
{
    using L = Smem<M, RB, false>;
    auto kern = patch_update_kernel<M, NT, RB, MINB, false>;
    static std::atomic<unsigned long long> attr_done{0};
    cudaError_t ae = smem_attr_per_device(kern, (int)L::BYTES, attr_done);
    if (ae != cudaSuccess) return ae;
    if (nwork <= 0) return cudaSuccess;
    const int grid = (max_ctas > 0 && max_ctas < nwork) ? max_ctas : nwork;
    kern<<<grid, NT, L::BYTES, st>>>(work, nwork, phys, dt, gdt, gpar, maux, cfl, gmax, err);
    return cudaGetLastError();
}

template <int M, int NT, int R, int MINB>
static cudaError_t launch_stream(const gf_patch_work* work, int nwork, const gf_phys* phys,
                                 double dt, const double* gdt, const int* gpar, int maux, double* cfl,
                                 unsigned long long* gmax, int* err, int max_ctas, cudaStream_t st)
{
    using L = StreamSmem<M, R>;
    auto kern = patch_update_stream_kernel<M, NT, R, MINB>;
    static std::atomic<unsigned long long> attr_done{0};
    cudaError_t ae = smem_attr_per_device(kern, (int)L::BYTES, attr_done);
    if (ae != cudaSuccess) return ae;
    if (nwork <= 0) return cudaSuccess;
    const int grid = (max_ctas > 0 && max_ctas < nwork) ? max_ctas : nwork;
    kern<<<grid, NT, L::BYTES, st>>>(work, nwork, phys, dt, gdt, gpar, maux, cfl, gmax, err);
    return cudaGetLastError();
}

/* The split form: each work item on a cluster of K CTAs (one window of
 * rows each); not persistent, so max_ctas does not apply. */
template <int M, int NT, int R, int K, int MINB>
static cudaError_t launch_window(const gf_patch_work* work, int nwork, const gf_phys* phys,
                                 double dt, const double* gdt, const int* gpar, int maux, double* cfl,
                                 unsigned long long* gmax, int* err, int max_ctas, cudaStream_t st)
{
    (void)max_ctas;
    using L = StreamSmem<M, R, K>;
    auto kern = patch_update_window_kernel<M, NT, R, K, MINB>;
    static std::atomic<unsigned long long> attr_done{0};
    cudaError_t ae = smem_attr_per_device(kern, (int)L::BYTES, attr_done);
    if (ae != cudaSuccess) return ae;
    if (nwork <= 0) return cudaSuccess;
    kern<<<nwork * K, NT, L::BYTES, st>>>(work, nwork, phys, dt, gdt, gpar, maux, cfl, gmax, err);
    return cudaGetLastError();
}

/* Patches one launch of the window kernel runs at once: the clusters of K
 * CTAs the device holds resident together (placement inside a GPC counted). */
template <int M, int NT, int R, int K, int MINB>
static int window_slots()
{
    using L = StreamSmem<M, R, K>;
    auto kern = patch_update_window_kernel<M, NT, R, K, MINB>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::BYTES) !=
        cudaSuccess)
        return 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(K * sm_count());
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = L::BYTES;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) return 0;
    return n;
}

template <int M, int NT, int R, int K, int MINB>
static int window_occupancy()
{
    using L = StreamSmem<M, R, K>;
    auto kern = patch_update_window_kernel<M, NT, R, K, MINB>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::BYTES) !=
        cudaSuccess)
        return 0;
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, NT, L::BYTES) != cudaSuccess) return 0;
    return n;
}

/* ---- tile shapes (threads per patch x slices per band) per patch size ----
 * Without a choice by hand a launch takes its tile by its number of patches
 * (pick_tile); gf_autotune measures them all and installs the fastest for
 * throughput (whole levels) and for latency (a lone small scenario, where one
 * patch's critical path is the step time). */
using UpdateFn = cudaError_t (*)(const gf_patch_work*, int, const gf_phys*, double, const double*,
                                 const int*, int, double*, unsigned long long*, int*, int, cudaStream_t);
using OccFn = int (*)();

template <int M, int NT, int RB, int MINB>
static int occupancy_of()
{
    using L = Smem<M, RB, false>;
    auto kern = patch_update_kernel<M, NT, RB, MINB, false>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::BYTES) !=
        cudaSuccess)
        return 0;
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, NT, L::BYTES) != cudaSuccess) return 0;
    return n;
}

template <int M, int NT, int R, int MINB>
static int stream_occupancy()
{
    using L = StreamSmem<M, R>;
    auto kern = patch_update_stream_kernel<M, NT, R, MINB>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::BYTES) !=
        cudaSuccess)
        return 0;
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, NT, L::BYTES) != cudaSuccess) return 0;
    return n;
}

template <int M, int NT, int R, int MINB>
static int stream_slots() { return stream_occupancy<M, NT, R, MINB>() * sm_count(); }

template <int M, int NT, int RB, int MINB>
static int tile_slots() { return occupancy_of<M, NT, RB, MINB>() * sm_count(); }

struct Tile {
    int nt, rb, k; /* k > 1: the patch split over a cluster of k CTAs */
    UpdateFn fn;
    OccFn occ;
    OccFn slots; /* patches resident at once in one launch */
};

#define GF_TILE(M, NT, RB, MINB)                                                              \
    {NT, RB, 1, &launch_update<M, NT, RB, MINB>, &occupancy_of<M, NT, RB, MINB>,              \
     &tile_slots<M, NT, RB, MINB>}
#define GF_STILE(M, NT, R, MINB)                                                              \
    {NT, R, 1, &launch_stream<M, NT, R, MINB>, &stream_occupancy<M, NT, R, MINB>,             \
     &stream_slots<M, NT, R, MINB>}
#define GF_WTILE(M, NT, R, K, MINB)                                                           \
    {NT, R, K, &launch_window<M, NT, R, K, MINB>, &window_occupancy<M, NT, R, K, MINB>,       \
     &window_slots<M, NT, R, K, MINB>}
static const Tile kTiles8[] = {GF_TILE(8, 64, 5, 6), GF_TILE(8, 128, 10, 4), GF_STILE(8, 128, 11, 4),
                               GF_WTILE(8, 128, 7, 2, 2), GF_WTILE(8, 128, 5, 4, 2)};
static const Tile kTiles16[] = {GF_STILE(16, 128, 5, 3), GF_STILE(16, 192, 7, 2), GF_TILE(16, 256, 9, 2),
                                GF_WTILE(16, 256, 11, 2, 2), GF_WTILE(16, 256, 7, 4, 1), GF_WTILE(16, 256, 5, 8, 1)};
static const Tile kTiles32[] = {GF_TILE(32, 256, 7, 1), GF_STILE(32, 256, 4, 2), GF_TILE(32, 384, 7, 1),
                                GF_TILE(32, 384, 9, 1), GF_WTILE(32, 384, 11, 4, 1), GF_WTILE(32, 384, 7, 8, 1),
                                GF_WTILE(32, 384, 10, 2, 1)};
#undef GF_TILE
#undef GF_STILE
#undef GF_WTILE

static const Tile* tiles_of(int m, int* n)
{
    switch (m) {
    case 8: *n = (int)(sizeof kTiles8 / sizeof kTiles8[0]); return kTiles8;
    case 16: *n = (int)(sizeof kTiles16 / sizeof kTiles16[0]); return kTiles16;
    case 32: *n = (int)(sizeof kTiles32 / sizeof kTiles32[0]); return kTiles32;
    default: *n = 0; return nullptr;
    }
}

/* Tile of a launch without a choice by hand, where the number of patches does
 * not name another one (pick_tile). 8^2 patches take the
 * streamed form, a whole patch in its one band, four CTAs an SM (4096 patches
 * 288 us, three CTAs 305, 128 x 10 swept 323), 16^2 its bands of five rows,
 * three CTAs an SM (5561 patches 1.27 ms at 80 % wet and 0.85 at 50 %, swept
 * 128 x 6 1.31 and 0.92, streamed 192 x 7 1.34 and 0.93), 32^2 patches 384 x 9
 * (4096 patches 3.43 ms, 256 x 7 3.61) or the streamed form, pick_tile. */
static const int kDefault[3] = {2, 0, 3};
/* Chosen per goal (0 throughput, 1 latency) and patch size: by hand (tile_set),
 * by gf_autotune; -1: not. */
static std::atomic<int> g_pin[2][3] = {{-1, -1, -1}, {-1, -1, -1}};
static std::atomic<int> g_tuned[2][3] = {{-1, -1, -1}, {-1, -1, -1}};
static inline int mcls(int m) { return m == 8 ? 0 : m == 16 ? 1 : 2; }

int tile_count(int m)
{
    int n = 0;
    tiles_of(m, &n);
    return n;
}

int tile_shape(int m, int v, int* nt, int* rb, int* k)
{
    int n = 0;
    const Tile* t = tiles_of(m, &n);
    if (!t || v < 0 || v >= n) return -1;
    *nt = t[v].nt;
    *rb = t[v].rb;
    if (k) *k = t[v].k;
    return 0;
}

static int chosen(int m, int goal) /* by hand, else tuned, else -1 */
{
    const int pin = g_pin[goal != 0][mcls(m)];
    return pin >= 0 ? pin : g_tuned[goal != 0][mcls(m)].load();
}

int tile_get(int m, int goal)
{
    const int v = chosen(m, goal);
    return v >= 0 ? v : GF_TILE_AUTO;
}

/* Patches that one launch of variant v runs at once on this device. */
static long tile_resident(int m, int v)
{
    int n = 0;
    const Tile* t = tiles_of(m, &n);
    static std::atomic<int> cache[64][3][GF_MAX_TILES] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64 || v >= GF_MAX_TILES) return sm_count() / t[v].k;
    std::atomic<int>& c = cache[dev][mcls(m)][v];
    int slots = c.load(std::memory_order_relaxed);
    if (!slots) {
        slots = t[v].slots();
        if (slots <= 0) slots = sm_count() / t[v].k;
        if (slots <= 0) slots = 1;
        c.store(slots, std::memory_order_relaxed);
    }
    return slots;
}

/* The latency tile pays for its split only while every patch of the launch
 * is resident at once; past one wave the throughput tile finishes sooner. */
int latency_goal_fits(int m, long npatch)
{
    int n = 0;
    if (!tiles_of(m, &n)) return 0;
    const int v = chosen(m, 1);
    return npatch <= tile_resident(m, v >= 0 ? v : kDefault[mcls(m)]) ? 1 : 0;
}

/* Launches that leave SMs idle take a tile that spreads a patch: the first of
 * these with at most per_2sm CTAs for two SMs (FP64 throughput is the SM's, so a
 * split pays while SMs are free), and, for one_wave, all of them resident at
 * once (clusters of 8 of 15 patches on this device, of 4 of 36). us for that many 32^2 patches, the next choice beside it: K = 8 42 (1;
 * 56), K = 4 55 (24; 90), K = 2 90 (72; 171), 167 (152; 188), 251 (247; 288), but
 * 325 (304; 289); 16^2: K = 8 29 (1; 31), K = 4 33 (24; 40), K = 2 41 (72; 64), 54
 * (152; 64), the streamed 192 x 7 94 (304; 102) and 166 (400; 134); 8^2: K = 4 29
 * (24; 35) and 31 (72; 31). */
struct SmallTile {
    int v, per_2sm;
    bool one_wave;
};
static const SmallTile kSmall8[] = {{4, 2, true}};
static const SmallTile kSmall16[] = {{5, 2, true}, {4, 2, true}, {3, 4, true}, {1, 4, true}};
static const SmallTile kSmall32[] = {{5, 2, true}, {4, 2, true}, {6, 7, false}};
/* Whole 32^2 levels: the streamed tile, two CTAs an SM, when it fills its slots
 * once (247 patches 286 us, 384 x 9 301) or many times (4096 patches 3.18 ms,
 * 3.34; 1215 1.07, 1.09); between, its half-empty last wave costs more than it
 * gains (400 patches 504 us against 442, 760 671 against 612). */
constexpr int kStream32 = 1, kStream32Waves = 6; /* patches an SM from which it always pays */

/* Tile of a capped launch, whose CTAs walk the list on part of the SMs: no rule
 * by the number of patches. */
static int capped_tile(int m)
{
    const int v = chosen(m, 0);
    return v >= 0 ? v : kDefault[mcls(m)];
}

/* A choice by hand always stands, the tuned latency tile where it is asked for.
 * The tuned throughput tile serves launches of the size it was measured on:
 * below, the number of patches decides as without it (400 patches of 32^2 442 us
 * so, 504 by the tile that is the fastest for 4096; 760 612 and 671). whole: the
 * patches of the level that the launch is a part of; parts follow one another
 * on two streams, without the last waves that decide for a launch by itself (host
 * step of 4096 patches, half of them wet, 2.76 ms by the part's number, 2.47 by the
 * level's). */
static int pick_tile(int m, long npatch, int max_ctas, int goal, long whole = 0)
{
    const int c = mcls(m);
    goal = goal != 0;
    const int pin = g_pin[goal][c], best = g_tuned[goal][c];
    if (pin >= 0) return pin;
    if (goal && best >= 0) return best;
    if (max_ctas > 0) return capped_tile(m);
    int nt = 0;
    const Tile* t = tiles_of(m, &nt);
    const SmallTile* s = c == 0 ? kSmall8 : c == 1 ? kSmall16 : kSmall32;
    const int ns = (int)(c == 0 ? sizeof kSmall8 : c == 1 ? sizeof kSmall16 : sizeof kSmall32) / (int)sizeof *s;
    for (int i = 0; i < ns; ++i)
        if (2 * npatch * t[s[i].v].k <= (long)s[i].per_2sm * sm_count() &&
            (!s[i].one_wave || npatch <= tile_resident(m, s[i].v)))
            return s[i].v;
    if (const int by_hand = g_pin[0][c]; by_hand >= 0) return by_hand; /* goal 1 */
    if (const int tuned = g_tuned[0][c]; tuned >= 0 && std::max(npatch, whole) * m * m >= kTuneCells) return tuned;
    if (c == 2 && (npatch <= tile_resident(m, kStream32) || npatch >= (long)kStream32Waves * sm_count()))
        return kStream32;
    return kDefault[c];
}

int tile_of(int m, long npatch, int goal) { return pick_tile(m, npatch, 0, goal); }

int tile_set(int m, int goal, int v)
{
    int n = 0;
    tiles_of(m, &n);
    if (v == GF_TILE_AUTO) {
        g_pin[goal != 0][mcls(m)] = -1;
        g_tuned[goal != 0][mcls(m)] = -1;
        return 0;
    }
    if (v < 0 || v >= n) return -1;
    g_pin[goal != 0][mcls(m)] = v;
    return 0;
}

void tile_install_tuned(int m, int throughput, int latency)
{
    const int c = mcls(m);
    g_tuned[0][c] = throughput;
    g_tuned[1][c] = latency;
    g_pin[0][c] = g_pin[1][c] = -1;
}

cudaError_t launch_patch_update_tile(int m, int v, const gf_patch_work* work, int nwork,
                                     const gf_phys* phys, double dt, const double* gdt,
                                     const int* gpar, int maux, double* cfl,
                                     unsigned long long* gmax, int* err, cudaStream_t st,
                                     int max_ctas)
{
    int n = 0;
    const Tile* t = tiles_of(m, &n);
    if (!t || v < 0 || v >= n) return cudaErrorInvalidValue;
    return t[v].fn(work, nwork, phys, dt, gdt, gpar, maux, cfl, gmax, err, max_ctas, st);
}

cudaError_t launch_patch_update(int m, const gf_patch_work* work, int nwork, const gf_phys* phys,
                                double dt, const double* gdt, const int* gpar, int maux, double* cfl,
                                unsigned long long* gmax, int* err, cudaStream_t st, int max_ctas,
                                int goal, long whole)
{
    if (!(m == 8 || m == 16 || m == 32)) return cudaErrorInvalidValue;
    if (nwork <= 0) { /* set every tile's attributes, ahead of a capture */
        int n = 0;
        const Tile* t = tiles_of(m, &n);
        for (int v = 0; v < n; ++v) {
            tile_resident(m, v);
            cudaError_t e = t[v].fn(work, 0, phys, dt, gdt, gpar, maux, cfl, gmax, err, 0, st);
            if (e != cudaSuccess) return e;
        }
        return cudaSuccess;
    }
    return launch_patch_update_tile(m, pick_tile(m, nwork, max_ctas, goal, whole), work, nwork, phys, dt, gdt,
                                    gpar, maux, cfl, gmax, err, st, max_ctas);
}

int sm_count()
{
    static int cache[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 1;
    if (!cache[dev]) {
        int n = 0;
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        cache[dev] = n > 0 ? n : 1;
    }
    return cache[dev];
}

/* One launch for every size, 256 threads. Uncapped: the streamed form, two
 * CTAs an SM (rows per band 11, 7, 4). With a cap, which leaves SMs free for
 * other launches: the swept form, one CTA an SM (mx = 8 a whole patch per band,
 * mx = 16 its 256-thread variant). */
constexpr int kMixNT = 256, kMixRB8 = 10, kMixRB16 = 13, kMixRB32 = 7;
constexpr int kMixR8 = 11, kMixR16 = 7, kMixR32 = 4;

cudaError_t launch_patch_update_mixed(const gf_patch_work* work, const int n[3], const gf_phys* phys,
                                      double dt, const double* gdt, const int* gpar, int maux,
                                      double* cfl, unsigned long long* gmax, int* err,
                                      unsigned int* sched, cudaStream_t st, int max_ctas)
{
    using X = MixedSmem<kMixRB8, kMixRB16, kMixRB32, false>;
    auto kern = patch_update_mixed_kernel<kMixNT, kMixRB8, kMixRB16, kMixRB32, false>;
    static std::atomic<unsigned long long> attr_done{0};
    cudaError_t ae = smem_attr_per_device(kern, (int)X::BYTES, attr_done);
    if (ae != cudaSuccess) return ae;
    using Y = MixedStreamSmem<kMixR8, kMixR16, kMixR32>;
    auto skern = patch_update_mixed_stream_kernel<kMixNT, kMixR8, kMixR16, kMixR32>;
    static std::atomic<unsigned long long> sattr_done{0};
    if ((ae = smem_attr_per_device(skern, (int)Y::BYTES, sattr_done)) != cudaSuccess) return ae;
    const int nwork = n[0] + n[1] + n[2];
    if (nwork <= 0) return cudaSuccess;
    int grid = sm_count();
    if (max_ctas <= 0 || max_ctas >= grid) {
        grid = std::min(2 * grid, nwork);
        skern<<<grid, kMixNT, Y::BYTES, st>>>(work, n[0], n[1], n[2], phys, dt, gdt, gpar, maux, cfl, gmax, err, sched);
        return cudaGetLastError();
    }
    grid = std::min(max_ctas, nwork);
    kern<<<grid, kMixNT, X::BYTES, st>>>(work, n[0], n[1], n[2], phys, dt, gdt, gpar, maux, cfl, gmax, err,
                                         sched);
    return cudaGetLastError();
}

int patch_update_occupancy(int m, bool capped)
{
    int n = 0;
    const Tile* t = tiles_of(m, &n);
    if (!t) return 0;
    const int pin = g_pin[0][mcls(m)];
    return t[capped ? capped_tile(m) : pin >= 0 ? pin : kDefault[mcls(m)]].occ();
}

/* ---- layout conversion at the boundary ----
 * Fortran layout a(nf, 0..nx-1, 0..ny-1) of npatch contiguous patches
 * <-> planes [patch][field][cell]. One thread per (patch, cell). */
__global__ void aos_to_soa_kernel(const double* __restrict__ src, double* __restrict__ dst,
                                  long npatch, int ncell, int nf, long src_stride, long dst_stride)
{
    const long total = npatch * (long)ncell;
    for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < total;
         e += (long)gridDim.x * blockDim.x) {
        const long p = e / ncell;
        const int k = (int)(e % ncell);
        const double* s = src + p * src_stride + (long)k * nf;
        double* d = dst + p * dst_stride + k;
        for (int f = 0; f < nf; ++f) d[(long)f * ncell] = s[f];
    }
}

__global__ void soa_to_aos_kernel(const double* __restrict__ src, double* __restrict__ dst,
                                  long npatch, int ncell, int nf, long src_stride, long dst_stride)
{
    const long total = npatch * (long)ncell;
    for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < total;
         e += (long)gridDim.x * blockDim.x) {
        const long p = e / ncell;
        const int k = (int)(e % ncell);
        const double* s = src + p * src_stride + k;
        double* d = dst + p * dst_stride + (long)k * nf;
        for (int f = 0; f < nf; ++f) d[f] = s[(long)f * ncell];
    }
}

static int conv_grid(long total)
{
    long b = (total + 255) / 256;
    if (b > 152L * 16) b = 152L * 16;
    if (b < 1) b = 1;
    return (int)b;
}

cudaError_t launch_aos_to_soa(const double* src, double* dst, long npatch, int ncell, int nf,
                              long src_stride, long dst_stride, cudaStream_t st)
{
    const long total = npatch * (long)ncell;
    if (total == 0) return cudaSuccess;
    aos_to_soa_kernel<<<conv_grid(total), 256, 0, st>>>(src, dst, npatch, ncell, nf, src_stride,
                                                        dst_stride);
    return cudaGetLastError();
}

/* A host batch's traffic, straight from and to its pinned host buffers: in one
 * launch q and aux into planes (reads in address order; also zeroes the batch's
 * status), in another the planes of q back (writes in address order) with the
 * status and the patch CFLs. Copies to and from a device buffer ahead of and
 * behind these cost two operations more a call (one 32^2 patch: 84 us a call, now 72). */
__global__ void batch_in_kernel(const double* __restrict__ hq, double* __restrict__ q, const double* __restrict__ ha,
                                double* __restrict__ aux, int maux, long npatch, int ncell,
                                unsigned long long* __restrict__ gmax, int* __restrict__ err)
{
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *gmax = 0ull;
        *err = 0;
    }
    const long nq = npatch * 3 * ncell, total = nq + npatch * (long)maux * ncell;
    for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < total; e += (long)gridDim.x * blockDim.x) {
        const bool second = e >= nq;
        const long ee = second ? e - nq : e;
        const int nf = second ? maux : 3;
        const long cell = ee / nf, p = cell / ncell;
        const int f = (int)(ee - cell * nf), k = (int)(cell - p * ncell);
        (second ? aux : q)[(p * nf + f) * ncell + k] = (second ? ha : hq)[ee];
    }
}

__global__ void batch_out_kernel(const double* __restrict__ q, double* __restrict__ hq, long npatch, int ncell,
                                 const double* __restrict__ cfl, double* __restrict__ hcfl,
                                 const unsigned long long* __restrict__ gmax, const int* __restrict__ err,
                                 unsigned long long* __restrict__ hgmax, int* __restrict__ herr)
{
    const long t = blockIdx.x * (long)blockDim.x + threadIdx.x, step = (long)gridDim.x * blockDim.x;
    if (t == 0) {
        *hgmax = *gmax;
        *herr = *err;
    }
    if (hcfl)
        for (long e = t; e < npatch; e += step) hcfl[e] = cfl[e];
    const long total = npatch * 3 * ncell;
    for (long e = t; e < total; e += step) {
        const long cell = e / 3, p = cell / ncell;
        const int f = (int)(e - cell * 3), k = (int)(cell - p * ncell);
        hq[e] = q[(p * 3 + f) * ncell + k];
    }
}

cudaError_t launch_batch_in(const double* hq, double* q, const double* ha, double* aux, int maux, long npatch,
                            int ncell, unsigned long long* gmax, int* err, cudaStream_t st)
{
    if (npatch <= 0) return cudaSuccess;
    batch_in_kernel<<<conv_grid(npatch * (3L + maux) * ncell), 256, 0, st>>>(hq, q, ha, aux, maux, npatch, ncell, gmax,
                                                                             err);
    return cudaGetLastError();
}

cudaError_t launch_batch_out(const double* q, double* hq, long npatch, int ncell, const double* cfl, double* hcfl,
                             const unsigned long long* gmax, const int* err, unsigned long long* hgmax, int* herr,
                             cudaStream_t st)
{
    if (npatch <= 0) return cudaSuccess;
    batch_out_kernel<<<conv_grid(npatch * 3L * ncell), 256, 0, st>>>(q, hq, npatch, ncell, cfl, hcfl, gmax, err, hgmax,
                                                                     herr);
    return cudaGetLastError();
}

cudaError_t launch_soa_to_aos(const double* src, double* dst, long npatch, int ncell, int nf,
                              long src_stride, long dst_stride, cudaStream_t st)
{
    const long total = npatch * (long)ncell;
    if (total == 0) return cudaSuccess;
    soa_to_aos_kernel<<<conv_grid(total), 256, 0, st>>>(src, dst, npatch, ncell, nf, src_stride,
                                                        dst_stride);
    return cudaGetLastError();
}

} // namespace gf
