/* Host build of the face solvers: random faces through the single-precision
 * classes; where a class allows a shorter solve (smooth, edge) it must give
 * the full one's speeds and f-waves bit for bit. Prints the faces of each
 * class and those that differ. */
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

#define GF_HOST_MATH
#define __device__
#define __forceinline__ inline
static inline long long __double_as_longlong(double x) { long long v; std::memcpy(&v, &x, 8); return v; }
static inline double __longlong_as_double(long long v) { double x; std::memcpy(&x, &v, 8); return x; }
static inline int __double2hiint(double x) { return (int)(__double_as_longlong(x) >> 32); }
static inline int __double2loint(double x) { return (int)__double_as_longlong(x); }
static inline double __hiloint2double(int hi, int lo)
{
    return __longlong_as_double((long long)(((unsigned long long)(unsigned)hi << 32) | (unsigned)lo));
}
static inline unsigned __funnelshift_l(unsigned lo, unsigned hi, unsigned s) { return (hi << s) | (lo >> (32 - s)); }
static inline float __uint_as_float(unsigned u) { float f; std::memcpy(&f, &u, 4); return f; }
static inline unsigned __float_as_uint(float f) { unsigned u; std::memcpy(&u, &f, 4); return u; }
static inline double __dmul_rn(double a, double b) { return a * b; }
static inline double rsqrt(double x) { return 1.0 / std::sqrt(x); }
static inline double __dadd_rn(double a, double b) { return a + b; }
using std::fmax;
using std::fmin;
/* the solves spell out what the device compiler fuses, the full one does not:
 * unfused, all of them are the same products and sums */
#define fma(a, b, c) ((a) * (b) + (c))
/* approximations as coarse as the hardware's (about 2^-20), and quotients and
 * roots of the test with an error of a few units of their last place */
static int g_wobble = 0;
static inline float wob(float x) { g_wobble = g_wobble * 1103515245 + 12345; return x * (1.0f + 2.4e-7f * (float)((g_wobble >> 16) % 3 - 1)); }
static inline float __fdividef(float a, float b) { return wob(a / b); }
static inline float gf_sqrtf(float a) { return wob(std::sqrt(a)); }
static inline double gf_rcp_seed(double y) { return (1.0 / y) * (1.0 + 7.0e-7); }
static inline double gf_rsqrt_seed(double a) { return (1.0 / std::sqrt(a)) * (1.0 - 7.0e-7); }

#include "gf_riemann.cuh"

static bool same(double a, double b) { return a == b || (std::isnan(a) && std::isnan(b)); }

int main(int argc, char** argv)
{
    const int kind = std::atoi(argv[1]);
    const long n = std::atol(argv[2]);
    std::mt19937_64 r(1234 + kind);
    std::uniform_real_distribution<double> U(0.0, 1.0);
    auto logu = [&](double a, double b) { return a * std::pow(b / a, U(r)); };
    auto sgn = [&] { return U(r) < 0.5 ? -1.0 : 1.0; };
    const double g = 9.81;
    long count[4] = {0, 0, 0, 0}, differ = 0;
    for (long k = 0; k < n; ++k) {
        const double drytol = kind == 4 ? logu(1e-6, 1e-1) : 1e-3;
        double h[2], u[2], v[2], b[2];
        const double base = kind == 3 ? 2000.0 * U(r) : 10.0 * U(r);
        const double h0 = drytol * 1.001 + logu(1e-4, 50.0), near = logu(1e-14, 1.0);
        for (int s = 0; s < 2; ++s) {
            const double c = std::sqrt(g * h0);
            switch (kind) {
            case 0: /* smooth flow: neighbours close to each other */
                h[s] = h0 * (1.0 + near * (U(r) - 0.5));
                u[s] = 0.6 * c * sgn() * near + (s ? u[0] * 0.0 : 0.0) + 0.5 * c * (near - 0.5);
                b[s] = base + h0 * near * (U(r) - 0.5);
                break;
            case 1: /* anything: strong shocks, rarefactions, steps */
                h[s] = drytol * 1.001 + logu(1e-4, 50.0);
                u[s] = sgn() * logu(1e-6, 30.0);
                b[s] = base + sgn() * logu(1e-6, 20.0);
                break;
            case 2: /* near critical flow */
                h[s] = h0 * (1.0 + 0.2 * near * (U(r) - 0.5));
                u[s] = (s ? (u[0] < 0 ? -1.0 : 1.0) : sgn()) * c * (1.0 + near * (U(r) - 0.5));
                b[s] = base + h0 * near * (U(r) - 0.5);
                break;
            case 3: /* thin water on a high bed */
                h[s] = drytol * 1.001 + logu(1e-5, 0.1);
                u[s] = sgn() * logu(1e-6, 2.0);
                b[s] = base + sgn() * logu(1e-6, 0.5);
                break;
            case 5: /* lake at rest, exact and almost exact */
                h[s] = h0 * (s ? U(r) + 0.2 : 1.0);
                u[s] = U(r) < 0.5 ? 0.0 : sgn() * logu(1e-300, 1e-6);
                b[s] = base + h0 - h[s];
                break;
            default: /* jumps at the edge of the bounds of the steady-state wave */
                h[s] = drytol * 1.001 + logu(1e-3, 5.0);
                u[s] = sgn() * logu(1e-3, 5.0);
                b[s] = base + (s ? sgn() * (h[0] + h[1]) * (0.8 + 0.4 * U(r)) : 0.0);
            }
            if (h[s] <= drytol) h[s] = drytol * 1.01;
            v[s] = sgn() * logu(1e-6, 5.0);
        }
        /* one cell dry, with every step between the levels */
        const int dry = kind >= 7 ? (int)(U(r) * 2.0) : -1;
        if (dry >= 0) {
            const int w = 1 - dry;
            h[dry] = U(r) < 0.5 ? 0.0 : drytol * U(r);
            const double c0 = std::sqrt(g * h[w]);
            if (kind == 8) u[w] = c0 * 4.0 * (U(r) - 0.5);
            const double reach = (c0 + 0.5 * std::fabs(u[w])) * (c0 + 0.5 * std::fabs(u[w])) / g;
            b[dry] = b[w] + (U(r) < 0.5 ? h[w] : reach) * (U(r) < 0.3 ? 1.0 + sgn() * logu(1e-16, 1e-3) : 2.0 * U(r) - 0.5);
        }
        gf_cell c[2];
        for (int s = 0; s < 2; ++s) {
            c[s].h = h[s]; c[s].b = b[s]; c[s].wet = h[s] > drytol;
            c[s].hun = c[s].hut = c[s].un = c[s].ut = c[s].c = c[s].rc = 0.0;
            if (!c[s].wet) continue;
            c[s].rc = 1.0 / std::sqrt(g * h[s]);
            c[s].c = g * h[s] * c[s].rc;
            const double rh = g * (c[s].rc * c[s].rc);
            c[s].hun = h[s] * u[s]; c[s].hut = h[s] * v[s];
            c[s].un = c[s].hun * rh; c[s].ut = c[s].hut * rh;
        }
        const double crit = fmax(drytol * g, 1e-6), crit2 = std::sqrt(crit);
        const int cls = gf_face_class(gf_f32(c[0].h), gf_f32(c[1].h), gf_f32(c[0].un), gf_f32(c[1].un),
                                      gf_f32(c[0].c), gf_f32(c[1].c), gf_f32(c[0].b), gf_f32(c[1].b), c[0].wet,
                                      c[1].wet, (float)g, (float)crit, (float)crit2);
        ++count[cls];
        if (cls == 3) continue;
        double s1[3], f1[3][3], s2[3], f2[3][3];
        gf_rpn2_face<true>(c[0], c[1], g, drytol, 1.0 / (16.0 * g), rsqrt(g), crit, crit2, s1, f1);
        for (int solve = 0; solve < 2; ++solve) {
            if (solve == 0) {
                if (cls != 0) continue;
                gf_rpn2_smooth(c[0], c[1], g, s2, f2);
            } else {
                gf_rpn2_edge(c[0], c[1], cls == 2, g, crit, crit2, s2, f2);
            }
            bool eq = true;
            for (int w = 0; w < 3; ++w) {
                eq = eq && same(s1[w], s2[w]);
                for (int m = 0; m < 3; ++m) eq = eq && same(f1[w][m], f2[w][m]);
            }
            if (!eq) ++differ;
        }
    }
    std::printf("%ld %ld %ld %ld %ld\n", count[0], count[1], count[2], count[3], differ);
    return 0;
}
