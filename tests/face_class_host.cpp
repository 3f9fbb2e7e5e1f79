/* Host build of the single-precision face classes: faces from bit patterns (no
 * arithmetic that a compiler could fuse), their classes as a hash. Prints the
 * faces of each class and the hash. */
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
static inline double __dadd_rn(double a, double b) { return a + b; }
static inline double rsqrt(double x) { return 1.0 / std::sqrt(x); }
using std::fma;
using std::fmax;
using std::fmin;
static inline float __fdividef(float a, float b) { return a / b; }
static inline float gf_sqrtf(float a) { return std::sqrt(a); }
static inline double gf_rcp_seed(double y) { return 1.0 / y; }
static inline double gf_rsqrt_seed(double a) { return 1.0 / std::sqrt(a); }

#include "gf_riemann.cuh"

int main(int argc, char** argv)
{
    const long n = std::atol(argv[1]);
    std::mt19937_64 r(4321);
    /* a random significand, the exponent in lo .. hi */
    auto bits = [&](int lo, int hi) -> float {
        const uint64_t v = r();
        return __uint_as_float((unsigned)(127 + lo + (int)((v >> 40) % (unsigned)(hi - lo + 1))) << 23 | (unsigned)(v & 0x7fffff));
    };
    const float g = 9.81f, crit = 9.81e-3f, crit2 = std::sqrt(crit);
    long count[4] = {0, 0, 0, 0};
    uint64_t hash = 1469598103934665603ull;
    for (long k = 0; k < n; ++k) {
        const uint64_t v = r();
        float h[2], u[2], c[2], b[2];
        for (int s = 0; s < 2; ++s) {
            h[s] = s && (v & 1) ? __uint_as_float(__float_as_uint(h[0]) ^ (unsigned)(v >> 8 & 0x3ffff)) : bits(-6, 4);
            u[s] = s && (v & 2) ? __uint_as_float(__float_as_uint(u[0]) ^ (unsigned)(v >> 26 & 0x3ffff)) : bits(-8, 4);
            if (v & (uint64_t)4 << s) u[s] = -u[s];
            b[s] = s && (v & 16) ? __uint_as_float(__float_as_uint(b[0]) ^ (unsigned)(v >> 44 & 0x1ffff)) : bits(-2, 6);
            const float gh = gf_fmul(g, h[s]);
            c[s] = std::sqrt(gh);
        }
        const int dry = (v >> 62) == 3 ? (int)(v >> 61 & 1) : -1;
        if (dry >= 0) h[dry] = u[dry] = c[dry] = 0.0f;
        const int cls = gf_face_class(h[0], h[1], u[0], u[1], c[0], c[1], b[0], b[1], dry != 0, dry != 1, g, crit, crit2);
        ++count[cls];
        hash = (hash ^ (uint64_t)cls) * 1099511628211ull;
    }
    std::printf("%ld %ld %ld %ld %llu\n", count[0], count[1], count[2], count[3], (unsigned long long)hash);
    return 0;
}
