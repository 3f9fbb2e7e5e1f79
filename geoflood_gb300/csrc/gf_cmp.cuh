/*
 * FP64 comparisons and min / max on the integer pipe.
 *
 * On this GPU an FP64 warp instruction occupies the FP64 pipe for tens of
 * cycles while an integer instruction issues in two; comparisons and
 * min / max of doubles are a quarter of the patch update's FP64-pipe
 * instructions. With FAST = true these helpers compare the IEEE bit
 * patterns instead:
 *   - against zero they are exact (x > 0, x < 0, x == 0 with either zero);
 *   - between two values they use the order-preserving integer key of the
 *     bit pattern, which agrees with IEEE ordering except that -0 sorts
 *     below +0 (IEEE: equal). A NaN sorts by its sign, above infinity or below
 *     minus infinity, where IEEE comparisons are false: a depth that is a
 *     negative NaN is dry (the inflow states without a root, gf_ghost.cu), a
 *     positive one wet. d_max_abs leaves a NaN out.
 * With FAST = false they are the IEEE operations themselves, so the
 * contraction-free build keeps the reference's arithmetic bit for bit.
 */
#ifndef GF_CMP_CUH
#define GF_CMP_CUH

__device__ __forceinline__ long long gf_bits(double x) { return __double_as_longlong(x); }

/* order-preserving signed key: larger double <=> larger key */
__device__ __forceinline__ long long gf_okey(double x)
{
    const long long b = __double_as_longlong(x);
    return b ^ ((b >> 63) & 0x7fffffffffffffffLL);
}

template <bool F> __device__ __forceinline__ bool d_lt(double a, double b)
{
    if (F) return gf_okey(a) < gf_okey(b);
    return a < b;
}
template <bool F> __device__ __forceinline__ bool d_le(double a, double b)
{
    if (F) return gf_okey(a) <= gf_okey(b);
    return a <= b;
}
template <bool F> __device__ __forceinline__ bool d_gt(double a, double b) { return d_lt<F>(b, a); }
template <bool F> __device__ __forceinline__ bool d_ge(double a, double b) { return d_le<F>(b, a); }

/* against zero: exact for both zeros */
template <bool F> __device__ __forceinline__ bool d_gtz(double x)
{
    if (F) return gf_bits(x) > 0;
    return x > 0.0;
}
template <bool F> __device__ __forceinline__ bool d_ltz(double x)
{
    if (F) {
        const long long b = gf_bits(x);
        return b < 0 && (b << 1) != 0;
    }
    return x < 0.0;
}
template <bool F> __device__ __forceinline__ bool d_lez(double x) { return !d_gtz<F>(x); }
template <bool F> __device__ __forceinline__ bool d_gez(double x) { return !d_ltz<F>(x); }
template <bool F> __device__ __forceinline__ bool d_eqz(double x)
{
    if (F) return (gf_bits(x) << 1) == 0;
    return x == 0.0;
}

template <bool F> __device__ __forceinline__ double d_max(double a, double b)
{
    if (F) return gf_okey(a) < gf_okey(b) ? b : a;
    return fmax(a, b);
}
template <bool F> __device__ __forceinline__ double d_min(double a, double b)
{
    if (F) return gf_okey(b) < gf_okey(a) ? b : a;
    return fmin(a, b);
}
/* both operands >= +0 (or -0): the raw bit patterns order correctly */
template <bool F> __device__ __forceinline__ double d_max_nn(double a, double b)
{
    if (F) return gf_bits(a) < gf_bits(b) ? b : a;
    return fmax(a, b);
}

/* the larger of a (a number >= 0) and |x|; a where x is not a number, as fmax */
template <bool F> __device__ __forceinline__ double d_max_abs(double a, double x)
{
    if (F) {
        const long long b = gf_bits(x) & 0x7fffffffffffffffLL;
        return b > gf_bits(a) && b <= 0x7ff0000000000000LL ? __longlong_as_double(b) : a;
    }
    return fmax(a, fabs(x));
}

/* The hardware's approximate FP64 reciprocal and reciprocal root (subnormal
 * arguments count as zero). A host build of these headers (tests) brings its
 * own. */
#ifndef GF_HOST_MATH
__device__ __forceinline__ double gf_rcp_seed(double y)
{
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(y));
    return r;
}
__device__ __forceinline__ double gf_rsqrt_seed(double a)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
    return y;
}
#endif

/* 1/y from the hardware's approximate FP64 reciprocal r refined once with
 * the third-order step r + r (e + e^2), e = 1 - y r (the geometric series of
 * 1 / (1 - e) cut after e^2): the remainder e^3 is far below the last
 * rounding (measured over every exponent: 0.50 ulp at most). One FP64
 * instruction fewer than two Newton-Raphson steps. For normal y up to 2^1022
 * only (beyond, 1/y is no normal number): the inputs here are depths, speeds and
 * their differences away from zero. */
__device__ __forceinline__ double gf_rcp(double y)
{
    const double r = gf_rcp_seed(y);
    const double e = fma(-y, r, 1.0);
    return fma(r, fma(e, e, e), r);
}

/* positive and normal (neither zero, subnormal, infinite, NaN nor negative) */
__device__ __forceinline__ bool gf_pos_normal(double x)
{
    return static_cast<unsigned>(__double2hiint(x)) - 0x00100000u < 0x7ff00000u - 0x00100000u;
}

/* The root and its reciprocal of a positive normal a from the hardware's
 * approximate FP64 reciprocal root y and one third-order step: with
 * e = 1 - a y^2, a^(-1/2) = y (1 - e)^(-1/2) = y (1 + e/2 + 3 e^2/8 + ...);
 * the remainder of order e^3 is far below the last rounding, half the rounding
 * of a y stays (measured over every exponent: 0.79 ulp at most, the root 0.72). */
__device__ __forceinline__ double gf_rsqrt_n(double a)
{
    const double y = gf_rsqrt_seed(a);
    const double e = fma(-(a * y), y, 1.0);
    return fma(y * e, fma(0.375, e, 0.5), y);
}
__device__ __forceinline__ double gf_sqrt_n(double a)
{
    const double y = gf_rsqrt_seed(a);
    const double t = a * y;
    const double e = fma(-t, y, 1.0);
    return fma(t * e, fma(0.375, e, 0.5), t);
}

/* Single-precision value of x, cut to its leading bits on the integer pipe
 * (a conversion instruction runs at the FP64 pipe's rate): below the normal
 * range zero, above it infinity. And a normal float as a double. */
__device__ __forceinline__ float gf_f32(double x)
{
    const unsigned hi = static_cast<unsigned>(__double2hiint(x)), lo = static_cast<unsigned>(__double2loint(x));
    const unsigned a = hi & 0x7fffffffu;
    unsigned r = __funnelshift_l(lo, a - 0x38000000u, 3);
    r = a < 0x38100000u ? 0u : a >= 0x47f00000u ? 0x7f800000u : r;
    return __uint_as_float(r | (hi & 0x80000000u));
}
__device__ __forceinline__ double gf_f64_pos(float x)
{
    const unsigned u = __float_as_uint(x);
    return __hiloint2double(static_cast<int>((u >> 3) + 0x38000000u), static_cast<int>(u << 29));
}

/* Products and sums of the contracted build that are written as the operation
 * they become: the compiler fuses none of them, so every kernel instantiated
 * from one source gives the same bits. */
__device__ __forceinline__ double gf_mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double gf_add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double gf_sub(double a, double b) { return __dadd_rn(a, -b); }

/* x / y: the IEEE quotient, or x * gf_rcp(y) in the production build */
template <bool F> __device__ __forceinline__ double d_div(double x, double y)
{
    if (F) return gf_mul(x, gf_rcp(y));
    return x / y;
}

#endif
