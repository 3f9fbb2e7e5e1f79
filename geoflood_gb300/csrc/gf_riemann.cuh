/*
 * Face-level shallow-water Riemann solvers, FP64, device side.
 *
 * Restates the reference's GeoClaw solvers for one face at a time:
 *   - normal solve: rpn2_geoclaw.f:84-330 with riemann_aug_JCP
 *     (geoclaw_riemann_utils.f:2-311, maxiter = 1) and riemanntype
 *     (geoclaw_riemann_utils.f:566-677);
 *   - transverse split: rpt2_geoclaw.f:61-187.
 *
 * Inputs per cell come pre-digested from shared memory (gf_cell): the
 * quotients hu/h, hv/h and sqrt(g h) are computed once per cell instead of
 * once per face side. Each is the same IEEE operation the Fortran performs,
 * so the values are identical. Cramer's rule in riemann_aug_JCP is written
 * out for the fixed eigenvector pattern r(:,2) = (0,0,1), r(1,:) = 1, which
 * removes multiplications by exact 0 and 1 only.
 *
 * Component order inside these routines is LOCAL: 0 = depth, 1 = momentum
 * normal to the face, 2 = momentum along the face.
 */
#ifndef GF_RIEMANN_CUH
#define GF_RIEMANN_CUH

#include "gf_types.h"
#include "gf_cmp.cuh"

struct gf_cell {
    double h;    /* depth after b4step2                         */
    double hun;  /* momentum normal to the face                 */
    double hut;  /* momentum along the face                     */
    double un;   /* hun/h if wet else 0                         */
    double ut;   /* hut/h if wet else 0                         */
    double c;    /* sqrt(g h) if wet else 0                     */
    double b;    /* bathymetry                                  */
    double rc;   /* 1/sqrt(g h) if wet (contracted build only)  */
    bool wet;    /* h > dry_tolerance                           */
};

/* sqrt(a): the IEEE root, or, in the contracted build and for positive
 * normal a, the approximate root refined (within an ulp or two, fewer FP64
 * instructions; zeros are their own root, the rest keeps the IEEE root: one
 * integer test on the bit pattern decides) */
template <bool FAST>
__device__ __forceinline__ double d_sqrt(double a)
{
    if (FAST) {
        if (gf_pos_normal(a)) return gf_sqrt_n(a);
        if (d_eqz<FAST>(a)) return a;
    }
    return sqrt(a);
}

/* a * b < 0 for nonzero finite factors, from the sign bits on the integer
 * pipe (a product that underflows to zero aside) */
__device__ __forceinline__ bool opposite_signs(double a, double b)
{
    const unsigned long long ia = static_cast<unsigned long long>(__double_as_longlong(a));
    const unsigned long long ib = static_cast<unsigned long long>(__double_as_longlong(b));
    return ((ia ^ ib) >> 63) != 0 && (ia << 1) != 0 && (ib << 1) != 0;
}

/* riemanntype (geoclaw_riemann_utils.f:566-677), maxiter = 1.
 * cL = sqrt(g hL), cR = sqrt(g hR) are supplied by the caller (they equal
 * the Fortran's sqrt(g*hL), sqrt(g*hR) bit for bit). Returns hm, s1m, s2m. */
template <bool FAST>
__device__ __forceinline__ void gf_riemanntype(double hL, double hR, double uL,
                                               double uR, double cL, double cR,
                                               double rhL, double rhR,
                                               double g, double drytol,
                                               double c16g, double rsg, double& hm,
                                               double& s1m, double& s2m)
{
    const double h_min = d_min<FAST>(hR, hL);
    const double h_max = d_max<FAST>(hR, hL);
    const double delu = uR - uL;
    if (d_le<FAST>(h_min, drytol)) {
        hm = 0.0;
        s1m = uR + uL - 2.0 * cR + 2.0 * cL;
        s2m = s1m;
        return;
    }
    /* sqrt is monotone, so sqrt(g*h_min) = min(cL, cR). */
    const double c_min = d_min<FAST>(cR, cL);
    const double c_max = d_max<FAST>(cR, cL);
    const double F_min = delu + 2.0 * (c_min - c_max);
    /* (h_max + h_min)/(h_max h_min) = 1/h_min + 1/h_max: the contracted
     * build uses the per-cell reciprocals instead of a division. */
    double F_max = 0.0, q_fm = 0.0, s_fm = 0.0;
    if (!FAST) F_max = delu + (h_max - h_min) * sqrt(0.5 * g * (h_max + h_min) / (h_max * h_min));
    /* the contracted build forms F_max only where it is read (not for two
     * rarefactions), its root through rsqrt, whose value the two-shock step
     * reuses */
    auto f_max = [&]() {
        if (FAST) {
            const double a_fm = 0.5 * g * (d_max<FAST>(rhL, rhR) + d_min<FAST>(rhL, rhR));
            q_fm = rsqrt(a_fm);
            s_fm = a_fm * q_fm;
            F_max = delu + (h_max - h_min) * s_fm;
        }
    };
    if (d_gtz<FAST>(F_min)) { /* 2-rarefactions */
        const double t = d_max<FAST>(0.0, -delu + 2.0 * (cL + cR));
        hm = c16g * (t * t);
        /* sqrt(g hm) = t / 4 up to rounding: the contracted build takes it */
        const double cm = FAST ? 0.25 * t : sqrt(g * hm);
        s1m = uL + 2.0 * cL - 3.0 * cm;
        s2m = uR - 2.0 * cR + 3.0 * cm;
    } else if ((f_max(), d_lez<FAST>(F_max))) { /* 2 shocks, one Newton step on sqrt(h) */
        const double h0 = h_max;
        double gL, gR, dfdh, sh0, rL, rR;
        if (FAST) {
            rL = rhL;
            rR = rhR;
            /* h0 = h_max: the deeper side's root is sqrt(g / h_max) = c_max / h_max
             * and its (h0 - h) terms vanish; the shallower side's root is
             * F_max's, sqrt(g (1/h_min + 1/h_max) / 2) */
            const double r0 = d_min<FAST>(rhL, rhR); /* 1/h_max */
            const double gmx = d_max<FAST>(cL, cR) * r0;
            const bool lmax = d_ge<FAST>(hL, hR);
            gL = lmax ? gmx : s_fm;
            gR = lmax ? s_fm : gmx;
            const double w = 0.25 * (r0 * r0) * g;
            dfdh = gmx + s_fm - (h0 - h_min) * w * q_fm;
            sh0 = d_max<FAST>(cL, cR) * rsg; /* sqrt(h_max) = sqrt(g h_max)/sqrt(g) */
        } else {
            rL = 1.0 / hL;
            rR = 1.0 / hR;
            const double r0 = 1.0 / h0; /* equals rL or rR */
            gL = sqrt(0.5 * g * (r0 + rL));
            gR = sqrt(0.5 * g * (r0 + rR));
            dfdh = gL - g * (h0 - hL) / (4.0 * (h0 * h0) * gL) + gR -
                   g * (h0 - hR) / (4.0 * (h0 * h0) * gR);
            sh0 = sqrt(h0);
        }
        const double F0 = delu + (h0 - hL) * gL + (h0 - hR) * gR;
        const double slope = 2.0 * sh0 * dfdh;
        const double t = sh0 - d_div<FAST>(F0, slope);
        hm = t * t;
        const double rm = d_div<FAST>(1.0, hm);
        const double u1m = uL - (hm - hL) * d_sqrt<FAST>((0.5 * g) * (rm + rL));
        const double u2m = uR + (hm - hR) * d_sqrt<FAST>((0.5 * g) * (rm + rR));
        /* hm = t^2: sqrt(g hm) = sqrt(g) |t| up to rounding in the contracted build */
        const double cm = FAST ? (g * rsg) * fabs(t) : sqrt(g * hm);
        s1m = u1m - cm;
        s2m = u2m + cm;
    } else { /* one shock, one rarefaction, one secant step.
                The first F0 has (h0 - h_min) = 0, so F0 = F_min exactly. */
        const double F0 = F_min;
        if (FAST) {
            hm = h_min - F0 * d_div<FAST>(h_max - h_min, F_max - F0);
        } else {
            const double slope = (F_max - F0) / (h_max - h_min);
            hm = h_min - F0 / slope;
        }
        const double cm = d_sqrt<FAST>(g * hm);
        if (d_gt<FAST>(hL, hR)) {
            s1m = uL + 2.0 * cL - 3.0 * cm;
            s2m = uL + 2.0 * cL - cm;
        } else {
            s2m = uR - 2.0 * cR + 3.0 * cm;
            s1m = uR - 2.0 * cR + cm;
        }
    }
}

/* Normal Riemann problem at one face: rpn2_geoclaw.f:110-315 + aug_JCP.
 * Outputs speeds s[3] and f-waves fw[mw][m] (LOCAL component order). */
template <bool FAST>
__device__ __forceinline__ void gf_rpn2_face(const gf_cell& Lc, const gf_cell& Rc,
                                             double g, double drytol,
                                             double c16g, double rsg, double crit,
                                             double crit2, double s[3],
                                             double fw[3][3])
{
    /* Riemann problem variables (rpn2_geoclaw.f:136-171). */
    double hL, huL, hvL, uL, vL, phiL, cL, rhL = 0.0; /* rhL, rhR: 1/h, contracted build */
    double hR, huR, hvR, uR, vR, phiR, cR, rhR = 0.0;
    double bL = Lc.b, bR = Rc.b;
    if (Rc.wet) {
        hR = Rc.h; huR = Rc.hun; hvR = Rc.hut; uR = Rc.un; vR = Rc.ut; cR = Rc.c;
        if (FAST) rhR = g * (Rc.rc * Rc.rc);
        /* hu^2/h = hu u: the contracted build reuses the cell quotient */
        phiR = FAST ? 0.0 : 0.5 * g * (hR * hR) + (huR * huR) / hR; /* contracted: delphi below */
    } else {
        hR = 0.0; huR = 0.0; hvR = 0.0; uR = 0.0; vR = 0.0; phiR = 0.0; cR = 0.0;
    }
    if (Lc.wet) {
        hL = Lc.h; huL = Lc.hun; hvL = Lc.hut; uL = Lc.un; vL = Lc.ut; cL = Lc.c;
        if (FAST) rhL = g * (Lc.rc * Lc.rc);
        phiL = FAST ? 0.0 : 0.5 * g * (hL * hL) + (huL * huL) / hL;
    } else {
        hL = 0.0; huL = 0.0; hvL = 0.0; uL = 0.0; vL = 0.0; phiL = 0.0; cL = 0.0;
    }
    (void)hvL; (void)hvR;

    /* Wet/dry interface: wall or overtopping (rpn2_geoclaw.f:185-242). */
    double wall0 = 1.0, wall1 = 1.0, wall2 = 1.0;
    if (!Rc.wet) {
        double hstar, s1x, s2x;
        gf_riemanntype<FAST>(hL, hL, uL, -uL, cL, cL, rhL, rhL, g, drytol, c16g, rsg, hstar, s1x, s2x);
        const double hstartest = d_max<FAST>(hL, hstar);
        if (d_lt<FAST>(hstartest + bL, bR)) {
            wall1 = 0.0; wall2 = 0.0;
            hR = hL; huR = -huL; bR = bL; phiR = phiL; uR = -uL; vR = vL; cR = cL; rhR = rhL;
        } else if (d_lt<FAST>(hL + bL, bR)) {
            bR = hL + bL;
        }
    } else if (!Lc.wet) {
        double hstar, s1x, s2x;
        gf_riemanntype<FAST>(hR, hR, -uR, uR, cR, cR, rhR, rhR, g, drytol, c16g, rsg, hstar, s1x, s2x);
        const double hstartest = d_max<FAST>(hR, hstar);
        if (d_lt<FAST>(hstartest + bR, bL)) {
            wall0 = 0.0; wall1 = 0.0;
            hL = hR; huL = -huR; bL = bR; phiL = phiR; uL = -uR; vL = vR; cL = cR; rhL = rhR;
        } else if (d_lt<FAST>(hR + bR, bL)) {
            bL = hR + bR;
        }
    }

    /* Einfeldt / Roe speeds (rpn2_geoclaw.f:257-266). */
    const double sL = uL - cL;
    const double sR = uR + cR;
    const double uhat = d_div<FAST>(cL * uL + cR * uR, cR + cL);
    /* hbar of the steady-state wave below; g (hL + hR) / 2 = g hbar for the
     * non-negative depths here, so the contracted build shares the product */
    const double hbar = d_max<FAST>(0.5 * (hL + hR), 0.0);
    const double chat = FAST ? d_sqrt<FAST>(g * hbar) : d_sqrt<FAST>(g * 0.5 * (hR + hL));
    double sE1 = d_min<FAST>(sL, uhat - chat);
    double sE2 = d_max<FAST>(sR, uhat + chat);

    /* ---- riemann_aug_JCP (geoclaw_riemann_utils.f:57-306) ---- */
    const double delh = hR - hL;
    const double delhu = huR - huL;
    /* phi = g h^2 / 2 + hu^2 / h: the contracted build forms the jump as
     * (g / 2) (hR - hL) (hR + hL) + (huR uR - huL uL), with hu^2 / h = hu u;
     * both products rounded, so a mirrored wall state gives exactly zero */
    const double delphi = FAST ? fma((0.5 * g) * delh, hR + hL, __dmul_rn(huR, uR) - __dmul_rn(huL, uL))
                               : phiR - phiL;
    const double delb = bR - bL;

    double hm, s1m, s2m;
    gf_riemanntype<FAST>(hL, hR, uL, uR, cL, cR, rhL, rhR, g, drytol, c16g, rsg, hm, s1m, s2m);
    (void)hm;

    const double l1 = d_min<FAST>(sE1, s2m);
    const double l3 = d_max<FAST>(sE2, s1m);
    sE1 = l1;
    sE2 = l3;
    /* One reciprocal serves h*_HLL and Cramer's rule in the contracted
     * build: sE2 - sE1 = l3 - l1 = -(l1 - l3). */
    const double rdet = FAST ? gf_rcp(l1 - l3) : 0.0;
    /* h*_HLL (sE2 - sE1) enters only as hsd: the contracted build takes it as
     * max(numerator, 0) (sE2 - sE1 = l3 - l1 > 0 for a wet face) */
    const double hll_num = huL - huR + sE2 * hR - sE1 * hL;
    const double hstarHLL = FAST ? 0.0 : fmax(hll_num / (sE2 - sE1), 0.0);
    const double l2 = 0.5 * (l1 + l3);

    /* steady-state wave, first (only) iteration: hLstar = hL etc. */
    const double s1s2bar = FAST ? fma(0.25 * (uL + uR), uL + uR, -(g * hbar))
                                : 0.25 * ((uL + uR) * (uL + uR)) - g * hbar;
    const double s1s2tilde = d_max<FAST>(0.0, uL * uR) - g * hbar;
    const double crit_sq = crit * crit;
    bool sonic;
    if (d_le<FAST>(fabs(s1s2bar), crit)) sonic = true;
    else if (d_le<FAST>(s1s2bar * s1s2tilde, crit_sq)) sonic = true;
    else if (d_le<FAST>(s1s2bar * sE1 * sE2, crit_sq)) sonic = true;
    else if (d_lt<FAST>(d_min<FAST>(fabs(sE1), fabs(sE2)), crit2)) sonic = true;
    else if (d_lt<FAST>(sE1, crit2) && d_gt<FAST>(s1m, -crit2)) sonic = true;
    else if (d_gt<FAST>(sE2, -crit2) && d_lt<FAST>(s2m, crit2)) sonic = true;
    else if (FAST ? opposite_signs(uL + cL, uR + cR) : d_ltz<FAST>((uL + cL) * (uR + cR))) sonic = true;
    else if (FAST ? opposite_signs(uL - cL, uR - cR) : d_ltz<FAST>((uL - cL) * (uR - cR))) sonic = true;
    else sonic = false;

    const double rs12 = (FAST && !sonic) ? gf_rcp(s1s2bar) : 0.0;
    /* contracted build: g hbar delb once; deldelphi below is -(g hbar delb /
     * s1s2bar) s1s2tilde, i.e. the unclamped deldelh times -s1s2tilde */
    const double ghd = FAST ? (g * hbar) * delb : 0.0;
    double deldelh = sonic ? -delb : (FAST ? ghd * rs12 : delb * g * hbar / s1s2bar);
    const double deldelh0 = deldelh;
    const double hsd = FAST ? d_max<FAST>(hll_num, 0.0) : hstarHLL * (sE2 - sE1);
    if (FAST) {
        /* The bounds hsd / sE clamp rarely: compare hsd with deldelh * sE (the
         * sign of sE is known in each branch) and divide only to clamp. */
        if (d_lt<FAST>(sE1, -crit) && d_gt<FAST>(sE2, crit)) {
            if (d_lt<FAST>(hsd, deldelh * sE2)) deldelh = d_div<FAST>(hsd, sE2); /* min, sE2 > 0 */
            if (d_lt<FAST>(hsd, deldelh * sE1)) deldelh = d_div<FAST>(hsd, sE1); /* max, sE1 < 0 */
        } else if (d_ge<FAST>(sE1, crit)) {
            if (d_lt<FAST>(hsd, deldelh * sE1)) deldelh = d_div<FAST>(hsd, sE1); /* min, sE1 > 0 */
            deldelh = d_max<FAST>(deldelh, -hL);
        } else if (d_le<FAST>(sE2, -crit)) {
            deldelh = d_min<FAST>(deldelh, hR);
            if (d_lt<FAST>(hsd, deldelh * sE2)) deldelh = d_div<FAST>(hsd, sE2); /* max, sE2 < 0 */
        }
    } else if (d_lt<FAST>(sE1, -crit) && d_gt<FAST>(sE2, crit)) {
        deldelh = d_min<FAST>(deldelh, d_div<FAST>(hsd, sE2));
        deldelh = d_max<FAST>(deldelh, d_div<FAST>(hsd, sE1));
    } else if (d_ge<FAST>(sE1, crit)) {
        deldelh = d_min<FAST>(deldelh, d_div<FAST>(hsd, sE1));
        deldelh = d_max<FAST>(deldelh, -hL);
    } else if (d_le<FAST>(sE2, -crit)) {
        deldelh = d_min<FAST>(deldelh, hR);
        deldelh = d_max<FAST>(deldelh, d_div<FAST>(hsd, sE2));
    }
    double deldelphi;
    if (FAST) {
        deldelphi = sonic ? -ghd : -deldelh0 * s1s2tilde;
        /* g max(-hL delb, -hR delb) = -g delb h_lo and g min(..) = -g delb h_hi,
         * with h_lo the smaller depth when delb > 0 (the larger otherwise) */
        const double mgd = -g * delb;
        const bool pos = d_gtz<FAST>(delb);
        const double hmn = d_min<FAST>(hL, hR), hmx = d_max<FAST>(hL, hR);
        deldelphi = d_min<FAST>(deldelphi, mgd * (pos ? hmn : hmx));
        deldelphi = d_max<FAST>(deldelphi, mgd * (pos ? hmx : hmn));
    } else {
        deldelphi = sonic ? -g * hbar * delb : -delb * g * hbar * s1s2tilde / s1s2bar;
        deldelphi = d_min<FAST>(deldelphi, g * d_max<FAST>(-hL * delb, -hR * delb));
        deldelphi = d_max<FAST>(deldelphi, g * d_min<FAST>(-hL * delb, -hR * delb));
    }

    const double d1 = delh - deldelh;
    const double d2 = delhu;
    const double d3 = delphi - deldelphi;

    /* Cramer's rule with r(:,1) = (1,l1,l1^2), r(:,2) = (0,0,1),
     * r(:,3) = (1,l3,l3^2): determinant = l1 - l3. */
    const double A2 = l1 * l1, C2 = l3 * l3;
    const double det = l1 - l3;
    /* n2 = (l1 - l3) (d3 + d1 l1 l3 - d2 (l1 + l3)): the contracted build
     * takes beta2 = n2 / det as that bracket, without the division */
    const double beta1 = FAST ? (d2 - d1 * l3) * rdet : (d2 - d1 * l3) / det;
    double beta2;
    if (FAST) {
        beta2 = fma(-d2, l1 + l3, fma(d1, l1 * l3, d3));
    } else {
        const double n2 = (d2 * C2 - l3 * d3) - d1 * (l1 * C2 - l3 * A2) + (l1 * d3 - d2 * A2);
        beta2 = n2 / det;
    }
    const double beta3 = FAST ? (d1 * l1 - d2) * rdet : (d1 * l1 - d2) / det;

    /* f-waves (geoclaw_riemann_utils.f:289-306). */
    /* contracted build: l^2 beta = (beta l) l, no squares */
    double f11 = beta1 * l1, f21 = FAST ? f11 * l1 : beta1 * A2, f31 = beta1 * l1 * vL;
    double f13 = beta3 * l3, f23 = FAST ? f13 * l3 : beta3 * C2, f33 = beta3 * l3 * vR;
    /* h u v: the contracted build takes hu v (hu = h u up to rounding) */
    const double corr = FAST ? (huR * vR - huL * vL - f31 - f33) : (hR * uR * vR - hL * uL * vL - f31 - f33);
    if (d_lez<FAST>(huL + f11)) f31 = f31 + corr;
    else f33 = f33 + corr;

    /* Wall masking (rpn2_geoclaw.f:303-309). Without a wall every mask is 1
     * and the products are the values themselves. */
    if (FAST && Lc.wet && Rc.wet) {
        s[0] = l1; s[1] = l2; s[2] = l3;
        fw[0][0] = f11; fw[0][1] = f21; fw[0][2] = f31;
        fw[1][0] = 0.0; fw[1][1] = beta2; fw[1][2] = 0.0;
        fw[2][0] = f13; fw[2][1] = f23; fw[2][2] = f33;
        return;
    }
    s[0] = l1 * wall0; s[1] = l2 * wall1; s[2] = l3 * wall2;
    fw[0][0] = f11 * wall0; fw[0][1] = f21 * wall0; fw[0][2] = f31 * wall0;
    fw[1][0] = 0.0 * wall1; fw[1][1] = beta2 * wall1; fw[1][2] = 0.0 * wall1;
    fw[2][0] = f13 * wall2; fw[2][1] = f23 * wall2; fw[2][2] = f33 * wall2;
}

/* Single-precision products, fused sums, quotients and roots written as the
 * operation they become, as gf_mul above: a face has the same class in every
 * kernel. A host build (tests) brings its own root and __fdividef. */
#ifndef GF_HOST_MATH
__device__ __forceinline__ float gf_sqrtf(float x)
{
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float gf_fmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float gf_ffma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float gf_fdiv(float a, float b)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(b));
    return __fmul_rn(a, r);
}
#else
__device__ __forceinline__ float gf_fmul(float a, float b)
{
    volatile float r = a * b;
    return r;
}
__device__ __forceinline__ float gf_ffma(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ float gf_fdiv(float a, float b)
{
    volatile float r = __fdividef(a, b);
    return r;
}
#endif

/* Class of a face with water (contracted build), decided in single precision:
 *   0 smooth: both cells wet, the Einfeldt speeds are the outer speeds (the
 *     middle-state speeds s1m, s2m of riemanntype neither the largest nor the
 *     smallest), no sonic point, the steady-state jump of h inside its bounds:
 *     gf_rpn2_smooth;
 *   1 edge: gf_rpn2_edge with flag 0; 2 edge with flag 1 (both wet: a sonic
 *     point by the middle-state speeds; one wet: a wall at the dry side);
 *   3 none of these for certain: gf_rpn2_face.
 * A class is given only with room for every rounding of its tests, so the
 * short solves return the full solve's values. The FP64 pipe takes two lanes
 * a clock (an FP64 instruction occupies its scheduler's pipe for 64 cycles)
 * and the single-precision pipes 128 lanes, which otherwise idle: the tests
 * cost about a fiftieth of the FP64 instructions they save, and a warp that
 * holds a shore face no longer runs both calls of riemanntype with all their
 * branches (375 FP64 instructions against 90 for smooth faces). Margins are at
 * least ten times the tests' rounding (inputs cut to 23 bits, approximate
 * roots and quotients); infinities and NaN fail the comparisons and end in
 * class 3. */
__device__ __forceinline__ int gf_face_class(float hL, float hR, float uL, float uR, float cL, float cR, float bL,
                                             float bR, bool wetL, bool wetR, float g, float crit, float crit2)
{
    const float S = fabsf(uL) + fabsf(uR) + cL + cR;
    if (wetL != wetR) {
        /* mirrored at the dry side, riemanntype's depth is (c + u/2)^2 / g in
         * both its branches (u towards the dry side, 0 below -2 c), and its
         * speeds lie 2 c inside the Einfeldt speeds */
        const float h = wetL ? hL : hR, u = wetL ? uL : -uR, c = wetL ? cL : cR;
        const float bw = wetL ? bL : bR, bd = wetL ? bR : bL;
        const float r = fmaxf(gf_ffma(0.5f, u, c), 0.0f);
        const float top = fmaxf(h, gf_fdiv(gf_fmul(r, r), g));
        const float gap = bd - (top + bw);
        const float e = gf_ffma(1.0e-5f, top, gf_fmul(1.0e-6f, fabsf(bw) + fabsf(bd)));
        const bool ok = (h > 1.0e-15f) & (h < 1.0e15f) & (S < 1.0e15f);
        return ok & (gap > e) ? 2 : ok & (gap < -e) ? 1 : 3;
    }
    const float ghb = gf_fmul(gf_fmul(0.5f, g), hL + hR);
    const float uhat = gf_fdiv(gf_ffma(cL, uL, gf_fmul(cR, uR)), cL + cR);
    const float chat = gf_sqrtf(ghb);
    const float l1 = fminf(uL - cL, uhat - chat), l3 = fmaxf(uR + cR, uhat + chat);
    /* middle-state speeds: the formulas of gf_riemanntype for two
     * rarefactions and for a shock and a rarefaction; for two shocks
     * (hm >= hmax there) an upper bound of s1m and a lower bound of s2m. No
     * branches: a warp holds all three. */
    const float hmin = fminf(hL, hR), hmax = fmaxf(hL, hR), dh = hmax - hmin;
    const float cmin = fminf(cL, cR), cmax = fmaxf(cL, cR);
    const float delu = uR - uL;
    const float Fmin = gf_ffma(2.0f, cmin - cmax, delu);
    const float dhs = gf_fmul(dh, gf_sqrtf(gf_fdiv(ghb, gf_fmul(hL, hR)))); /* dh sqrt(g (1/hL + 1/hR) / 2) */
    const float Fmax = delu + dhs;
    const float hm = fminf(fmaxf(hmin - gf_fdiv(gf_fmul(Fmin, dh), Fmax - Fmin), hmin), hmax);
    const float cm = gf_sqrtf(gf_fmul(g, hm));
    const float c3 = gf_fmul(0.75f, fmaxf(0.0f, gf_ffma(2.0f, cL + cR, -delu)));
    const float wL = gf_ffma(2.0f, cL, uL), wR = gf_ffma(-2.0f, cR, uR);
    const bool left = hL > hR, rare = Fmin > 0.0f, shock = !rare & (Fmax <= 0.0f);
    const float s1m = rare    ? wL - c3
                      : shock ? (left ? uL : uL - dhs) - cmax
                              : (left ? gf_ffma(-3.0f, cm, wL) : wR + cm);
    const float s2m = rare    ? wR + c3
                      : shock ? (left ? uR + dhs : uR) + cmax
                              : (left ? wL - cm : gf_ffma(3.0f, cm, wR));
    const float em = gf_fmul(1.0e-4f, S + fabsf(s1m) + fabsf(s2m)), e = gf_fmul(1.0e-5f, S);
    const bool mid = (hmin > 1.0e-15f) & (hmax < 1.0e15f) & (S < 1.0e15f) & (s2m > l1 + em) & (s1m < l3 - em);
    /* the sonic tests with the middle-state speeds: clearly false, clearly
     * true (a bound of two shocks proves no truth) */
    const bool no1 = (l1 > crit2 + e) | (s1m < -crit2 - em), no2 = (l3 < -crit2 - e) | (s2m > crit2 + em);
    const bool yes = !shock & (((l1 < crit2 - e) & (s1m > -crit2 + em)) | ((l3 > -crit2 + e) & (s2m < crit2 - em)));
    /* the other sonic tests clearly false */
    const float us = uL + uR, uu = gf_fmul(uL, uR), us4 = gf_fmul(0.25f, us), cc = gf_fmul(crit, crit);
    const float sb = gf_ffma(us4, us, -ghb), st = fmaxf(0.0f, uu) - ghb;
    const float A = gf_ffma(us4, us, ghb), B = fabsf(uu) + ghb, ab = fabsf(sb), A4 = gf_fmul(1.0e-4f, A);
    bool ok = no1 & no2 & (ab > gf_ffma(1.0e-3f, A, crit));
    ok = ok & (gf_fmul(sb, st) > gf_ffma(A4, B, cc));
    ok = ok & (gf_fmul(gf_fmul(sb, l1), l3) > gf_ffma(gf_fmul(A4, S), S, cc));
    ok = ok & (fminf(fabsf(l1), fabsf(l3)) > crit2 + e);
    const float pL = uL + cL, pR = uR + cR, mL = uL - cL, mR = uR - cR;
    ok = ok & ((fminf(pL, pR) > e) | (fmaxf(pL, pR) < -e));
    ok = ok & ((fminf(mL, mR) > e) | (fmaxf(mL, mR) < -e));
    /* the jump of h within hsd / l1, hsd / l3 (or -hL, hR) */
    const float rsb = gf_fdiv(ghb, sb);
    const float dd = gf_fmul(bR - bL, rsb);
    const float de = gf_ffma(0.02f, fabsf(dd), gf_fmul(gf_fmul(1.0e-5f, fabsf(bL) + fabsf(bR)), fabsf(rsb)));
    const float num = gf_ffma(hL, uL - l1, gf_fmul(hR, l3 - uR));
    const float en = gf_fmul(1.0e-5f, gf_ffma(hL, fabsf(uL) + fabsf(l1), gf_fmul(hR, fabsf(uR) + fabsf(l3))));
    const bool t1 = gf_ffma(-fabsf(l1), de, gf_ffma(-dd, l1, num)) > en;
    const bool t3 = gf_ffma(-fabsf(l3), de, gf_ffma(-dd, l3, num)) > en;
    const bool sub = (l1 < -crit - e) & (l3 > crit + e), right = l1 > crit + e, leftw = l3 < -crit - e;
    ok = ok & (num > en) & (sub | right | leftw);
    ok = ok & (t1 | !(sub | right)) & (t3 | !(sub | leftw));
    ok = ok & ((dd - de > gf_fmul(-0.999f, hL)) | !right) & ((dd + de < gf_fmul(0.999f, hR)) | !leftw);
    return !mid ? 3 : ok ? 0 : yes ? 2 : no1 & no2 ? 1 : 3;
}

/* The parts that gf_rpn2_smooth and gf_rpn2_edge share. A smooth face may be
 * solved by either (which one depends on the faces listed beside it): with
 * every operation spelled out both give the same bits. */
/* Roe mean speed uhat; sum of the depths hs and gh = g hs / 2 */
__device__ __forceinline__ void gf_roe(double hL, double hR, double uL, double uR, double cL, double cR, double g,
                                       double& uhat, double& hs, double& gh)
{
    uhat = gf_mul(fma(cL, uL, gf_mul(cR, uR)), gf_rcp(gf_add(cR, cL)));
    hs = gf_add(hL, hR);
    gh = gf_mul(0.5 * g, hs);
}
__device__ __forceinline__ double gf_s1s2bar(double uL, double uR, double gh)
{
    const double us = gf_add(uL, uR);
    return fma(gf_mul(0.25, us), us, -gh);
}
__device__ __forceinline__ double gf_s1s2tilde(double uL, double uR, double gh)
{
    return gf_sub(d_max<true>(0.0, gf_mul(uL, uR)), gh);
}

/* From the outer speeds and the steady-state jumps to speeds and f-waves. */
__device__ __forceinline__ void gf_waves(double hL, double hR, double huL, double huR, double uL, double uR,
                                         double vL, double vR, double delb, double hs, double l1, double l3,
                                         double deldelh, double deldelphi, double g, double s[3], double fw[3][3])
{
    constexpr bool F = true;
    const double delh = gf_sub(hR, hL), d2 = gf_sub(huR, huL);
    const double delphi = fma(gf_mul(0.5 * g, delh), hs, gf_sub(gf_mul(huR, uR), gf_mul(huL, uL)));
    const double rdet = gf_rcp(gf_sub(l1, l3));
    const double mgd = gf_mul(-g, delb);
    const bool pos = d_gtz<F>(delb);
    const double hmn = d_min<F>(hL, hR), hmx = d_max<F>(hL, hR);
    deldelphi = d_min<F>(deldelphi, gf_mul(mgd, pos ? hmn : hmx));
    deldelphi = d_max<F>(deldelphi, gf_mul(mgd, pos ? hmx : hmn));
    const double d1 = gf_sub(delh, deldelh), d3 = gf_sub(delphi, deldelphi);
    const double beta1 = gf_mul(fma(-d1, l3, d2), rdet), beta3 = gf_mul(fma(d1, l1, -d2), rdet);
    const double f11 = gf_mul(beta1, l1), f13 = gf_mul(beta3, l3);
    double f31 = gf_mul(f11, vL), f33 = gf_mul(f13, vR);
    /* the correction goes to the wave on the side the interface moves to */
    const bool left = d_lez<F>(gf_add(huL, f11));
    const double corr = gf_sub(gf_sub(fma(huR, vR, -gf_mul(huL, vL)), f31), f33);
    const double upd = gf_add(left ? f31 : f33, corr);
    f31 = left ? upd : f31;
    f33 = left ? f33 : upd;
    const double ls = gf_add(l1, l3);
    s[0] = l1; s[1] = gf_mul(0.5, ls); s[2] = l3;
    fw[0][0] = f11; fw[0][1] = gf_mul(f11, l1); fw[0][2] = f31;
    fw[1][0] = 0.0; fw[1][1] = fma(-d2, ls, fma(d1, gf_mul(l1, l3), d3)); fw[1][2] = 0.0;
    fw[2][0] = f13; fw[2][1] = gf_mul(f13, l3); fw[2][2] = f33;
}

/* gf_rpn2_face<true> at a face of class 0 (gf_face_class). */
__device__ __forceinline__ void gf_rpn2_smooth(const gf_cell& Lc, const gf_cell& Rc, double g, double s[3],
                                               double fw[3][3])
{
    constexpr bool F = true;
    double uhat, hs, gh;
    gf_roe(Lc.h, Rc.h, Lc.un, Rc.un, Lc.c, Rc.c, g, uhat, hs, gh);
    const double chat = gf_sqrt_n(gh);
    const double l1 = d_min<F>(gf_sub(Lc.un, Lc.c), gf_sub(uhat, chat));
    const double l3 = d_max<F>(gf_add(Rc.un, Rc.c), gf_add(uhat, chat));
    const double delb = gf_sub(Rc.b, Lc.b);
    const double deldelh = gf_mul(gf_mul(gh, delb), gf_rcp(gf_s1s2bar(Lc.un, Rc.un, gh)));
    const double deldelphi = gf_mul(-deldelh, gf_s1s2tilde(Lc.un, Rc.un, gh));
    gf_waves(Lc.h, Rc.h, Lc.hun, Rc.hun, Lc.un, Rc.un, Lc.ut, Rc.ut, delb, hs, l1, l3, deldelh, deldelphi, g, s, fw);
}

/* gf_rpn2_face<true> at a face of class 0, 1 (flag false) or 2 (flag true):
 * the speeds of riemanntype are those of a dry side, uL + 2 cL or uR - 2 cR,
 * or do not matter, and the wall test is decided. */
__device__ __forceinline__ void gf_rpn2_edge(const gf_cell& Lc, const gf_cell& Rc, bool flag, double g, double crit,
                                             double crit2, double s[3], double fw[3][3])
{
    constexpr bool F = true;
    const bool one = Lc.wet != Rc.wet, wall = one && flag;
    const bool wl = Lc.wet, wr = Rc.wet;
    /* a dry cell's u, v and c are zero; its h and momenta are not read */
    double hL = wl ? Lc.h : 0.0, huL = wl ? Lc.hun : 0.0, uL = Lc.un, vL = Lc.ut, cL = Lc.c, bL = Lc.b;
    double hR = wr ? Rc.h : 0.0, huR = wr ? Rc.hun : 0.0, uR = Rc.un, vR = Rc.ut, cR = Rc.c, bR = Rc.b;
    if (one) {
        const double top = wl ? gf_add(hL, bL) : gf_add(hR, bR);
        if (!wr) {
            if (wall) { hR = hL; huR = -huL; bR = bL; uR = -uL; vR = vL; cR = cL; }
            else if (d_lt<F>(top, bR)) bR = top;
        } else {
            if (wall) { hL = hR; huL = -huR; bL = bR; uL = -uR; vL = vR; cL = cR; }
            else if (d_lt<F>(top, bL)) bL = top;
        }
    }
    double uhat, hs, gh;
    gf_roe(hL, hR, uL, uR, cL, cR, g, uhat, hs, gh);
    const double chat = d_sqrt<F>(gh);
    const double mL = gf_sub(uL, cL), pR = gf_add(uR, cR);
    double l1 = d_min<F>(mL, gf_sub(uhat, chat));
    double l3 = d_max<F>(pR, gf_add(uhat, chat));
    bool sonic = flag && !one;
    if (one && !wall) {
        const double sm = fma(2.0, cL, fma(-2.0, cR, gf_add(uR, uL)));
        l1 = d_min<F>(l1, sm);
        l3 = d_max<F>(l3, sm);
        sonic = (d_lt<F>(l1, crit2) && d_gt<F>(sm, -crit2)) || (d_gt<F>(l3, -crit2) && d_lt<F>(sm, crit2));
    }
    const double delb = gf_sub(bR, bL);
    const double hsd = d_max<F>(fma(-l1, hL, fma(l3, hR, gf_sub(huL, huR))), 0.0);
    const double s1s2bar = gf_s1s2bar(uL, uR, gh), s1s2tilde = gf_s1s2tilde(uL, uR, gh);
    const double crit_sq = gf_mul(crit, crit);
    sonic = sonic || d_le<F>(fabs(s1s2bar), crit) || d_le<F>(gf_mul(s1s2bar, s1s2tilde), crit_sq) ||
            d_le<F>(gf_mul(gf_mul(s1s2bar, l1), l3), crit_sq) || d_lt<F>(d_min<F>(fabs(l1), fabs(l3)), crit2) ||
            opposite_signs(gf_add(uL, cL), pR) || opposite_signs(mL, gf_sub(uR, cR));
    const double ghd = gf_mul(gh, delb);
    double deldelh = sonic ? -delb : gf_mul(ghd, gf_rcp(s1s2bar));
    const double deldelphi = sonic ? -ghd : gf_mul(-deldelh, s1s2tilde);
    /* the bounds of deldelh: the one quotient that can bind */
    const bool right = d_ge<F>(l1, crit), left = d_le<F>(l3, -crit);
    if ((d_lt<F>(l1, -crit) && d_gt<F>(l3, crit)) || right || left) {
        if (left) deldelh = d_min<F>(deldelh, hR);
        const double den = right ? l1 : left ? l3 : d_gtz<F>(deldelh) ? l3 : l1;
        if (d_lt<F>(hsd, gf_mul(deldelh, den))) deldelh = gf_mul(hsd, gf_rcp(den));
        if (right) deldelh = d_max<F>(deldelh, -hL);
    }
    gf_waves(hL, hR, huL, huR, uL, uR, vL, vR, delb, hs, l1, l3, deldelh, deldelphi, g, s, fw);
    /* waves behind a wall are dropped (rpn2_geoclaw.f:303-309) */
    if (wall) {
        const int k = wl ? 2 : 0; /* the dry side's outer wave */
        s[1] = 0.0; fw[1][1] = 0.0;
        s[0] = k == 0 ? 0.0 : s[0]; s[2] = k == 2 ? 0.0 : s[2];
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            fw[0][m] = k == 0 ? 0.0 : fw[0][m];
            fw[2][m] = k == 2 ? 0.0 : fw[2][m];
        }
    }
}

/* Transverse split of one fluctuation (rpt2_geoclaw.f:63-182), one face, in the
 * reference's expressions (exact build).
 * cell: the cell the fluctuation enters; topo_lo / topo_hi: bathymetry of
 * the transverse neighbours below / above it. asdq in LOCAL order (0 = h,
 * 1 = momentum normal to the face, 2 = momentum along the face; "along the
 * face" is the transverse sweep direction). Accumulates into bm / bp. */
__device__ __forceinline__ void gf_rpt2_face(const gf_cell& cl, double topo_lo,
                                             double topo_hi, double tol,
                                             const double asdq[3], double bm[3],
                                             double bp[3])
{
    bm[0] = bm[1] = bm[2] = 0.0;
    bp[0] = bp[1] = bp[2] = 0.0;
    if (d_le<false>(cl.h, tol)) return;
    const double eta = cl.h + cl.b;
    if (d_lt<false>(eta, d_min<false>(topo_lo, topo_hi))) return;
    const bool up_lo = d_ge<false>(eta, topo_lo), up_hi = d_ge<false>(eta, topo_hi);
    const double u = cl.un;  /* q(mu)/h */
    const double v = cl.ut;  /* q(mv)/h */
    const double s1 = v - cl.c;
    const double s2 = v;
    const double s3 = v + cl.c;
    const double delf1 = asdq[0], delf2 = asdq[1], delf3 = asdq[2];
    const double den = s3 - s1;
    const double beta1 = (s3 * delf1 - delf3) / den;
    const double beta2 = -u * delf1 + delf2;
    const double beta3 = (delf3 - s1 * delf1) / den;
    /* r(:,1) = (1, u, s1); r(:,2) = (0, 1, 0); r(:,3) = (1, u, s3). */
    if (d_ltz<false>(s1) && up_lo) {
        const double a = s1 * beta1;
        bm[0] += a; bm[1] += a * u; bm[2] += a * s1;
    } else if (d_gtz<false>(s1) && up_hi) {
        const double a = s1 * beta1;
        bp[0] += a; bp[1] += a * u; bp[2] += a * s1;
    }
    if (d_ltz<false>(s2) && up_lo) {
        bm[1] += s2 * beta2;
    } else if (d_gtz<false>(s2) && up_hi) {
        bp[1] += s2 * beta2;
    }
    if (d_ltz<false>(s3) && up_lo) {
        const double a = s3 * beta3;
        bm[0] += a; bm[1] += a * u; bm[2] += a * s3;
    } else if (d_gtz<false>(s3) && up_hi) {
        const double a = s3 * beta3;
        bp[0] += a; bp[1] += a * u; bp[2] += a * s3;
    }
}

/* gf_rpt2_face in the contracted build: every operation spelled out, the
 * first wave assigned, the two quotients by s3 - s1 = 2 sqrt(g h) products with
 * the cell's 1 / sqrt(g h). h > tol. */
__device__ __forceinline__ void gf_rpt2_fast(const gf_cell& cl, double topo_lo, double topo_hi, const double x[3],
                                             double bm[3], double bp[3])
{
    constexpr bool F = true;
    bm[0] = bm[1] = bm[2] = 0.0;
    bp[0] = bp[1] = bp[2] = 0.0;
    const double eta = gf_add(cl.h, cl.b);
    const bool up_lo = d_ge<F>(eta, topo_lo), up_hi = d_ge<F>(eta, topo_hi);
    if (!(up_lo || up_hi)) return;
    const double u = cl.un, s2 = cl.ut;
    const double s1 = gf_sub(s2, cl.c), s3 = gf_add(s2, cl.c);
    const double rden = gf_mul(0.5, cl.rc);
    const double a1 = gf_mul(s1, gf_mul(fma(s3, x[0], -x[2]), rden));
    const double a2 = gf_mul(s2, fma(-u, x[0], x[1]));
    const double a3 = gf_mul(s3, gf_mul(fma(-s1, x[0], x[2]), rden));
    if (d_ltz<F>(s1)) {
        if (up_lo) { bm[0] = a1; bm[1] = gf_mul(a1, u); bm[2] = gf_mul(a1, s1); }
    } else if (d_gtz<F>(s1) && up_hi) {
        bp[0] = a1; bp[1] = gf_mul(a1, u); bp[2] = gf_mul(a1, s1);
    }
    if (d_gtz<F>(s3)) {
        if (up_hi) {
            if (d_gtz<F>(s1)) { /* both outer waves up */
                bp[0] = gf_add(bp[0], a3); bp[1] = fma(a3, u, bp[1]); bp[2] = fma(a3, s3, bp[2]);
            } else {
                bp[0] = a3; bp[1] = gf_mul(a3, u); bp[2] = gf_mul(a3, s3);
            }
        }
    } else if (d_ltz<F>(s3) && up_lo) { /* both down */
        bm[0] = gf_add(bm[0], a3); bm[1] = fma(a3, u, bm[1]); bm[2] = fma(a3, s3, bm[2]);
    }
    const bool d2 = d_ltz<F>(s2);
    const double v = gf_add(d2 ? bm[1] : bp[1], a2); /* a2 = 0 where s2 = 0 */
    if (d2 ? up_lo : up_hi) {
        bm[1] = d2 ? v : bm[1];
        bp[1] = d2 ? bp[1] : v;
    }
}

/* philim (philim.f:4-65): limiter value for wave strengths a (= |w|^2) and
 * b (= projection of the upwind wave), as its ratio r = b / a, a != 0. */
template <bool FAST>
__device__ __forceinline__ double gf_philim_r(double r, int meth)
{
    switch (meth) {
    case 2: return d_max<FAST>(d_max<FAST>(0.0, d_min<FAST>(1.0, 2.0 * r)), d_min<FAST>(2.0, r));
    case 3: return (r + fabs(r)) / (1.0 + fabs(r));
    case 4: {
        /* (1 + r) / 2 or 2 r, whichever is smaller: the lines cross at 1/3.
         * One fused form with the line's coefficients in the contracted build
         * (halving and doubling are exact). */
        if (FAST) {
            const bool low = d_lt<FAST>(r, 1.0 / 3.0);
            const double c = fma(r, low ? 2.0 : 0.5, low ? 0.0 : 0.5);
            return d_max<FAST>(0.0, d_min<FAST>(c, 2.0));
        }
        const double c = (1.0 + r) * 0.5;
        return d_max<FAST>(0.0, d_min<FAST>(d_min<FAST>(c, 2.0), 2.0 * r));
    }
    case 5: return r;
    default: return d_max<FAST>(0.0, d_min<FAST>(1.0, r));
    }
}
template <bool FAST>
__device__ __forceinline__ double gf_philim(double a, double b, int meth)
{
    if (d_eqz<FAST>(a)) return 0.0;
    /* MC with b <= 0: r <= 0 and the limiter is zero; the contracted build
     * skips the division (a zero's sign aside) */
    if (FAST && meth == 4 && d_lez<FAST>(b)) return 0.0;
    return gf_philim_r<FAST>(d_div<FAST>(b, a), meth);
}

#endif
