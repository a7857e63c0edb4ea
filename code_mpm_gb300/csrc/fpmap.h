// The von Mises hardening return map (ConstitutiveRelation_calculateIncrement_VonMisesHardening.cpp:4-92)
// of float states in pairs of floats.
//
// The FP32 form's fallback path asks for the map of a float state computed
// far below float resolution, each output then rounded once to float.  In
// FP64 that map bounds pass 2 wherever the particles sit near the yield
// surface: GB300 issues FP64 at about 1/60 of the FP32 rate, and one lane of
// a warp is enough to pay for it.  Here every quantity is an unevaluated sum
// h + l of two floats (48 significand bits), from the error-free sums and
// products of Dekker (Numer. Math. 18, 1971) and Knuth (TAOCP 2, 4.2.2) with
// the products' error by FMA.
//
// Two steps keep the small results exact where plain substitution would
// cancel: with the trial stress tr = sig + D de, its deviator d and the
// surface radius rad, the correction is w = d q with
//   q = 1 - rad / sqrt(J2) = (J2 - rad^2) / (sqrt(J2) (sqrt(J2) + rad)),
// so dsig = D de - w (not d rad / sqrt(J2) + hyd - sig) and the plastic
// strain is w / 2G (w / G for the engineering shears), which is what
// de - C^-1 dsig equals.  J2 is summed from the deviator.
//
// Stresses are scaled by a power of two that brings k0 into [1, 2), so the
// squares and their error terms stay far from the float range's ends for any
// system of units.  That needs a material whose moduli are within reach of its
// yield stress, and a state within reach of its yield surface: fps_vmh_fits
// says whether they are, and the caller takes the map in FP64 where not
// (yield 0 or next to nothing, stresses far past the surface).
//
// Measured against the exact value in long double (tests/csrc/fpmap_check.c,
// three runs of 4M random states from 0.9 to 1.02 of the surface, six
// materials): rounded to float, the outputs of the pairs are off by 0.288692,
// 0.288679 and 0.288658 ulp RMS, those of the map in FP64 by 0.288691,
// 0.288679 and 0.288658 (rounding alone gives 0.288675); the largest errors,
// of corrections near zero, are 2.8 ulp in both.  The two round differently
// in 2.4e-5 of the outputs.
//
// The header compiles as C (gcc) and as CUDA, so the CPU test checks the code
// that the kernels run.
#ifndef MPM_FPMAP_H
#define MPM_FPMAP_H

#include "fpsplit.h"

typedef struct {
    float h, l;
} fps_df;

// The material's constants (stresses and moduli times `s`), from doubles on the host.
typedef struct {
    fps_df twoG, lam, G, inv_2G, k0, s23C1, C0, third, irt2, f23;
    float s23C1_ll;  // s23C1's bits below its pair: near saturation the difference from R is all there is
    float s, inv_s;
    float rad_min, rad_max;  // radii the map is taken for (unscaled); none (1 and 0) for a material it does not suit
} fps_map_const;

typedef struct {
    float dsig[6], deps_p[6], dR;
} fps_map_out;

FPS_HD fps_df fps_two_sum(float a, float b) {
    fps_df r;
    r.h = fps_add(a, b);
    const float bb = fps_add(r.h, -a);
    r.l = fps_add(fps_add(a, -fps_add(r.h, -bb)), fps_add(b, -bb));
    return r;
}

// |a| >= |b| (or a = 0)
FPS_HD fps_df fps_fast_sum(float a, float b) {
    fps_df r;
    r.h = fps_add(a, b);
    r.l = fps_add(b, -fps_add(r.h, -a));
    return r;
}

FPS_HD fps_df fps_df_add(fps_df a, fps_df b) {
    const fps_df s = fps_two_sum(a.h, b.h);
    return fps_fast_sum(s.h, fps_add(s.l, fps_add(a.l, b.l)));
}

FPS_HD fps_df fps_df_sub(fps_df a, fps_df b) {
    fps_df n;
    n.h = -b.h;
    n.l = -b.l;
    return fps_df_add(a, n);
}

FPS_HD fps_df fps_df_addf(fps_df a, float b) {
    const fps_df s = fps_two_sum(a.h, b);
    return fps_fast_sum(s.h, fps_add(s.l, a.l));
}

FPS_HD fps_df fps_df_mul(fps_df a, fps_df b) {
    const float p = fps_mul(a.h, b.h);
    float e = fmaf(a.h, b.h, -p);
    e = fmaf(a.h, b.l, e);
    e = fmaf(a.l, b.h, e);
    return fps_fast_sum(p, e);
}

FPS_HD fps_df fps_df_mulf(fps_df a, float b) {
    const float p = fps_mul(a.h, b);
    return fps_fast_sum(p, fmaf(a.l, b, fmaf(a.h, b, -p)));
}

FPS_HD fps_df fps_df_sqr(fps_df a) {
    const float p = fps_mul(a.h, a.h);
    return fps_fast_sum(p, fmaf(fps_add(a.h, a.h), a.l, fmaf(a.h, a.h, -p)));
}

// sqrt of a >= 0: one correction of the float root
FPS_HD fps_df fps_df_sqrt(fps_df a) {
    fps_df z;
    z.h = z.l = 0.0f;
    if (!(a.h > 0.0f)) return z;
    const float s = sqrtf(a.h);
    const float r = fps_add(fmaf(-s, s, a.h), a.l);
    return fps_fast_sum(s, fps_mul(r, 0.5f / s));
}

FPS_HD fps_df fps_df_div(fps_df a, fps_df b) {
    const float inv = 1.0f / b.h;
    const float q = fps_mul(a.h, inv);
    const float r = fps_add(fmaf(-q, b.h, a.h), fmaf(-q, b.l, a.l));
    return fps_fast_sum(q, fps_mul(r, inv));
}

// Whether the pairs serve a state of this radius, stress and trial stress
// (unscaled floats; the trial stress to float accuracy).  The bound, 1024 radii,
// leaves the sums at 2^-36 of the radius or better, 2^12 below what the float
// stress itself resolves; NaN fits (either map gives NaN).
FPS_HD int fps_vmh_fits(const fps_map_const* m, float rad, const float sig[6], const float tr[6]) {
    float a = 0.0f;
    for (int i = 0; i < 6; ++i) a = fmaxf(a, fmaxf(fabsf(sig[i]), fabsf(tr[i])));
    return rad >= m->rad_min && rad <= m->rad_max && a <= 1024.0f * rad;
}

// The map of (sig, R, de): the float state's increments, each rounded once.
// Returns 1 for a plastic step, 0 for an elastic one (deps_p and dR are then
// zero); elastic as in the reference when J2 <= rad^2.
FPS_HD int fps_vmh_map(const fps_map_const* m, float R, const float sig[6], const float e[6], fps_map_out* o) {
    fps_df d[6];  // D de, then kept beside the deviator
    {
        const fps_df tr = fps_df_addf(fps_two_sum(e[0], e[1]), e[2]);
        const fps_df lt = fps_df_mul(m->lam, tr);
        d[0] = fps_df_add(fps_df_mulf(m->twoG, e[0]), lt);
        d[1] = fps_df_add(fps_df_mulf(m->twoG, e[1]), lt);
        d[2] = fps_df_add(fps_df_mulf(m->twoG, e[2]), lt);
        d[3] = fps_df_mulf(m->G, e[3]);
        d[4] = fps_df_mulf(m->G, e[4]);
        d[5] = fps_df_mulf(m->G, e[5]);
    }
    fps_df t[6];  // the trial stress, then its deviator
    for (int i = 0; i < 6; ++i) t[i] = fps_df_addf(d[i], fps_mul(sig[i], m->s));
    {
        const fps_df hyd = fps_df_mul(m->third, fps_df_add(fps_df_add(t[0], t[1]), t[2]));
        for (int i = 0; i < 3; ++i) t[i] = fps_df_sub(t[i], hyd);
    }
    fps_df J2 = fps_df_add(fps_df_add(fps_df_sqr(t[0]), fps_df_sqr(t[1])), fps_df_sqr(t[2]));
    J2.h = fps_mul(0.5f, J2.h);
    J2.l = fps_mul(0.5f, J2.l);
    J2 = fps_df_add(J2, fps_df_add(fps_df_add(fps_df_sqr(t[3]), fps_df_sqr(t[4])), fps_df_sqr(t[5])));
    const float Rs = fps_mul(R, m->s);
    const fps_df rad = fps_df_add(m->k0, fps_df_mulf(m->irt2, Rs));
    const fps_df D = fps_df_sub(J2, fps_df_sqr(rad));
    o->dR = 0.0f;
    if (D.h <= 0.0f) {
        for (int i = 0; i < 6; ++i) {
            o->dsig[i] = fps_mul(d[i].h, m->inv_s);
            o->deps_p[i] = 0.0f;
        }
        return 0;
    }
    const fps_df root = fps_df_sqrt(J2);
    const fps_df q = fps_df_div(D, fps_df_mul(root, fps_df_add(root, rad)));
    fps_df n2, s2;  // sums of w^2 over the normal and the shear components
    for (int i = 0; i < 6; ++i) {
        const fps_df w = fps_df_mul(t[i], q);
        const fps_df ep = fps_df_mul(w, m->inv_2G);
        o->dsig[i] = fps_mul(fps_df_sub(d[i], w).h, m->inv_s);
        o->deps_p[i] = i < 3 ? ep.h : fps_mul(2.0f, ep.h);
        const fps_df w2 = fps_df_sqr(w);
        if (i < 3) n2 = i == 0 ? w2 : fps_df_add(n2, w2);
        else s2 = i == 3 ? w2 : fps_df_add(s2, w2);
    }
    const fps_df sat = fps_df_addf(fps_df_addf(fps_two_sum(m->s23C1.h, -Rs), m->s23C1.l), m->s23C1_ll);
    if (sat.h > 0.0f) {
        s2.h = fps_mul(4.0f, s2.h);
        s2.l = fps_mul(4.0f, s2.l);
        const fps_df ep = fps_df_mul(fps_df_sqrt(fps_df_mul(m->f23, fps_df_add(n2, s2))), m->inv_2G);
        o->dR = fps_mul(fps_df_mul(fps_df_mul(m->C0, sat), ep).h, m->inv_s);
    }
    return 1;
}

// ---- host: the constants of a material ------------------------------------
static inline fps_df fps_df_of(double v) {
    fps_df r;
    r.h = (float)v;
    r.l = (float)(v - (double)r.h);
    return r;
}

static inline void fps_map_constants(double E, double nu, double yield, double C0, double C1, fps_map_const* m) {
    const double k0 = yield / sqrt(3.0), G = 0.5 * E / (1.0 + nu);
    int ex = 0;
    if (k0 > 0.0 && k0 < 1.0e300) (void)frexp(k0, &ex);
    if (ex > 100) ex = 100;
    if (ex < -100) ex = -100;
    const double s = ldexp(1.0, 1 - ex);
    m->s = (float)s;
    m->inv_s = (float)(1.0 / s);
    m->G = fps_df_of(G * s);
    m->twoG = fps_df_of(2.0 * G * s);
    m->lam = fps_df_of(E / (1.0 + nu) / (1.0 - 2.0 * nu) * nu * s);
    m->inv_2G = fps_df_of(1.0 / (2.0 * G * s));
    m->k0 = fps_df_of(k0 * s);
    m->s23C1 = fps_df_of(sqrt(2.0 / 3.0) * C1 * s);
    m->s23C1_ll = (float)(sqrt(2.0 / 3.0) * C1 * s - (double)m->s23C1.h - (double)m->s23C1.l);
    m->C0 = fps_df_of(C0);
    m->third = fps_df_of(1.0 / 3.0);
    m->irt2 = fps_df_of(1.0 / sqrt(2.0));
    m->f23 = fps_df_of(2.0 / 3.0);
    // suited: k0 within the scale's range; yield strains from 2^-45 (3e-14) to 2^20, saturation and hardening rate
    // inside the float range with their low parts; Poisson ratios away from -1 and 0.5 (no modulus 2^12 of another)
    const int fits = k0 * s >= 1.0 && k0 * s < 2.0 && G * s >= 0x1p-20 && G * s <= 0x1p45 && nu >= -0.95 &&
                     1.0 - 2.0 * nu >= 0x1p-11 && fabs(C1) * s <= 0x1p60 && (C1 == 0.0 || fabs(C1) * s >= 0x1p-60) &&
                     (C0 == 0.0 || (fabs(C0) >= 0x1p-60 && fabs(C0) <= 0x1p60));
    m->rad_min = fits ? (float)(0.5 * k0) : 1.0f;
    m->rad_max = fits ? (float)(0x1p40 * k0) : 0.0f;
}

#endif
