/* CPU check of the return map in pairs of floats (code_mpm_gb300/csrc/fpmap.h), compiled with gcc -O2
 * -ffp-contract=off: random float states around the yield surface, several materials and systems of units, against the
 * map in long double.  Prints, for the pairs and for the map in double as the reference orders it: the RMS and the
 * largest error in float ulps of the exact value, and the share of outputs that the two round differently.
 * Usage: fpmap_check <samples> <seed> */
#include <stdio.h>
#include <stdlib.h>
#include "../../code_mpm_gb300/csrc/fpmap.h"

static uint64_t s_state;
static uint64_t rnd(void) { /* splitmix64 */
    uint64_t z = (s_state += 0x9e3779b97f4a7c15ULL);
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
    return z ^ (z >> 31);
}
static double unif(void) { return (double)(rnd() >> 11) * (1.0 / 9007199254740992.0); }
static double normal(void) {
    double s = -6.0;
    for (int i = 0; i < 12; ++i) s += unif();
    return s;
}

#define MAP(NAME, T, SQRT)                                                                                       \
    static int NAME(double E, double nu, double Y, double C0, double C1, float R_, const float s_[6],            \
                    const float e_[6], T out[13]) {                                                              \
        const T C = (T)E / (1 + (T)nu) / (1 - 2 * (T)nu), a = 1 - (T)nu, hb = (T)0.5 - (T)nu, n = nu;            \
        const T G = (T)0.5 * (T)E / (1 + (T)nu), R = R_;                                                         \
        T s[6], e[6], d[6], t[6];                                                                                \
        for (int i = 0; i < 6; ++i) s[i] = s_[i], e[i] = e_[i], out[i] = out[6 + i] = 0;                         \
        out[12] = 0;                                                                                             \
        d[0] = C * (a * e[0] + n * e[1] + n * e[2]);                                                             \
        d[1] = C * (a * e[1] + n * e[0] + n * e[2]);                                                             \
        d[2] = C * (a * e[2] + n * e[0] + n * e[1]);                                                             \
        for (int i = 3; i < 6; ++i) d[i] = C * hb * e[i];                                                        \
        for (int i = 0; i < 6; ++i) t[i] = s[i] + d[i];                                                          \
        const T x = t[0] - t[1], y = t[1] - t[2], z = t[2] - t[0];                                               \
        const T J2 = (x * x + y * y + z * z) / 6 + t[3] * t[3] + t[4] * t[4] + t[5] * t[5];                      \
        const T rad = (T)Y / SQRT((T)3) + R / SQRT((T)2);                                                        \
        if (J2 <= rad * rad) {                                                                                   \
            for (int i = 0; i < 6; ++i) out[i] = d[i];                                                           \
            return 0;                                                                                            \
        }                                                                                                        \
        const T hyd = (t[0] + t[1] + t[2]) / 3, sc = rad / SQRT(J2);                                             \
        for (int i = 0; i < 6; ++i) out[i] = (t[i] - (i < 3 ? hyd : 0)) * sc - s[i] + (i < 3 ? hyd : 0);         \
        T ee[6], ep = 0;                                                                                         \
        ee[0] = (out[0] - (T)nu * out[1] - (T)nu * out[2]) / (T)E;                                               \
        ee[1] = (out[1] - (T)nu * out[0] - (T)nu * out[2]) / (T)E;                                               \
        ee[2] = (out[2] - (T)nu * out[0] - (T)nu * out[1]) / (T)E;                                               \
        for (int i = 3; i < 6; ++i) ee[i] = out[i] / G;                                                          \
        for (int i = 0; i < 6; ++i) out[6 + i] = e[i] - ee[i], ep += out[6 + i] * out[6 + i];                    \
        const T sat = SQRT((T)2 / 3) * (T)C1 - R;                                                                \
        out[12] = sat > 0 ? (T)C0 * sat * SQRT(ep * 2 / 3) : 0;                                                  \
        return 1;                                                                                                \
    }
MAP(map_ld, long double, sqrtl)
MAP(map_d, double, sqrt)

int main(int argc, char** argv) {
    const long long n = argc > 1 ? atoll(argv[1]) : 1000000;
    s_state = argc > 2 ? strtoull(argv[2], 0, 10) : 1;
    /* E, nu, yield, C0, C1: structural steel, aluminium foam, a strongly saturating law, steel in MPa and in GPa,
     * a material without hardening */
    const double mats[6][5] = {{200e9, 0.3, 250e6, 2e-3, 1e12}, {70e9, 0.33, 120e6, 7e-4, 1e12},
                               {70e9, 0.33, 70e6, 35.0, 55e6},  {200e3, 0.3, 250.0, 2e-3, 1e6},
                               {200.0, 0.3, 0.25, 2e-3, 1e3},   {200e9, 0.3, 250e6, 0.0, 0.0}};
    double sq[2] = {0, 0}, mx[2] = {0, 0};
    long long cnt = 0, differ = 0, plastic = 0, branch = 0;
    for (long long it = 0; it < n; ++it) {
        const double* m = mats[rnd() % 6];
        fps_map_const mc;
        fps_map_constants(m[0], m[1], m[2], m[3], m[4], &mc);
        const double ep = unif() * 0.05, C1 = m[4];
        const float R = (float)(sqrt(2.0 / 3.0) * C1 * (1.0 - exp(-m[3] * ep)));
        const double rad = m[2] / sqrt(3.0) + R / sqrt(2.0);
        double dv[6], j = 0, tr;
        for (int i = 0; i < 6; ++i) dv[i] = normal();
        tr = (dv[0] + dv[1] + dv[2]) / 3;
        for (int i = 0; i < 3; ++i) dv[i] -= tr, j += 0.5 * dv[i] * dv[i];
        for (int i = 3; i < 6; ++i) j += dv[i] * dv[i];
        const double f = (0.9 + 0.12 * unif()) * rad / sqrt(j), p = (2 * unif() - 1) * m[2];
        float s[6], e[6];
        const double de = pow(10.0, -6.0 + 3.0 * unif());  /* strain increments from 1e-6 to 1e-3 */
        for (int i = 0; i < 6; ++i) s[i] = (float)(f * dv[i] + (i < 3 ? p : 0)), e[i] = (float)(de * normal());
        fps_map_out o;
        long double x[13];
        double d[13];
        const int a = fps_vmh_map(&mc, R, s, e, &o), b = map_ld(m[0], m[1], m[2], m[3], m[4], R, s, e, x);
        const int c = map_d(m[0], m[1], m[2], m[3], m[4], R, s, e, d);
        if (a != b || c != b) {
            ++branch;
            continue;
        }
        plastic += a;
        for (int i = 0; i < 13; ++i) {
            const float got = i < 6 ? o.dsig[i] : i < 12 ? o.deps_p[i - 6] : o.dR, ref = (float)d[i];
            if (x[i] == 0) continue;
            const float xf = fabsf((float)x[i]);
            const double ulp = (double)nextafterf(xf, INFINITY) - (double)xf;
            const double g = (double)((long double)got - x[i]) / ulp, r = (double)((long double)ref - x[i]) / ulp;
            sq[0] += g * g, sq[1] += r * r;
            if (fabs(g) > mx[0]) mx[0] = fabs(g);
            if (fabs(r) > mx[1]) mx[1] = fabs(r);
            ++cnt;
            differ += got != ref;
        }
    }
    printf("pairs rms %.6f max %.6f double rms %.6f max %.6f differ %.3e plastic %.3f branch %lld outputs %lld\n",
           sqrt(sq[0] / cnt), mx[0], sqrt(sq[1] / cnt), mx[1], (double)differ / cnt, (double)plastic / n, branch, cnt);
    return 0;
}
