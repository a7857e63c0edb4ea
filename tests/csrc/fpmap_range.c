/* CPU check of where the return map in pairs of floats is taken (fps_vmh_fits in code_mpm_gb300/csrc/fpmap.h), compiled
 * with gcc -O2 -ffp-contract=off: materials from no yield stress at all to yield strains of 0.1, in units from 1e-20 to
 * 1e20, Poisson ratios from -0.5 to 0.4999, with and without saturation; states from well inside the surface to 1e20
 * times past it, under pressures up to 1e6 radii, back stresses up to saturation.  Each state that fits is mapped; the
 * errors against long double are taken in units of 2^-42 of the largest stress in hand (deps_p: over 2G or G; dR: with
 * the rounding to double of sqrt(2/3) C1, which either map starts from).
 * Prints the states that fit, those with an output that is not finite, those on the wrong side of the surface (beyond
 * 2^-40 of it), and the largest errors; then how many states near the surface of ordinary materials do not fit.
 * Usage: fpmap_range <samples> <seed> */
#include <stdio.h>
#include <stdlib.h>
#include "../../code_mpm_gb300/csrc/fpmap.h"

#ifdef TAKE_ALL
#define FITS(m, rad, s, t) 1
#else
#define FITS(m, rad, s, t) fps_vmh_fits(m, rad, s, t)
#endif

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
static double pick(const double* v, int n) { return v[rnd() % (uint64_t)n]; }

typedef long double L;

int main(int argc, char** argv) {
    const long long n = argc > 1 ? atoll(argv[1]) : 1000000;
    s_state = argc > 2 ? strtoull(argv[2], 0, 10) : 1;
    static const double yields[] = {0, 1e-30, 1e-20, 1e-14, 1e-12, 1e-10, 1e-8, 1e-6, 1e-4, 1e-3, 2e-3, 1e-2, 1e-1};
    static const double units[] = {1e-20, 1e-6, 1, 1e3, 2e11, 1e20}, nus[] = {-0.5, 0, 0.3, 0.45, 0.4999};
    static const double past[] = {0.5, 0.99, 1, 1.01, 1.5, 3, 30, 100, 1e4, 1e8, 1e20}, press[] = {0, 1, 10, 100, 1e4, 1e6};
    long long fit = 0, bad = 0, side = 0, near = 0, left = 0;
    L worst[3] = {0, 0, 0};
    for (long long it = 0; it < n; ++it) {
        const double E = pick(units, 6), nu = pick(nus, 5), yE = pick(yields, 13), Y = yE * E;
        const double C1 = rnd() % 3 ? E * pick(yields + 4, 9) * 3.0 : 0.0, C0 = rnd() % 4 ? pow(10.0, 4.0 * unif() - 3.0) : 0.0;
        fps_map_const mc;
        fps_map_constants(E, nu, Y, C0, C1, &mc);
        const double sat = sqrt(2.0 / 3.0) * C1;
        static const double frac[] = {0, 0.3, 0.999, 0.9999999, 1};
        const float R = (float)(sat * pick(frac, 5) * (rnd() % 2 ? 1.0 : unif()));
        const double rad0 = Y / sqrt(3.0) + R / sqrt(2.0), ratio = pick(past, 11), pr = pick(press, 6);
        double dv[6], j = 0;
        for (int i = 0; i < 6; ++i) dv[i] = normal();
        const double tr0 = (dv[0] + dv[1] + dv[2]) / 3;
        for (int i = 0; i < 3; ++i) dv[i] -= tr0, j += 0.5 * dv[i] * dv[i];
        for (int i = 3; i < 6; ++i) j += dv[i] * dv[i];
        const double base = rad0 > 0 ? rad0 : 1e-3 * E, f = ratio * base / sqrt(j), p = (2 * unif() - 1) * pr * base;
        const double de = pow(10.0, -8.0 + 7.0 * unif()) * (yE > 0 && rnd() % 2 ? yE * 1e3 : 1.0); /* up to 0.1, or of the yield strain's size */
        float s[6], e[6], tf[6];
        int finite_in = isfinite(R);
        for (int i = 0; i < 6; ++i) {
            s[i] = (float)(f * dv[i] + (i < 3 ? p : 0)), e[i] = (float)(de * normal());
            finite_in = finite_in && isfinite(s[i]);
        }
        if (!finite_in) continue;
        const L C = (L)E / (1 + (L)nu) / (1 - 2 * (L)nu), G = (L)0.5 * (L)E / (1 + (L)nu);
        L d[6], t[6], x[13] = {0}, big = 0, ep = 0;
        for (int i = 0; i < 3; ++i) d[i] = 2 * G * e[i] + C * (L)nu * ((L)e[0] + e[1] + e[2]);
        for (int i = 3; i < 6; ++i) d[i] = G * e[i];
        for (int i = 0; i < 6; ++i) {
            t[i] = s[i] + d[i], tf[i] = (float)t[i];
            if (fabsl(t[i]) > big) big = fabsl(t[i]);
            if (fabsl((L)s[i]) > big) big = fabsl((L)s[i]);
        }
        const L rad = (L)Y / sqrtl(3) + (L)R / sqrtl(2), hyd = (t[0] + t[1] + t[2]) / 3;
        if (rad > big) big = rad;
        L J2 = 0;
        for (int i = 0; i < 3; ++i) J2 += (t[i] - hyd) * (t[i] - hyd) / 2;
        for (int i = 3; i < 6; ++i) J2 += t[i] * t[i];
        const int ordinary = yE >= 1e-6 && pr <= 10 && ratio <= 3 && nu < 0.499 && E >= 1e-6 && big <= 50 * rad;
        near += ordinary;
        if (!FITS(&mc, (float)rad, s, tf)) {
            left += ordinary;
            continue;
        }
        ++fit;
        fps_map_out o;
        const int a = fps_vmh_map(&mc, R, s, e, &o);
        int ok = isfinite(o.dR);
        for (int i = 0; i < 6; ++i) ok = ok && isfinite(o.dsig[i]) && isfinite(o.deps_p[i]);
        if (!ok) {
            ++bad;
            continue;
        }
        const L over = (sqrtl(J2) - rad) / big;
        if (a != (over > 0)) {
            if (fabsl(over) > 0x1p-40L) ++side;
            continue;
        }
        if (a) {
            const L q = 1 - rad / sqrtl(J2);
            L n2 = 0;
            for (int i = 0; i < 6; ++i) {
                const L w = (t[i] - (i < 3 ? hyd : 0)) * q;
                x[i] = d[i] - w;
                x[6 + i] = i < 3 ? w / (2 * G) : w / G;
                n2 += x[6 + i] * x[6 + i];
            }
            const L st = sqrtl(2.0L / 3) * (L)C1 - R;
            ep = sqrtl(n2 * 2 / 3);
            x[12] = st > 0 ? (L)C0 * st * ep : 0;
        } else {
            for (int i = 0; i < 6; ++i) x[i] = d[i];
        }
        for (int i = 0; i < 13; ++i) {
            const float got = i < 6 ? o.dsig[i] : i < 12 ? o.deps_p[i - 6] : o.dR, xf = fabsf((float)x[i]);
            /* its own rounding; below the normal floats, twice (to 24 bits, then unscaled) */
            const L half = 0.5L * ((L)nextafterf(xf, INFINITY) - xf) + (xf < 0x1p-126f ? 0x1p-24L * xf : 0), err = fabsl((L)got - x[i]) - half * (1 + 0x1p-20L);
            /* what an error of 2^-42 of the largest stress is worth in this output */
            L unit = 0x1p-42L * big / (i < 6 ? 1 : i < 9 ? 2 * G : G);
            if (i == 12)
                unit = 0x1p-42L * (fabsl(x[12]) + (L)C0 * fabsl(sqrtl(2.0L / 3) * (L)C1 - R) * big / G) +
                       0x1p-52L * (L)C0 * (ep + 0x1p-42L * big / G) * sat;
            const int k = i < 6 ? 0 : i < 12 ? 1 : 2;
            if (err > 0 && unit > 0 && err / unit > worst[k]) worst[k] = err / unit;
        }
    }
    printf("fit %lld notfinite %lld side %lld dsig %.3Lf deps_p %.3Lf dR %.3Lf ordinary %lld left %lld\n", fit, bad, side,
           worst[0], worst[1], worst[2], near, left);
    return 0;
}
