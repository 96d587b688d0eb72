// Checks fixed_stencil (csrc/sf_f64_int.cuh), n x minus its six neighbours in 64-bit integers, against the exact sum
// (128-bit integers), next to the same sum in FP64 arithmetic.  Bound of a sum: six units of 2^-58 of the largest
// magnitude M among the seven, and half a unit in the last place of the result.  Over each class of values (all of one
// size, sizes spread over 2^s, a small centre, a small neighbourhood of a large value, a smooth field), at scales from
// 2^300 down to 2^-300: the root mean square error is no larger than that of the FP64 form.
// Prints the violations and the number of sums.
#include <cmath>
#include <cstdio>
#include <random>

#include "sf_f64_int.cuh"

typedef __int128 wide;

static wide to_wide(double v, int base) {  // v / 2^base, exact
    int e;
    const double f = std::frexp(v, &e);
    const wide m = (wide)(int64_t)std::ldexp(f, 53);
    const int s = e - 53 - base;
    return s >= 0 ? m << s : m >> -s;
}

int main() {
    std::mt19937_64 rng(11);
    std::uniform_real_distribution<double> one(1.0, 2.0);
    long long bad = 0, n = 0;
    for (int kind = 0; kind < 8; kind++)
        for (int scale : {0, 300, -30, -300}) {
            double sq_int = 0, sq_fp = 0;
            for (int t = 0; t < 200000; t++) {
                double v[7];
                int lo = 10000, hi = -10000;
                for (int q = 0; q < 7; q++) {
                    int e = 0;
                    if (kind == 1) e = -(int)(rng() % 4);
                    if (kind == 2) e = -(int)(rng() % 12);
                    if (kind == 3) e = -(int)(rng() % 40);
                    if (kind == 4) e = q == 0 ? -20 : 0;
                    if (kind == 5) e = q == 3 ? 0 : -20;
                    if (kind == 6) e = q == 0 ? 0 : -(int)(rng() % 56);
                    e += scale;
                    v[q] = std::ldexp(one(rng) * (rng() & 1 ? 1 : -1), e);
                    if (kind == 7) v[q] = std::ldexp(1.5 + 1e-6 * one(rng), e);  // a smooth field: cancellation
                    lo = e < lo ? e : lo;
                    hi = e > hi ? e : hi;
                }
                const int c = 3 + (int)(rng() % 4);  // in-grid neighbours; the others are zero
                for (int q = 1 + c; q < 7; q++) v[q] = 0.;
                double got;
                sf::F64Fixed f[7];
                for (int q = 0; q < 7; q++) f[q] = sf::f64_fixed(v[q]);
                n++;
                if (!sf::fixed_stencil(c, f[0], f[1], f[2], f[3], f[4], f[5], f[6], got)) {
                    bad++;
                    continue;
                }
                int base = lo - 53 < hi - 60 ? lo - 53 : hi - 60;
                wide exact = (wide)c * to_wide(v[0], base);
                double fp = c * v[0], s = 0, top = 0;
                for (int q = 0; q < 7; q++) top = std::fmax(top, std::fabs(v[q]));
                for (int q = 1; q <= c; q++) {
                    exact -= to_wide(v[q], base);
                    s += v[q];
                }
                fp -= s;
                const double unit = std::ldexp(1.0, std::ilogb(top) - 58 - base);
                const double err = std::fabs((double)(to_wide(got, base) - exact)), size = std::fabs((double)exact);
                if (err > 6 * unit + 0x1p-53 * size * 1.0001) bad++;
                sq_int += std::pow(err / std::ldexp(top, -base), 2);
                sq_fp += std::pow((double)(to_wide(fp, base) - exact) / std::ldexp(top, -base), 2);
            }
            if (sq_int > sq_fp) {
                std::printf("class %d, scale %d: %g against %g\n", kind, scale, std::sqrt(sq_int / 2e5), std::sqrt(sq_fp / 2e5));
                bad++;
            }
        }
    // zeros, and what the integer form leaves to FP64
    double s;
    const sf::F64Fixed z = sf::f64_fixed(0.), w = sf::f64_fixed(3.), y = sf::f64_fixed(-0.);
    n += 6;
    bad += !sf::fixed_stencil(6, w, z, z, z, z, z, z, s) || s != 18.;
    bad += !sf::fixed_stencil(6, z, w, z, z, z, z, z, s) || s != -3.;
    bad += !sf::fixed_stencil(6, w, w, w, w, w, w, w, s) || s != 0.;
    bad += !sf::fixed_stencil(5, w, y, y, y, y, y, z, s) || std::fabs(s - 15.) > 5 * 0x1p-57;
    bad += sf::fixed_stencil(6, z, z, z, z, z, z, z, s) || sf::fixed_stencil(6, sf::f64_fixed(1e-300), z, z, z, z, z, z, s);
    bad += sf::fixed_stencil(6, w, sf::f64_fixed(INFINITY), w, w, w, w, w, s) ||
           sf::fixed_stencil(6, sf::f64_fixed(NAN), w, w, w, w, w, w, s);
    std::printf("%lld %lld\n", bad, n);
    return bad != 0;
}
