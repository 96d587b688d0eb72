// Checks the integer-pipe double-precision functions (csrc/sf_f64_int.cuh) against the host's own arithmetic, bit
// for bit, with a reciprocal that is off by up to four units in the last place either way (the device's is off by
// one).  Significands at the ends of the binade, with few set bits and at random; exponents over the range the
// callers accept.  Prints the number of mismatches and the number of values checked.
#include <cinttypes>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>

#define SF_F64_TEST_RCP test_rcp
namespace sf {
float test_rcp(float y);
}
#include "sf_f64_int.cuh"

static int g_off = 0;
namespace sf {
float test_rcp(float y) {
    for (int i = 0; i < std::abs(g_off); i++) y = std::nextafterf(y, g_off > 0 ? 2.f : 0.f);
    return y;
}
}  // namespace sf

static uint64_t bits(double v) {
    uint64_t u;
    std::memcpy(&u, &v, 8);
    return u;
}

int main() {
    long long bad = 0, n = 0;
    std::mt19937_64 rng(2025);
    auto draw = [&]() {
        uint64_t m = rng() & 0xfffffffffffffull;
        switch (rng() % 7) {
            case 0: m = 0; break;
            case 1: m = 0xfffffffffffffull; break;
            case 2: m = rng() & 15; break;
            case 3: m = 0xfffffffffffffull - (rng() & 15); break;
            case 4: m &= ~0xffffffffull; break;
            default: break;
        }
        const uint64_t u = ((rng() & 1) << 63) | ((uint64_t)(1023 - 250 + (int)(rng() % 500)) << 52) | m;
        double v;
        std::memcpy(&v, &u, 8);
        return rng() % 40 == 0 ? std::copysign(0.0, v) : v;
    };
    auto check = [&](const char *what, double got, double want, double a, double b) {
        n++;
        if (bits(got) != bits(want)) {
            if (bad < 10) std::printf("%s(%a, %a) = %a, expected %a\n", what, a, b, got, want);
            bad++;
        }
    };
    for (int t = 0; t < 6000000; t++) {
        g_off = (int)(rng() % 9) - 4;
        const double a = draw(), b = draw();
        if (b != 0) {
            check("div", sf::f64_div(a, b), a / b, a, b);
            // a quotient next to a representable value and next to a midpoint
            const double q = a / b, c = q * b;
            if (c != 0) check("div", sf::f64_div(c, b), c / b, c, b);
        }
        check("mul", sf::f64_mul(a, b), a * b, a, b);
        check("third", sf::f64_third(a), a / 3, a, 0);
        check("times_third<5>", sf::f64_times_third<5>(a), a * 5 / 3, a, 0);
        check("times_third<7>", sf::f64_times_third<7>(a), a * 7 / 3, a, 0);
        check("times_third<11>", sf::f64_times_third<11>(a), a * 11 / 3, a, 0);
        check("times_third<13>", sf::f64_times_third<13>(a), a * 13 / 3, a, 0);
        check("sqr", sf::f64_sqr(a), a * a, a, a);
        check("half", sf::f64_half(a), a / 2, a, 0);
        check("-half", sf::f64_half<true>(a), a / -2, a, 0);
        check("div_any", sf::f64_div_any(a, b != 0 ? b : 1), a / (b != 0 ? b : 1), a, b);
        check("sqrt_any", sf::f64_sqrt_any(std::fabs(a)), std::sqrt(std::fabs(a)), a, 0);
        check("third_any", sf::f64_third_any(a), a / 3, a, 0);
        if (a != 0 && b != 0) check("mul nonzero", sf::f64_mul<false, false>(a, b), a * b, a, b);
        if (a != 0) {
            const double r = std::fabs(a);
            check("sqrt", sf::f64_sqrt(r), std::sqrt(r), r, 0);
            // a radicand next to a square and next to the square of a midpoint
            const double w = std::sqrt(r), near = w * w, next = std::nextafter(w, 1e300) * w;
            check("sqrt", sf::f64_sqrt(near), std::sqrt(near), near, 0);
            check("sqrt", sf::f64_sqrt(next), std::sqrt(next), next, 0);
        }
        const bool in = a == 0 || (std::fabs(a) >= 0x1p-100 && std::fabs(a) < 0x1p60);
        n++;
        bad += sf::f64_in_range(a, -100, 60) != in;
        n++;
        bad += (sf::f64_above(a, -100) < (160u << 20)) != (in && a != 0);
    }
    auto check_floor = [&](double v) {
        double fl;
        const int i = sf::f64_floor(v, fl), w = (int)std::floor(v);
        n++;
        if (i != w || fl != (double)w) {
            if (bad < 10) std::printf("floor(%a) = %d, %a, expected %d\n", v, i, fl, w);
            bad++;
        }
    };
    auto check_order = [&](double v) {
        n++;
        bad += sf::f64_le0(v) != (v <= 0) || sf::f64_lt0(v) != (v < 0) || sf::f64_lt1(v) != (v < 1) ||
               sf::f64_is_one(v) != (v == 1);
    };
    for (int t = 0; t < 3000000; t++) {
        const double v = std::ldexp((double)(int64_t)rng(), -33 - (int)(rng() % 60));  // |v| < 2^30
        check_floor(v);
        check_floor(std::rint(v));
        check_floor(std::nextafter(std::rint(v), rng() & 1 ? 1e9 : -1e9));
        check_order(v);
    }
    for (double v : {0.0, -0.0, 0x1p-1074, -0x1p-1074, 1.0, -1.0, 0x1p30, -0x1p30, 2147483647.0, -2147483648.0 + 0.5,
                     2147483646.5, -2147483647.0, 0x1p20, 0x1p21, -0x1p20 - 0.5, 0x1.fffffffffffffp-1}) {
        check_floor(v);
        check_order(v);
    }
    for (double v : {(double)NAN, -(double)NAN, (double)INFINITY, -(double)INFINITY, 1 + 0x1p-52, -1e308, 1e308}) check_order(v);
    for (double v : {0x1p-1074, -0x1p-1030, 1e308, -1e308, (double)INFINITY, -0.0, 0x1p-1022, 0x1p1023}) {
        check("div_any", sf::f64_div_any(v, 3.0), v / 3.0, v, 3);
        check("div_any", sf::f64_div_any(1.0, v), 1.0 / v, 1, v);
        check("sqrt_any", sf::f64_sqrt_any(std::fabs(v)), std::sqrt(std::fabs(v)), v, 0);
        check("third_any", sf::f64_third_any(v), v / 3, v, 0);
    }
    n++;
    bad += !std::isnan(sf::f64_sqrt_any(-1.0)) || !std::isnan(sf::f64_div_any(NAN, 1.0));
    const double outside[] = {0x1p-1074, -0x1p-1030, 0x1p-101, 0x1p60, -0x1p60, 1e300, INFINITY, -INFINITY, NAN};
    for (double v : outside) {
        n++;
        bad += sf::f64_in_range(v, -100, 60);
    }
    std::printf("%lld %lld\n", bad, n);
    return bad != 0;
}
