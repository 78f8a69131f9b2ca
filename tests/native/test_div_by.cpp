// dm::div_by (csrc/khs_device_math.cuh) against the IEEE division, bit for bit,
// over random significands and exponents, those around the limits past which it
// divides, quotients next to a midpoint, and zeros, infinities and NaN.  Built
// and run by tests/test_div_by.py.
#include "khs_device_math.cuh"

#include <cmath>
#include <cstdio>
#include <cstring>
#include <limits>
#include <random>

namespace dm = khs::dm;

int main()
{
    std::mt19937_64 rng(21);
    long bad = 0, checked = 0;
    auto check = [&](double a, double n) {
        const double got = dm::div_by(a, n, 1.0 / n), want = a / n;
        ++checked;
        if (std::isnan(want) ? !std::isnan(got) : std::memcmp(&got, &want, 8) != 0) {
            if (++bad < 5) std::printf("%a / %a = %a, not %a\n", a, n, want, got);
        }
    };
    auto value = [&](int exponent) {
        const double m = 1.0 + double(rng() & 0xfffffffffffffull) * 0x1p-52;
        return std::ldexp(rng() & 1 ? m : -m, exponent);
    };
    const int edges[] = {-1022, -824, -823, -822, -301, -300, -1, 0, 1, 300, 301, 776, 777, 778, 1023};
    for (int k = 0; k < 4000000; ++k) {
        check(value(int(rng() % 40) - 20), value(int(rng() % 40) - 20));
        if (k % 16 == 0) check(value(edges[rng() % 15]), value(edges[rng() % 15]));
    }
    // Significands of few bits, and quotients a unit in the last place from a
    // midpoint: a = n q, rounded, for q of 54 bits.
    for (int k = 0; k < 1000000; ++k) {
        check(double(rng() % 4096), double(1 + rng() % 4096));
        const double n = value(0), q = value(0);
        check(std::fma(n, q, n * 0x1p-53), n);
        check(std::fma(n, q, n * -0x1p-53), n);
    }
    const double inf = std::numeric_limits<double>::infinity(), special[] = {0.0, -0.0, inf, -inf, std::nan(""), 5e-324, -1e-310, 1.7e308, 1.0, -3.0};
    for (double a : special)
        for (double n : special) check(a, n);
    std::printf("division by a reciprocal: %ld checks, %ld mismatches\n%s\n", checked, bad, bad ? "FAIL" : "PASS");
    return bad != 0;
}
