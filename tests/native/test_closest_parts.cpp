// The closest pair of a segment and a triangle (csrc/khs_device_math.cuh):
// integer comparisons on the bits, squared distances and the shared parts,
// against the plain form with floating comparisons and a square root a part,
// bit for bit.  Inputs: random at several scales; on a small lattice, where
// zeros of either sign, exact ties and degenerate segments and triangles
// abound; squared distances a few units in the last place apart; huge,
// infinite and NaN coordinates.  Built and run by tests/test_closest_parts.py.
#include "khs_device_math.cuh"

#include <cstdio>
#include <limits>
#include <random>

namespace dm = khs::dm;
using dm::V;

static dm::ClosestPair plain(V p0, V p1, V a, V b, V c)
{
    dm::ClosestPair out;
    out.distance = 1.0e300; out.t = 0.0; out.bary = dm::v(1, 0, 0);
    V bary;
    for (int k = 0; k < 2; ++k) {
        const V p = k ? p1 : p0;
        const double d = dm::gnorm(dm::gsub(p, dm::closest_point_triangle<false>(p, a, b, c, bary)));
        if (d < out.distance) { out.distance = d; out.t = k; out.bary = bary; }
    }
    const V d1 = dm::gsub(p1, p0);
    for (int e = 0; e < 3; ++e) {
        const V p2 = e == 0 ? a : (e == 1 ? b : c), q2 = e == 0 ? b : (e == 1 ? c : a);
        double s, t;
        dm::segment_segment_params<false>(p0, p1, p2, q2, s, t);
        const double d = dm::gnorm(dm::gsub(dm::gadd(p0, dm::gmul(d1, s)), dm::gadd(p2, dm::gmul(dm::gsub(q2, p2), t))));
        if (d < out.distance) {
            out.distance = d;
            out.t = s;
            out.bary = e == 0 ? dm::v(1.0 - t, t, 0) : (e == 1 ? dm::v(0, 1.0 - t, t) : dm::v(t, 0, 1.0 - t));
        }
    }
    return out;
}

static bool same(double x, double y) { return dm::bits_of(x) == dm::bits_of(y) || (x != x && y != y); }

int main()
{
    std::mt19937_64 rng(7);
    std::normal_distribution<double> normal;
    const double special[] = {0.0, -0.0, std::numeric_limits<double>::infinity(), -std::numeric_limits<double>::infinity(),
                              std::numeric_limits<double>::quiet_NaN(), 1e70, -1e160, 1e300, 5e-324, 1e-200};
    long bad = 0, total = 0;
    for (int kind = 0; kind < 6; ++kind)
        for (int n = 0; n < 400000; ++n) {
            const double scale = kind == 0 ? 1e-3 : kind == 1 ? 50.0 : 1.0;
            V p[5];
            for (V &q : p) {
                double x[3];
                for (double &y : x) {
                    y = scale * normal(rng);
                    if (kind == 2) y = double(int(rng() % 5) - 2) * (rng() & 1 ? 1.0 : -1.0);
                    if (kind == 3) y = double(int(rng() % 3) - 1) + double(int(rng() % 5) - 2) * 0x1p-52;
                    if (kind == 4 && rng() % 12 == 0) y = special[rng() % 10];
                }
                q = dm::v(x[0], x[1], x[2]);
            }
            if (kind == 5) {  // slivers and short segments
                p[1] = dm::gadd(p[0], dm::gmul(p[1], rng() & 1 ? 1e-8 : 1e-6));
                p[4] = dm::gadd(p[3], dm::gmul(p[4], rng() & 1 ? 1e-9 : 1e-5));
            }
            const dm::ClosestPair x = dm::closest_segment_triangle(p[0], p[1], p[2], p[3], p[4]), y = plain(p[0], p[1], p[2], p[3], p[4]);
            ++total;
            if (!(same(x.distance, y.distance) && same(x.t, y.t) && same(x.bary.x, y.bary.x) && same(x.bary.y, y.bary.y) &&
                  same(x.bary.z, y.bary.z))) {
                if (bad++ < 5) std::printf("kind %d: %a %a against %a %a\n", kind, x.distance, x.t, y.distance, y.t);
            }
        }
    // root_less around ties.
    for (int n = 0; n < 400000; ++n) {
        const double x = std::ldexp(1.0 + (rng() >> 12) * 0x1p-52, int(rng() % 40) - 20);
        const double y = dm::double_of(dm::bits_of(x) + rng() % 40 - 20);
        ++total;
        if (dm::root_less(x, y) != (std::sqrt(x) < std::sqrt(y))) ++bad;
    }
    std::printf("%ld values, %ld mismatches\n", total, bad);
    if (!bad) std::printf("PASS\n");
    return bad != 0;
}
