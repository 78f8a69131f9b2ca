// The two-thread form of an element's gradient and Hessian (element_end and the
// mixed block from both ends' rows) against the one-thread form, bit for bit:
// built without contraction, so both round every product and sum alike.
// Random states, straight and nearly folded elements, weights from thin to
// thick hair.  Built and run by tests/test_element_ends.py.
#include "khs_device_math.cuh"

#include <cstdio>
#include <cstring>
#include <random>

using namespace khs;

int main()
{
    std::mt19937_64 rng(5);
    std::normal_distribution<double> normal;
    int bad = 0;
    for (int trial = 0; trial < 4000; ++trial) {
        const double bend = trial % 4 == 0 ? 0.0 : trial % 4 == 1 ? 1.0e-6 : trial % 4 == 2 ? 0.7 : 3.0;
        const dm::V ri = dm::v(normal(rng), normal(rng), normal(rng));
        const dm::V rj = ri + dm::v(bend * normal(rng), bend * normal(rng), bend * normal(rng));
        const double L0 = 0.001 * (1.0 + 30.0 * double(trial % 7));
        const dm::V xi = dm::v(normal(rng), normal(rng), normal(rng));
        const dm::V xj = xi + dm::v(L0 * normal(rng), L0 * normal(rng), L0 * normal(rng));
        dm::M Ri, Rj, Jli, Jlj;
        const double unit[9] = {1, 0, 0, 0, 1, 0, 0, 0, 1};
        dm::rotation_and_jacobian(ri, unit, Ri, &Jli);
        dm::rotation_and_jacobian(rj, unit, Rj, &Jlj);
        const dm::V gamma0 = dm::v(0.01 * normal(rng), 0.01 * normal(rng), 1.0), kappa0 = dm::v(normal(rng), normal(rng), normal(rng));
        const dm::Weights w = dm::strain_weights(1.0e-5 * (1 + trial % 50), 4.0e9, 0.35, 0.9);
        const double invL = 1.0 / L0;
        double eps[6], gi[6], gj[6], Hii[36], Hjj[36], Hij[36];
        dm::ElementJacobian J;
        dm::element_strain_inv(Ri, Rj, xi, xj, invL, gamma0, kappa0, eps, &J, &Jli, &Jlj);
        dm::element_gradient(J, eps, w, L0, gi, gj);
        dm::element_hessian(J, w, L0, Hii, Hjj, Hij);
        double e2[6], g[2][6], H[2][36], mixed[36];
        dm::V t;
        dm::M S, K, A2, S2[2], Kk[2], x[2], WS[2], WK[2];
        dm::element_strain_shared(Ri, Rj, xi, xj, invL, gamma0, kappa0, e2, t, S, &K);
        for (int k = 0; k < 9; ++k) A2.m[k] = S.m[k] * invL;
        for (int right = 0; right < 2; ++right) {
            dm::element_strain_end(right ? Rj : Ri, Ri, right ? Jlj : Jli, t, K, right ? invL : -invL, S2[right], Kk[right]);
            dm::element_end(right, A2, S2[right], Kk[right], e2, w, L0, g[right], H[right], x[right], WS[right], WK[right]);
        }
        for (int r = 0; r < 3; ++r)
            for (int c = 0; c < 3; ++c) {
                mixed[6 * r + c] = -H[0][6 * r + c];
                mixed[6 * r + 3 + c] = -x[1].m[3 * r + c];
                mixed[6 * (3 + r) + c] = x[0].m[3 * c + r];
                mixed[6 * (3 + r) + 3 + c] = dm::dot3w(S2[0], r, WS[1], c) + dm::dot3w(Kk[0], r, WK[1], c);
            }
        const bool same = !std::memcmp(eps, e2, sizeof eps) && !std::memcmp(gi, g[0], sizeof gi) && !std::memcmp(gj, g[1], sizeof gj) &&
                          !std::memcmp(Hii, H[0], sizeof Hii) && !std::memcmp(Hjj, H[1], sizeof Hjj) && !std::memcmp(Hij, mixed, sizeof Hij);
        if (!same && ++bad < 5) std::printf("trial %d differs\n", trial);
    }
    std::printf(bad ? "%d differ\n" : "PASS\n", bad);
    return bad != 0;
}
