// Strands that fail in the FP64 block solve (csrc/khs_block_solve.cuh) and their
// neighbours, in every layout: a pivot that is not a number, a finite pivot below
// 1e-30 and pivots that are zero are reported, a pivot just above 1e-30 is not, and every
// other strand, those that share a warp with a failing one among them, equals
// the host recurrence bit for bit.  Built and run by
// tests/test_gpu_block_solve_failures.py.
#define main layouts_match_the_host  // the recurrence and the launches of the layouts
#include "test_block_solve.cu"
#undef main

int main()
{
    enum { NOT_A_NUMBER, BELOW, ABOVE, ZERO, KINDS };
    const uint32_t S = 27, lens[] = {1, 2, 6, 7, 8, 9, 15, 33, 70};
    int bad = 0;
    for (int kind = 0; kind < KINDS; ++kind)
        for (uint32_t where : {0u, 13u, 26u}) {
            std::mt19937_64 rng(31 + kind);
            std::normal_distribution<double> normal;
            std::vector<uint32_t> first, count, fixed, order;
            uint32_t N = 0;
            for (uint32_t s = 0; s < S; ++s) {
                order.push_back(s);
                first.push_back(N);
                fixed.push_back(s % 3);
                count.push_back(lens[s % 9] + s % 3);
                N += count.back();
            }
            std::vector<double> D(36 * size_t(N)), U(36 * size_t(N)), g(6 * size_t(N)), x(6 * size_t(N), 0.0);
            for (size_t n = 0; n < N; ++n)
                for (int k = 0; k < 36; ++k) {
                    D[36 * n + k] = normal(rng) + (k % 7 == 0 ? 6.0 : 0.0);
                    U[36 * n + k] = 0.4 * normal(rng);
                }
            for (double &v : g) v = normal(rng);
            // The first free node of one strand: a diagonal block below 1e-12,
            // so that the shift is 1e-24, which its first entry takes away but
            // for the pivot wanted.
            double *B = &D[36 * size_t(first[where] + fixed[where])];
            for (int k = 0; k < 36; ++k) B[k] = kind == NOT_A_NUMBER ? std::nan("") : k % 7 == 0 ? 1.0e-13 : 0.0;
            if (kind == BELOW) B[0] = -(1.0e-24 - 9.0e-31);
            if (kind == ABOVE) B[0] = -(1.0e-24 - 2.0e-30);
            if (kind == ZERO) B[0] = -1.0e-24;
            std::vector<bool> good(S);
            bool failed = false;
            for (uint32_t s = 0; s < S; ++s) {
                const size_t n = first[s] + fixed[s];
                good[s] = solve_host(&D[36 * n], &U[36 * n], &g[6 * n], count[s] - fixed[s], &x[6 * n]);
                failed = failed || !good[s];
            }
            if (failed != (kind != ABOVE) || good[where] != (kind == ABOVE)) {
                std::printf("kind %d: the input does not do what it is for\n", kind);
                ++bad;
            }
            Arrays a;
            a.S = S;
            a.diag = device(D); a.upper = device(U); a.grad = device(g);
            a.cprime = device(D); a.dprime = device(g);
            a.sorder = device(order); a.sfirst = device(first); a.scount = device(count); a.sfixed = device(fixed);
            for (int layout = 0; layout < 3; ++layout) {
                a.dir = device(std::vector<double>(x.size(), 0.0));
                a.sc = device(std::vector<Flags>(1, Flags{0}));
                if (layout == 2) k_team<<<S, kTeam>>>(a);
                else if (layout == 1) k_five<<<(S + kStrandsPerWarp - 1) / kStrandsPerWarp, 32>>>(a);
                else k_alone<<<S, 32>>>(a);
                if (cudaDeviceSynchronize() != cudaSuccess) { std::printf("CUDA error\n"); return 1; }
                std::vector<double> got(x.size());
                Flags f;
                cudaMemcpy(got.data(), a.dir, got.size() * 8, cudaMemcpyDeviceToHost);
                cudaMemcpy(&f, a.sc, sizeof(f), cudaMemcpyDeviceToHost);
                size_t differ = 0, compared = 0;
                for (uint32_t s = 0; s < S; ++s) {
                    if (!good[s]) continue;
                    const size_t begin = 6 * size_t(first[s] + fixed[s]), end = 6 * size_t(first[s] + count[s]);
                    compared += end - begin;
                    for (size_t i = begin; i < end; ++i) differ += std::memcmp(&got[i], &x[i], 8) != 0;
                }
                std::printf("kind %d strand %u layout %d: %zu of %zu differ, failed %d / %d\n", kind, where, layout, differ, compared,
                            f.solve_failed, int(failed));
                if (differ || (f.solve_failed != 0) != failed) ++bad;
            }
        }
    if (!bad) std::printf("PASS\n");
    return bad != 0;
}
