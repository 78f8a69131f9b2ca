// The three layouts of the FP64 block solve (csrc/khs_block_solve.cuh) against the
// same recurrence on the host, entry by entry with std::fma and IEEE division,
// bit for bit: random blocks; blocks of small integers, where pivot candidates
// tie exactly; candidates that differ only below the bits the warp's pivot
// search compares first; pivots with reciprocals below the normal range; and
// a singular block, which every layout reports.  Strand lengths around the
// back substitution's ring.  Built and run by tests/test_gpu_block_solve.py.
#include "khs_block_solve.cuh"

#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

using namespace khs;

struct Flags { int solve_failed; };
struct Arrays {
    uint32_t S;
    double *diag, *upper, *cprime, *grad, *dprime, *dir;
    uint32_t *sorder, *sfirst, *scount, *sfixed;
    Flags *sc;
};

__global__ void __launch_bounds__(32) k_alone(Arrays d)
{
    __shared__ __align__(16) BackRing ring;
    solve_strand_warp(d, blockIdx.x, ring);
}
__global__ void __launch_bounds__(kTeam) k_team(Arrays d)
{
    __shared__ __align__(16) TeamShared sh;
    solve_strand_team(d, blockIdx.x, sh);
}
__global__ void __launch_bounds__(32) k_five(Arrays d) { solve_strands_five(d, kStrandsPerWarp * blockIdx.x); }

// The recurrence of one strand on the host; false when a pivot fails.
static bool solve_host(const double *D, const double *U, const double *g, uint32_t len, double *x)
{
    std::vector<double> C(36 * size_t(len)), dp(6 * size_t(len));
    for (uint32_t n = 0; n < len; ++n) {
        double a[6][13];
        for (int r = 0; r < 6; ++r) {
            for (int c = 0; c < 6; ++c) a[r][c] = D[36 * n + 6 * r + c];
            for (int c = 0; c < 6; ++c) a[r][6 + c] = n + 1 < len ? U[36 * n + 6 * r + c] : 0.0;
            a[r][12] = -g[6 * n + r];
            if (n)
                for (int q = 0; q < 6; ++q) {
                    const double u = -U[36 * (n - 1) + 6 * q + r];
                    for (int c = 0; c < 6; ++c) a[r][c] = std::fma(u, C[36 * (n - 1) + 6 * q + c], a[r][c]);
                    a[r][12] = std::fma(u, dp[6 * (n - 1) + q], a[r][12]);
                }
        }
        double most = 0.0;
        for (int r = 0; r < 6; ++r) most = std::fmax(most, std::fabs(a[r][r]));
        const double shift = std::fmax(1.0e-12 * most, 1.0e-24);
        for (int r = 0; r < 6; ++r) a[r][r] += shift;
        double ipiv[6];
        for (int col = 0; col < 6; ++col) {
            int pivot = col;
            for (int r = col + 1; r < 6; ++r)
                if (std::fabs(a[r][col]) > std::fabs(a[pivot][col])) pivot = r;
            if (!(std::fabs(a[pivot][col]) >= 1.0e-30) || !std::isfinite(a[pivot][col])) return false;
            if (pivot != col)
                for (int c = 0; c < 13; ++c) std::swap(a[col][c], a[pivot][c]);
            ipiv[col] = 1.0 / a[col][col];
            for (int r = 0; r < 6; ++r) {
                if (r == col) continue;
                const double f = -(a[r][col] * ipiv[col]);
                for (int c = col + 1; c < 13; ++c) a[r][c] = std::fma(f, a[col][c], a[r][c]);
            }
        }
        for (int r = 0; r < 6; ++r) {
            for (int c = 0; c < 6; ++c) C[36 * n + 6 * r + c] = a[r][6 + c] * ipiv[r];
            dp[6 * n + r] = a[r][12] * ipiv[r];
        }
    }
    for (uint32_t n = len; n-- > 0;)
        for (int r = 0; r < 6; ++r) {
            double v = dp[6 * n + r];
            if (n + 1 < len)
                for (int q = 0; q < 6; ++q) v = std::fma(-C[36 * n + 6 * r + q], x[6 * (n + 1) + q], v);
            x[6 * n + r] = v;
        }
    return true;
}

template<class T> static T *device(const std::vector<T> &h)
{
    T *p = nullptr;
    cudaMalloc(&p, h.size() * sizeof(T));
    cudaMemcpy(p, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice);
    return p;
}

int main()
{
    enum { RANDOM, TIES, NEAR, HUGE_PIVOT, SINGULAR, KINDS };
    const uint32_t lens[] = {1, 2, 6, 7, 8, 9, 15, 33, 70};
    int bad = 0;
    for (int kind = 0; kind < KINDS; ++kind) {
        std::mt19937_64 rng(11 + kind);
        std::normal_distribution<double> normal;
        std::vector<uint32_t> first, count, fixed, order;
        uint32_t N = 0;
        for (uint32_t s = 0; s < 27; ++s) {
            order.push_back(s);
            first.push_back(N);
            fixed.push_back(s % 3);
            count.push_back(lens[s % 9] + s % 3);
            N += count.back();
        }
        std::vector<double> D(36 * size_t(N)), U(36 * size_t(N)), g(6 * size_t(N)), x(6 * size_t(N), 0.0);
        auto entry = [&](bool diagonal) {
            double v = kind == TIES ? double(int(rng() % 5) - 2) : normal(rng);
            if (kind == NEAR) v = (rng() & 1 ? 1.0 : -1.0) * (1.0 + double(rng() % 64) * 0x1p-40);
            if (diagonal && kind != TIES && kind != NEAR) v += 6.0;
            if (kind == HUGE_PIVOT) v *= diagonal ? 0x1.3p1020 : 0x1p400;
            return v;
        };
        for (size_t n = 0; n < N; ++n)
            for (int k = 0; k < 36; ++k) {
                D[36 * n + k] = entry(k % 7 == 0);
                U[36 * n + k] = kind == HUGE_PIVOT ? 0x1p300 * normal(rng) : 0.4 * (kind == TIES ? double(int(rng() % 3) - 1) : normal(rng));
            }
        for (double &v : g) v = normal(rng);
        if (kind == SINGULAR)
            for (int k = 0; k < 36; ++k) D[36 * size_t(first[13] + fixed[13]) + k] = std::nan("");
        bool failed = false;
        for (uint32_t s = 0; s < 27; ++s) {
            const size_t n = first[s] + fixed[s];
            if (!solve_host(&D[36 * n], &U[36 * n], &g[6 * n], count[s] - fixed[s], &x[6 * n])) failed = true;
        }
        Arrays a;
        a.S = 27;
        a.diag = device(D); a.upper = device(U); a.grad = device(g);
        a.cprime = device(D); a.dprime = device(g);
        a.sorder = device(order); a.sfirst = device(first); a.scount = device(count); a.sfixed = device(fixed);
        for (int layout = 0; layout < 3; ++layout) {
            a.dir = device(std::vector<double>(x.size(), 0.0));
            a.sc = device(std::vector<Flags>(1, Flags{0}));
            if (layout == 2) k_team<<<27, kTeam>>>(a);
            else if (layout == 1) k_five<<<(27 + kStrandsPerWarp - 1) / kStrandsPerWarp, 32>>>(a);
            else k_alone<<<27, 32>>>(a);
            if (cudaDeviceSynchronize() != cudaSuccess) { std::printf("CUDA error\n"); return 1; }
            std::vector<double> got(x.size());
            Flags f;
            cudaMemcpy(got.data(), a.dir, got.size() * 8, cudaMemcpyDeviceToHost);
            cudaMemcpy(&f, a.sc, sizeof(f), cudaMemcpyDeviceToHost);
            size_t differ = 0;
            if (!failed)
                for (size_t i = 0; i < x.size(); ++i) differ += std::memcmp(&got[i], &x[i], 8) != 0;
            const bool ok = differ == 0 && (f.solve_failed != 0) == failed;
            std::printf("kind %d layout %d: %zu of %zu differ, failed %d / %d\n", kind, layout, differ, x.size(), f.solve_failed, int(failed));
            if (!ok) ++bad;
        }
    }
    if (!bad) std::printf("PASS\n");
    return bad != 0;
}
