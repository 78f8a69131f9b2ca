// Kernels that share one result between threads against the form that one
// thread takes, bit for bit, on the device's own contraction of sums:
// * k_elem_ends (two threads an element) against k_elem_eval, gradient,
//   Hessian blocks and energy, and the energy form's energy against both: the
//   line search compares energies of either form, and the launch changes from
//   one kernel to the other with the number of elements;
// * k_root_frames (three lanes a strand, divisions by a shared reciprocal)
//   against the walk by one thread on the host, which divides.
// Compiled as the library is.  Built and run by tests/test_gpu_kernel_forms.py.
#include "khs_engine.cu"

#include <cstdio>
#include <random>
#include <vector>

using namespace khs;

template<class T> static T *device(const std::vector<T> &h)
{
    T *p = nullptr;
    cudaMalloc(&p, std::max<size_t>(1, h.size()) * sizeof(T));
    cudaMemcpy(p, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice);
    return p;
}
static std::vector<double> host(const double *p, size_t n)
{
    std::vector<double> h(n);
    cudaMemcpy(h.data(), p, n * 8, cudaMemcpyDeviceToHost);
    return h;
}
static size_t differing(const std::vector<double> &a, const std::vector<double> &b)
{
    size_t n = 0;
    for (size_t k = 0; k < a.size(); ++k) n += std::memcmp(&a[k], &b[k], 8) != 0;
    return n;
}

// One strand of E + 1 nodes, the first two fixed and one in the middle.
static bool elements(uint32_t E, unsigned seed)
{
    const uint32_t N = E + 1;
    std::mt19937_64 rng(seed);
    std::normal_distribution<double> normal;
    View v{};
    v.N = N; v.E = E;
    std::vector<double> q, rot, jl, L0, invL, gamma0, kappa0;
    std::vector<uint8_t> fixed(N, 0);
    std::vector<uint32_t> ei, ej;
    fixed[0] = fixed[1] = fixed[N / 2] = 1;
    const double unit[9] = {1, 0, 0, 0, 1, 0, 0, 0, 1};
    dm::V x = dm::v(0, 0, 0), u = dm::v(normal(rng), normal(rng), normal(rng));
    for (uint32_t n = 0; n < N; ++n) {
        const double bend = n % 4 == 0 ? 0.0 : n % 4 == 1 ? 1.0e-6 : n % 4 == 2 ? 0.3 : 3.0;
        u = u + dm::v(bend * normal(rng), bend * normal(rng), bend * normal(rng));
        x = x + dm::v(0.002 * normal(rng), 0.002 * normal(rng), 0.002 * normal(rng));
        dm::M R, J;
        dm::rotation_and_jacobian(u, unit, R, &J);
        for (double value : {x.x, x.y, x.z, u.x, u.y, u.z}) q.push_back(value);
        rot.insert(rot.end(), R.m, R.m + 9);
        jl.insert(jl.end(), J.m, J.m + 9);
    }
    for (uint32_t e = 0; e < E; ++e) {
        ei.push_back(e); ej.push_back(e + 1);
        L0.push_back(0.002 * (1.0 + 0.1 * normal(rng)));
        invL.push_back(1.0 / L0.back());
        for (int k = 0; k < 3; ++k) { gamma0.push_back(k == 2 ? 1.0 : 0.01 * normal(rng)); kappa0.push_back(normal(rng)); }
    }
    v.q = device(q); v.rot = device(rot); v.jl = device(jl);
    v.fixed = device(fixed); v.ei = device(ei); v.ej = device(ej);
    v.L0 = device(L0); v.invL = device(invL); v.gamma0 = device(gamma0); v.kappa0 = device(kappa0);
    v.w = dm::strain_weights(4.0e-5, 3.0e9, 0.25, 0.9);
    struct Out { std::vector<double> gi, gj, hi, hj, upper, energy; };
    auto run = [&](int form) {
        auto blank = [&](size_t n) { return device(std::vector<double>(n, 0.0)); };
        v.as_i_g = blank(6 * N); v.as_j_g = blank(6 * N);
        v.as_i_h = blank(36 * N); v.as_j_h = blank(36 * N); v.upper = blank(36 * N);
        v.e_el = blank(E);
        if (form == 2) k_elem_ends<<<grid_for(E, kEndElements), kEndBlock>>>(v);
        else k_elem_eval<<<grid_for(E, kEvalBlock), kEvalBlock>>>(v, form);
        if (cudaDeviceSynchronize() != cudaSuccess) std::printf("CUDA error\n");
        Out o{host(v.as_i_g, 6 * N), host(v.as_j_g, 6 * N), host(v.as_i_h, 36 * N), host(v.as_j_h, 36 * N), host(v.upper, 36 * N),
              host(v.e_el, E)};
        for (double *p : {v.as_i_g, v.as_j_g, v.as_i_h, v.as_j_h, v.upper, v.e_el}) cudaFree(p);
        return o;
    };
    const Out energy = run(0), one = run(1), two = run(2);
    const size_t d[6] = {differing(one.gi, two.gi) + differing(one.gj, two.gj), differing(one.hi, two.hi), differing(one.hj, two.hj),
                         differing(one.upper, two.upper), differing(one.energy, two.energy), differing(one.energy, energy.energy)};
    std::printf("%u elements: gradient %zu, left %zu, right %zu, coupling %zu, energy %zu, energy form %zu differ\n", E, d[0], d[1],
                d[2], d[3], d[4], d[5]);
    size_t sum = 0;
    for (size_t k : d) sum += k;
    double largest = 0.0;
    for (double x : one.hi) largest = std::fmax(largest, std::fabs(x));
    return sum == 0 && (E < 4 || largest > 0.0);
}

// Strands of 2 to 90 points, some with straight runs, kinks and reversals.
static bool frames(uint32_t S, unsigned seed)
{
    std::mt19937_64 rng(seed);
    std::normal_distribution<double> normal;
    std::uniform_real_distribution<double> uniform;
    std::vector<double> points, ref, t;
    std::vector<uint32_t> left, right, strand, first, count, order;
    std::vector<dm::V> x;
    std::vector<dm::M> rest;
    for (uint32_t s = 0; s < S; ++s) {
        first.push_back(uint32_t(x.size()));
        count.push_back(s % 11 == 0 ? 2 : 2 + uint32_t(uniform(rng) * 89));
        dm::V at = dm::v(normal(rng), normal(rng), normal(rng));
        dm::V dir = dm::gunit(dm::v(normal(rng), normal(rng), normal(rng)));
        if (s % 5 == 2) dir = dm::v(1, 0, 0);
        const double bend = s % 4 == 0 ? 1e-9 : s % 4 == 1 ? 0.05 : s % 4 == 2 ? 0.5 : 2.0;
        for (uint32_t k = 0; k < count[s]; ++k) {
            const uint32_t n = uint32_t(x.size());
            left.push_back(n); right.push_back(n); t.push_back(0.0); strand.push_back(s);
            x.push_back(at);
            for (double value : {at.x, at.y, at.z}) points.push_back(value);
            rest.push_back(dm::frame_from_tangent(dm::gunit(dm::v(normal(rng), normal(rng), normal(rng))),
                                                  s % 5 == 2 && k == 0 ? dm::v(1, 0, 0) : dm::v(normal(rng), normal(rng), normal(rng))));
            ref.insert(ref.end(), rest.back().m, rest.back().m + 9);
            if (s % 7 == 3 && k % 9 == 4) dir = dir * -1.0;
            else if (!(s % 5 == 1 && k % 3 == 0)) dir = dm::gunit(dir + dm::v(bend * normal(rng), bend * normal(rng), bend * normal(rng)));
            at = at + dir * (0.002 * (0.5 + uniform(rng)));
        }
        order.push_back(s);
    }
    std::stable_sort(order.begin(), order.end(), [&](uint32_t a, uint32_t b) { return count[a] > count[b]; });
    const uint32_t N = uint32_t(x.size());
    RootArgs a{};
    a.N = N; a.S = S; a.P = N;
    a.points = device(points); a.bind_l = device(left); a.bind_r = device(right); a.bind_t = device(t);
    a.node_strand = device(strand); a.sfirst = device(first); a.scount = device(count); a.sorder = device(order);
    a.ref = device(ref);
    auto blank = [&](size_t n) { return device(std::vector<double>(n, 0.0)); };
    a.x = blank(3 * N); a.tangent = blank(3 * N); a.frame = blank(9 * N); a.rot = blank(3 * N);
    a.bad = device(std::vector<uint32_t>(1, 0));
    k_root_tangents<<<grid_for(N), kBlock>>>(a);
    k_root_transport<<<grid_for(N), kBlock>>>(a);
    k_root_frames<<<grid_for(S, kRootStrands), 32>>>(a);
    if (cudaDeviceSynchronize() != cudaSuccess) std::printf("CUDA error\n");
    const std::vector<double> tangent = host(a.tangent, 3 * N), frame = host(a.frame, 9 * N);
    std::vector<double> want_t, want_f;
    for (uint32_t s = 0; s < S; ++s) {
        dm::M f;
        dm::V before;
        for (uint32_t k = 0; k < count[s]; ++k) {
            const uint32_t n = first[s] + k;
            const dm::V d = k == 0 ? dm::gsub(x[n + 1], x[n]) : k + 1 == count[s] ? dm::gsub(x[n], x[n - 1]) : dm::gsub(x[n + 1], x[n - 1]);
            const dm::V tan = dm::gunit(d);
            const dm::V hint = k == 0 ? dm::v(rest[n].m[0], rest[n].m[3], rest[n].m[6])
                                      : dm::parallel_transport(dm::v(f.m[0], f.m[3], f.m[6]), before, tan);
            f = dm::frame_from_tangent(tan, hint);
            before = tan;
            for (double value : {tan.x, tan.y, tan.z}) want_t.push_back(value);
            want_f.insert(want_f.end(), f.m, f.m + 9);
        }
    }
    const size_t dt = differing(tangent, want_t), df = differing(frame, want_f);
    std::printf("%u strands, %u nodes: tangents %zu, frames %zu differ\n", S, N, dt, df);
    return dt == 0 && df == 0;
}

int main()
{
    bool ok = true;
    for (uint32_t E : {1u, 31u, 32u, 33u, 64u, 65u, 1000u, 64u * 152u, 64u * 152u + 1u}) ok = elements(E, 3 + E) && ok;
    for (uint32_t S : {1u, 9u, 10u, 11u, 800u}) ok = frames(S, 17 + S) && ok;
    std::printf(ok ? "PASS\n" : "FAIL\n");
    return ok ? 0 : 1;
}
