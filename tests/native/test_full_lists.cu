// The bounded lists of the contact and CCD passes (leaf pool, FP64 pairs, CCD
// pairs) once their counters have gone past 2^32: a full list stays full.
// Four elements among forty leaves of one triangle each, through the kernels
// that ask for room (csrc/khs_engine.cu).  Built and run by
// tests/test_gpu_full_lists.py.
#include "khs_engine.cu"

#include <cstdio>
#include <vector>

using namespace khs;

template<class T> static T *device(const std::vector<T> &h)
{
    T *p = nullptr;
    cudaMalloc(&p, h.size() * sizeof(T));
    cudaMemcpy(p, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice);
    return p;
}
template<class T> static std::vector<T> host(const T *p, size_t n)
{
    std::vector<T> h(n);
    cudaMemcpy(h.data(), p, n * sizeof(T), cudaMemcpyDeviceToHost);
    return h;
}

int main()
{
    constexpr uint32_t E = 4, N = 2 * E, L = 40, kCapacity = 100;
    static_assert(L > kCacheLeaves && 2 * L <= kCapacity, "a list in the pool, room for two");
    static_assert(sizeof(Mailbox::pair_count) == sizeof(Scalars::pair_count), "the host sees the whole count");
    constexpr unsigned long long kNearly = (1ull << 32) - L;
    View v{};
    v.N = N; v.E = E; v.B = L; v.L = L; v.T = L;
    std::vector<double> q(6 * N, 0.0), zeros(6 * N, 0.0);
    std::vector<float> q32(3 * N, 0.0f), x32(6 * E, 0.0f);
    std::vector<uint32_t> ei, ej;
    for (uint32_t e = 0; e < E; ++e) {
        ei.push_back(2 * e);
        ej.push_back(2 * e + 1);
        q[6 * ej[e]] = 0x1p-10;
        q32[3 * ej[e]] = x32[6 * e + 3] = 0x1p-10f;
    }
    std::vector<float4> nodes, records;
    std::vector<double> lo, hi;
    for (uint32_t k = 0; k < L; ++k) {
        const uint32_t escape = k + 1, leaf = k << 4 | 1u;
        float escape_f, leaf_f, t_f;
        std::memcpy(&escape_f, &escape, 4); std::memcpy(&leaf_f, &leaf, 4); std::memcpy(&t_f, &k, 4);
        nodes.push_back(make_float4(-0.01f, -0.01f, -0.01f, escape_f));
        nodes.push_back(make_float4(0.01f, 0.01f, 0.01f, leaf_f));
        for (int c = 0; c < 3; ++c) {
            lo.push_back(-0.009);
            hi.push_back(0.009);
            records.push_back(make_float4(0.001f * c, 0.002f * (c == 1), 0.0f, c == 0 ? t_f : 0.0f));
        }
    }
    v.q = device(q); v.dir = device(zeros); v.q32 = device(q32); v.e32 = device(q32);
    v.ei = device(ei); v.ej = device(ej);
    v.fixed = device(std::vector<uint8_t>(N, 0)); v.econtact = device(std::vector<uint8_t>(E, 1));
    v.bnode = device(nodes); v.blo = device(lo); v.bhi = device(hi); v.tri32 = device(records);
    v.contact_pad = v.ccd_pad = View::Padding{0x1p-10, 0x1p-10f, 0x1p-10f};
    v.dhat = 1.0e-3; v.has_collider = 1;
    // Element 0 holds its list at the pool's start; the others ask for room.
    std::vector<uint32_t> slots(kCacheLeaves * E, 0);
    slots[1] = L;
    v.cache_leaf = device(slots); v.cache_x32 = device(x32);
    v.cache_n = device(std::vector<uint8_t>{kCacheBig, kCacheInvalid, kCacheInvalid, kCacheInvalid});
    v.leaf_pool = device(std::vector<uint32_t>(kCapacity, 7)); v.leaf_pool_capacity = kCapacity;
    v.near_list = device(std::vector<uint32_t>(E, 0));
    v.surv_elem = device(std::vector<uint32_t>(kCapacity, 9)); v.surv_tri = device(std::vector<uint32_t>(kCapacity, 9));
    v.surv_n = device(std::vector<uint32_t>(E, 0)); v.surv_off = device(std::vector<uint32_t>(E, 0)); v.surv_capacity = kCapacity;
    v.pair_elem = device(std::vector<uint32_t>(kCapacity, 9)); v.pair_tri = device(std::vector<uint32_t>(kCapacity, 9));
    v.pair_capacity = kCapacity;
    v.c_cand = device(std::vector<uint32_t>(E, 0)); v.c_tri = device(std::vector<uint32_t>(E, 0));
    v.c_flags = device(std::vector<uint8_t>(E, 0)); v.c_gap = device(std::vector<double>(E, 0.0));
    v.c_t = device(std::vector<double>(E, 0.0)); v.c_dist = device(std::vector<double>(E, 0.0));
    v.c_bary = device(std::vector<double>(3 * E, 0.0)); v.e_co = device(std::vector<double>(E, 0.0));
    int bad = 0;
    auto check = [&](bool ok, const char *what) {
        if (!ok) { std::printf("FAIL: %s\n", what); ++bad; }
    };
    auto all = [](const std::vector<uint32_t> &x, uint32_t value) { return std::count(x.begin(), x.end(), value) == long(x.size()); };
    auto scalars = [&](Scalars s) { v.sc = device(std::vector<Scalars>(1, s)); };

    // The leaf pool: elements 1 to 3 find it full.
    Scalars s{};
    s.pool_used = kNearly;
    scalars(s);
    k_contact_filter<<<1, kBlock>>>(v, v.q, 0);
    check(cudaDeviceSynchronize() == cudaSuccess, "k_contact_filter");
    check(all(host(v.leaf_pool, kCapacity), 7), "lists in use are left alone");
    check(host(v.cache_n, E) == std::vector<uint8_t>({kCacheBig, kCacheInvalid, kCacheInvalid, kCacheInvalid}), "no room, no list");
    const std::vector<uint32_t> held = host(v.surv_n, E);
    check(held[1] == kSurvOverflow && held[2] == kSurvOverflow && held[3] == kSurvOverflow, "elements without a list are searched");
    check(host(v.sc, 1)[0].pool_used > kNearly, "the count goes on");

    // The FP64 pairs: every element has a list of forty leaves and finds the
    // pool full.
    std::vector<uint32_t> everyone(kCacheLeaves * E, 0);
    for (uint32_t e = 0; e < E; ++e) everyone[kCacheLeaves * e + 1] = L;
    v.cache_leaf = device(everyone);
    v.cache_n = device(std::vector<uint8_t>(E, kCacheBig));
    std::vector<uint32_t> order(kCapacity, 0);
    for (uint32_t k = 0; k < L; ++k) order[k] = k;
    v.leaf_pool = device(order);
    v.near_list = device(std::vector<uint32_t>{3, 2, 1, 0});
    s = Scalars{};
    s.surv_count = kNearly;
    s.wide_count = E;
    scalars(s);
    k_contact_near<false><<<2, kBlock>>>(v);
    check(cudaDeviceSynchronize() == cudaSuccess, "k_contact_near");
    check(all(host(v.surv_n, E), kSurvOverflow), "no room, no pairs");
    check(all(host(v.c_cand, E), L), "every candidate counted");
    check(all(host(v.surv_elem, kCapacity), 9) && all(host(v.surv_tri, kCapacity), 9), "pairs in use are left alone");

    // The CCD pairs: the list is reported as overfull.
    s = Scalars{};
    s.pair_count = kNearly;
    s.ccd_near = E;
    scalars(s);
    k_ccd_near<false><<<2, kBlock>>>(v);
    check(cudaDeviceSynchronize() == cudaSuccess, "k_ccd_near");
    check(host(v.sc, 1)[0].pair_count == kNearly + E * L, "every pair counted");
    check(all(host(v.pair_elem, kCapacity), 9) && all(host(v.pair_tri, kCapacity), 9), "listed pairs are left alone");

    // And with room, ranges up to the last entry.
    s = Scalars{};
    s.surv_count = kCapacity - L;
    s.wide_count = 1;
    scalars(s);
    k_contact_near<false><<<2, kBlock>>>(v);
    check(cudaDeviceSynchronize() == cudaSuccess, "k_contact_near with room");
    check(host(v.surv_n, E)[0] == L && host(v.surv_off, E)[0] == kCapacity - L, "the last range is handed out");
    const std::vector<uint32_t> tri = host(v.surv_tri, kCapacity);
    bool listed = true;
    for (uint32_t k = 0; k < L; ++k) listed = listed && tri[kCapacity - L + k] == k;
    check(listed, "in traversal order");
    if (!bad) std::printf("PASS\n");
    return bad != 0;
}
