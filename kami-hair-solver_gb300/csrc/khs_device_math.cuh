// Per-element and per-contact FP64 math of the GB300 solver.
//
// Everything here is __host__ __device__ so the same source runs in the
// sm_103a kernels and in host-side unit tests.  It evaluates the Cosserat rod
// strains of the reference (src/cuda_backend.cu:234-245), their energy, the
// gradient and the Gauss-Newton Hessian blocks (src/cuda_backend.cu:899-919)
// with closed-form derivatives of the SO(3) exponential (left Jacobian)
// and of the regularised Cayley map instead of the reference's Dual<12>
// forward-mode AD, plus the log-barrier contact term
// (src/cuda_backend.cu:255-265, 920-938) and the device segment-triangle
// distance (src/cuda_backend.cu:200-223).
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#if defined(__CUDACC__)
#define KHS_HD __host__ __device__ __forceinline__
#define KHS_HD_SLOW inline __host__ __device__ __noinline__  // a rare path, kept out of line
#else
#define KHS_HD inline
#define KHS_HD_SLOW inline
#endif

namespace khs {
namespace dm {

constexpr double kPi = 3.1415926535897932384626433832795;

struct V {
    double x, y, z;
};

KHS_HD V v(double x, double y, double z) { V r; r.x = x; r.y = y; r.z = z; return r; }
KHS_HD V operator+(V a, V b) { return v(a.x + b.x, a.y + b.y, a.z + b.z); }
KHS_HD V operator-(V a, V b) { return v(a.x - b.x, a.y - b.y, a.z - b.z); }
KHS_HD V operator*(V a, double s) { return v(a.x * s, a.y * s, a.z * s); }
KHS_HD double dot(V a, V b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
KHS_HD V cross(V a, V b) { return v(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x); }
KHS_HD double norm(V a) { return sqrt(dot(a, a)); }
KHS_HD V vmin(V a, V b) { return v(fmin(a.x, b.x), fmin(a.y, b.y), fmin(a.z, b.z)); }
KHS_HD V vmax(V a, V b) { return v(fmax(a.x, b.x), fmax(a.y, b.y), fmax(a.z, b.z)); }
KHS_HD double at(V a, int k) { return k == 0 ? a.x : (k == 1 ? a.y : a.z); }

// 3x3 row-major.
struct M {
    double m[9];
};

KHS_HD M mmul(const M &a, const M &b)
{
    M r;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) r.m[3 * i + j] = a.m[3 * i] * b.m[j] + a.m[3 * i + 1] * b.m[3 + j] + a.m[3 * i + 2] * b.m[6 + j];
    return r;
}
// a^T b
KHS_HD M mtmul(const M &a, const M &b)
{
    M r;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) r.m[3 * i + j] = a.m[i] * b.m[j] + a.m[3 + i] * b.m[3 + j] + a.m[6 + i] * b.m[6 + j];
    return r;
}
// a^T x
KHS_HD V mtvec(const M &a, V x)
{
    return v(a.m[0] * x.x + a.m[3] * x.y + a.m[6] * x.z, a.m[1] * x.x + a.m[4] * x.y + a.m[7] * x.z,
             a.m[2] * x.x + a.m[5] * x.y + a.m[8] * x.z);
}
KHS_HD V mvec(const M &a, V x)
{
    return v(a.m[0] * x.x + a.m[1] * x.y + a.m[2] * x.z, a.m[3] * x.x + a.m[4] * x.y + a.m[5] * x.z,
             a.m[6] * x.x + a.m[7] * x.y + a.m[8] * x.z);
}

#if defined(__CUDA_ARCH__)
KHS_HD uint64_t bits_of(double x) { return uint64_t(__double_as_longlong(x)); }
KHS_HD double double_of(uint64_t b) { return __longlong_as_double((long long)b); }
KHS_HD uint32_t bits_of(float x) { return __float_as_uint(x); }
KHS_HD float float_of(uint32_t b) { return __uint_as_float(b); }
#else
KHS_HD uint64_t bits_of(double x) { uint64_t b; std::memcpy(&b, &x, 8); return b; }
KHS_HD double double_of(uint64_t b) { double x; std::memcpy(&x, &b, 8); return x; }
KHS_HD uint32_t bits_of(float x) { uint32_t b; std::memcpy(&b, &x, 4); return b; }
KHS_HD float float_of(uint32_t b) { float x; std::memcpy(&x, &b, 4); return x; }
#endif

// ---- correctly rounded reciprocal on the integer pipes -----------------
//
// 1/x rounded to nearest, computed without FP64 instructions: on GB300 one
// FP64 warp instruction occupies a sub-partition's pipe for ~64 cycles, and a
// reciprocal is on the chain of every pivot step of the block solve.
// For x = (-1)^s * M * 2^(E-1075) with M the 53-bit significand,
// 1/x = (-1)^s * T * 2^(970-E) with T = 2^105 / M in (2^52, 2^53]:
// * seed: an FP32 reciprocal of the top 24 bits of M as the integer
//   t ~ 2^23 * 2^52 / M, so T0 = 2^30 t; its relative error e = 1 - T0 / T
//   is below 2^-20 (one ulp of the seed, the bits of M cut off, the rounding
//   of t, and three further ulps of the seed to spare);
// * residual: d = 2^75 - t M = 2^75 e, exact in 64 bits modulo 2^64 (2^75
//   vanishes, |d| < 2^55), so one 24 x 53 bit product;
// * Q = T0 (1 + e + e^2), rounded to an integer: e carried to 2^-62, e^2
//   from the top 27 bits of d; with the cubic term left out the sum is within
//   0.01 of T before the rounding, so Q is the nearest integer or next to it;
// * the remainder R = 2^105 - Q M (exact modulo 2^64, |R| < 2^53) moves Q by
//   one where |R| > M / 2.  No ties: M is odd times a power of two and T
//   has more bits than a midpoint, or M = 2^52 and R = 0.
// The steps are chosen for latency: 156 cycles of dependent instructions
// (the FP64 reciprocal takes 352, the 128-bit form this replaces 382).  Reciprocals below the normal range (|x| >= 2^1022) are rounded from
// floor(T) and its remainder to nearest-even on a branch of their own.
// The result equals the IEEE division 1.0 / x for every finite normal x
// (against 1.0 / x on the host, tests/native/test_recip.cpp); zero,
// subnormal and non-finite inputs give an unspecified bit pattern (the block
// solve fails such pivots before using the result).
#if defined(__CUDA_ARCH__)
KHS_HD int32_t smulhi32(int32_t a, int32_t b) { return __mulhi(a, b); }
KHS_HD float recip_seed(float m)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(m));
    return r;
}
#else
KHS_HD int32_t smulhi32(int32_t a, int32_t b) { return int32_t((int64_t(a) * b) >> 32); }
// Host seed: the correctly rounded float reciprocal (tests may substitute a
// perturbed one through KHS_RECIP_SEED_HOST).
#ifndef KHS_RECIP_SEED_HOST
#define KHS_RECIP_SEED_HOST(m) (1.0f / (m))
#endif
KHS_HD float recip_seed(float m) { return KHS_RECIP_SEED_HOST(m); }
#endif

// The reciprocal where it is normal too (2^-1022 <= |x| < 2^1022), without
// a branch.  Q and nR: the rounded T and minus its remainder.
KHS_HD double recip_normal(double x, uint64_t &Q, int64_t &nR)
{
    const uint64_t b = bits_of(x);
    const uint32_t hi = uint32_t(b >> 32), mlo = uint32_t(b);
    const uint32_t E = (hi >> 20) & 0x7ff, mhi = (hi & 0xfffffu) | 0x100000u;
    const uint64_t M = (uint64_t(mhi) << 32) | mlo, half = M >> 1;
    const float seed = recip_seed(float_of((127u << 23) | ((hi << 3 | mlo >> 29) & 0x7fffffu)));
    // 2^23 * seed as an integer: the bits of 1 + seed count it from those of 1.
    const uint32_t t = bits_of(1.0f + seed) - 0x3f800000u;
    // -d, and s = 2^62 (e + e^2) from it.
    const uint64_t tm = uint64_t(t) * mlo;
    const int64_t nd = int64_t((uint64_t(uint32_t(tm >> 32) + t * mhi) << 32) | uint32_t(tm));
    const int32_t dh = int32_t(nd >> 28);
    const int64_t s = int64_t(smulhi32(dh, dh)) - (nd >> 13);
    // Q = round(2^30 t + t s / 2^32), the low and high words of s apart.
    const uint64_t low = uint64_t(t) * uint32_t(s) + 0x80000000u;
    Q = (uint64_t(t) << 30) + uint64_t(int64_t(int32_t(t)) * int32_t(s >> 32)) + (low >> 32);
    nR = int64_t(Q * M);
    // Q counts its implicit bit into the exponent field (Q = 2^53 as well).
    const uint64_t out = (b & 0x8000000000000000ull) | ((uint64_t(2044 - E) << 52) + Q);
    const uint64_t above = out + 1, below = out - 1;
    return double_of(nR < -int64_t(half) ? above : (nR > int64_t(half) ? below : out));
}
KHS_HD double recip_normal(double x)
{
    uint64_t Q;
    int64_t nR;
    return recip_normal(x, Q, nR);
}

KHS_HD double recip_rn(double x)
{
    uint64_t F;
    int64_t nR;
    const double normal = recip_normal(x, F, nR);
    const uint64_t b = bits_of(x);
    const int E = int((b >> 52) & 0x7ff);
    if (E < 2045) return normal;
    // floor(T) and the remainder below M, then the subnormal's bits.
    const int64_t M = int64_t((b & 0xfffffffffffffull) | (1ull << 52));
    int64_t R = -nR;
    if (R < 0) { --F; R += M; }
    if (R >= M) { ++F; R -= M; }
    const int k = E - 2044;
    const uint64_t mant = F >> k;
    const uint64_t dropped = F & ((1ull << k) - 1), mid = 1ull << (k - 1);
    const bool up = dropped > mid || (dropped == mid && (R > 0 || (mant & 1)));
    return double_of((b & 0x8000000000000000ull) | (mant + uint64_t(up)));
}

// 1 / x with the integer-pipe reciprocal where it is exact and the division
// elsewhere (zero, subnormal, not finite, a result below the normal range).
KHS_HD double recip_any(double x)
{
#if defined(__CUDA_ARCH__)
    const uint32_t E = uint32_t(bits_of(x) >> 52) & 0x7ffu;
    return E - 1u < 2044u ? recip_normal(x) : 1.0 / x;
#else
    return 1.0 / x;
#endif
}

// Rotation R = exp([u]x) Ref with the reference's Rodrigues coefficients and
// small-angle Taylor branch below theta^2 = 1e-10 (cuda_backend.cu:130-136).
// Also returns the left Jacobian Jl(u), defined by
// exp(u + du) = exp([Jl du]x) exp(u) + O(du^2), as I + p W + r W^2 with
// p = 2 sin^2(t/2) / t^2 (cancellation-free form of (1 - cos t) / t^2) and
// r = (t - sin t) / t^3, both from their Taylor series below t^2 = 1e-4.
KHS_HD void rotation_and_jacobian(V u, const double *ref, M &R, M *Jl)
{
    const double t2 = dot(u, u);
    double a, b;
    double s, t = 0.0, it = 0.0;
    if (t2 < 1.0e-10) {
        a = 1.0 - t2 / 6.0 + t2 * t2 / 120.0;
        b = 0.5 - t2 / 24.0 + t2 * t2 / 720.0;
        s = 0.0;
    } else {
        // Half-angle form: one sincos, and 1 - cos t = 2 sin^2(t/2) without
        // cancellation (it is also the left Jacobian's coefficient p).
        t = sqrt(t2);
        it = recip_any(t);
        double sh, ch;
        sincos(0.5 * t, &sh, &ch);
        s = 2.0 * sh * ch;
        a = s * it;
        b = 2.0 * sh * sh * (it * it);
    }
    // E = I + a W + b W^2 with W = [u]x.
    const double wx = u.x, wy = u.y, wz = u.z;
    const double w2[9] = {-(wy * wy + wz * wz), wx * wy, wx * wz,
                          wx * wy, -(wx * wx + wz * wz), wy * wz,
                          wx * wz, wy * wz, -(wx * wx + wy * wy)};
    M E;
    E.m[0] = 1.0 + b * w2[0]; E.m[1] = -a * wz + b * w2[1]; E.m[2] = a * wy + b * w2[2];
    E.m[3] = a * wz + b * w2[3]; E.m[4] = 1.0 + b * w2[4]; E.m[5] = -a * wx + b * w2[5];
    E.m[6] = -a * wy + b * w2[6]; E.m[7] = a * wx + b * w2[7]; E.m[8] = 1.0 + b * w2[8];
    M Rf;
#pragma unroll
    for (int k = 0; k < 9; ++k) Rf.m[k] = ref[k];
    R = mmul(E, Rf);
    if (Jl) {
        double p, r;  // Jl = I + p W + r W^2
        if (t2 < 1.0e-4) {
            p = 0.5 - t2 / 24.0 + t2 * t2 / 720.0 - t2 * t2 * t2 / 40320.0;
            r = 1.0 / 6.0 - t2 / 120.0 + t2 * t2 / 5040.0 - t2 * t2 * t2 / 362880.0;
        } else {
            p = b;
            r = (t - s) * (it * it * it);
        }
        M &J = *Jl;
        J.m[0] = 1.0 + r * w2[0]; J.m[1] = -p * wz + r * w2[1]; J.m[2] = p * wy + r * w2[2];
        J.m[3] = p * wz + r * w2[3]; J.m[4] = 1.0 + r * w2[4]; J.m[5] = -p * wx + r * w2[5];
        J.m[6] = -p * wy + r * w2[6]; J.m[7] = p * wx + r * w2[7]; J.m[8] = 1.0 + r * w2[8];
    }
}

// Material weights of the six strains (cuda_backend.cu:905-907):
// shear, shear, stretch, bend, bend, twist.
struct Weights {
    double w[6];
};

KHS_HD Weights strain_weights(double radius, double young, double poisson, double shear_correction)
{
    const double area = kPi * radius * radius;
    const double inertia = kPi * radius * radius * radius * radius / 4.0;
    const double G = young / (2.0 * (1.0 + poisson));
    Weights r;
    r.w[0] = shear_correction * G * area;
    r.w[1] = r.w[0];
    r.w[2] = young * area;
    r.w[3] = young * inertia;
    r.w[4] = r.w[3];
    r.w[5] = 2.0 * G * inertia;
    return r;
}

// Strain of one element and, optionally, its Jacobian.
//   gamma = 0.5 (Ri^T + Rj^T) t - gamma0,    t = (xj - xi) / L0
//   kappa = cay(Ri^T Rj) / L0 - kappa0
// Jacobian (per 3x3 block; [.]x = cross-product matrix):
//   d gamma / d xj = -d gamma / d xi = A = 0.5 (Ri^T + Rj^T) / L0
//   d gamma / d ui = 0.5 Ri^T [t]x Jl(ui),  d gamma / d uj = 0.5 Rj^T [t]x Jl(uj)
//   d kappa / d uj = -d kappa / d ui|_(Jl(ui) -> Jl(uj)) = K Ri^T Jl(uj) / L0
//   with K = ((tr Q) I - Q) / s + 2 c c^T / s^2, Q = Ri^T Rj, c = axial(Q),
//   s = 1 + (tr Q - 1) / 2 + 1e-12 (differential of the regularised Cayley
//   map along dQ = [w]x Q).
// The Jacobian blocks, A, S and T with the factors of a half left out: a
// product with a power of two is exact, so the sums that use them take it up
// in their other factor without a change of rounding (A2 = 2 A, S2 = 2 d gamma
// / d u).
struct ElementJacobian {
    M A2, S2i, S2j, Kki, Kkj;
};

// What both ends of an element need of its strain (invL = 1 / L0): t, S = Ri^T
// + Rj^T and, with a Jacobian, K.
KHS_HD void element_strain_shared(const M &Ri, const M &Rj, V xi, V xj, double invL, V gamma0, V kappa0, double eps[6], V &t,
                                  M &S, M *K)
{
    t = (xj - xi) * invL;
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) S.m[3 * r + c] = Ri.m[3 * c + r] + Rj.m[3 * c + r];
    const V shear = mvec(S, t) * 0.5;
    const M Q = mtmul(Ri, Rj);
    const V ax2 = v(Q.m[7] - Q.m[5], Q.m[2] - Q.m[6], Q.m[3] - Q.m[1]);  // 2 axial(Q)
    const double trQ = Q.m[0] + Q.m[4] + Q.m[8];
    const double s = 1.0 + (trQ - 1.0) * 0.5 + 1.0e-12;
    const double is = recip_any(s);
    eps[0] = shear.x - gamma0.x;
    eps[1] = shear.y - gamma0.y;
    eps[2] = shear.z - gamma0.z;
    eps[3] = ax2.x * is * invL - kappa0.x;
    eps[4] = ax2.y * is * invL - kappa0.y;
    eps[5] = ax2.z * is * invL - kappa0.z;
    if (!K) return;
    // K = ((tr Q) I - Q) / s + 2 c c^T / s^2 with c = ax2 / 2
    const double is2 = 0.5 * is * is;
    const double axv[3] = {ax2.x, ax2.y, ax2.z};
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) K->m[3 * r + c] = ((r == c ? trQ : 0.0) - Q.m[3 * r + c]) * is + is2 * axv[r] * axv[c];
}

// The Jacobian blocks of one end, with its rotation R and left Jacobian Jl
// (scale: invL, negative for node i).
KHS_HD void element_strain_end(const M &R, const M &Ri, const M &Jl, V t, const M &K, double scale, M &S2, M &Kk)
{
    M TJ;  // [t]x Jl: column k = t x Jl_col(k)
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const V c = cross(t, v(Jl.m[k], Jl.m[3 + k], Jl.m[6 + k]));
        TJ.m[k] = c.x; TJ.m[3 + k] = c.y; TJ.m[6 + k] = c.z;
    }
    S2 = mtmul(R, TJ);
    Kk = mmul(K, mtmul(Ri, Jl));
#pragma unroll
    for (int k = 0; k < 9; ++k) Kk.m[k] *= scale;
}

KHS_HD void element_strain_inv(const M &Ri, const M &Rj, V xi, V xj, double invL, V gamma0, V kappa0, double eps[6],
                               ElementJacobian *J, const M *Jli, const M *Jlj)
{
    V t;
    M S, K;
    element_strain_shared(Ri, Rj, xi, xj, invL, gamma0, kappa0, eps, t, S, J ? &K : nullptr);
    if (!J) return;
#pragma unroll
    for (int k = 0; k < 9; ++k) J->A2.m[k] = S.m[k] * invL;
    element_strain_end(Ri, Ri, *Jli, t, K, -invL, J->S2i, J->Kki);
    element_strain_end(Rj, Ri, *Jlj, t, K, invL, J->S2j, J->Kkj);
}

KHS_HD void element_strain(const M &Ri, const M &Rj, V xi, V xj, double L0, V gamma0, V kappa0, double eps[6],
                           ElementJacobian *J, const M *Jli, const M *Jlj)
{
    element_strain_inv(Ri, Rj, xi, xj, 1.0 / L0, gamma0, kappa0, eps, J, Jli, Jlj);
}

// Half the weights times the length; the first two strains' weights are equal
// and so are the fourth's and fifth's (strain_weights).
struct HalfWeights {
    double shear, stretch, bend, twist;
};
KHS_HD HalfWeights half_weights(const Weights &w, double L0)
{
    HalfWeights h;
    h.shear = 0.5 * L0 * w.w[0]; h.stretch = 0.5 * L0 * w.w[2]; h.bend = 0.5 * L0 * w.w[3]; h.twist = 0.5 * L0 * w.w[5];
    return h;
}

// Elastic energy 0.5 L0 sum w eps^2.
KHS_HD double element_energy(const double eps[6], const Weights &w, double L0)
{
    const HalfWeights h = half_weights(w, L0);
    const double hw[6] = {h.shear, h.shear, h.stretch, h.bend, h.bend, h.twist};
    double e = 0.0;
#pragma unroll
    for (int s = 0; s < 6; ++s) e += hw[s] * eps[s] * eps[s];
    return e;
}

// Gradient of the element energy: gi, gj (6 each; translation then
// rotation) = L0 J^T diag(w) eps.
KHS_HD void element_gradient(const ElementJacobian &J, const double eps[6], const Weights &w, double L0, double gi[6],
                             double gj[6])
{
    const HalfWeights h = half_weights(w, L0);
    const double hs[3] = {h.shear, h.shear, h.stretch}, hb[3] = {h.bend, h.bend, h.twist};
    double se[3], ke[3];  // se: half of L0 w eps, for A2 and S2
#pragma unroll
    for (int k = 0; k < 3; ++k) { se[k] = hs[k] * eps[k]; ke[k] = 2.0 * (hb[k] * eps[3 + k]); }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const double ax = J.A2.m[c] * se[0] + J.A2.m[3 + c] * se[1] + J.A2.m[6 + c] * se[2];
        gi[c] = -ax;
        gj[c] = ax;
        gi[3 + c] = J.S2i.m[c] * se[0] + J.S2i.m[3 + c] * se[1] + J.S2i.m[6 + c] * se[2] +
                    J.Kki.m[c] * ke[0] + J.Kki.m[3 + c] * ke[1] + J.Kki.m[6 + c] * ke[2];
        gj[3 + c] = J.S2j.m[c] * se[0] + J.S2j.m[3 + c] * se[1] + J.S2j.m[6 + c] * se[2] +
                    J.Kkj.m[c] * ke[0] + J.Kkj.m[3 + c] * ke[1] + J.Kkj.m[6 + c] * ke[2];
    }
}

// Gauss-Newton Hessian blocks L0 J^T diag(w) J of one element, as 6x6
// row-major blocks: Hii, Hjj (diagonal blocks of the two nodes) and Hij
// (rows of node i, columns of node j).  With the strain Jacobian's
// structure (shear/stretch rows -A, Sgi, A, Sgj; curvature rows 0, Kki, 0,
// Kkj) the blocks reduce to six 3x3 products:
//   P = A^T Wg A, Xi = A^T Wg Sgi, Xj = A^T Wg Sgj,
//   Rii = Sgi^T Wg Sgi + Kki^T Wk Kki, Rjj likewise, Rij = Sgi^T Wg Sgj + Kki^T Wk Kkj,
//   Hii = [P, -Xi; -Xi^T, Rii], Hjj = [P, Xj; Xj^T, Rjj], Hij = [-P, -Xj; Xi^T, Rij],
// with the symmetric ones (P, Rii, Rjj) evaluated on one triangle and mirrored.
// (On the doubled A2, S2 with a quarter of the weights.)
KHS_HD double dot3w(const M &X, int r, const M &WY, int c)
{
    return X.m[r] * WY.m[c] + X.m[3 + r] * WY.m[3 + c] + X.m[6 + r] * WY.m[6 + c];
}

KHS_HD void element_hessian(const ElementJacobian &J, const Weights &w, double L0, double *Hii, double *Hjj, double *Hij)
{
    M WA, WSi, WSj, WKi, WKj;  // rows scaled by L0 w / 4 and, for K, L0 w
    const HalfWeights h = half_weights(w, L0);
    const double hs[3] = {h.shear, h.shear, h.stretch}, hb[3] = {h.bend, h.bend, h.twist};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const double g = 0.5 * hs[k], kk = 2.0 * hb[k];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            WA.m[3 * k + c] = g * J.A2.m[3 * k + c];
            WSi.m[3 * k + c] = g * J.S2i.m[3 * k + c];
            WSj.m[3 * k + c] = g * J.S2j.m[3 * k + c];
            WKi.m[3 * k + c] = kk * J.Kki.m[3 * k + c];
            WKj.m[3 * k + c] = kk * J.Kkj.m[3 * k + c];
        }
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double xi = dot3w(J.A2, r, WSi, c), xj = dot3w(J.A2, r, WSj, c);
            Hii[6 * r + 3 + c] = -xi;
            Hii[6 * (3 + c) + r] = -xi;
            Hjj[6 * r + 3 + c] = xj;
            Hjj[6 * (3 + c) + r] = xj;
            Hij[6 * r + 3 + c] = -xj;
            Hij[6 * (3 + c) + r] = xi;
            Hij[6 * (3 + r) + 3 + c] = dot3w(J.S2i, r, WSj, c) + dot3w(J.Kki, r, WKj, c);
            if (c < r) continue;
            const double p = dot3w(J.A2, r, WA, c);
            const double rii = dot3w(J.S2i, r, WSi, c) + dot3w(J.Kki, r, WKi, c);
            const double rjj = dot3w(J.S2j, r, WSj, c) + dot3w(J.Kkj, r, WKj, c);
            Hii[6 * r + c] = p; Hii[6 * c + r] = p;
            Hjj[6 * r + c] = p; Hjj[6 * c + r] = p;
            Hij[6 * r + c] = -p; Hij[6 * c + r] = -p;
            Hii[6 * (3 + r) + 3 + c] = rii; Hii[6 * (3 + c) + 3 + r] = rii;
            Hjj[6 * (3 + r) + 3 + c] = rjj; Hjj[6 * (3 + c) + 3 + r] = rjj;
        }
    }
}

// One end's share of the gradient and the Hessian blocks, for two threads an
// element: right 0 for node i, 1 for node j.  g: the node's gradient; H: its
// diagonal block; x = A^T Wg Sg; WS, WK: the rows scaled for the mixed block.
KHS_HD void element_end(bool right, const M &A2, const M &S2, const M &Kk, const double eps[6], const Weights &w, double L0,
                        double g[6], double H[36], M &x, M &WS, M &WK)
{
    M WA;
    const HalfWeights h = half_weights(w, L0);
    const double hs[3] = {h.shear, h.shear, h.stretch}, hb[3] = {h.bend, h.bend, h.twist};
    double se[3], ke[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) { se[k] = hs[k] * eps[k]; ke[k] = 2.0 * (hb[k] * eps[3 + k]); }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const double ax = A2.m[c] * se[0] + A2.m[3 + c] * se[1] + A2.m[6 + c] * se[2];
        g[c] = right ? ax : -ax;
        g[3 + c] = S2.m[c] * se[0] + S2.m[3 + c] * se[1] + S2.m[6 + c] * se[2] +
                   Kk.m[c] * ke[0] + Kk.m[3 + c] * ke[1] + Kk.m[6 + c] * ke[2];
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const double gk = 0.5 * hs[k], kk = 2.0 * hb[k];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            WA.m[3 * k + c] = gk * A2.m[3 * k + c];
            WS.m[3 * k + c] = gk * S2.m[3 * k + c];
            WK.m[3 * k + c] = kk * Kk.m[3 * k + c];
        }
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double xc = dot3w(A2, r, WS, c);
            x.m[3 * r + c] = xc;
            H[6 * r + 3 + c] = H[6 * (3 + c) + r] = right ? xc : -xc;
            if (c < r) continue;
            const double p = dot3w(A2, r, WA, c);
            const double rr = dot3w(S2, r, WS, c) + dot3w(Kk, r, WK, c);
            H[6 * r + c] = H[6 * c + r] = p;
            H[6 * (3 + r) + 3 + c] = H[6 * (3 + c) + 3 + r] = rr;
        }
    }
}

// ---- geometry (device flavour, cuda_backend.cu:200-223) ----------------
//
// The proximity tests decide integer outputs (candidate sets, closest
// triangle, active flags), so they are evaluated without FMA contraction:
// every product and sum is rounded on its own (__dmul_rn / __dadd_rn on the
// device, plain operations in host code built with -ffp-contract=off).
// Given the same inputs the device then produces the same bits as a
// correctly rounded host evaluation, including exact-distance ties.

#if defined(__CUDA_ARCH__)
KHS_HD double xm(double a, double b) { return __dmul_rn(a, b); }
KHS_HD double xa(double a, double b) { return __dadd_rn(a, b); }
KHS_HD double xs(double a, double b) { return __dsub_rn(a, b); }
KHS_HD double xf(double a, double b, double c) { return __fma_rn(a, b, c); }
#else
KHS_HD double xm(double a, double b) { return a * b; }
KHS_HD double xa(double a, double b) { return a + b; }
KHS_HD double xs(double a, double b) { return a - b; }
KHS_HD double xf(double a, double b, double c) { return fma(a, b, c); }
#endif
KHS_HD V gadd(V a, V b) { return v(xa(a.x, b.x), xa(a.y, b.y), xa(a.z, b.z)); }
KHS_HD V gsub(V a, V b) { return v(xs(a.x, b.x), xs(a.y, b.y), xs(a.z, b.z)); }
KHS_HD V gmul(V a, double s) { return v(xm(a.x, s), xm(a.y, s), xm(a.z, s)); }
KHS_HD double gdot(V a, V b) { return xa(xa(xm(a.x, b.x), xm(a.y, b.y)), xm(a.z, b.z)); }
KHS_HD double gnorm(V a) { return sqrt(gdot(a, a)); }

struct ClosestPair {
    double distance, t;
    V bary;
};

// Comparisons of the closest-point code.  On GB300 an FP64 comparison takes an
// FP64 issue slot (64 cycles) like a multiply-add, and fmin / fmax several, so
// FAST decides on the bits with integer instructions.  The answers are those
// of the floating comparisons for everything but NaN (zeros of either sign
// and infinities included); callers take FAST only for coordinates that
// sane_coordinate admits, which cannot produce a NaN before the last division.
template<bool FAST> KHS_HD bool le0(double x) { return FAST ? int64_t(bits_of(x)) <= 0 : x <= 0; }
template<bool FAST> KHS_HD bool ge0(double x) { return FAST ? bits_of(x) <= 0x8000000000000000ull : x >= 0; }
template<bool FAST> KHS_HD bool lt0(double x) { return FAST ? bits_of(x) > 0x8000000000000000ull : x < 0; }
// x <= y for y >= 0.
template<bool FAST> KHS_HD bool le_nonneg(double x, double y)
{
    return FAST ? int64_t(bits_of(x)) <= int64_t(bits_of(y) & 0x7fffffffffffffffull) : x <= y;
}
template<bool FAST> KHS_HD bool nonzero(double x) { return FAST ? (bits_of(x) << 1) != 0 : x != 0; }
template<bool FAST> KHS_HD bool gt1(double x) { return FAST ? int64_t(bits_of(x)) > 0x3ff0000000000000ll : x > 1; }
// fmin(1, fmax(0, x)).
template<bool FAST> KHS_HD double clamp01(double x)
{
    if (!FAST) return fmin(1.0, fmax(0.0, x));
    return int64_t(bits_of(x)) <= 0 ? 0.0 : (gt1<true>(x) ? 1.0 : x);
}
// Finite and below 2^200: sums of products of four differences stay finite.
KHS_HD bool sane_coordinate(double x) { return (uint32_t(bits_of(x) >> 32) & 0x7fffffffu) < ((1023u + 200u) << 20); }
KHS_HD bool sane(V a) { return sane_coordinate(a.x) && sane_coordinate(a.y) && sane_coordinate(a.z); }

template<bool FAST> KHS_HD V closest_point_triangle(V p, V a, V b, V c, V &bary)
{
    const V ab = gsub(b, a), ac = gsub(c, a), ap = gsub(p, a);
    const double d1 = gdot(ab, ap), d2 = gdot(ac, ap);
    if (le0<FAST>(d1) && le0<FAST>(d2)) { bary = v(1, 0, 0); return a; }
    const V bp = gsub(p, b);
    const double d3 = gdot(ab, bp), d4 = gdot(ac, bp);
    if (ge0<FAST>(d3) && le_nonneg<FAST>(d4, d3)) { bary = v(0, 1, 0); return b; }
    const double vc = xs(xm(d1, d4), xm(d3, d2));
    if (le0<FAST>(vc) && ge0<FAST>(d1) && le0<FAST>(d3)) {
        const double w = d1 / xs(d1, d3);
        bary = v(xs(1.0, w), w, 0);
        return gadd(a, gmul(ab, w));
    }
    const V cp = gsub(p, c);
    const double d5 = gdot(ab, cp), d6 = gdot(ac, cp);
    if (ge0<FAST>(d6) && le_nonneg<FAST>(d5, d6)) { bary = v(0, 0, 1); return c; }
    const double vb = xs(xm(d5, d2), xm(d1, d6));
    if (le0<FAST>(vb) && ge0<FAST>(d2) && le0<FAST>(d6)) {
        const double w = d2 / xs(d2, d6);
        bary = v(xs(1.0, w), 0, w);
        return gadd(a, gmul(ac, w));
    }
    const double va = xs(xm(d3, d6), xm(d5, d4));
    const double d43 = xs(d4, d3), d56 = xs(d5, d6);
    if (le0<FAST>(va) && ge0<FAST>(d43) && ge0<FAST>(d56)) {
        const double w = d43 / xa(d43, d56);
        bary = v(0, xs(1.0, w), w);
        return gadd(b, gmul(gsub(c, b), w));
    }
    const double inv = 1.0 / xa(xa(va, vb), vc), vv = xm(vb, inv), ww = xm(vc, inv);
    bary = v(xs(xs(1.0, vv), ww), vv, ww);
    return gadd(gadd(a, gmul(ab, vv)), gmul(ac, ww));
}

template<bool FAST> KHS_HD void segment_segment_params(V p1, V q1, V p2, V q2, double &s, double &t)
{
    const V d1 = gsub(q1, p1), d2 = gsub(q2, p2), r = gsub(p1, p2);
    const double a = gdot(d1, d1), e = gdot(d2, d2), f = gdot(d2, r);
    s = 0.0; t = 0.0;
    const bool point1 = le_nonneg<FAST>(a, 1e-14), point2 = le_nonneg<FAST>(e, 1e-14);
    if (point1 && point2) return;
    if (point1) { t = clamp01<FAST>(f / e); return; }
    const double c = gdot(d1, r);
    if (point2) { s = clamp01<FAST>(-c / a); return; }
    const double b = gdot(d1, d2), den = xs(xm(a, e), xm(b, b));
    if (nonzero<FAST>(den)) s = clamp01<FAST>(xs(xm(b, f), xm(c, e)) / den);
    t = xa(xm(b, s), f) / e;
    if (lt0<FAST>(t)) { t = 0; s = clamp01<FAST>(-c / a); }
    else if (gt1<FAST>(t)) { t = 1; s = clamp01<FAST>(xs(b, c) / a); }
}

// Closest pair between segment p0-p1 and triangle abc: end points against
// the face, then the segment against the three edges, keeping the first
// strictly smaller distance.  No interior-crossing test (device semantics of
// the reference).
//
// The five tests as parts of their own, so that threads can share a pair:
// part 0 and 1 the end points, 2 ... 4 the edges.  dist2 is the squared
// distance before the square root.
struct PairPart {
    double dist2, t;
    V bary;
};

template<bool FAST> KHS_HD PairPart point_part(V p, double t, V a, V b, V c)
{
    PairPart out;
    const V cp = closest_point_triangle<FAST>(p, a, b, c, out.bary);
    const V w = gsub(p, cp);
    out.dist2 = gdot(w, w);
    out.t = t;
    return out;
}

template<bool FAST> KHS_HD PairPart edge_part(int e, V p0, V p1, V a, V b, V c)
{
    const V p2 = e == 0 ? a : (e == 1 ? b : c);
    const V q2 = e == 0 ? b : (e == 1 ? c : a);
    PairPart out;
    double t;
    segment_segment_params<FAST>(p0, p1, p2, q2, out.t, t);
    const V w = gsub(gadd(p0, gmul(gsub(p1, p0), out.t)), gadd(p2, gmul(gsub(q2, p2), t)));
    out.dist2 = gdot(w, w);
    const double u = xs(1.0, t);
    out.bary = e == 0 ? v(u, t, 0) : (e == 1 ? v(0, u, t) : v(t, 0, u));
    return out;
}

template<bool FAST> KHS_HD PairPart pair_part(int part, V p0, V p1, V a, V b, V c)
{
    return part < 2 ? point_part<FAST>(part ? p1 : p0, part ? 1.0 : 0.0, a, b, c) : edge_part<FAST>(part - 2, p0, p1, a, b, c);
}

// sqrt(x) < sqrt(best) of two squared distances, or NaN (never smaller), for
// best >= 0 and not NaN.  The rounded square root does not decrease, and more
// than 16 units in the last place apart it differs; closer ones are compared
// as roots.
KHS_HD bool root_less(double x, double best)
{
    const uint64_t bx = bits_of(x), bb = bits_of(best);
    if (bx >= bb) return false;  // NaN included
    return bb - bx > 16 || sqrt(x) < sqrt(best);
}

template<bool FAST> KHS_HD ClosestPair closest_of_parts(V p0, V p1, V a, V b, V c)
{
    // No part found: the distance stays at 1e300, whose square is infinite.
    PairPart best;
    best.dist2 = double_of(0x7ff0000000000000ull); best.t = 0.0; best.bary = v(1, 0, 0);
#pragma unroll
    for (int part = 0; part < 5; ++part) {
        const PairPart x = pair_part<FAST>(part, p0, p1, a, b, c);
        if (root_less(x.dist2, best.dist2)) best = x;
    }
    ClosestPair out;
    out.distance = bits_of(best.dist2) < 0x7ff0000000000000ull ? sqrt(best.dist2) : 1.0e300;
    out.t = best.t;
    out.bary = best.bary;
    return out;
}
KHS_HD_SLOW ClosestPair closest_of_parts_slow(V p0, V p1, V a, V b, V c) { return closest_of_parts<false>(p0, p1, a, b, c); }
KHS_HD_SLOW PairPart pair_part_slow(int part, V p0, V p1, V a, V b, V c) { return pair_part<false>(part, p0, p1, a, b, c); }

KHS_HD bool sane_pair(V p0, V p1, V a, V b, V c) { return sane(p0) && sane(p1) && sane(a) && sane(b) && sane(c); }

KHS_HD ClosestPair closest_segment_triangle(V p0, V p1, V a, V b, V c)
{
    if (!sane_pair(p0, p1, a, b, c)) return closest_of_parts_slow(p0, p1, a, b, c);
    return closest_of_parts<true>(p0, p1, a, b, c);
}

// ---- FP32 filters for the mixed form -----------------------------------
//
// Single-precision segment-triangle distance on coordinates taken relative
// to a local origin (the segment start, subtracted in FP64).  Used only to
// discard candidates that provably cannot be the closest one, with a
// relative margin far above the FP32 rounding of these few operations; the
// decision among the survivors is taken in FP64 with the exact code above.
struct F3 {
    float x, y, z;
};
KHS_HD F3 f3(float x, float y, float z) { F3 r; r.x = x; r.y = y; r.z = z; return r; }
KHS_HD F3 fsub(F3 a, F3 b) { return f3(a.x - b.x, a.y - b.y, a.z - b.z); }
KHS_HD F3 fadd(F3 a, F3 b) { return f3(a.x + b.x, a.y + b.y, a.z + b.z); }
KHS_HD F3 fmulv(F3 a, float s) { return f3(a.x * s, a.y * s, a.z * s); }
KHS_HD float fdot(F3 a, F3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
KHS_HD F3 to_local(V p, V origin) { return f3(float(p.x - origin.x), float(p.y - origin.y), float(p.z - origin.z)); }

KHS_HD F3 closest_point_triangle_f(F3 p, F3 a, F3 b, F3 c)
{
    const F3 ab = fsub(b, a), ac = fsub(c, a), ap = fsub(p, a);
    const float d1 = fdot(ab, ap), d2 = fdot(ac, ap);
    if (d1 <= 0.f && d2 <= 0.f) return a;
    const F3 bp = fsub(p, b);
    const float d3 = fdot(ab, bp), d4 = fdot(ac, bp);
    if (d3 >= 0.f && d4 <= d3) return b;
    const float vc = d1 * d4 - d3 * d2;
    if (vc <= 0.f && d1 >= 0.f && d3 <= 0.f) return fadd(a, fmulv(ab, d1 / (d1 - d3)));
    const F3 cp = fsub(p, c);
    const float d5 = fdot(ab, cp), d6 = fdot(ac, cp);
    if (d6 >= 0.f && d5 <= d6) return c;
    const float vb = d5 * d2 - d1 * d6;
    if (vb <= 0.f && d2 >= 0.f && d6 <= 0.f) return fadd(a, fmulv(ac, d2 / (d2 - d6)));
    const float va = d3 * d6 - d5 * d4;
    if (va <= 0.f && (d4 - d3) >= 0.f && (d5 - d6) >= 0.f)
        return fadd(b, fmulv(fsub(c, b), (d4 - d3) / ((d4 - d3) + (d5 - d6))));
    const float inv = 1.f / (va + vb + vc);
    return fadd(fadd(a, fmulv(ab, vb * inv)), fmulv(ac, vc * inv));
}

KHS_HD float segment_segment_distance_f(F3 p1, F3 q1, F3 p2, F3 q2)
{
    const F3 d1 = fsub(q1, p1), d2 = fsub(q2, p2), r = fsub(p1, p2);
    const float a = fdot(d1, d1), e = fdot(d2, d2), f = fdot(d2, r);
    float s = 0.f, t = 0.f;
    if (!(a <= 1e-20f && e <= 1e-20f)) {
        if (a <= 1e-20f) t = fminf(1.f, fmaxf(0.f, f / e));
        else {
            const float c = fdot(d1, r);
            if (e <= 1e-20f) s = fminf(1.f, fmaxf(0.f, -c / a));
            else {
                const float b = fdot(d1, d2), den = a * e - b * b;
                if (den > 0.f) s = fminf(1.f, fmaxf(0.f, (b * f - c * e) / den));
                t = (b * s + f) / e;
                if (t < 0.f) { t = 0.f; s = fminf(1.f, fmaxf(0.f, -c / a)); }
                else if (t > 1.f) { t = 1.f; s = fminf(1.f, fmaxf(0.f, (b - c) / a)); }
            }
        }
    }
    const F3 w = fsub(fadd(p1, fmulv(d1, s)), fadd(p2, fmulv(d2, t)));
    return sqrtf(fdot(w, w));
}

// FP32 segment-triangle distance (local coordinates) and the absolute
// margin that bounds its deviation from the FP64 distance.
KHS_HD float segment_triangle_distance_f(F3 p0, F3 p1, F3 a, F3 b, F3 c, float &margin)
{
    F3 w = fsub(p0, closest_point_triangle_f(p0, a, b, c));
    float dist = sqrtf(fdot(w, w));
    w = fsub(p1, closest_point_triangle_f(p1, a, b, c));
    dist = fminf(dist, sqrtf(fdot(w, w)));
    dist = fminf(dist, segment_segment_distance_f(p0, p1, a, b));
    dist = fminf(dist, segment_segment_distance_f(p0, p1, b, c));
    dist = fminf(dist, segment_segment_distance_f(p0, p1, c, a));
    const float scale = fmaxf(fmaxf(fabsf(p1.x), fmaxf(fabsf(p1.y), fabsf(p1.z))),
                              fmaxf(fmaxf(fabsf(a.x), fmaxf(fabsf(a.y), fabsf(a.z))),
                                    fmaxf(fmaxf(fabsf(b.x), fmaxf(fabsf(b.y), fabsf(b.z))),
                                          fmaxf(fabsf(c.x), fmaxf(fabsf(c.y), fabsf(c.z))))));
    margin = 1.0e-4f * (scale + dist) + 1.0e-9f;
    return dist;
}

KHS_HD bool boxes_overlap(V al, V au, V bl, V bu, double p)
{
    return al.x <= bu.x + p && bl.x <= au.x + p && al.y <= bu.y + p && bl.y <= au.y + p && al.z <= bu.z + p &&
           bl.z <= au.z + p;
}

// Offset of a segment's point at t from a triangle's point at the barycentric
// weights.  Which products its sums take into a multiply-add is written out
// here and in the barrier: left to the compiler it depends on what stands
// around them, and stiff contacts carry a changed bit into the step counts.
KHS_HD V contact_offset(V x0, V x1, double t, V a, V b, V c, V bary)
{
    const double w = 1.0 - t;
    auto one = [&](double p0, double p1, double va, double vb, double vc) {
        const double p = xf(p1, t, xm(p0, w));
        return xs(p, xf(vc, bary.z, xf(va, bary.x, xm(vb, bary.y))));
    };
    return v(one(x0.x, x1.x, a.x, b.x, c.x), one(x0.y, x1.y, a.y, b.y, c.y), one(x0.z, x1.z, a.z, b.z, c.z));
}

// Log barrier b(g) = -kc (dh - g)^2 ln(g / dh) of the contact gap and its
// gradient with respect to the two segment end points at fixed (t, bary), from
// their offset (cuda_backend.cu:255-265: the distance is regularised by 1e-30
// inside the square root).  Returns the energy; g0, g1 get the gradients.
KHS_HD double barrier_energy_gradient(V offset, double t, double radius_offset, double dh, double kc, double g0[3], double g1[3])
{
    const double dist = sqrt(xa(xf(offset.z, offset.z, xf(offset.x, offset.x, xm(offset.y, offset.y))), 1e-30));
    const double gap = dist - radius_offset;
    if (gap >= dh) {
        g0[0] = g0[1] = g0[2] = g1[0] = g1[1] = g1[2] = 0.0;
        return 0.0;
    }
    const double aa = dh - gap, lg = log(gap / dh), w = 1.0 - t;
    const double energy = xm(xm(xm(-kc, aa), aa), lg);
    const double db = xm(kc, xs(xm(2.0 * aa, lg), xm(aa, aa) / gap));  // d energy / d gap
    const double s = db / dist;
    const double f[3] = {xm(s, offset.x), xm(s, offset.y), xm(s, offset.z)};
#pragma unroll
    for (int k = 0; k < 3; ++k) { g0[k] = xm(f[k], w); g1[k] = xm(f[k], t); }
    return energy;
}

// ---- root targets (src/solver.cpp:416-447, src/math.hpp:26-58) -----------
//
// Frames of the driven nodes: a frame per node whose third column is the
// unit tangent, the first column carried from node to node by the minimal
// rotation between consecutive tangents, and the rotation vector of
// frame * reference^T (src/solver.cpp:19-26 goes through Eigen's AngleAxis;
// restated with Shepperd's method, J. Guidance and Control 1(3), 1978).
// Written with the non-contracting operations above and correctly rounded
// division and square root, so the device rounds like host code built with
// -ffp-contract=off: positions, tangents and frames agree bit for bit and the
// rotation vectors differ only through atan2.

#if defined(__CUDA_ARCH__)
KHS_HD bool gfinite(double x) { return isfinite(x); }
#else
KHS_HD bool gfinite(double x) { return std::isfinite(x); }
#endif

KHS_HD V gcross(V a, V b)
{
    return v(xs(xm(a.y, b.z), xm(a.z, b.y)), xs(xm(a.z, b.x), xm(a.x, b.z)), xs(xm(a.x, b.y), xm(a.y, b.x)));
}

// a / n rounded to nearest with r = 1 / n rounded to nearest: the quotient
// a r, its exact remainder, and one correction by it, which Markstein
// (Computation of elementary functions on the IBM RISC System/6000, 1990)
// shows to round correctly when r does.  Three multiply-adds where a division
// takes a dozen FP64 instructions, and several numerators share r.  The
// division itself where the remainder or the quotient could leave the normal
// range (a zero, tiny or huge a or n, a NaN).
KHS_HD double div_by(double a, double n, double r)
{
    const int ea = int((bits_of(a) >> 52) & 0x7ff), en = int((bits_of(n) >> 52) & 0x7ff);
    if (ea < 200 || ea > 1800 || en < 200 || en > 1800 || ea - en > 600 || en - ea > 600) return a / n;
#if defined(__CUDA_ARCH__)
    const double q = __dmul_rn(a, r);
    return __fma_rn(__fma_rn(-q, n, a), r, q);
#else
    const double q = a * r;
    return std::fma(std::fma(-q, n, a), r, q);
#endif
}

// a / n for each component.
KHS_HD V gdiv(V a, double n)
{
#if defined(__CUDA_ARCH__)
    const double r = recip_any(n);
    return v(div_by(a.x, n, r), div_by(a.y, n, r), div_by(a.z, n, r));
#else
    return v(a.x / n, a.y / n, a.z / n);
#endif
}

// Unit vector with Eigen's normalized() semantics: a zero (or NaN) squared
// norm leaves the vector unchanged; each component is divided.
KHS_HD V gunit(V a)
{
    const double n2 = gdot(a, a);
    if (!(n2 > 0.0)) return a;
    return gdiv(a, sqrt(n2));
}

// (1 - t) a + t b, each product and the sum rounded on its own.
KHS_HD V glerp(V a, V b, double t)
{
    const double u = xs(1.0, t);
    return v(xa(xm(a.x, u), xm(b.x, t)), xa(xm(a.y, u), xm(b.y, t)), xa(xm(a.z, u), xm(b.z, t)));
}

// Frame (row-major, columns d1 d2 d3) from d3 = the normalised tangent and
// d1 the hint made orthogonal to it (math.hpp:26-43).
KHS_HD M frame_from_d3(V d3, V hint)
{
    V d1 = gsub(hint, gmul(d3, gdot(hint, d3)));
    if (gdot(d1, d1) < 1.0e-16) {
        const V axis = fabs(d3.x) < 0.8 ? v(1.0, 0.0, 0.0) : v(0.0, 1.0, 0.0);
        d1 = gsub(axis, gmul(d3, gdot(axis, d3)));
    }
    d1 = gunit(d1);
    const V d2 = gunit(gcross(d3, d1));
    d1 = gunit(gcross(d2, d3));
    M r;
    r.m[0] = d1.x; r.m[1] = d2.x; r.m[2] = d3.x;
    r.m[3] = d1.y; r.m[4] = d2.y; r.m[5] = d3.y;
    r.m[6] = d1.z; r.m[7] = d2.z; r.m[8] = d3.z;
    return r;
}

KHS_HD M frame_from_tangent(V tangent, V hint) { return frame_from_d3(gunit(tangent), hint); }

// A unit vector orthogonal to s, chosen like Eigen's unitOrthogonal.
KHS_HD V unit_orthogonal(V s)
{
    const double eps = 1e-12;
    if (!(fabs(s.x) <= xm(fabs(s.z), eps)) || !(fabs(s.y) <= xm(fabs(s.z), eps))) {
        const double inv = 1.0 / sqrt(xa(xm(s.x, s.x), xm(s.y, s.y)));
        return v(xm(-s.y, inv), xm(s.x, inv), 0.0);
    }
    const double inv = 1.0 / sqrt(xa(xm(s.y, s.y), xm(s.z, s.z)));
    return v(0.0, xm(-s.z, inv), xm(s.y, inv));
}

// The minimal rotation taking `from` to `to` (math.hpp:45-58), split into
// the part that depends on the two tangents only and its application to a
// director: Rodrigues' formula about n = from x to / |from x to| (kind 0),
// the identity for parallel tangents (kind 1), a half turn about an
// orthogonal axis n for opposite ones (kind 2).
struct Transport {
    V n;
    double s, c;
    int kind;
};

KHS_HD Transport transport_between(V from, V to)
{
    const V a = gunit(from), b = gunit(to);
    const V axis = gcross(a, b);
    Transport t;
    t.s = sqrt(gdot(axis, axis));
    const double c = gdot(a, b);
    t.c = c < -1.0 ? -1.0 : (1.0 < c ? 1.0 : c);
    t.kind = 0;
    if (t.s < 1.0e-12) {
        t.kind = t.c > 0.0 ? 1 : 2;
        t.n = t.kind == 2 ? unit_orthogonal(a) : v(0.0, 0.0, 0.0);
    } else {
        t.n = gdiv(axis, t.s);
    }
    return t;
}

KHS_HD V transport_apply(const Transport &t, V director)
{
    if (t.kind == 1) return director;
    if (t.kind == 2) return gsub(gmul(gmul(t.n, 2.0), gdot(t.n, director)), director);
    return gadd(gadd(gmul(director, t.c), gmul(gcross(t.n, director), t.s)), gmul(gmul(t.n, gdot(t.n, director)), xs(1.0, t.c)));
}

KHS_HD V parallel_transport(V director, V from, V to) { return transport_apply(transport_between(from, to), director); }

// a * b^T for row-major 3x3 matrices.
KHS_HD M times_transpose(const M &a, const M &b)
{
    M r;
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j)
            r.m[3 * i + j] = xa(xa(xm(a.m[3 * i], b.m[3 * j]), xm(a.m[3 * i + 1], b.m[3 * j + 1])), xm(a.m[3 * i + 2], b.m[3 * j + 2]));
    return r;
}

// Rotation vector (axis * angle, angle in (-pi, pi]) of a rotation matrix:
// the quaternion from the largest of its four squared components, then
// angle = 2 atan2(|v|, |w|) with the axis carrying the sign of w.
KHS_HD V rotation_vector(const M &r)
{
    double q[4];  // x y z w
    const double tr = xa(xa(r.m[0], r.m[4]), r.m[8]);
    if (tr > 0.0) {
        double s = sqrt(xa(tr, 1.0));
        q[3] = xm(0.5, s);
        s = 0.5 / s;
        q[0] = xm(xs(r.m[7], r.m[5]), s);
        q[1] = xm(xs(r.m[2], r.m[6]), s);
        q[2] = xm(xs(r.m[3], r.m[1]), s);
    } else {
        int i = 0;
        if (r.m[4] > r.m[0]) i = 1;
        if (r.m[8] > r.m[4 * i]) i = 2;
        const int j = (i + 1) % 3, k = (j + 1) % 3;
        double s = sqrt(xa(xs(xs(r.m[4 * i], r.m[4 * j]), r.m[4 * k]), 1.0));
        q[i] = xm(0.5, s);
        s = 0.5 / s;
        q[3] = xm(xs(r.m[3 * k + j], r.m[3 * j + k]), s);
        q[j] = xm(xa(r.m[3 * j + i], r.m[3 * i + j]), s);
        q[k] = xm(xa(r.m[3 * k + i], r.m[3 * i + k]), s);
    }
    double n = sqrt(xa(xa(xm(q[0], q[0]), xm(q[1], q[1])), xm(q[2], q[2])));
    if (!(n != 0.0)) return v(0.0, 0.0, 0.0);
    double angle = xm(2.0, atan2(n, fabs(q[3])));
    if (q[3] < 0.0) n = -n;
    const V axis = gdiv(v(q[0], q[1], q[2]), n);
    if (!gfinite(angle) || !gfinite(axis.x) || !gfinite(axis.y) || !gfinite(axis.z)) return v(0.0, 0.0, 0.0);
    if (angle > kPi) angle = xs(angle, xm(2.0, kPi));
    return gmul(axis, angle);
}

}  // namespace dm
}  // namespace khs
