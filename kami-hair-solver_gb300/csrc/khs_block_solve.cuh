// FP64 block-tridiagonal solve of the Gauss-Newton direction: the device code
// of k_block_solve and k_block_solve_team (khs_engine.cu), for a view D of the
// solver's arrays (diag, upper, cprime [N][36]; grad, dprime, dir [N][6]; the
// strands' order and ranges; sc->solve_failed).
#pragma once

#include "khs_device_math.cuh"

#include <cstdint>

namespace khs {
namespace {

constexpr int kStrandsPerWarp = 5;  // solve_strands_five: 6 lanes per strand

// Block Thomas solve with Gauss-Jordan elimination on the augmented block
// [B_n | U_n | rhs_n]: the elimination leaves C_n = B_n^-1 U_n and
// d'_n = B_n^-1 rhs_n in place of U_n and rhs_n (the reference forms
// B_n^-1 first and multiplies; the operations per result entry differ in
// order only).  Pivot rows stay unscaled until one scaling per row at the end,
// so each column costs one reciprocal, one product and one fused
// multiply-add per live entry; finished pivot columns are not updated.
//
// On GB300 an FP64 warp instruction holds its sub-partition's pipe for 64
// cycles whatever the number of active lanes (76 with all four
// sub-partitions busy), and a dependent one waits as long, so a strand's time
// is its chain of nodes and the machine's throughput is instructions times 76
// cycles.  Three layouts:
// * solve_strand_team: one strand on three warps, the pivot chain on one and
//   what follows it on the others, 4,000 cycles a node alone and 4,550 with
//   608 strands;
// * solve_strand_warp: one strand on a warp, one matrix entry per lane, 42
//   FP64 instructions and 4,950 cycles a node alone, 3,200 of a
//   sub-partition's cycles when the machine is full;
// * solve_strands_five: five strands on a warp, a lane per block row, 127
//   FP64 instructions and 14,700 cycles a node of five strands alone, 2,020
//   of a sub-partition's cycles per strand and node when it is full.
// (160-node strands.  The layouts they replace, with 6 H lanes a strand and
// four warps on the longest, took 12,000 cycles a node on one warp, 8,800 on
// four.)
// All take the pivot's reciprocal on the integer pipes (dm::recip_rn, equal
// to the FP64 division) for every candidate of the column while the pivot
// search runs.  Shuffles, reductions and FP64 instructions share a queue that
// issues in order, so shuffles are counted like arithmetic.  Every entry goes
// through the same operations in the same order in every layout, so the
// results are identical bit for bit and the split between them changes no
// result.

// The relative diagonal shift max(1e-12 smax, 1e-24) of the largest diagonal
// magnitude (compared as bits; a NaN product gives 1e-24, as fmax does).
__device__ __forceinline__ double diagonal_shift(unsigned long long smax)
{
    const long long p = __double_as_longlong(__dmul_rn(1.0e-12, __longlong_as_double((long long)smax)));
    const long long least = 0x3af357c299a88ea7ll;  // 1e-24
    return __longlong_as_double(p > least && p <= 0x7ff0000000000000ll ? p : least);
}

// A pivot below 1e-30 or not finite (exponent all ones) fails the node.
__device__ __forceinline__ bool pivot_fails(unsigned long long best)
{
    return best < 0x39b4484bfeebc2a0ull || best >= 0x7ff0000000000000ull;
}

// Free nodes of the strand at place k of the solve order.
template<class D> __device__ __forceinline__ void strand_range(const D &d, uint32_t k, uint32_t &begin, uint32_t &len)
{
    const uint32_t s = d.sorder[k];
    begin = d.sfirst[s] + d.sfixed[s];
    const uint32_t end = d.sfirst[s] + d.scount[s];
    len = end > begin ? end - begin : 0;
}

// Rows of C and d' read back through shared memory, kRing nodes ahead.
constexpr int kRing = 8;
struct BackRing {
    double row[kRing][42];  // C_n row-major, then d'_n
};

__device__ __forceinline__ void copy16_async(double *shared, const double *global)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(uint32_t(__cvta_generic_to_shared(shared))), "l"(global) : "memory");
}

// The state of one node's elimination on a warp (solve_strand_warp).
struct WarpNode {
    double b, bx, u, ux, ipiv;
};

// Gauss-Jordan on one node: the six pivot steps on b, bx, u, ux.  The pivot
// search compares the top 29 bits of the magnitudes with the row beside them,
// in one warp reduction; EXACT compares all bits and checks the pivots.
// Returns whether, for !EXACT, some step needs EXACT (candidates equal in
// those bits, or a pivot outside [1e-30, 2^1022)), and for EXACT, whether a
// pivot failed.
template<bool EXACT> __device__ __forceinline__ bool eliminate_node(WarpNode &w, int lane, int g, int r)
{
    const unsigned FULL = 0xffffffffu;
    double b = w.b, u = w.u, ux = w.ux, ipiv = 1.0, fp = 0.0, xu = 0.0, xx = 0.0;
    bool flag = false;
#pragma unroll
    for (int col = 0; col < 6; ++col) {
        const int base = col == 0 ? 0 : 6 * (col - 1);  // first lane of the pivot column
        const double mine = col == 0 ? w.bx : b;
        // The first row of the largest magnitude, among rows col ... 5.
        const bool cand = lane >= base + col && lane < base + 6;
        const unsigned hi = cand ? unsigned(__double2hiint(mine)) & 0x7fffffffu : 0u;
        const unsigned key = EXACT ? hi : cand ? (hi & ~7u) | unsigned(5 - r) : 0u;
        const unsigned best = __reduce_max_sync(FULL, key);
        int pivot = 5 - int(best & 7u);
        if (EXACT) {
            const unsigned lo = cand && hi == best ? unsigned(__double2loint(mine)) : 0u;
            const unsigned ml = __reduce_max_sync(FULL, lo);
            pivot = 5 - int(__reduce_max_sync(FULL, cand && hi == best && lo == ml ? unsigned(5 - r) : 0u));
            flag |= pivot_fails((unsigned long long)best << 32 | ml);
        }
        const int partner = r == col ? pivot : (r == pivot ? col : r);
        const int row = 6 * g + pivot, swap = 6 * g + partner;
        // The pivot row's entries and the row swap of B.
        const double fcol = __shfl_sync(FULL, mine, base + partner);
        if (col == 2) {
            // Lanes 0-11 have no live entry of B left: ux rides there.
            ux = r == 1 ? ux : __fma_rn(-fp, xx, ux);
            if (g < 2) b = ux;
        }
        const double xb = __shfl_sync(FULL, b, row);
        b = __shfl_sync(FULL, b, swap);
        const double rc = EXACT ? dm::recip_rn(mine) : dm::recip_normal(mine);
        // The last step's update of U.
        if (col > 0) u = r == col - 1 ? u : __fma_rn(-fp, xu, u);
        if (col == 1) ux = r == 0 ? ux : __fma_rn(-fp, xx, ux);
        const double ip = __shfl_sync(FULL, rc, base + pivot);
        fp = __dmul_rn(fcol, ip);
        xu = __shfl_sync(FULL, u, row);
        u = __shfl_sync(FULL, u, swap);
        if (col < 2) {
            xx = __shfl_sync(FULL, ux, row);
            ux = __shfl_sync(FULL, ux, swap);
        }
        if (r == col) ipiv = ip;
        b = r == col ? b : __fma_rn(-fp, xb, b);
        if (!EXACT) {
            const unsigned off = (r != pivot) & cand ? key ^ best : 8u;
            const unsigned low = best - 0x39b44850u;  // wraps below the least pivot
            flag |= (off < 8u) | (low >= 0x7fd00000u - 0x39b44850u);
        }
    }
    w.u = r == 5 ? u : __fma_rn(-fp, xu, u);
    w.ux = b;
    w.ipiv = ipiv;
    return EXACT ? flag : __any_sync(FULL, flag);
}

// Back substitution d_n = d'_n - C_n d_{n+1} of one strand on a warp, every
// lane of row r: a chain of six multiply-adds a node, shorter than a read from
// L2, so the rows come through a ring of asynchronous copies (16 bytes a lane),
// and from there to registers one node ahead.  C and d' are visible to the
// warp.
template<class D>
__device__ __forceinline__ void substitute_back(const D &d, uint32_t begin, uint32_t len, BackRing &ring, int lane, int r)
{
    const unsigned FULL = 0xffffffffu;
    const uint32_t last = begin + len - 1;
    const double *src = lane < 18 ? d.cprime + 36 * size_t(last) + 2 * lane : d.dprime + 6 * size_t(last) + 2 * (lane - 18);
    const int back = lane < 18 ? 36 : 6;
    uint32_t asked = 0;
    auto request = [&]() {
        if (lane < 21 && asked < len) copy16_async(ring.row[asked % kRing] + 2 * lane, src);
        asm volatile("cp.async.commit_group;" ::: "memory");
        src -= back;
        ++asked;
    };
    double next = 0.0, nv, nc[6];
    auto take = [&](uint32_t done) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kRing - 2) : "memory");
        __syncwarp();
        const double *row = ring.row[done % kRing];
        nv = row[36 + r];
        const double2 *pair = reinterpret_cast<const double2 *>(row + 6 * r);
#pragma unroll
        for (int q = 0; q < 3; ++q) { nc[2 * q] = pair[q].x; nc[2 * q + 1] = pair[q].y; }
    };
    for (int a = 0; a < kRing - 1; ++a) request();
    take(0);
    double *out = d.dir + 6 * size_t(last) + r;
    for (uint32_t done = 0; done < len; ++done) {
        double value = nv, crow[6];
#pragma unroll
        for (int q = 0; q < 6; ++q) crow[q] = nc[q];
        // The slot of kRing - 1 ahead is that of the row before this one,
        // which every lane took before the __syncwarp of the last take.
        request();
        take(done + 1);  // past the last row: an old slot, unused
        if (done > 0) {
#pragma unroll
            for (int q = 0; q < 6; ++q) value = __fma_rn(-crow[q], __shfl_sync(FULL, next, q), value);
        }
        if (lane < 6) *out = value;
        out -= 6;
        next = value;
    }
    __syncwarp();  // the ring is free for the next strand
}

// One strand on one warp.  Lane 6 g + r holds row r of column g + 1 of B_n
// and U_n (g < 5) in b and u, and of an extra column in bx and ux: column 0
// for g = 0, the right-hand side for g = 1 (the other lanes' extra entries
// and lanes 30 and 31 carry values that nothing reads).  After pivot column
// 2 the lanes of columns 1 and 2 have nothing left in b, so ux rides there
// and one multiply-add updates both.  What bounds it, of 4,950 cycles a node:
// six pivot steps of 490 (reciprocal 156, the pivot search beside it, a
// product, two multiply-adds, six shuffles), twelve multiply-adds of the next
// Schur complement in two chains 970, the shift 240, loads, stores and
// scaling 300, the back substitution 520.
template<class D> __device__ __forceinline__ void solve_strand_warp(const D &d, uint32_t k, BackRing &ring)
{
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int g = lane / 6, r = lane - 6 * g;
    const bool wide = g < 5;
    uint32_t begin, len;
    strand_range(d, k, begin, len);
    if (len == 0) return;
    // Every lane reads through pointers of its own, without conditions (a
    // divergent one costs more than the read): lanes without an entry read a
    // neighbour's and nothing uses it.  sx flips the sign of the gradient.
    const double *pd = d.diag + 36 * size_t(begin) + 6 * r + (wide ? g + 1 : 0);
    const double *pu = d.upper + 36 * size_t(begin) + 6 * r + (wide ? g + 1 : 0);
    const double *pux = d.upper + 36 * size_t(begin) + 6 * r;
    const double *puc = d.upper + 36 * size_t(begin) + r;
    const double *px = g == 1 ? d.grad + 6 * size_t(begin) + r : d.diag + 36 * size_t(begin) + 6 * r;
    const int step = g == 1 ? 6 : 36, sx = g == 1 ? int(0x80000000) : 0;
    double *pc = d.cprime + 36 * size_t(begin) + 6 * r + (wide ? g + 1 : 0);
    double *pcx = g == 1 ? d.dprime + 6 * size_t(begin) + r : d.cprime + 36 * size_t(begin) + 6 * r;
    double nd = *pd, nx = *px, nu = *pu, nux = *pux, nuc[6];
    double cu = 0.0, cx = 0.0;  // row r of C_{n-1} (columns as u, ux) and d'_{n-1}
    bool failed = false;
    for (uint32_t t = 0; t < len; ++t) {
        const bool tip = t + 1 == len;  // U_n couples to nothing there
        WarpNode w;
        w.b = nd;
        w.bx = __hiloint2double(__double2hiint(nx) ^ sx, __double2loint(nx));
        w.u = tip ? 0.0 : nu;
        w.ux = tip || g != 0 ? 0.0 : nux;
        if (t > 0) {
            // B = D - U_{n-1}^T C_{n-1}, rhs = -g - U_{n-1}^T d'_{n-1}
#pragma unroll
            for (int q = 0; q < 6; ++q) {
                w.bx = __fma_rn(-nuc[q], __shfl_sync(FULL, cx, 6 * g + q), w.bx);
                w.b = __fma_rn(-nuc[q], __shfl_sync(FULL, cu, 6 * g + q), w.b);
            }
        }
        // The next node's entries are requested only now: a wait for this
        // node's would otherwise wait for them too.
        if (!tip) {
            pd += 36; pu += 36; pux += 36; px += step;
            nd = *pd; nx = *px; nu = *pu; nux = *pux;
#pragma unroll
            for (int q = 0; q < 6; ++q) nuc[q] = puc[6 * q];
            puc += 36;
        }
        if (g == 1) w.ux = w.bx;
        {
            const bool first = lane == 0, diagonal = first || (wide && r == g + 1);
            const unsigned long long mag =
                (unsigned long long)__double_as_longlong(first ? w.bx : w.b) & 0x7fffffffffffffffull;
            const unsigned hi = diagonal ? unsigned(mag >> 32) : 0u;
            const unsigned mh = __reduce_max_sync(FULL, hi);
            const unsigned ml = __reduce_max_sync(FULL, diagonal && hi == mh ? unsigned(mag) : 0u);
            const double shifted = __dadd_rn(first ? w.bx : w.b, diagonal_shift((unsigned long long)mh << 32 | ml));
            if (first) w.bx = shifted;
            else if (diagonal) w.b = shifted;
        }
        WarpNode x = w;
        if (eliminate_node<false>(x, lane, g, r)) {
            x = w;
            if (eliminate_node<true>(x, lane, g, r) && !failed) {
                failed = true;
                if (lane == 0) atomicExch(&d.sc->solve_failed, 1);
            }
        }
        cu = __dmul_rn(x.u, x.ipiv);
        cx = __dmul_rn(x.ux, x.ipiv);
        if (wide) *pc = cu;  // of a failed strand nothing is read
        if (g < 2) *pcx = cx;
        pc += 36;
        pcx += step;
    }
    if (failed) return;
    __syncwarp();  // C_n and d'_n written by the other lanes of this warp
    substitute_back(d, begin, len, ring, lane, r);
}

// One strand on a team of three warps (on three sub-partitions):
// * the pivot warp holds B_n, row r of columns 1 ... 5 in lane 6 g + r and
//   column 0 in the lanes g = 0 once more, adds the shift and runs the six
//   pivot steps; the reciprocal of every candidate is taken beside the pivot
//   search.  It publishes each step's row factors, pivot and reciprocal and
//   goes on without waiting;
// * two column warps hold one entry of [U_n | rhs_n] a lane (columns 0 ... 4;
//   column 5 and the right-hand side), follow the published steps, scale the
//   rows, store C_n and d'_n and form the same entries of the next Schur
//   complement and right-hand side (column c of B_{n+1} needs column c of C_n
//   only), which goes back to the pivot warp.
// On one warp the updates of U sit in the pivot chain, since FP64 instructions
// and shuffles issue in order, and each node's Schur complement waits for all
// of them.  What bounds the team is the chain of six pivot steps (2,700 of the
// 4,000 cycles a node), then the Schur complement (540), the scaling (160) and
// the hand-overs.  It has more FP64 instructions in flight for the same
// result, so it pays while a sub-partition has less work than the longest
// chain: a solve of 100 strands of 16-160 nodes 384 -> 311 us, of 1,200 451 ->
// 413, of 2,200 495 -> 513.
struct TeamShared {
    double B[36];      // B_n row-major, from the column warps
    double fp[6][6];   // row factors a[r][col] / pivot of each step
    double ip[6];      // pivot reciprocals
    int pivot[6];      // pivot rows
    int redo;          // the node is eliminated again with the exact search
    BackRing ring;
};

// Named barriers of a team: 1 ... 6 the pivot steps (the pivot warp arrives,
// the column warps wait), 7 all three warps.
constexpr int kTeam = 96;
__device__ __forceinline__ void team_wait(int id) { asm volatile("bar.sync %0, 96;" ::"r"(id) : "memory"); }
__device__ __forceinline__ void team_arrive(int id) { asm volatile("bar.arrive %0, 96;" ::"r"(id) : "memory"); }

// The six pivot steps on b and (column 0) bx.  The pivot search compares the
// top 29 bits of the magnitudes with the row beside them, in one warp
// reduction; EXACT compares all bits and checks the pivots.  Returns whether,
// for !EXACT, some step needs EXACT (candidates equal in those bits, or a
// pivot outside [1e-30, 2^1022)), which the column warps learn with the last
// step, and for EXACT, whether a pivot failed.
template<bool EXACT> __device__ __forceinline__ bool team_pivots(double b, double bx, TeamShared &sh, int lane, int g, int r)
{
    const unsigned FULL = 0xffffffffu;
    bool flag = false;
#pragma unroll
    for (int col = 0; col < 6; ++col) {
        const int base = col == 0 ? 0 : 6 * (col - 1);  // first lane of the pivot column
        const double mine = col == 0 ? bx : b;
        // The first row of the largest magnitude, among rows col ... 5.
        const bool cand = lane >= base + col && lane < base + 6;
        const unsigned hi = cand ? unsigned(__double2hiint(mine)) & 0x7fffffffu : 0u;
        const unsigned key = EXACT ? hi : cand ? (hi & ~7u) | unsigned(5 - r) : 0u;
        const unsigned best = __reduce_max_sync(FULL, key);
        int pivot = 5 - int(best & 7u);
        if (EXACT) {
            const unsigned lo = cand && hi == best ? unsigned(__double2loint(mine)) : 0u;
            const unsigned ml = __reduce_max_sync(FULL, lo);
            pivot = 5 - int(__reduce_max_sync(FULL, cand && hi == best && lo == ml ? unsigned(5 - r) : 0u));
            flag |= pivot_fails((unsigned long long)best << 32 | ml);
        } else {
            const unsigned off = (r != pivot) & cand ? key ^ best : 8u;
            const unsigned low = best - 0x39b44850u;  // wraps below the least pivot
            flag |= (off < 8u) | (low >= 0x7fd00000u - 0x39b44850u);
        }
        const int partner = r == col ? pivot : (r == pivot ? col : r);
        const double fcol = __shfl_sync(FULL, mine, base + partner);
        double xb = 0.0;
        if (col < 5) {
            xb = __shfl_sync(FULL, b, 6 * g + pivot);
            if (pivot != col) b = __shfl_sync(FULL, b, 6 * g + partner);
        }
        const double rc = EXACT ? dm::recip_rn(mine) : dm::recip_normal(mine);
        if (col == 5 && !EXACT) flag = __any_sync(FULL, flag);
        const double ip = __shfl_sync(FULL, rc, base + pivot);
        const double fp = __dmul_rn(fcol, ip);
        if (col < 5) b = r == col ? b : __fma_rn(-fp, xb, b);
        // Lanes that hold the same value write the same word: no branch.
        sh.fp[col][r] = fp;
        sh.ip[col] = ip;
        sh.pivot[col] = pivot;
        if (col == 5) sh.redo = !EXACT && flag ? 1 : 0;
        team_arrive(1 + col);
    }
    return flag;
}

template<class D> __device__ __forceinline__ void team_pivot_warp(const D &d, uint32_t len, TeamShared &sh, int lane, int g, int r)
{
    const unsigned FULL = 0xffffffffu;
    const bool wide = g < 5;
    for (uint32_t t = 0; t < len; ++t) {
        team_wait(7);  // B_t is in shared memory
        double b = sh.B[6 * r + (wide ? g + 1 : 0)], bx = sh.B[6 * r];
        {
            const bool first = lane == 0, diagonal = first || (wide && r == g + 1);
            const unsigned long long mag = (unsigned long long)__double_as_longlong(first ? bx : b) & 0x7fffffffffffffffull;
            const unsigned hi = diagonal ? unsigned(mag >> 32) : 0u;
            const unsigned mh = __reduce_max_sync(FULL, hi);
            const unsigned ml = __reduce_max_sync(FULL, diagonal && hi == mh ? unsigned(mag) : 0u);
            const double shifted = __dadd_rn(first ? bx : b, diagonal_shift((unsigned long long)mh << 32 | ml));
            if (first) bx = shifted;
            else if (diagonal) b = shifted;
        }
        if (team_pivots<false>(b, bx, sh, lane, g, r)) {
            team_wait(7);  // the column warps have read every step
            if (team_pivots<true>(b, bx, sh, lane, g, r) && lane == 0) atomicExch(&d.sc->solve_failed, 1);
        }
    }
}

// Column warp w (0 or 1).  Every lane reads through pointers of its own,
// without conditions (a divergent one costs more than the read): lanes without
// an entry read a neighbour's and nothing uses it.
template<class D>
__device__ __forceinline__ void team_column_warp(const D &d, uint32_t begin, uint32_t len, TeamShared &sh, int lane, int g, int r, int w)
{
    const unsigned FULL = 0xffffffffu;
    const bool rhs = w == 1 && g == 1;                     // this lane holds the right-hand side
    const bool entry = w == 0 ? g < 5 : g < 2;             // ... something at all
    const int c = w == 0 ? (g < 5 ? g : 0) : 5;            // column of B and U
    const double *pd = rhs ? d.grad + 6 * size_t(begin) + r : d.diag + 36 * size_t(begin) + 6 * r + c;
    const double *pu = d.upper + 36 * size_t(begin) + 6 * r + c, *puc = d.upper + 36 * size_t(begin) + r;
    double *pc = rhs ? d.dprime + 6 * size_t(begin) + r : d.cprime + 36 * size_t(begin) + 6 * r + c;
    const int step = rhs ? 6 : 36, sign = rhs ? int(0x80000000) : 0;
    double nd = *pd, nu = *pu, nuc[6];
    double acc = __hiloint2double(__double2hiint(nd) ^ sign, __double2loint(nd));
    for (uint32_t t = 0; t < len; ++t) {
        const bool tip = t + 1 == len;  // U_n couples to nothing there
        if (entry && !rhs) sh.B[6 * r + c] = acc;
        const double start = rhs ? acc : tip ? 0.0 : nu;
        team_wait(7);  // hand B_t over
        if (!tip) {
            // U_t's column r for the Schur complement, the next D and U.
#pragma unroll
            for (int q = 0; q < 6; ++q) nuc[q] = puc[6 * q];
            pd += step; pu += 36; puc += 36;
            nd = *pd; nu = *pu;
        }
        double u;
        for (;;) {
            u = start;
#pragma unroll
            for (int col = 0; col < 6; ++col) {
                team_wait(1 + col);
                const int pivot = sh.pivot[col];
                const double fp = sh.fp[col][r];
                const double x = __shfl_sync(FULL, u, 6 * g + pivot);
                if (pivot != col) u = __shfl_sync(FULL, u, 6 * g + (r == col ? pivot : (r == pivot ? col : r)));
                u = r == col ? u : __fma_rn(-fp, x, u);
            }
            if (sh.redo == 0) break;
            team_wait(7);
        }
        const double scaled = __dmul_rn(u, sh.ip[r]);  // row r of C_t, or d'_t
        if (entry) *pc = scaled;
        pc += step;
        if (!tip) {
            // B = D - U_t^T C_t, rhs = -g - U_t^T d'_t
            acc = __hiloint2double(__double2hiint(nd) ^ sign, __double2loint(nd));
#pragma unroll
            for (int q = 0; q < 6; ++q) acc = __fma_rn(-nuc[q], __shfl_sync(FULL, scaled, 6 * g + q), acc);
        }
    }
}

template<class D> __device__ __forceinline__ void solve_strand_team(const D &d, uint32_t k, TeamShared &sh)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane / 6, r = lane - 6 * g;
    uint32_t begin, len;
    strand_range(d, k, begin, len);
    if (len == 0) return;
    if (warp == 0) team_pivot_warp(d, len, sh, lane, g, r);
    else team_column_warp(d, begin, len, sh, lane, g, r, warp - 1);
    team_wait(7);  // C and d' are stored
    if (warp != 0) return;
    substitute_back(d, begin, len, sh.ring, lane, r);
}

// Five strands on one warp: lane 6 s + r holds row r of strand first + s of
// the solve order (up to the last one); lanes 30 and 31 are idle.
template<class D> __device__ __forceinline__ void solve_strands_five(const D &d, uint32_t first)
{
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int grp = lane / 6, r = lane - 6 * grp, base = 6 * grp;
    const uint32_t k = first + uint32_t(grp);
    uint32_t begin = 0, len = 0;
    if (grp < kStrandsPerWarp && k < d.S) strand_range(d, k, begin, len);
    const uint32_t maxlen = __reduce_max_sync(FULL, len);
    double nd[6], nu[6], nuc[6], ng = 0.0;
    auto fetch = [&](uint32_t t) {
        const bool on = t < len;
        const size_t n = begin + t;
#pragma unroll
        for (int j = 0; j < 6; ++j) nd[j] = on ? d.diag[36 * n + 6 * r + j] : 0.0;
        ng = on ? d.grad[6 * n + r] : 0.0;
        const bool up = on && t + 1 < len;
#pragma unroll
        for (int j = 0; j < 6; ++j) nu[j] = up ? d.upper[36 * n + 6 * r + j] : 0.0;
#pragma unroll
        for (int q = 0; q < 6; ++q) nuc[q] = (on && t > 0) ? d.upper[36 * (n - 1) + 6 * q + r] : 0.0;
    };
    fetch(0);
    double Cprev[6], dprev = 0.0;
#pragma unroll
    for (int j = 0; j < 6; ++j) Cprev[j] = 0.0;
    bool failed = false;
    for (uint32_t t = 0; t < maxlen; ++t) {
        const bool on = t < len && !failed;
        const size_t n = begin + t;
        double a[6], u[6], ucol[6], rhs = -ng;
#pragma unroll
        for (int j = 0; j < 6; ++j) { a[j] = nd[j]; u[j] = nu[j]; }
#pragma unroll
        for (int q = 0; q < 6; ++q) ucol[q] = nuc[q];
        if (t + 1 < maxlen) fetch(t + 1);
        if (t > 0) {
            // B = D - U_{n-1}^T C_{n-1}, rhs = -g - U_{n-1}^T d'_{n-1}
#pragma unroll
            for (int q = 0; q < 6; ++q) {
#pragma unroll
                for (int j = 0; j < 6; ++j) a[j] = __fma_rn(-ucol[q], __shfl_sync(FULL, Cprev[j], base + q), a[j]);
                rhs = __fma_rn(-ucol[q], __shfl_sync(FULL, dprev, base + q), rhs);
            }
        }
        double diag_r = 0.0;
#pragma unroll
        for (int j = 0; j < 6; ++j) if (j == r) diag_r = a[j];
        unsigned long long smax = 0ull;
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            const unsigned long long b = (unsigned long long)__double_as_longlong(__shfl_sync(FULL, diag_r, base + q)) & 0x7fffffffffffffffull;
            smax = b > smax ? b : smax;
        }
        const double shifted = __dadd_rn(diag_r, diagonal_shift(smax));
#pragma unroll
        for (int j = 0; j < 6; ++j) if (j == r) a[j] = shifted;
        bool ok = true;
        double ipiv = 1.0;
#pragma unroll
        for (int col = 0; col < 6; ++col) {
            const double rc = dm::recip_rn(a[col]);
            const unsigned long long mb = (unsigned long long)__double_as_longlong(a[col]) & 0x7fffffffffffffffull;
            int pivot = col;
            unsigned long long best = __shfl_sync(FULL, mb, base + col);
#pragma unroll
            for (int row = col + 1; row < 6; ++row) {
                const unsigned long long vrow = __shfl_sync(FULL, mb, base + row);
                if (vrow > best) { best = vrow; pivot = row; }
            }
            if (pivot_fails(best)) ok = false;
            const int partner = r == col ? pivot : (r == pivot ? col : r);
            const int src = base + partner, prow = base + pivot;
            const double ip = __shfl_sync(FULL, rc, prow);
            const double fp = __dmul_rn(__shfl_sync(FULL, a[col], src), ip);
            if (r == col) ipiv = ip;
            // The pivot row's entries are read before the swap: row col of
            // the swapped block is row pivot of this one.
            double xa[6], xu[6];
#pragma unroll
            for (int j = col + 1; j < 6; ++j) xa[j] = __shfl_sync(FULL, a[j], prow);
#pragma unroll
            for (int j = 0; j < 6; ++j) xu[j] = __shfl_sync(FULL, u[j], prow);
            const double xr = __shfl_sync(FULL, rhs, prow);
            if (__any_sync(FULL, pivot != col)) {
#pragma unroll
                for (int j = col + 1; j < 6; ++j) a[j] = __shfl_sync(FULL, a[j], src);
#pragma unroll
                for (int j = 0; j < 6; ++j) u[j] = __shfl_sync(FULL, u[j], src);
                rhs = __shfl_sync(FULL, rhs, src);
            }
#pragma unroll
            for (int j = col + 1; j < 6; ++j) a[j] = (r == col) ? a[j] : __fma_rn(-fp, xa[j], a[j]);
#pragma unroll
            for (int j = 0; j < 6; ++j) u[j] = (r == col) ? u[j] : __fma_rn(-fp, xu[j], u[j]);
            rhs = (r == col) ? rhs : __fma_rn(-fp, xr, rhs);
        }
#pragma unroll
        for (int j = 0; j < 6; ++j) u[j] = __dmul_rn(u[j], ipiv);
        rhs = __dmul_rn(rhs, ipiv);
        if (on && !ok) {
            failed = true;
            if (r == 0) atomicExch(&d.sc->solve_failed, 1);
        }
        // u now holds row r of C_n (zero at the strand tip), rhs = d'_n[r].
#pragma unroll
        for (int j = 0; j < 6; ++j) Cprev[j] = u[j];
        dprev = rhs;
        if (on && !failed) {
#pragma unroll
            for (int j = 0; j < 6; ++j) d.cprime[36 * n + 6 * r + j] = u[j];
            d.dprime[6 * n + r] = rhs;
        }
    }
    // Back substitution d_n = d'_n - C_n d_{n+1}.
    double next = 0.0;
    double pc[6], pd = 0.0;
    auto fetch_back = [&](uint32_t t) {
        const bool on = t < len && !failed;
        const size_t n = begin + t;
        pd = on ? d.dprime[6 * n + r] : 0.0;
#pragma unroll
        for (int q = 0; q < 6; ++q) pc[q] = on ? d.cprime[36 * n + 6 * r + q] : 0.0;
    };
    if (maxlen) fetch_back(maxlen - 1);
    for (uint32_t t = maxlen; t-- > 0;) {
        const bool on = t < len && !failed;
        const size_t n = begin + t;
        double value = pd, crow[6];
#pragma unroll
        for (int q = 0; q < 6; ++q) crow[q] = pc[q];
        if (t > 0) fetch_back(t - 1);
        const bool coupled = on && t + 1 < len;
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            const double dq = __shfl_sync(FULL, next, base + q);
            if (coupled) value = __fma_rn(-crow[q], dq, value);
        }
        if (on) d.dir[6 * n + r] = value;
        next = on ? value : 0.0;
    }
}

}  // namespace
}  // namespace khs
