// GB300 device engine (see khs_engine.hpp).
//
// Device data layout (one arena allocation, 256-byte aligned sub-arrays):
//   node state     q, q_old, v, q_snap, v_snap, q_base   [N][6] FP64
//   solver vectors grad, dir, precond, dprime            [N][6] FP64
//   block matrices diag, upper, cprime                   [N][36] FP64
//   rotation cache R = exp(u) Ref, left Jacobian Jl      [N][9] FP64
//   element parts  contributions of the element whose left node is n
//                  (as_i_*) and whose right node is n (as_j_*) so every
//                  node sums its two incident elements in a fixed order
//                  without atomics
//   elements       (i, j, contact flag, L0, gamma0, kappa0), energies,
//                  contact records                        [E]
//   strands        first, count, fixed prefix, length-sorted order [S]
//   collider       triangles [T][3], current/old/frame-start/pending
//                  vertices [V][3], BVH in right-first preorder with escape
//                  indices (stackless traversal) and parent links (one-launch
//                  bottom-up refit)
//
// Kernels (thread per node / element / BVH leaf unless noted):
//   per substep   k_begin_substep, k_refit (eight lanes per leaf),
//                 k_sweep_collect, k_sweep_near, k_advance_pairs,
//                 k_sweep_record, k_update_velocity, k_friction(+apply)
//   evaluation    k_positions, k_node_eval, k_contact_filter, k_contact_near
//                 (warp per element with cached leaves, block where they are
//                 many), k_contact_exact (five warps to 32 pairs),
//                 k_contact_select, k_elem_eval or k_elem_ends (two threads
//                 per element), k_node_sum (thread per two block entries),
//                 k_reduce_eval (both levels: the last block to finish
//                 reduces the partials)
//   direction     k_block_solve (blocks of one warp, a strand or five at a
//                 time from a longest-first queue) or k_block_solve_team
//                 (three warps per strand),
//                 [float-float form: k_ff_factor, k_ff_residual, k_ff_correct],
//                 k_steepest, k_scale, k_reduce_dir, k_limit
//   CCD           k_ccd_collect, k_ccd_near, k_advance_pairs; k_ccd where the
//                 pair list is full
//   queries       k_contact, k_contact_query_records, k_gather
//   root targets  k_root_tangents, k_root_transport, k_root_frames (three
//                 lanes per strand), k_root_rotations: per call of
//                 khsUpdateRootTargets / khsSetRootAnimationFrame
// Reductions are two-level (fixed per-block trees, then one block over the
// partials) and therefore deterministic.
#include "khs_engine.hpp"
#include "khs_device_math.cuh"
#include "khs_ff.cuh"
#include "khs_block_solve.cuh"

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <limits>
#include <mutex>
#include <numeric>
#include <stdexcept>

namespace khs {
namespace {

#define KHS_CUDA(call)                                                                         \
    do {                                                                                       \
        const cudaError_t khs_err = (call);                                                    \
        if (khs_err != cudaSuccess) throw std::runtime_error(std::string("CUDA: ") + cudaGetErrorString(khs_err)); \
    } while (0)

using dm::V;
using dm::M;

constexpr int kBlock = 256;
// Element and node evaluation: FP64 bound with few registers to spare, so one
// or two warps keep a sub-partition's FP64 pipe busy and small blocks spread a
// small scene over all of them.
constexpr int kEvalBlock = 64;
// Every kernel starts with this.  The launches of an evaluation or a step of
// the search are small and follow one another on a stream; they are launched
// with programmatic serialization, so a kernel's blocks are brought up while
// the previous kernel drains and wait here until it has completed and its
// writes are visible.  A kernel lets its successor come up only after its own
// wait, so one kernel at most is waiting behind the running one.
// A frame with it: 64 strands on a sphere 2.89 -> 2.55 ms (220 launches), 12
// strands at a mesh pole 79.8 -> 74.4 (3,700), 700 strands of the body scene
// 73.0 -> 69.9, all 6,757 310.0 -> 305.7.
__device__ __forceinline__ void follow_previous()
{
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
}

constexpr int kPartials = 304;  // 2 reduction blocks per SM on a 152-SM GB300
constexpr uint32_t kNone = 0xffffffffu;
constexpr uint64_t kCheckpointMagic = 0x3154504348534bULL;  // same blob header as the reference
constexpr uint8_t kFlagActive = 1, kFlagInfeasible = 2, kFlagEnergy = 4, kFlagClosest = 8;

inline unsigned grid_for(size_t n, int block = kBlock) { return unsigned((n + block - 1) / block); }
// Every solver runs on device 0 (Engine::initialize selects it).
constexpr int kDevice = 0;

// Scalars produced by one evaluation / direction pass (host-mapped).
struct Mailbox {
    double objective, elastic, contact, kinetic, minimum_gap, grad_norm2;
    unsigned long long candidates, active;
    int feasible;
    int solve_failed;
    double slope, dir_norm2, max_translation;
    unsigned long long ccd_bits;
    unsigned long long pair_count;
    uint32_t sweep_fail;
    uint32_t refine_bits;
    // The direction as solved (k_reduce_dir); slope, dir_norm2 and
    // max_translation are those of the limited one after k_limit.
    double dir_slope, dir_max_translation;
    int dir_solve_failed;
    int dir_pad;
};

// Atomic targets live in device memory; the publishing kernels copy them to
// the host-mapped mailbox and reset them for the next use.
struct Scalars {
    unsigned long long ccd_bits;
    // Room asked for in the bounded lists, in 64 bits: a full list goes on
    // counting (claim_range, append_slot), with elements asking again at every
    // evaluation of a substep, and a count that came round would hand out
    // ranges in use.
    unsigned long long pair_count;
    unsigned long long surv_count;  // pairs of the contact pass's FP64 pool
    unsigned long long pool_used;   // entries of the leaf pool, since the last cache rebuild
    uint32_t sweep_fail;
    int solve_failed;
    uint32_t solve_next;  // next strand group of the block-solve work queue
    uint32_t refine_bits; // largest relative refinement correction (FP32 bits)
    uint32_t near_count;  // elements queued for the warp-cooperative contact pass
    uint32_t ccd_near;    // elements queued for the warp-cooperative CCD pass
    uint32_t eval_done;   // blocks of k_reduce_eval finished (the last one reduces the partials)
    uint32_t dir_done, ccd_done;  // the same for the direction's sums and the CCD pairs
    double trial_alpha;   // first line-search step from the last CCD bound (publish_ccd)
    double max_translation;  // largest free-node translation of the last reduced direction
    uint32_t wide_count;  // elements queued for k_contact_near that take a block each
};

struct Partial {
    double node_energy, kinetic, elastic, contact, min_gap, grad2;
    unsigned long long candidates, active;
    int infeasible;
    int pad;
};

struct DirPartial {
    double slope, dnorm2, max_translation;
};

struct SweepRecord {
    uint32_t claimed, strand, element, triangle;
    double distance, required, clearance, displacement;
    double hair_start[3], hair_end[3], collider_point[3];
};

// POD view of every device array (passed by value to kernels).
struct View {
    uint32_t N, E, S, V, T, B;
    double *q, *q_old, *v, *q_base, *grad, *dir, *precond;
    double *inertia;  // inertia + damping diagonal of each node's block [N][6]
    float *q32, *e32;  // FP32 copies of the node positions and of positions + direction [N][3]
    double *rot, *jl, *node_energy, *node_kinetic;
    double *diag, *upper, *cprime, *dprime;
    double *as_i_g, *as_j_g, *as_i_h, *as_j_h, *as_i_f, *as_j_f;
    const double *ref, *mass, *rmass;
    const uint8_t *fixed;
    const int32_t *elem_left, *elem_right;
    const uint32_t *ei, *ej, *estrand;
    const uint8_t *econtact;
    const double *L0, *invL, *gamma0, *kappa0;  // invL = 1 / L0
    double *e_el, *e_co, *c_gap;
    double *push;  // the barrier's gradient and curvature [E][kPush] (element_barrier)
    uint32_t *c_cand, *c_tri;
    uint8_t *c_flags;
    const uint32_t *sfirst, *scount, *sfixed, *sorder;
    const uint32_t *tri;
    double *col_cur, *col_old;
    float *col32;  // FP32 copy of col_cur for the FP32 search by one thread (closest_triangle)
    double *blo, *bhi;  // leaves only: the FP64 boxes of the exact leaf test
    // The tree over old and new positions, for the moving-collider sweep.
    double *swept_lo, *swept_hi;
    float4 *swept_node;
    // Each BVH node packed in 32 bytes (FP32 outward-rounded box,
    // escape index, leaf range), the per-element contact result of the
    // separate contact pass, and the CCD (element, triangle) work list.
    float4 *bnode;
    double *c_t, *c_bary, *c_dist;
    uint32_t *pair_elem, *pair_tri;
    uint32_t pair_capacity;
    // Per-substep leaf cache of the contact pass: the leaves (DFS
    // order) whose FP32 box overlaps the element box grown by kCacheSlack,
    // and the element's node positions when they were collected.
    uint32_t *cache_leaf;
    uint8_t *cache_n;
    // Leaf lists of elements with more than kCacheLeaves leaves: a bump
    // pool (reset at each cache rebuild); such an element's first two
    // cache_leaf slots hold its offset and count.
    uint32_t *leaf_pool;
    uint32_t leaf_pool_capacity;
    float *cache_x32;  // FP32 node positions when the leaves were collected [E][6]
    // Contact pass in several launches: FP32 vertex records of every triangle
    // in leaf order (a, b, c as three float4, the triangle index in the first
    // .w), and a pool of (element, triangle) pairs for the FP64 pass with
    // their closest pairs (distance, t, barycentrics).  An element's pairs
    // are surv_n from surv_off on, in traversal order.
    float4 *tri32, *tri32_old;  // FP32 records of col_cur and col_old
    // Mixed-form factors in float-float (hi, lo): B_n^-1 and C_n rows [N][36],
    // d'_n [N][6], and the diagonal shift used at each node.
    float2 *ff_inv, *ff_c, *ff_d;
    float *ff_shift;
    uint32_t *surv_elem, *surv_tri;
    uint32_t surv_capacity;
    uint32_t *surv_off, *surv_n;
    uint32_t *near_list;  // elements with cached leaves, one warp each in k_contact_near (from the end: a block each)
    double *surv_res;
    const uint32_t *solve_items;  // work items of the block solve, at most one per strand
    const uint32_t *bfirst, *bcount, *border, *bleaves;
    const int32_t *bparent;
    const uint32_t *bleft, *bright;
    uint32_t *brefit;
    uint32_t L;
    Partial *partials;
    DirPartial *dpartials;
    Scalars *sc;          // device
    Mailbox *mail;        // host-mapped
    SweepRecord *sweep;   // host-mapped
    // material / desc
    double radius, offset, dhat, kc, friction, smoothing, damping, min_gap;
    double gx, gy, gz;
    dm::Weights w;
    double young, poisson, shear_corr;
    int has_collider;
    struct Padding { double exact; float up, down; } contact_pad, ccd_pad;  // radius + offset + dhat, ... + min_gap
};

// Next free slot of a work list whose length is *count, for every lane that
// calls it: the lanes that arrive together take consecutive slots with one
// atomic (a per-lane atomic on one address serialises at L2 when tens of
// thousands of elements append in one launch).  Slot order within a list is
// not meaningful to any of its consumers.
template<class T> __device__ __forceinline__ T append_slot(T *count)
{
    namespace cg = cooperative_groups;
    const cg::coalesced_group g = cg::coalesced_threads();
    T base = 0;
    if (g.thread_rank() == 0) base = atomicAdd(count, T(g.size()));
    return g.shfl(base, 0) + g.thread_rank();
}

// n entries of a list of `capacity` entries, *used of which were asked for so
// far: their offset, or kNone without room.
__device__ __forceinline__ uint32_t claim_range(unsigned long long *used, uint32_t n, uint32_t capacity)
{
    const unsigned long long off = atomicAdd(used, (unsigned long long)n);
    return off + n <= capacity ? uint32_t(off) : kNone;
}

__device__ __forceinline__ V load3(const double *p) { return dm::v(p[0], p[1], p[2]); }
__device__ __forceinline__ void store3(double *p, V a) { p[0] = a.x; p[1] = a.y; p[2] = a.z; }
__device__ __forceinline__ M load9(const double *p)
{
    M r;
#pragma unroll
    for (int k = 0; k < 9; ++k) r.m[k] = p[k];
    return r;
}
__device__ __forceinline__ V tri_vertex(const View &d, uint32_t t, int c) { return load3(d.col_cur + 3 * size_t(d.tri[3 * t + c])); }

// Next node of a stackless walk after skipping node i's subtree.  In the
// preorder layout a node's escape index is the end of its subtree, so it is
// always greater than i; anything else (a corrupted or uninitialised tree)
// ends the walk instead of restarting it.
__device__ __forceinline__ uint32_t escape_from(uint32_t i, uint32_t escape) { return escape > i ? escape : 0xffffffffu; }

// Exact FP64 leaf test of the reference (al <= bu + p && bl <= au + p per
// axis) decided in FP32 when possible: if the query box rounded inwards
// still overlaps the leaf box rounded inwards (one ulp inside the stored
// outward box) with the padding rounded down, the FP64 test is true; if the
// outward FP32 test failed it is false; only inside the rounding band is
// the FP64 test evaluated.
struct QueryBox {
    float olx, oly, olz, ohx, ohy, ohz, opad;  // outward-rounded box and padding
    float ilx, ily, ilz, ihx, ihy, ihz, ipad;  // inward-rounded box and padding
};

using Pad = View::Padding;  // with its roundings

__device__ __forceinline__ QueryBox make_query(V lo, V hi, Pad pad)
{
    QueryBox qb;
    qb.olx = __double2float_rd(lo.x); qb.oly = __double2float_rd(lo.y); qb.olz = __double2float_rd(lo.z);
    qb.ohx = __double2float_ru(hi.x); qb.ohy = __double2float_ru(hi.y); qb.ohz = __double2float_ru(hi.z);
    qb.opad = pad.up;
    qb.ilx = __double2float_ru(lo.x); qb.ily = __double2float_ru(lo.y); qb.ilz = __double2float_ru(lo.z);
    qb.ihx = __double2float_rd(hi.x); qb.ihy = __double2float_rd(hi.y); qb.ihz = __double2float_rd(hi.z);
    qb.ipad = pad.down;
    return qb;
}

// The same box from FP32 copies of the points it spans (lo32, hi32 =
// componentwise min / max of the rounded coordinates): rounding to nearest
// moved each coordinate by at most 2^-24 of its magnitude, so widening by
// 2^-23 of the magnitude (plus 1e-30) bounds the FP64 box from outside and
// narrowing by the same bounds it from inside.
__device__ __forceinline__ QueryBox make_query_f(const float lo32[3], const float hi32[3], Pad pad)
{
    QueryBox qb;
    const float k = 1.1920929e-7f;  // 2^-23
    qb.olx = __fsub_rd(lo32[0], __fmaf_ru(fabsf(lo32[0]), k, 1e-30f));
    qb.oly = __fsub_rd(lo32[1], __fmaf_ru(fabsf(lo32[1]), k, 1e-30f));
    qb.olz = __fsub_rd(lo32[2], __fmaf_ru(fabsf(lo32[2]), k, 1e-30f));
    qb.ohx = __fadd_ru(hi32[0], __fmaf_ru(fabsf(hi32[0]), k, 1e-30f));
    qb.ohy = __fadd_ru(hi32[1], __fmaf_ru(fabsf(hi32[1]), k, 1e-30f));
    qb.ohz = __fadd_ru(hi32[2], __fmaf_ru(fabsf(hi32[2]), k, 1e-30f));
    qb.ilx = __fadd_ru(lo32[0], __fmaf_ru(fabsf(lo32[0]), k, 1e-30f));
    qb.ily = __fadd_ru(lo32[1], __fmaf_ru(fabsf(lo32[1]), k, 1e-30f));
    qb.ilz = __fadd_ru(lo32[2], __fmaf_ru(fabsf(lo32[2]), k, 1e-30f));
    qb.ihx = __fsub_rd(hi32[0], __fmaf_ru(fabsf(hi32[0]), k, 1e-30f));
    qb.ihy = __fsub_rd(hi32[1], __fmaf_ru(fabsf(hi32[1]), k, 1e-30f));
    qb.ihz = __fsub_rd(hi32[2], __fmaf_ru(fabsf(hi32[2]), k, 1e-30f));
    qb.opad = pad.up;
    qb.ipad = pad.down;
    return qb;
}

__device__ __forceinline__ bool maybe_overlap(const QueryBox &q, float4 a, float4 b)
{
    return q.olx <= __fadd_ru(b.x, q.opad) && a.x <= __fadd_ru(q.ohx, q.opad) && q.oly <= __fadd_ru(b.y, q.opad) &&
           a.y <= __fadd_ru(q.ohy, q.opad) && q.olz <= __fadd_ru(b.z, q.opad) && a.z <= __fadd_ru(q.ohz, q.opad);
}

// box(lo, hi) gives the FP64 box, which the FP32 bounds nearly always make
// unnecessary (an FP64 minimum costs several FP64 issue slots).
template<class Box>
__device__ __forceinline__ bool leaf_overlap_exact(const View &d, uint32_t node, float4 a, float4 b, const QueryBox &q, double pad,
                                                   Box &&box)
{
    const bool surely = q.ilx <= __fadd_rd(nextafterf(b.x, -INFINITY), q.ipad) &&
                        nextafterf(a.x, INFINITY) <= __fadd_rd(q.ihx, q.ipad) &&
                        q.ily <= __fadd_rd(nextafterf(b.y, -INFINITY), q.ipad) &&
                        nextafterf(a.y, INFINITY) <= __fadd_rd(q.ihy, q.ipad) &&
                        q.ilz <= __fadd_rd(nextafterf(b.z, -INFINITY), q.ipad) &&
                        nextafterf(a.z, INFINITY) <= __fadd_rd(q.ihz, q.ipad);
    if (surely) return true;
    V lo, hi;
    box(lo, hi);
    return dm::boxes_overlap(lo, hi, load3(d.blo + 3 * size_t(node)), load3(d.bhi + 3 * size_t(node)), pad);
}

// Stackless BVH walk in the reference's visiting order over packed 32-byte
// nodes: one pair of 16-byte loads per visited node (box + escape, box + leaf
// range (first << 4 | count)).  Nodes are tested on outward-rounded FP32 boxes
// (a superset of the FP64 test, and an FP64 overlap of a leaf implies FP64
// overlap of every ancestor), leaves exactly, so the candidates and their
// order are those of a walk over FP64 boxes; an FP64 comparison costs as much
// as a multiply-add, twelve of them a node.  f receives the position of each
// candidate in leaf order (index into border and tri32).
template<class Box, class F> __device__ void bvh_positions_packed(const View &d, const QueryBox &q, double pad, Box &&box, F &&f)
{
    uint32_t i = 0;
    while (i < d.B) {
        const float4 a = __ldg(d.bnode + 2 * size_t(i)), b = __ldg(d.bnode + 2 * size_t(i) + 1);
        const uint32_t escape = __float_as_uint(a.w), leaf = __float_as_uint(b.w);
        if (!maybe_overlap(q, a, b)) { i = escape_from(i, escape); continue; }
        if (leaf == 0) { ++i; continue; }
        if (leaf_overlap_exact(d, i, a, b, q, pad, box)) {
            const uint32_t first = leaf >> 4, cnt = leaf & 15u;
            for (uint32_t k = first; k < first + cnt; ++k) f(k);
        }
        i = escape_from(i, escape);
    }
}

template<class F> __device__ void bvh_query_packed(const View &d, V lo, V hi, Pad pad, F &&f)
{
    bvh_positions_packed(d, make_query(lo, hi, pad), pad.exact, [&](V &l, V &h) { l = lo; h = hi; },
                         [&](uint32_t k) { f(d.border[k]); });
}

constexpr int kCacheLeaves = 32;
constexpr double kCacheSlack = 1.0e-3;  // metres each node may move before the cache is bypassed
constexpr uint8_t kCacheInvalid = 0xff;
constexpr uint8_t kCacheBig = 0xfe;     // cache_n of an element whose leaves live in the leaf pool

// Leaves whose FP32 outward box overlaps (lo, hi) padded by pad, in DFS
// order; the first cap are written to out, and the return value is the
// count of all of them.
__device__ uint32_t collect_leaves(const View &d, V lo, V hi, Pad pad, uint32_t *out, uint32_t cap)
{
    const QueryBox q = make_query(lo, hi, pad);
    uint32_t i = 0, n = 0;
    while (i < d.B) {
        const float4 a = __ldg(d.bnode + 2 * size_t(i)), b = __ldg(d.bnode + 2 * size_t(i) + 1);
        const uint32_t escape = __float_as_uint(a.w), leaf = __float_as_uint(b.w);
        if (!maybe_overlap(q, a, b)) { i = escape_from(i, escape); continue; }
        if (leaf == 0) { ++i; continue; }
        if (n < cap) out[n] = i;
        ++n;
        i = escape_from(i, escape);
    }
    return n;
}

// Collects the leaves around (lo, hi) into the element's cache slots; returns
// its cache_n.  More than kCacheLeaves, at a dense patch of the collider (a
// mesh pole, a seam), go to the pool, which the warp passes take 32 at a time.
__device__ __forceinline__ uint8_t leaves_to_cache(const View &d, uint32_t e, V lo, V hi, Pad pad)
{
    uint32_t *slots = d.cache_leaf + size_t(kCacheLeaves) * e;
    const uint32_t c = collect_leaves(d, lo, hi, pad, slots, kCacheLeaves);
    uint8_t nl = uint8_t(c);
    if (c > uint32_t(kCacheLeaves)) {
        const uint32_t off = claim_range(&d.sc->pool_used, c, d.leaf_pool_capacity);
        nl = kCacheInvalid;
        if (off != kNone) {
            collect_leaves(d, lo, hi, pad, d.leaf_pool + off, c);
            slots[0] = off;
            slots[1] = c;
            nl = kCacheBig;
        }
    }
    d.cache_n[e] = nl;
    return nl;
}

// The cached leaf list of element e with cache state nl (its cache_n):
// the element's own slots, or its range of the leaf pool; nullptr without
// a cache.
__device__ __forceinline__ const uint32_t *cached_leaves(const View &d, uint32_t e, uint8_t nl, uint32_t &count)
{
    const uint32_t *slots = d.cache_leaf + size_t(kCacheLeaves) * e;
    if (nl == kCacheInvalid) { count = 0; return nullptr; }
    if (nl == kCacheBig) { count = slots[1]; return d.leaf_pool + slots[0]; }
    count = nl;
    return slots;
}

// FP32 distance of a candidate from the FP32 vertex copy, relative to an
// FP32 origin (the segment start): no FP64 instruction.  Rounding the
// vertices, the origin and the segment end to FP32 moves each coordinate by
// at most 2^-24 of its magnitude, so the distance moves by at most
// sqrt(3) * 2^-24 * (|vertex| + |origin| + |end|)_inf < 2.5e-7 * M, with M
// bounding the absolute coordinates involved; that term is added to the
// relative margin of the FP32 distance itself.
__device__ __forceinline__ float candidate_distance_f(const View &d, uint32_t t, dm::F3 origin, dm::F3 p0, dm::F3 p1, float &m)
{
    const float *c32 = d.col32;
    const uint32_t i0 = d.tri[3 * t], i1 = d.tri[3 * t + 1], i2 = d.tri[3 * t + 2];
    const float ax = c32[3 * i0], ay = c32[3 * i0 + 1], az = c32[3 * i0 + 2];
    const float bx = c32[3 * i1], by = c32[3 * i1 + 1], bz = c32[3 * i1 + 2];
    const float cx = c32[3 * i2], cy = c32[3 * i2 + 1], cz = c32[3 * i2 + 2];
    const dm::F3 a = dm::f3(ax - origin.x, ay - origin.y, az - origin.z);
    const dm::F3 b = dm::f3(bx - origin.x, by - origin.y, bz - origin.z);
    const dm::F3 c = dm::f3(cx - origin.x, cy - origin.y, cz - origin.z);
    const float df = dm::segment_triangle_distance_f(p0, p1, a, b, c, m);
    const float vmax = fmaxf(fmaxf(fmaxf(fabsf(ax), fabsf(ay)), fmaxf(fabsf(az), fabsf(bx))),
                             fmaxf(fmaxf(fabsf(by), fabsf(bz)), fmaxf(fmaxf(fabsf(cx), fabsf(cy)), fabsf(cz))));
    const float omax = fmaxf(fmaxf(fabsf(origin.x), fabsf(origin.y)), fabsf(origin.z));
    const float emax = fmaxf(fmaxf(fabsf(p1.x), fabsf(p1.y)), fabsf(p1.z)) + omax;
    m += 2.5e-7f * (vmax + omax + emax) + 1.0e-9f;
    return df;
}

// ---- per-substep set-up ---------------------------------------------------

// Start of a substep, thread per node and per collider vertex.  Uncontracted
// lerps: the root targets and collider vertices feed the integer contact work,
// so they round exactly like a host evaluation.
struct SubstepTargets {
    const double *root_a, *rot_a, *root_b, *rot_b;  // [N][3]
    const double *col_a, *col_b;                    // [V][3]
    double f, dt;
};

__global__ void __launch_bounds__(kBlock) k_begin_substep(View d, SubstepTargets s)
{
    follow_previous();
    const uint32_t n = blockIdx.x * blockDim.x + threadIdx.x;
    const double f = s.f;
    if (d.has_collider && n < d.V) {
        const V cur = load3(d.col_cur + 3 * size_t(n));
        store3(d.col_old + 3 * size_t(n), cur);
        const V nv = dm::gadd(dm::gmul(load3(s.col_a + 3 * size_t(n)), 1.0 - f), dm::gmul(load3(s.col_b + 3 * size_t(n)), f));
        store3(d.col_cur + 3 * size_t(n), nv);
        d.col32[3 * size_t(n)] = float(nv.x); d.col32[3 * size_t(n) + 1] = float(nv.y); d.col32[3 * size_t(n) + 2] = float(nv.z);
    }
    if (n >= d.N) return;
    double q[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) { q[k] = d.q[6 * size_t(n) + k]; d.q_old[6 * size_t(n) + k] = q[k]; }
    if (!d.fixed[n]) return;
    const V p = dm::gadd(dm::gmul(load3(s.root_a + 3 * size_t(n)), 1.0 - f), dm::gmul(load3(s.root_b + 3 * size_t(n)), f));
    const V r = dm::gadd(dm::gmul(load3(s.rot_a + 3 * size_t(n)), 1.0 - f), dm::gmul(load3(s.rot_b + 3 * size_t(n)), f));
    const double vals[6] = {p.x, p.y, p.z, r.x, r.y, r.z};
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        d.q[6 * size_t(n) + k] = vals[k];
        d.v[6 * size_t(n) + k] = (vals[k] - q[k]) / s.dt;
    }
}

// Minima and maxima of coordinates on order-preserving integers: an FP64
// minimum costs several FP64 issue slots, 144 to 288 of them a leaf.  A NaN is
// skipped, as fmin and fmax do.
__device__ __forceinline__ long long order_key(double x)
{
    const long long b = __double_as_longlong(x);
    return b ^ ((b >> 63) & 0x7fffffffffffffffll);
}
__device__ __forceinline__ double from_key(long long k) { return __longlong_as_double(k ^ ((k >> 63) & 0x7fffffffffffffffll)); }

struct KeyBox {
    long long lo[3], hi[3];
    __device__ void clear()
    {
#pragma unroll
        for (int k = 0; k < 3; ++k) { lo[k] = order_key(1e300); hi[k] = order_key(-1e300); }
    }
    __device__ void add(V p)
    {
        const double x[3] = {p.x, p.y, p.z};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const long long b = __double_as_longlong(x[k]), key = order_key(x[k]);
            if ((b & 0x7fffffffffffffffll) > 0x7ff0000000000000ll) continue;
            lo[k] = min(lo[k], key);
            hi[k] = max(hi[k], key);
        }
    }
    // Over the eight lanes of a leaf.
    __device__ void reduce8()
    {
#pragma unroll
        for (int o = 1; o < 8; o <<= 1)
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                lo[k] = min(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], o));
                hi[k] = max(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], o));
            }
    }
};

// A leaf's FP64 box and its outward-rounded FP32 copy in the packed node,
// whose .w words (escape index and leaf range) are the build's.
__device__ __forceinline__ void put_leaf(float4 *bnode, double *blo, double *bhi, uint32_t node, const KeyBox &box)
{
    const V lo = dm::v(from_key(box.lo[0]), from_key(box.lo[1]), from_key(box.lo[2]));
    const V hi = dm::v(from_key(box.hi[0]), from_key(box.hi[1]), from_key(box.hi[2]));
    store3(blo + 3 * size_t(node), lo);
    store3(bhi + 3 * size_t(node), hi);
    float4 *pn = bnode + 2 * size_t(node);
    pn[0].x = __double2float_rd(lo.x); pn[0].y = __double2float_rd(lo.y); pn[0].z = __double2float_rd(lo.z);
    pn[1].x = __double2float_ru(hi.x); pn[1].y = __double2float_ru(hi.y); pn[1].z = __double2float_ru(hi.z);
}

// An inner node's FP32 box from its children's: rounding is monotone, so the
// merge of the rounded boxes is the rounded merge.  Inner boxes are only ever
// tested in FP32.
__device__ __forceinline__ void merge_children(float4 *bnode, uint32_t p, uint32_t l, uint32_t r)
{
    const float4 la = __ldcg(bnode + 2 * size_t(l)), lb = __ldcg(bnode + 2 * size_t(l) + 1);
    const float4 ra = __ldcg(bnode + 2 * size_t(r)), rb = __ldcg(bnode + 2 * size_t(r) + 1);
    float4 *pn = bnode + 2 * size_t(p);
    pn[0].x = fminf(la.x, ra.x); pn[0].y = fminf(la.y, ra.y); pn[0].z = fminf(la.z, ra.z);
    pn[1].x = fmaxf(lb.x, rb.x); pn[1].y = fmaxf(lb.y, rb.y); pn[1].z = fmaxf(lb.z, rb.z);
}

// Bottom-up refit of both trees (at the new positions, and swept over old and
// new ones) and the FP32 records of every triangle, in one launch: eight lanes
// a leaf, a triangle each; the first one walks up, the second child to arrive
// at a parent (atomic counter) merges the two children, resets the counter for
// the next launch and continues.  Two launches with a thread a leaf, and a
// third for the records, took 90 us a substep on 1,280 triangles and 204 on
// 449,940; this one 25 and 127.
constexpr int kLeafTriangles = 8;  // BVH leaves hold at most 8 triangles (cuda_backend.cu:305)
__global__ void __launch_bounds__(kBlock) k_refit(View d)
{
    follow_previous();
    const uint32_t thread = blockIdx.x * blockDim.x + threadIdx.x, leaf = thread / kLeafTriangles, sub = thread % kLeafTriangles;
    const bool live = leaf < d.L;
    uint32_t node = 0;
    KeyBox now, swept;
    now.clear();
    swept.clear();
    if (live) {
        node = d.bleaves[leaf];
        const uint32_t p = d.bfirst[node] + sub;
        if (sub < d.bcount[node]) {
            const uint32_t t = d.border[p];
            float4 *rec = d.tri32 + 3 * size_t(p), *rec_old = d.tri32_old + 3 * size_t(p);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const uint32_t vi = d.tri[3 * t + c];
                const V a = load3(d.col_cur + 3 * size_t(vi)), o = load3(d.col_old + 3 * size_t(vi));
                const float w = c == 0 ? __uint_as_float(t) : 0.0f;
                rec[c] = make_float4(float(a.x), float(a.y), float(a.z), w);
                rec_old[c] = make_float4(float(o.x), float(o.y), float(o.z), w);
                now.add(a);
                swept.add(a);
                swept.add(o);
            }
        }
    }
    now.reduce8();
    swept.reduce8();
    if (!live || sub != 0) return;
    put_leaf(d.bnode, d.blo, d.bhi, node, now);
    put_leaf(d.swept_node, d.swept_lo, d.swept_hi, node, swept);
    for (;;) {
        const int32_t p = d.bparent[node];
        if (p < 0) return;
        __threadfence();
        if (atomicAdd(&d.brefit[p], 1u) == 0) return;
        d.brefit[p] = 0;
        __threadfence();
        const uint32_t l = d.bleft[p], r = d.bright[p];
        merge_children(d.bnode, uint32_t(p), l, r);
        merge_children(d.swept_node, uint32_t(p), l, r);
        node = uint32_t(p);
    }
}

// Conservative advancement of each moving triangle against the stationary
// hair at the start of the substep (cuda_backend.cu:975-987).  Returns the
// first failing triangle of this element in traversal order.
// FP32 pre-test of the mixed sweep for the candidate at leaf-order position
// p: true when the first conservative-advancement step of the exact pass is
// certain to reach the end of the substep (no failure from this triangle).
// It needs a lower bound of the segment's distance to the triangle at its
// old position (tri32_old records, margins as record_distance_f) and an
// upper bound of the largest vertex displacement (FP32 differences of the
// rounded copies, widened by their rounding).
__device__ __forceinline__ bool sweep_skip_f(const View &d, uint32_t p, dm::F3 origin, dm::F3 f1, float target_ru)
{
    const float4 n0 = __ldg(d.tri32 + 3 * size_t(p)), n1 = __ldg(d.tri32 + 3 * size_t(p) + 1),
                 n2 = __ldg(d.tri32 + 3 * size_t(p) + 2);
    const float4 o0 = __ldg(d.tri32_old + 3 * size_t(p)), o1 = __ldg(d.tri32_old + 3 * size_t(p) + 1),
                 o2 = __ldg(d.tri32_old + 3 * size_t(p) + 2);
    auto disp = [](float4 a, float4 b) {
        const float dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z;
        const float mag = fmaxf(fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fabsf(a.z)), fmaxf(fmaxf(fabsf(b.x), fabsf(b.y)), fabsf(b.z)));
        return __fadd_ru(__fmul_ru(sqrtf(dx * dx + dy * dy + dz * dz), 1.00001f), __fmaf_ru(mag, 5.0e-7f, 1.0e-12f));
    };
    const float speed_ub = fmaxf(disp(n0, o0), fmaxf(disp(n1, o1), disp(n2, o2)));
    const dm::F3 a = dm::f3(o0.x - origin.x, o0.y - origin.y, o0.z - origin.z);
    const dm::F3 b = dm::f3(o1.x - origin.x, o1.y - origin.y, o1.z - origin.z);
    const dm::F3 c = dm::f3(o2.x - origin.x, o2.y - origin.y, o2.z - origin.z);
    float m;
    const float df = dm::segment_triangle_distance_f(dm::f3(0.f, 0.f, 0.f), f1, a, b, c, m);
    const float vmax = fmaxf(fmaxf(fmaxf(fabsf(o0.x), fabsf(o0.y)), fmaxf(fabsf(o0.z), fabsf(o1.x))),
                             fmaxf(fmaxf(fabsf(o1.y), fabsf(o1.z)), fmaxf(fmaxf(fabsf(o2.x), fabsf(o2.y)), fabsf(o2.z))));
    const float omax = fmaxf(fmaxf(fabsf(origin.x), fabsf(origin.y)), fabsf(origin.z));
    const float emax = fmaxf(fmaxf(fabsf(f1.x), fabsf(f1.y)), fabsf(f1.z)) + omax;
    m += 2.5e-7f * (vmax + omax + emax) + 1.0e-9f;
    return __fmul_rd(0.8f, __fsub_rd(__fsub_rd(df, m), target_ru)) >= __fmul_ru(speed_ub, 1.000002f);
}

__device__ bool sweep_element(const View &d, uint32_t e, SweepRecord *rec)
{
    const uint32_t i = d.ei[e], j = d.ej[e];
    const V p0 = load3(d.q + 6 * size_t(i)), p1 = load3(d.q + 6 * size_t(j));
    const double target = d.radius + d.offset + d.min_gap;
    bool failed = false;
    bvh_query_packed(d, dm::vmin(p0, p1), dm::vmax(p0, p1), d.ccd_pad, [&](uint32_t t) {
        if (failed) return;
        const V oa = load3(d.col_old + 3 * size_t(d.tri[3 * t])), ob = load3(d.col_old + 3 * size_t(d.tri[3 * t + 1])),
                oc = load3(d.col_old + 3 * size_t(d.tri[3 * t + 2]));
        const V da = dm::gsub(tri_vertex(d, t, 0), oa), db = dm::gsub(tri_vertex(d, t, 1), ob),
                dc = dm::gsub(tri_vertex(d, t, 2), oc);
        const double speed = fmax(dm::gnorm(da), fmax(dm::gnorm(db), dm::gnorm(dc)));
        if (speed < 1e-30) return;
        double alpha = 0.0;
        bool end = false;
        dm::ClosestPair pair;
        V a, b, c;
        for (int k = 0; k < 80; ++k) {
            a = dm::gadd(oa, dm::gmul(da, alpha)); b = dm::gadd(ob, dm::gmul(db, alpha)); c = dm::gadd(oc, dm::gmul(dc, alpha));
            pair = dm::closest_segment_triangle(p0, p1, a, b, c);
            const double clearance = pair.distance - target;
            if (clearance <= 0) { failed = true; break; }
            const double advance = 0.8 * clearance / speed;
            if (alpha + advance >= 1) { end = true; break; }
            if (advance < 1e-12) { failed = true; break; }
            alpha += advance;
        }
        if (!end) failed = true;
        if (failed && rec) {
            rec->claimed = 1; rec->strand = d.estrand[e]; rec->element = e; rec->triangle = t;
            rec->distance = pair.distance; rec->required = target; rec->clearance = pair.distance - target;
            rec->displacement = speed;
            store3(rec->hair_start, p0); store3(rec->hair_end, p1);
            store3(rec->collider_point, dm::gadd(dm::gadd(dm::gmul(a, pair.bary.x), dm::gmul(b, pair.bary.y)), dm::gmul(c, pair.bary.z)));
        }
    });
    return failed;
}

__global__ void __launch_bounds__(kBlock) k_sweep(View d)
{
    follow_previous();
    const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= d.E) return;
    if (d.fixed[d.ei[e]] || !d.econtact[e]) return;
    if (sweep_element(d, e, nullptr)) atomicMin(&d.sc->sweep_fail, e);
}

// Diagonal preconditioner (cuda_backend.cu:815-841): node term then the
// left and right incident elements, inverted; 0 at fixed nodes.
__global__ void __launch_bounds__(kBlock) k_precond(View d, double dt)
{
    follow_previous();
    const uint32_t n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= d.N) return;
    const double inv = 1.0 / dt, inv2 = inv * inv;
    double t = d.mass[n] * (inv2 + d.damping * inv), r = d.rmass[n] * (inv2 + d.damping * inv);
    const double area = dm::kPi * d.radius * d.radius;
    const double inertia = dm::kPi * d.radius * d.radius * d.radius * d.radius / 4.0;
    const double G = d.young / (2.0 * (1.0 + d.poisson));
    const int32_t es[2] = {d.elem_left[n], d.elem_right[n]};
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        if (es[k] < 0) continue;
        const double L = d.L0[es[k]];
        t += fmax(d.young * area, d.shear_corr * G * area) / L;
        r += d.shear_corr * G * area * L + fmax(d.young * inertia, 2.0 * G * inertia) / L;
    }
    const bool fx = d.fixed[n];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        d.precond[6 * size_t(n) + k] = fx ? 0.0 : 1.0 / fmax(t, 1.0e-30);
        d.precond[6 * size_t(n) + 3 + k] = fx ? 0.0 : 1.0 / fmax(r, 1.0e-30);
    }
}

// ---- energy / gradient / Gauss-Newton Hessian -----------------------------

// Per node: optional line-search update q = q_base + alpha dir, rotation
// cache, inertia + damping energy, gradient and diagonal
// (cuda_backend.cu:883-897).
// Trial state q = q_base + alpha dir (trial) and the FP32 position copy.
// alpha_dev (if set) holds the trial step in device memory (the pipelined
// first trial of an iteration, whose step the host has not read yet).
__device__ __forceinline__ void node_positions(const View &d, uint32_t n, int trial, double alpha, double q[6])
{
    const size_t o = 6 * size_t(n);
    if (trial) {
#pragma unroll
        for (int k = 0; k < 6; ++k) { q[k] = d.q_base[o + k] + alpha * d.dir[o + k]; d.q[o + k] = q[k]; }
    } else {
#pragma unroll
        for (int k = 0; k < 6; ++k) q[k] = d.q[o + k];
    }
    d.q32[3 * size_t(n)] = float(q[0]); d.q32[3 * size_t(n) + 1] = float(q[1]); d.q32[3 * size_t(n) + 2] = float(q[2]);
}

// The positions alone, so that the contact passes (which read q and the
// FP32 copy) can run beside the rest of k_node_eval.
__global__ void __launch_bounds__(kBlock) k_positions(View d, int trial, double alpha, const double *alpha_dev)
{
    follow_previous();
    const uint32_t n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= d.N) return;
    double q[6];
    node_positions(d, n, trial, alpha_dev ? *alpha_dev : alpha, q);
}

// positions_done: k_positions has written q and the FP32 copy.
__global__ void __launch_bounds__(kEvalBlock) k_node_eval(View d, int gradient, int trial, double alpha, double dt,
                                                      const double *alpha_dev, int positions_done)
{
    follow_previous();
    const uint32_t n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= d.N) return;
    if (alpha_dev) alpha = *alpha_dev;
    double q[6];
    const size_t o = 6 * size_t(n);
    if (positions_done) {
#pragma unroll
        for (int k = 0; k < 6; ++k) q[k] = d.q[o + k];
    } else {
        node_positions(d, n, trial, alpha, q);
    }
    M R, J;
    dm::rotation_and_jacobian(dm::v(q[3], q[4], q[5]), d.ref + 9 * size_t(n), R, gradient ? &J : nullptr);
#pragma unroll
    for (int k = 0; k < 9; ++k) d.rot[9 * size_t(n) + k] = R.m[k];
    if (gradient) {
#pragma unroll
        for (int k = 0; k < 9; ++k) d.jl[9 * size_t(n) + k] = J.m[k];
    }
    if (d.fixed[n]) {
        d.node_energy[n] = 0.0;
        d.node_kinetic[n] = 0.0;
        if (gradient) {
#pragma unroll
            for (int k = 0; k < 6; ++k) { d.grad[o + k] = 0.0; d.inertia[o + k] = 0.0; }
        }
        return;
    }
    const double inv = 1.0 / dt, inv2 = inv * inv, m = d.mass[n], mr = d.rmass[n];
    const double kx = m * inv2, kr = mr * inv2, cx = m * d.damping * inv, cr = mr * d.damping * inv;
    const double grav[3] = {d.gx, d.gy, d.gz};
    double obj = 0.0, kin = 0.0;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        const double g = k < 3 ? grav[k] * dt * dt : 0.0;
        const double qo = d.q_old[o + k];
        const double predicted = qo + dt * d.v[o + k] + g;
        const double delta = q[k] - predicted, damp = q[k] - qo;
        const double kk = k < 3 ? kx : kr, c = k < 3 ? cx : cr;
        obj += 0.5 * kk * delta * delta + 0.5 * c * damp * damp;
        if (k < 3) kin += 0.5 * m * damp * damp * inv2;
        if (gradient) {
            d.grad[o + k] = kk * delta + c * damp;
            d.inertia[o + k] = kk + c;
        }
    }
    d.node_energy[n] = obj;
    d.node_kinetic[n] = kin;
}

// Two-pass closest search of the mixed form over a candidate source
// (source(fn) calls fn(triangle) for each candidate in traversal order):
// FP32 distances with margins bound the FP64 minimum, then FP64 is evaluated
// only for candidates whose lower bound does not exceed that bound.
template<class Source>
__device__ __forceinline__ uint32_t closest_triangle_in(const View &d, V xi, V xj, uint32_t &cand, dm::ClosestPair &pair,
                                                        Source &&source)
{
    uint32_t closest = kNone;
    cand = 0;
    pair.distance = 1.0e300; pair.t = 0.0; pair.bary = dm::v(1, 0, 0);
    const dm::F3 origin = dm::f3(float(xi.x), float(xi.y), float(xi.z));
    const dm::F3 p0 = dm::f3(0.f, 0.f, 0.f), p1 = dm::f3(float(xj.x) - origin.x, float(xj.y) - origin.y, float(xj.z) - origin.z);
    float bound = 3.0e38f;
    source([&](uint32_t t) {
        ++cand;
        float m;
        const float df = candidate_distance_f(d, t, origin, p0, p1, m);
        bound = fminf(bound, df + m);
    });
    if (cand == 0) return kNone;
    source([&](uint32_t t) {
        float m;
        const float df = candidate_distance_f(d, t, origin, p0, p1, m);
        if (df - m > bound) return;
        const dm::ClosestPair c = dm::closest_segment_triangle(xi, xj, tri_vertex(d, t, 0), tri_vertex(d, t, 1), tri_vertex(d, t, 2));
        if (c.distance < pair.distance) { pair = c; closest = t; }
    });
    return closest;
}

// Broad + narrow phase of one element: every candidate in traversal order,
// the first strictly closest triangle kept (cuda_backend.cu:920-926).
// Mixed form: a first pass bounds the FP64 minimum by FP32 distances with
// margins; the second pass evaluates in FP64 only the candidates whose lower
// bound does not exceed that bound, in the same order, so the result (and
// the first-found tie-break) equals the all-FP64 search.
template<bool MIXED>
__device__ __forceinline__ uint32_t closest_triangle(const View &d, V xi, V xj, Pad pad, uint32_t &cand,
                                                     dm::ClosestPair &pair)
{
    uint32_t closest = kNone;
    cand = 0;
    pair.distance = 1.0e300; pair.t = 0.0; pair.bary = dm::v(1, 0, 0);
    const V lo = dm::vmin(xi, xj), hi = dm::vmax(xi, xj);
    if (!MIXED) {
        bvh_query_packed(d, lo, hi, pad, [&](uint32_t t) {
            ++cand;
            const dm::ClosestPair c = dm::closest_segment_triangle(xi, xj, tri_vertex(d, t, 0), tri_vertex(d, t, 1), tri_vertex(d, t, 2));
            if (c.distance < pair.distance) { pair = c; closest = t; }
        });
        return closest;
    }
    return closest_triangle_in(d, xi, xj, cand, pair, [&](auto &&fn) { bvh_query_packed(d, lo, hi, pad, fn); });
}

// Contact classification of every element at the state q: candidate count,
// closest triangle with its closest pair, gap and flags, by one thread an
// element (the contact-query entry point).
template<bool MIXED> __global__ void __launch_bounds__(kBlock) k_contact(View d, const double *q)
{
    follow_previous();
    const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= d.E) return;
    const uint32_t i = d.ei[e], j = d.ej[e];
    uint32_t cand = 0, closest = kNone;
    uint8_t flags = 0;
    double gap = 0.0;
    dm::ClosestPair pair;
    pair.distance = 1.0e300; pair.t = 0.0; pair.bary = dm::v(1, 0, 0);
    if (d.has_collider && !d.fixed[i] && d.econtact[e]) {
        const V xi = load3(q + 6 * size_t(i)), xj = load3(q + 6 * size_t(j));
        closest = closest_triangle<MIXED>(d, xi, xj, d.contact_pad, cand, pair);
        if (closest != kNone) {
            flags |= kFlagClosest;
            gap = pair.distance - d.radius - d.offset;
            if (gap <= d.min_gap) flags |= kFlagInfeasible;
            else if (gap < d.dhat) flags |= kFlagActive;
        }
    }
    d.c_cand[e] = cand;
    d.c_tri[e] = closest;
    d.c_flags[e] = flags;
    d.c_gap[e] = gap;
    d.c_t[e] = pair.t;
    d.c_dist[e] = pair.distance;
    store3(d.c_bary + 3 * size_t(e), pair.bary);
}

// ---- contact pass of an evaluation ------------------------------------------
//
// k_contact_filter (thread per element): the element's cached leaves are still
// valid, or are collected again; elements with leaves are queued.
// k_contact_near (warp per queued element, a block per element with many
// leaves): lane l tests leaf l exactly, so
// the candidates are counted in traversal order; in the mixed form an FP32
// filter over the triangle records keeps every candidate whose lower bound
// does not exceed the smallest upper bound, in the plain form all stay.  They
// go to a pool of (element, triangle) pairs.  k_contact_exact (thread per
// pair): the FP64 closest pair.  k_contact_select (thread per element): the
// first strictly closest of the element's pairs, and its barrier.  Candidates
// the mixed form drops are strictly farther in FP64 than the minimum, so either
// way the result, tie-break included, equals k_contact's.
//
// The plain form used to search inside the element kernel, one thread walking
// the FP64 boxes and evaluating every candidate in turn: on 80 strands among
// contacts that took 2.0 ms an evaluation; the pairs are few (7,000 there) and
// independent.

constexpr uint32_t kSurvOverflow = 0xffffffffu;  // surv_n: no room in a pool, k_contact_select searches

// candidate_distance_f on the record at leaf-order position p (one 48-byte
// record instead of an index triple and three vertex reads).
__device__ __forceinline__ float record_distance_f(const View &d, uint32_t p, dm::F3 origin, dm::F3 p0, dm::F3 p1, float &m,
                                                   uint32_t &t)
{
    const float4 r0 = __ldg(d.tri32 + 3 * size_t(p)), r1 = __ldg(d.tri32 + 3 * size_t(p) + 1),
                 r2 = __ldg(d.tri32 + 3 * size_t(p) + 2);
    t = __float_as_uint(r0.w);
    const dm::F3 a = dm::f3(r0.x - origin.x, r0.y - origin.y, r0.z - origin.z);
    const dm::F3 b = dm::f3(r1.x - origin.x, r1.y - origin.y, r1.z - origin.z);
    const dm::F3 c = dm::f3(r2.x - origin.x, r2.y - origin.y, r2.z - origin.z);
    const float df = dm::segment_triangle_distance_f(p0, p1, a, b, c, m);
    const float vmax = fmaxf(fmaxf(fmaxf(fabsf(r0.x), fabsf(r0.y)), fmaxf(fabsf(r0.z), fabsf(r1.x))),
                             fmaxf(fmaxf(fabsf(r1.y), fabsf(r1.z)), fmaxf(fmaxf(fabsf(r2.x), fabsf(r2.y)), fabsf(r2.z))));
    const float omax = fmaxf(fmaxf(fabsf(origin.x), fabsf(origin.y)), fabsf(origin.z));
    const float emax = fmaxf(fmaxf(fabsf(p1.x), fabsf(p1.y)), fabsf(p1.z)) + omax;
    m += 2.5e-7f * (vmax + omax + emax) + 1.0e-9f;
    return df;
}

__device__ __forceinline__ uint8_t write_contact(const View &d, uint32_t e, uint32_t closest, const dm::ClosestPair &pair)
{
    uint8_t flags = 0;
    double gap = 0.0;
    if (closest != kNone) {
        flags |= kFlagClosest;
        gap = pair.distance - d.radius - d.offset;
        if (gap <= d.min_gap) flags |= kFlagInfeasible;
        else if (gap < d.dhat) flags |= kFlagActive;
    }
    d.c_tri[e] = closest;
    d.c_flags[e] = flags;
    d.c_gap[e] = gap;
    d.c_t[e] = pair.t;
    d.c_dist[e] = pair.distance;
    store3(d.c_bary + 3 * size_t(e), pair.bary);
    d.e_co[e] = 0.0;
    return flags;
}

// Slack test of the leaf cache on the FP32 copies: below kCacheReach metres
// they differ from the FP64 positions by at most 2^-24 of that, 4e-6 m, so the
// margin of 1e-5 m keeps every accepted displacement within kCacheSlack.
// Elements further out collect their leaves at every evaluation.
constexpr float kCacheReach = 64.0f;
__device__ __forceinline__ bool within_cache_slack(const float *c, dm::F3 xi, dm::F3 xj)
{
    const float s = float(kCacheSlack) - 1.0e-5f;
    const float far = fmaxf(fmaxf(fmaxf(fabsf(xi.x), fabsf(xi.y)), fmaxf(fabsf(xi.z), fabsf(xj.x))), fmaxf(fabsf(xj.y), fabsf(xj.z)));
    return far <= kCacheReach && fabsf(xi.x - c[0]) <= s && fabsf(xi.y - c[1]) <= s && fabsf(xi.z - c[2]) <= s &&
           fabsf(xj.x - c[3]) <= s && fabsf(xj.y - c[4]) <= s && fabsf(xj.z - c[5]) <= s;
}

// The element's cached leaves: collected around its box grown by the slack
// (always with force, else where it has left the slack), so that the passes of
// many evaluations read a short list.  Returns cache_n.  q must be d.q (its
// FP32 copy d.q32 is read).
__device__ __forceinline__ uint8_t refresh_leaves(const View &d, const double *q, uint32_t e, uint32_t i, uint32_t j, bool force)
{
    const dm::F3 xi32 = dm::f3(d.q32[3 * size_t(i)], d.q32[3 * size_t(i) + 1], d.q32[3 * size_t(i) + 2]);
    const dm::F3 xj32 = dm::f3(d.q32[3 * size_t(j)], d.q32[3 * size_t(j) + 1], d.q32[3 * size_t(j) + 2]);
    float *c32 = d.cache_x32 + 6 * size_t(e);
    uint8_t nl = d.cache_n[e];
    if (!force && nl != kCacheInvalid && within_cache_slack(c32, xi32, xj32)) return nl;
    const V xi = load3(q + 6 * size_t(i)), xj = load3(q + 6 * size_t(j));
    const V s3 = dm::v(kCacheSlack, kCacheSlack, kCacheSlack);
    nl = leaves_to_cache(d, e, dm::vmin(xi, xj) - s3, dm::vmax(xi, xj) + s3, d.contact_pad);
    c32[0] = xi32.x; c32[1] = xi32.y; c32[2] = xi32.z; c32[3] = xj32.x; c32[4] = xj32.y; c32[5] = xj32.z;
    return nl;
}

// Queues an element with leaves for k_contact_near.
__device__ __forceinline__ void queue_near(const View &d, uint32_t e, uint8_t nl)
{
    if (nl == kCacheBig) d.near_list[d.E - 1 - atomicAdd(&d.sc->wide_count, 1u)] = e;
    else d.near_list[append_slot(&d.sc->near_count)] = e;
}

// cache 1: collect every element's leaves (the first evaluation of a
// substep); 0: only where the element has left its slack.
__global__ void __launch_bounds__(kBlock) k_contact_filter(View d, const double *q, int cache)
{
    follow_previous();
    const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= d.E) return;
    const uint32_t i = d.ei[e], j = d.ej[e];
    if (!d.fixed[i] && d.econtact[e]) {
        const uint8_t nl = refresh_leaves(d, q, e, i, j, cache == 1);
        if (nl == kCacheInvalid) {  // the leaf pool is full
            d.surv_n[e] = kSurvOverflow;
            return;
        }
        if (nl > 0) {
            queue_near(d, e, nl);
            return;
        }
    } else if (cache == 1 && !d.fixed[j] && d.econtact[e]) {
        refresh_leaves(d, q, e, i, j, true);  // for k_friction_collect
    }
    d.c_cand[e] = 0;
    d.surv_n[e] = 0;
    dm::ClosestPair pair;
    pair.distance = 1.0e300; pair.t = 0.0; pair.bary = dm::v(1, 0, 0);
    write_contact(d, e, kNone, pair);
}

// Triangle range (first, cnt) of cached leaf k of a list of `count` when
// its box passes the query's exact per-leaf test; cnt = 0 otherwise.
template<class Box>
__device__ __forceinline__ void near_leaf(const View &d, const uint32_t *leaves, uint32_t k, uint32_t count, const QueryBox &qb,
                                          double pad, Box &&box, uint32_t &first, uint32_t &cnt)
{
    first = 0;
    cnt = 0;
    if (k >= count) return;
    const uint32_t node = leaves[k];
    const float4 a = __ldg(d.bnode + 2 * size_t(node)), b = __ldg(d.bnode + 2 * size_t(node) + 1);
    if (maybe_overlap(qb, a, b) && leaf_overlap_exact(d, node, a, b, qb, pad, box)) {
        const uint32_t leaf = __float_as_uint(b.w);
        first = leaf >> 4;
        cnt = leaf & 15u;
    }
}

__device__ __forceinline__ uint32_t warp_inclusive_sum(uint32_t v, int lane)
{
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
    }
    return v;
}

// The pool range of an element's n pairs of total candidates (lane 0 writes
// the element's record): its offset, or kNone without room or pairs.
__device__ __forceinline__ uint32_t near_claim(const View &d, uint32_t e, uint32_t total, uint32_t n, int lane)
{
    uint32_t off = kNone;
    if (lane == 0) {
        d.c_cand[e] = total;
        uint32_t held = n;
        if (n == 0) {
            dm::ClosestPair pair;
            pair.distance = 1.0e300; pair.t = 0.0; pair.bary = dm::v(1, 0, 0);
            write_contact(d, e, kNone, pair);
        } else {
            off = claim_range(&d.sc->surv_count, n, d.surv_capacity);
            if (off == kNone) held = kSurvOverflow;
            d.surv_off[e] = off;
        }
        d.surv_n[e] = held;
    }
    return __shfl_sync(0xffffffffu, off, 0);
}

__device__ __forceinline__ void put_pair(const View &d, uint32_t slot, uint32_t e, uint32_t t)
{
    d.surv_elem[slot] = e;
    d.surv_tri[slot] = t;
}

// Candidates of up to 32 leaves, spread over the warp: lane l brings leaf l's
// triangle range (first, cnt <= kLeafTriangles); pos lists the leaf-order
// positions of all of them in traversal order.  Returns their number.  A leaf
// a lane would leave most lanes idle: one or two leaves pass of thirty.
constexpr int kNearList = 32 * kLeafTriangles;
__device__ __forceinline__ uint32_t spread_candidates(uint32_t first, uint32_t cnt, uint32_t *pos, int lane)
{
    const uint32_t incl = warp_inclusive_sum(cnt, lane);
    __syncwarp();  // the list's last readers are done
    for (uint32_t r = 0; r < cnt; ++r) pos[incl - cnt + r] = first + r;
    __syncwarp();
    return __shfl_sync(0xffffffffu, incl, 31);
}

// The leaves of an element queued by k_contact_filter are tested 32 at a time,
// lane by lane, their candidates taken 32 at a time, lane by lane: with FILTER
// once for the smallest upper bound, once to count the survivors, and once to
// write the pairs, in traversal order (leaf, then triangle), so the first-found
// tie-break is kept.  With at most 32 candidates, the common case, the first
// round's bounds are kept instead.  An element has a warp; one with more than
// kCacheLeaves leaves (a mesh pole), queued at the list's other end, has a
// block, whose warps take runs of its leaves: the longest list of a pole bound
// the launch at 67 us with one warp, 26 with eight.
constexpr int kNearWarps = kBlock / 32;
// Four blocks an SM are resident.  Where their warps have several elements each,
// that many blocks spread the work better than twice as many (a frame of 1,000
// strands, 68,000 elements: 177.6 ms against 181.5); beside a half-empty
// element kernel, twice as many start sooner (27,000: 66.7 against 67.5).
inline unsigned near_grid(uint32_t E) { return E > 40000u ? 152u * 4u : 152u * 8u; }
template<bool FILTER> __global__ void __launch_bounds__(kBlock, 4) k_contact_near(View d)
{
    follow_previous();
    __shared__ uint32_t lists[kNearWarps][kNearList];
    __shared__ uint32_t totals[kNearWarps], counts[kNearWarps], slot;
    __shared__ float ubs[kNearWarps];
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t *pos = lists[w];
    const uint32_t nwide = d.sc->wide_count, count = d.sc->near_count;
    // Wide elements block by block, the others warp by warp from the next
    // block on.
    uint32_t kw = blockIdx.x, k = (blockIdx.x + gridDim.x - nwide % gridDim.x) % gridDim.x * kNearWarps + w;
    for (;;) {
        const bool wide = kw < nwide;
        if (!wide && k >= count) break;
        const uint32_t e = wide ? d.near_list[d.E - 1 - kw] : d.near_list[k];
        if (wide) kw += gridDim.x;
        else k += gridDim.x * kNearWarps;
        const uint32_t i = d.ei[e], j = d.ej[e];
        const dm::F3 xi32 = dm::f3(d.q32[3 * size_t(i)], d.q32[3 * size_t(i) + 1], d.q32[3 * size_t(i) + 2]);
        const dm::F3 xj32 = dm::f3(d.q32[3 * size_t(j)], d.q32[3 * size_t(j) + 1], d.q32[3 * size_t(j) + 2]);
        const float lo32[3] = {fminf(xi32.x, xj32.x), fminf(xi32.y, xj32.y), fminf(xi32.z, xj32.z)};
        const float hi32[3] = {fmaxf(xi32.x, xj32.x), fmaxf(xi32.y, xj32.y), fmaxf(xi32.z, xj32.z)};
        const QueryBox qb = make_query_f(lo32, hi32, d.contact_pad);
        auto box = [&](V &lo, V &hi) {
            const V xi = load3(d.q + 6 * size_t(i)), xj = load3(d.q + 6 * size_t(j));
            lo = dm::vmin(xi, xj); hi = dm::vmax(xi, xj);
        };
        const dm::F3 origin = xi32, p0 = dm::f3(0.f, 0.f, 0.f);
        const dm::F3 p1 = dm::f3(xj32.x - origin.x, xj32.y - origin.y, xj32.z - origin.z);
        uint32_t nleaves = 0;
        const uint32_t *leaves = cached_leaves(d, e, d.cache_n[e], nleaves);
        const uint32_t begin = wide ? uint32_t(uint64_t(nleaves) * w / kNearWarps) : 0;
        const uint32_t end = wide ? uint32_t(uint64_t(nleaves) * (w + 1) / kNearWarps) : nleaves;
        uint32_t total = 0, n = 0, at = 0, here = 0, t = 0;
        float ub = 3.0e38f, lb = 3.0e38f;
        for (int pass = 0; pass < 3; ++pass) {  // bounds, count, write
            if (pass == 1 && !FILTER) n = total;
            for (uint32_t r0 = begin; r0 < end && !(pass == 1 && !FILTER); r0 += 32) {
                if (pass == 0 || end - begin > 32) {
                    uint32_t first, cnt;
                    near_leaf(d, leaves, r0 + lane, end, qb, d.contact_pad.exact, box, first, cnt);
                    here = spread_candidates(first, cnt, pos, lane);
                }
                if (pass == 0) total += here;
                if (pass == 0 && !FILTER) continue;
                for (uint32_t c0 = 0; c0 < here; c0 += 32) {
                    const uint32_t c = c0 + lane;
                    bool stays = c < here;
                    if (stays) {
                        if (FILTER) {
                            float m;
                            const float df = record_distance_f(d, pos[c], origin, p0, p1, m, t);
                            lb = df - m;
                            if (pass == 0) ub = fminf(ub, df + m);
                            stays = !(lb > ub);
                        } else {
                            t = __float_as_uint(__ldg(d.tri32 + 3 * size_t(pos[c])).w);
                        }
                    }
                    if (pass == 0) continue;
                    const uint32_t mask = __ballot_sync(FULL, stays);
                    if (pass == 1) n += __popc(mask);
                    else {
                        if (stays) put_pair(d, at + __popc(mask & ((1u << lane) - 1u)), e, t);
                        at += __popc(mask);
                    }
                }
            }
            if (pass == 0) {
                if (FILTER) {
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) ub = fminf(ub, __shfl_xor_sync(FULL, ub, o));
                }
                if (wide) {
                    if (lane == 0) { totals[w] = total; ubs[w] = ub; }
                    __syncthreads();
#pragma unroll
                    for (int o = 0; o < kNearWarps; ++o) ub = fminf(ub, ubs[o]);
                } else if (total <= 32) {
                    const bool stays = uint32_t(lane) < total && !(FILTER && lb > ub);
                    const uint32_t mask = __ballot_sync(FULL, stays);
                    const uint32_t base = near_claim(d, e, total, __popc(mask), lane);
                    if (base != kNone && stays) {
                        if (!FILTER) t = __float_as_uint(__ldg(d.tri32 + 3 * size_t(pos[lane])).w);
                        put_pair(d, base + __popc(mask & ((1u << lane) - 1u)), e, t);
                    }
                    break;
                }
            } else if (pass == 1) {
                uint32_t before = 0;
                if (wide) {
                    if (lane == 0) counts[w] = n;
                    __syncthreads();
                    uint32_t every = 0, all = 0;
#pragma unroll
                    for (int o = 0; o < kNearWarps; ++o) {
                        every += totals[o];
                        before += o < w ? counts[o] : 0;
                        all += counts[o];
                    }
                    if (w == 0) {
                        at = near_claim(d, e, every, all, lane);
                        if (lane == 0) slot = at;
                    }
                    __syncthreads();
                    at = slot;
                } else {
                    at = near_claim(d, e, total, n, lane);
                }
                if (at == kNone) break;
                at += before;
            }
        }
        if (wide) __syncthreads();  // the shared values are read
    }
}

// FP64 passes over pairs: a block of five warps takes 32 pairs, warp w part w
// of each (the segment's ends against the face, the segment against an edge),
// so the parts of a pair run on as many sub-partitions and no lane waits for
// another's kind of part.  A whole pair in one thread is a chain of some 600
// FP64 instructions of 64 cycles (54 us for however few pairs); a part is
// about 80, with its comparisons on the integer pipes.
constexpr int kPairWarps = 5, kPairBlock = 32 * kPairWarps;
constexpr unsigned kPairGrid = 152 * 4;

__device__ __forceinline__ dm::PairPart part_of(bool fast, int part, V p0, V p1, V a, V b, V c)
{
    return fast ? dm::pair_part<true>(part, p0, p1, a, b, c) : dm::pair_part_slow(part, p0, p1, a, b, c);
}

__global__ void __launch_bounds__(kPairBlock) k_contact_exact(View d, const double *q)
{
    follow_previous();
    __shared__ double sh[kPairWarps][5][32];
    const int part = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t count = uint32_t(min(d.sc->surv_count, (unsigned long long)d.surv_capacity));
    for (uint32_t base = 32 * blockIdx.x; base < count; base += 32 * gridDim.x) {
        const uint32_t k = base + lane;
        if (k < count) {
            const uint32_t e = d.surv_elem[k], t = d.surv_tri[k];
            const V xi = load3(q + 6 * size_t(d.ei[e])), xj = load3(q + 6 * size_t(d.ej[e]));
            const V a = tri_vertex(d, t, 0), b = tri_vertex(d, t, 1), c = tri_vertex(d, t, 2);
            const dm::PairPart x = part_of(dm::sane_pair(xi, xj, a, b, c), part, xi, xj, a, b, c);
            sh[part][0][lane] = x.dist2; sh[part][1][lane] = x.t;
            sh[part][2][lane] = x.bary.x; sh[part][3][lane] = x.bary.y; sh[part][4][lane] = x.bary.z;
        }
        __syncthreads();
        if (part == 0 && k < count) {
            double best = __longlong_as_double(0x7ff0000000000000ll);
            int from = -1;
#pragma unroll
            for (int w = 0; w < kPairWarps; ++w)
                if (dm::root_less(sh[w][0][lane], best)) { best = sh[w][0][lane]; from = w; }
            double *r = d.surv_res + 5 * size_t(k);
            r[0] = from < 0 ? 1.0e300 : sqrt(best);
#pragma unroll
            for (int f = 1; f < 5; ++f) r[f] = from < 0 ? (f == 2 ? 1.0 : 0.0) : sh[from][f][lane];
        }
        __syncthreads();
    }
}

// The first strictly closest of element e's n pairs, or the search by one
// thread where a pool was full (which also counts the candidates).
template<bool FILTER>
__device__ __forceinline__ uint32_t select_pair(const View &d, const double *q, uint32_t e, uint32_t n, dm::ClosestPair &pair)
{
    pair.distance = 1.0e300; pair.t = 0.0; pair.bary = dm::v(1, 0, 0);
    if (n == kSurvOverflow) {
        const uint32_t i = d.ei[e], j = d.ej[e];
        uint32_t cand = 0;
        const uint32_t closest = closest_triangle<FILTER>(d, load3(q + 6 * size_t(i)), load3(q + 6 * size_t(j)), d.contact_pad,
                                                          cand, pair);
        d.c_cand[e] = cand;
        return closest;
    }
    const uint32_t off = n ? d.surv_off[e] : 0;
    uint32_t best = kNone;
    for (uint32_t k = off; k < off + n; ++k) {
        const double dist = d.surv_res[5 * size_t(k)];
        if (dist < pair.distance) { pair.distance = dist; best = k; }
    }
    if (best == kNone) return kNone;
    const double *r = d.surv_res + 5 * size_t(best);
    pair.t = r[1]; pair.bary = dm::v(r[2], r[3], r[4]);
    return d.surv_tri[best];
}

// The barrier of an active element (cuda_backend.cu:899-939), with a gradient
// also what it adds, for k_node_sum: g0 and g1 to the gradients of the ends'
// positions, curv dg dg^T (dg: node i, then node j) to the position parts of
// the blocks.  In its own record, so that the element kernel, whose chain of
// FP64 instructions bounds small scenes, runs beside the contact pass.
// Within the element kernel the barrier's logarithm and divisions added 8 us to
// an evaluation of 3,200 elements (39.0 us, then 30.7), and the element kernel
// waited for the contact pass.
constexpr int kPush = 13;  // g0, g1, curv, dg
__device__ __forceinline__ void element_barrier(const View &d, const double *q, uint32_t e, uint32_t closest,
                                                const dm::ClosestPair &pair, bool gradient)
{
    const V xi = load3(q + 6 * size_t(d.ei[e])), xj = load3(q + 6 * size_t(d.ej[e]));
    const double gap = pair.distance - d.radius - d.offset;
    const V offset = dm::contact_offset(xi, xj, pair.t, tri_vertex(d, closest, 0), tri_vertex(d, closest, 1),
                                        tri_vertex(d, closest, 2), pair.bary);
    double g0[3], g1[3];
    const double energy = dm::barrier_energy_gradient(offset, pair.t, d.radius + d.offset, d.dhat, d.kc, g0, g1);
    if (!isfinite(energy)) {
        d.c_flags[e] |= kFlagInfeasible;
        return;
    }
    d.c_flags[e] |= kFlagEnergy;
    d.e_co[e] = energy;
    if (!gradient) return;
    double *push = d.push + kPush * size_t(e);
    const V normal = offset * (1.0 / fmax(pair.distance, 1e-15));
    const double aa = d.dhat - gap;
#pragma unroll
    for (int k = 0; k < 3; ++k) { push[k] = g0[k]; push[3 + k] = g1[k]; }
    push[6] = d.kc * (-2.0 * log(gap / d.dhat) + 4.0 * aa / gap + aa * aa / (gap * gap));
    push[7] = normal.x * (1.0 - pair.t); push[8] = normal.y * (1.0 - pair.t); push[9] = normal.z * (1.0 - pair.t);
    push[10] = normal.x * pair.t; push[11] = normal.y * pair.t; push[12] = normal.z * pair.t;
}

constexpr int kSelectBlock = 64;
template<bool FILTER> __global__ void __launch_bounds__(kSelectBlock) k_contact_select(View d, const double *q, int gradient)
{
    follow_previous();
    const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e == 0) {  // k_contact_near and k_contact_exact, their only readers, have completed
        d.sc->surv_count = 0;
        d.sc->near_count = 0;
        d.sc->wide_count = 0;
    }
    if (e >= d.E) return;
    const uint32_t n = d.surv_n[e];
    if (n == 0) return;
    dm::ClosestPair pair;
    const uint32_t closest = select_pair<FILTER>(d, q, e, n, pair);
    if (write_contact(d, e, closest, pair) & kFlagActive) element_barrier(d, q, e, closest, pair, gradient);
}

// ---- contact query without allocation -------------------------------------
//
// Scratch of khsxQueryContactsNoAlloc: the caller's state (48 bytes per
// node) followed by the records (24 bytes per element), in a file-scope
// device array of KHSX_NO_ALLOC_SCRATCH_BYTES.  One array per device and
// process, shared by every solver on that device: calls that overlap in
// time on one device race on it.
__device__ __align__(256) unsigned char g_no_alloc_scratch[KHSX_NO_ALLOC_SCRATCH_BYTES];

// k_contact without the leaf cache, writing the caller-facing record of each
// element straight into the scratch instead of the solver's contact arrays
// (the solver's own records are left as they are).  Every record below E is
// written in full, so nothing in the scratch has to start at zero.
template<bool MIXED> __global__ void __launch_bounds__(kBlock) k_contact_query_records(View d, const double *q,
                                                                                        KhsxContactRecord *out)
{
    follow_previous();
    const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= d.E) return;
    const uint32_t i = d.ei[e], j = d.ej[e];
    uint32_t cand = 0, closest = kNone, active = 0;
    double gap = __longlong_as_double(0x7ff0000000000000LL);  // +infinity
    dm::ClosestPair pair;
    if (d.has_collider && !d.fixed[i] && d.econtact[e]) {
        const V xi = load3(q + 6 * size_t(i)), xj = load3(q + 6 * size_t(j));
        closest = closest_triangle<MIXED>(d, xi, xj, d.contact_pad, cand, pair);
        if (closest != kNone) {
            gap = pair.distance - d.radius - d.offset;
            active = gap > d.min_gap && gap < d.dhat ? 1u : 0u;
        }
    }
    KhsxContactRecord r;
    r.candidate_count = cand;
    r.closest_triangle = closest;
    r.active = active;
    r.reserved = 0;
    r.gap = gap;
    out[e] = r;
}

// Per element: elastic energy (+ gradient and GN blocks) (cuda_backend.cu:899-939).
__global__ void __launch_bounds__(kEvalBlock) k_elem_eval(View d, int gradient)
{
    follow_previous();
    const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= d.E) return;
    const uint32_t i = d.ei[e], j = d.ej[e];
    const bool fi = d.fixed[i], fj = d.fixed[j];
    const V xi = load3(d.q + 6 * size_t(i)), xj = load3(d.q + 6 * size_t(j));
    const M Ri = load9(d.rot + 9 * size_t(i)), Rj = load9(d.rot + 9 * size_t(j));
    const double L0 = d.L0[e];
    double eps[6];
    double *gi = d.as_i_g + 6 * size_t(i), *gj = d.as_j_g + 6 * size_t(j);
    double *Hii = d.as_i_h + 36 * size_t(i), *Hjj = d.as_j_h + 36 * size_t(j), *Hij = d.upper + 36 * size_t(i);
    if (gradient) {
        const M Jli = load9(d.jl + 9 * size_t(i)), Jlj = load9(d.jl + 9 * size_t(j));
        dm::ElementJacobian J;
        dm::element_strain_inv(Ri, Rj, xi, xj, d.invL[e], load3(d.gamma0 + 3 * size_t(e)), load3(d.kappa0 + 3 * size_t(e)), eps,
                               &J, &Jli, &Jlj);
        double a[6], b[6];
        dm::element_gradient(J, eps, d.w, L0, a, b);
        // 16-byte stores: every block starts on a 16-byte boundary (36 and
        // 6 doubles per node from 256-byte aligned arrays).
        double2 *gi2 = reinterpret_cast<double2 *>(gi), *gj2 = reinterpret_cast<double2 *>(gj);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            gi2[k] = fi ? make_double2(0.0, 0.0) : make_double2(a[2 * k], a[2 * k + 1]);
            gj2[k] = fj ? make_double2(0.0, 0.0) : make_double2(b[2 * k], b[2 * k + 1]);
        }
        double hii[36], hjj[36], hij[36];
        dm::element_hessian(J, d.w, L0, hii, hjj, hij);
        double2 *Hii2 = reinterpret_cast<double2 *>(Hii), *Hjj2 = reinterpret_cast<double2 *>(Hjj);
        double2 *Hij2 = reinterpret_cast<double2 *>(Hij);
        const bool fij = fi || fj;
#pragma unroll
        for (int k = 0; k < 18; ++k) {
            Hii2[k] = fi ? make_double2(0.0, 0.0) : make_double2(hii[2 * k], hii[2 * k + 1]);
            Hjj2[k] = fj ? make_double2(0.0, 0.0) : make_double2(hjj[2 * k], hjj[2 * k + 1]);
            Hij2[k] = fij ? make_double2(0.0, 0.0) : make_double2(hij[2 * k], hij[2 * k + 1]);
        }
    } else {
        dm::element_strain_inv(Ri, Rj, xi, xj, d.invL[e], load3(d.gamma0 + 3 * size_t(e)), load3(d.kappa0 + 3 * size_t(e)), eps,
                               nullptr, nullptr, nullptr);
    }
    d.e_el[e] = dm::element_energy(eps, d.w, L0);
}

// The gradient form with two threads an element: warp 0 of a block takes the
// left ends of 32 elements, warp 1 the right ones.  What both need (the strain
// and K) is evaluated twice; the mixed block, which needs both ends' rows, is
// shared out through shared memory.  One thread an element is a chain of 720
// FP64 instructions of 64 cycles, two a chain of 360, with 15% more of them in
// all; so two are taken while every warp has a sub-partition to itself (two
// blocks on each SM).  us a launch: 2,000 elements 30.7 -> 20.4, 6,200 30.6 ->
// 22.5; beyond the line one thread is the faster: 15,500 34.8 against 38.9,
// 66,000 106 against 115, 258,000 358 against 426.
constexpr int kEndElements = 32, kEndBlock = 2 * kEndElements;
__global__ void __launch_bounds__(kEndBlock) k_elem_ends(View d)
{
    follow_previous();
    __shared__ double rows[2][18][kEndElements];  // S2, Kk of the left end; the scaled rows of the right one
    const int lane = threadIdx.x & 31;
    const bool right = threadIdx.x >= 32;
    const uint32_t e = blockIdx.x * kEndElements + lane;
    const bool on = e < d.E;
    bool fij = false;
    M WS, WK, S2, Kk;
    double eps[6], L0 = 0.0, *Hij = nullptr;
    if (on) {
        const uint32_t i = d.ei[e], j = d.ej[e], n = right ? j : i;
        const bool fi = d.fixed[i], fj = d.fixed[j], fixed = right ? fj : fi;
        fij = fi || fj;
        const V xi = load3(d.q + 6 * size_t(i)), xj = load3(d.q + 6 * size_t(j));
        const M Ri = load9(d.rot + 9 * size_t(i)), Rj = load9(d.rot + 9 * size_t(j)), R = load9(d.rot + 9 * size_t(n));
        const M Jl = load9(d.jl + 9 * size_t(n));
        const double invL = d.invL[e];
        L0 = d.L0[e];
        V t;
        M A2, S, K, x;
        dm::element_strain_shared(Ri, Rj, xi, xj, invL, load3(d.gamma0 + 3 * size_t(e)), load3(d.kappa0 + 3 * size_t(e)), eps, t, S, &K);
#pragma unroll
        for (int k = 0; k < 9; ++k) A2.m[k] = S.m[k] * invL;
        dm::element_strain_end(R, Ri, Jl, t, K, right ? invL : -invL, S2, Kk);
        double g[6], H[36];
        dm::element_end(right, A2, S2, Kk, eps, d.w, L0, g, H, x, WS, WK);
        double2 *g2 = reinterpret_cast<double2 *>((right ? d.as_j_g : d.as_i_g) + 6 * size_t(n));
        double2 *H2 = reinterpret_cast<double2 *>((right ? d.as_j_h : d.as_i_h) + 36 * size_t(n));
#pragma unroll
        for (int k = 0; k < 3; ++k) g2[k] = fixed ? make_double2(0.0, 0.0) : make_double2(g[2 * k], g[2 * k + 1]);
#pragma unroll
        for (int k = 0; k < 18; ++k) H2[k] = fixed ? make_double2(0.0, 0.0) : make_double2(H[2 * k], H[2 * k + 1]);
        // Top left (-P) and bottom left (Xi^T) of the mixed block with the left
        // end, top right (-Xj) with the right one.
        Hij = d.upper + 36 * size_t(i);
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                if (right) Hij[6 * r + 3 + c] = fij ? 0.0 : -x.m[3 * r + c];
                else {
                    Hij[6 * r + c] = fij ? 0.0 : -H[6 * r + c];
                    Hij[6 * (3 + r) + c] = fij ? 0.0 : x.m[3 * c + r];
                }
            }
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            rows[right][k][lane] = right ? WS.m[k] : S2.m[k];
            rows[right][9 + k][lane] = right ? WK.m[k] : Kk.m[k];
        }
    }
    __syncthreads();
    if (!on) return;
    // Bottom right: four entries with the left end (and the energy), five with
    // the right one.
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        M &a = right ? S2 : WS, &b = right ? Kk : WK;
        a.m[k] = rows[!right][k][lane];
        b.m[k] = rows[!right][9 + k][lane];
    }
    auto mixed = [&](int k) {
        const int r = k / 3, c = k % 3;
        Hij[6 * (3 + r) + 3 + c] = fij ? 0.0 : dm::dot3w(S2, r, WS, c) + dm::dot3w(Kk, r, WK, c);
    };
    if (right) {
#pragma unroll
        for (int k = 4; k < 9; ++k) mixed(k);
    } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) mixed(k);
        d.e_el[e] = dm::element_energy(eps, d.w, L0);
    }
}

// Node sums in a fixed order: inertia, then the element on the left (this
// node as its right end), then the element on the right.
// One thread per two entries (18 N of the diagonal blocks, then 3 N of the
// gradient) so every access is coalesced; memory bounds it (265,000 nodes: 293
// MB, 57 us).  Diagonal block = inertia diagonal
// + the contribution of the element whose right node is n + that of the
// element whose left node is n, in that order, each with what its barrier adds
// to the position part (element_barrier), as does the coupling block.
__device__ __forceinline__ const double *pushed(const View &d, int32_t e)
{
    return e >= 0 && (d.c_flags[e] & kFlagEnergy) ? d.push + kPush * size_t(e) : nullptr;
}

__global__ void __launch_bounds__(kBlock) k_node_sum(View d)
{
    follow_previous();
    const size_t idx = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const size_t nh = 18 * size_t(d.N);
    if (idx < nh) {
        const size_t n = idx / 18;
        const int k = int(idx % 18), r = k / 3, c = 2 * (k % 3);  // entries (r, c) and (r, c + 1)
        const bool position = r < 3 && c < 3;
        const int32_t left = position ? d.elem_left[n] : -1, right = position ? d.elem_right[n] : -1;
        double2 hj = reinterpret_cast<const double2 *>(d.as_j_h)[idx], hi = reinterpret_cast<const double2 *>(d.as_i_h)[idx];
        double2 sum = make_double2(0.0, 0.0);
        if (r == c) sum.x = d.inertia[6 * n + r];
        if (r == c + 1) sum.y = d.inertia[6 * n + r];
        if (const double *p = pushed(d, left)) {
            const double cr = p[6] * p[10 + r];
            hj.x += cr * p[10 + c];
            if (c == 0) hj.y += cr * p[11];
        }
        if (const double *p = pushed(d, right)) {
            const double cr = p[6] * p[7 + r];
            double2 &u = reinterpret_cast<double2 *>(d.upper)[idx];
            hi.x += cr * p[7 + c];
            u.x += cr * p[10 + c];
            if (c == 0) { hi.y += cr * p[8]; u.y += cr * p[11]; }
        }
        reinterpret_cast<double2 *>(d.diag)[idx] = make_double2((sum.x + hj.x) + hi.x, (sum.y + hj.y) + hi.y);
    } else if (idx < nh + 3 * size_t(d.N)) {
        const size_t i = idx - nh, n = i / 3;
        const int k = 2 * int(i % 3);
        const int32_t left = k < 3 ? d.elem_left[n] : -1, right = k < 3 ? d.elem_right[n] : -1;
        double2 gj = reinterpret_cast<const double2 *>(d.as_j_g)[i], gi = reinterpret_cast<const double2 *>(d.as_i_g)[i];
        double2 &g = reinterpret_cast<double2 *>(d.grad)[i];
        if (const double *p = pushed(d, left)) { gj.x += p[3 + k]; if (k == 0) gj.y += p[4]; }
        if (const double *p = pushed(d, right)) { gi.x += p[k]; if (k == 0) gi.y += p[1]; }
        g = make_double2((g.x + gj.x) + gi.x, (g.y + gj.y) + gi.y);
    }
}

// Sum (or smallest key) over a block of 256 threads' values of one kind, by one
// warp: levels 128, 64 and 32 on a lane's eight values, then 16 ... 1 by
// shuffles, each element combined with the one that far above it, as in a tree
// over shared memory.  Lane 0 holds the result.
struct OpSum { template<class T> __device__ static T f(T a, T b) { return a + b; } };
struct OpMin { __device__ static long long f(long long a, long long b) { return a < b ? a : b; } };
struct OpMax { __device__ static long long f(long long a, long long b) { return a > b ? a : b; } };

template<class Op, class T> __device__ __forceinline__ T warp_tree(const T *sh, int lane)
{
    T y[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) y[k] = Op::f(sh[lane + 32 * k], sh[lane + 32 * k + 128]);
    T v = Op::f(Op::f(y[0], y[2]), Op::f(y[1], y[3]));
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) v = Op::f(v, __shfl_down_sync(0xffffffffu, v, s));
    return v;
}

// The block's sums: every thread brings its values, a warp of its own reduces
// each kind.  All kinds on the first warp, and fmin on the FP64 pipe, put some
// 45 FP64 instructions of 64 cycles in a row there: k_reduce_eval took 18.3 us
// on 2,000 elements and takes 12.2, k_reduce_dir 15.2 and 10.6.  An evaluation
// has five FP64 sums, the smallest gap's key and three counts, a direction two
// FP64 sums and the largest square as bits.  Thread 0 finds the results in
// element 0 of each row; the rows may be used again after a barrier.
constexpr int kEvalSums = 5, kEvalCounts = 3, kDirSums = 2;
struct EvalRows {
    double sum[kEvalSums][kBlock];
    long long gap[kBlock];
    unsigned long long count[kEvalCounts][kBlock];
};
struct DirRows {
    double sum[kDirSums][kBlock];
    long long top[kBlock];
};
__device__ __forceinline__ void block_sums(EvalRows &r, const double (&s)[kEvalSums], long long gap, const unsigned long long (&u)[kEvalCounts])
{
    const int t = threadIdx.x, w = t >> 5, lane = t & 31;
#pragma unroll
    for (int k = 0; k < kEvalSums; ++k) r.sum[k][t] = s[k];
    r.gap[t] = gap;
#pragma unroll
    for (int k = 0; k < kEvalCounts; ++k) r.count[k][t] = u[k];
    __syncthreads();
    if (w < kEvalSums) {
        const double v = warp_tree<OpSum>(r.sum[w], lane);
        if (lane == 0) r.sum[w][0] = v;
    } else if (w == kEvalSums) {
        const long long v = warp_tree<OpMin>(r.gap, lane);
        if (lane == 0) r.gap[0] = v;
    } else {
        for (int k = w - kEvalSums - 1; k < kEvalCounts; k += 2) {
            const unsigned long long v = warp_tree<OpSum>(r.count[k], lane);
            if (lane == 0) r.count[k][0] = v;
        }
    }
    __syncthreads();
}
__device__ __forceinline__ void block_sums(DirRows &r, const double (&s)[kDirSums], long long top)
{
    const int t = threadIdx.x, w = t >> 5, lane = t & 31;
#pragma unroll
    for (int k = 0; k < kDirSums; ++k) r.sum[k][t] = s[k];
    r.top[t] = top;
    __syncthreads();
    if (w < kDirSums) {
        const double v = warp_tree<OpSum>(r.sum[w], lane);
        if (lane == 0) r.sum[w][0] = v;
    } else if (w == kDirSums) {
        const long long v = warp_tree<OpMax>(r.top, lane);
        if (lane == 0) r.top[0] = v;
    }
    __syncthreads();
}

// A NaN orders above everything, so it loses every minimum as it does in fmin.
__device__ __forceinline__ long long gap_key(double x)
{
    const bool nan = (__double_as_longlong(x) & 0x7fffffffffffffffll) > 0x7ff0000000000000ll;
    return nan ? 0x7fffffffffffffffll : order_key(x);
}
constexpr long long kInfKey = 0x7ff0000000000000ll;

__device__ __forceinline__ void chunk(uint32_t count, uint32_t &begin, uint32_t &end)
{
    const uint64_t b = uint64_t(blockIdx.x) * count / gridDim.x, e = uint64_t(blockIdx.x + 1) * count / gridDim.x;
    begin = uint32_t(b);
    end = uint32_t(e);
}

// First reduction level over nodes and elements of this block's chunk.
// Final level of the evaluation sums over the per-block partials, in block
// order, published to the host mailbox (run by the last block of
// k_reduce_eval to finish).
__device__ void final_eval(const View &d, EvalRows &rows)
{
    double v[kEvalSums] = {0, 0, 0, 0, 0};  // energy, kinetic, grad2, elastic, contact
    long long gap = kInfKey;
    unsigned long long u[kEvalCounts] = {0, 0, 0};
    for (int b = threadIdx.x; b < kPartials; b += kBlock) {
        const Partial *p = d.partials + b;
        v[0] += __ldcg(&p->node_energy); v[1] += __ldcg(&p->kinetic); v[2] += __ldcg(&p->grad2);
        v[3] += __ldcg(&p->elastic); v[4] += __ldcg(&p->contact);
        gap = OpMin::f(gap, gap_key(__ldcg(&p->min_gap)));
        u[0] += __ldcg(&p->candidates); u[1] += __ldcg(&p->active); u[2] += (unsigned long long)__ldcg(&p->infeasible);
    }
    block_sums(rows, v, gap, u);
    if (threadIdx.x == 0) {
        Mailbox *m = d.mail;
        m->objective = (rows.sum[0][0] + rows.sum[3][0]) + rows.sum[4][0];
        m->elastic = rows.sum[3][0]; m->contact = rows.sum[4][0]; m->kinetic = rows.sum[1][0];
        m->minimum_gap = from_key(rows.gap[0]); m->grad_norm2 = rows.sum[2][0];
        m->candidates = rows.count[0][0]; m->active = rows.count[1][0]; m->feasible = rows.count[2][0] ? 0 : 1;
    }
}

// Both reduction levels of an evaluation in one launch: each block sums its
// chunk of nodes and elements into a partial; the last block to finish
// (counted with an atomic after a fence) reduces the partials in block
// order, so the result does not depend on which block that is.
__global__ void __launch_bounds__(kBlock) k_reduce_eval(View d, int gradient)
{
    follow_previous();
    __shared__ EvalRows rows;
    __shared__ bool last;
    uint32_t nb, ne, eb, ee;
    chunk(d.N, nb, ne);
    chunk(d.E, eb, ee);
    double en = 0.0, ki = 0.0, g2 = 0.0, el = 0.0, co = 0.0;
    long long gap = kInfKey;
    unsigned long long cand = 0, act = 0;
    int inf = 0;
    for (uint32_t n = nb + threadIdx.x; n < ne; n += kBlock) {
        en += d.node_energy[n];
        ki += d.node_kinetic[n];
        if (gradient)
            for (int k = 0; k < 6; ++k) { const double g = d.grad[6 * size_t(n) + k]; g2 += g * g; }
    }
    for (uint32_t e = eb + threadIdx.x; e < ee; e += kBlock) {
        el += d.e_el[e];
        co += d.e_co[e];
        cand += d.c_cand[e];
        const uint8_t f = d.c_flags[e];
        if (f & kFlagClosest) gap = OpMin::f(gap, gap_key(d.c_gap[e]));
        if (f & kFlagActive) ++act;
        if (f & kFlagInfeasible) inf = 1;
    }
    const double sums[kEvalSums] = {en, ki, g2, el, co};
    const unsigned long long u[kEvalCounts] = {cand, act, (unsigned long long)inf};
    block_sums(rows, sums, gap, u);
    if (threadIdx.x == 0) {
        Partial p;
        p.node_energy = rows.sum[0][0]; p.kinetic = rows.sum[1][0]; p.grad2 = rows.sum[2][0];
        p.elastic = rows.sum[3][0]; p.contact = rows.sum[4][0];
        p.min_gap = from_key(rows.gap[0]);
        p.candidates = rows.count[0][0]; p.active = rows.count[1][0]; p.infeasible = int(rows.count[2][0] != 0); p.pad = 0;
        d.partials[blockIdx.x] = p;
        __threadfence();
        last = atomicAdd(&d.sc->eval_done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    final_eval(d, rows);
    if (threadIdx.x == 0) d.sc->eval_done = 0;
}

// ---- direction ----------------------------------------------------------

// Block-tridiagonal Thomas solve per strand (cuda_backend.cu:866-881) with
// the reference's Gauss-Jordan elimination, partial pivoting on the first
// largest |pivot|, after the relative diagonal shift max(1e-12 max|a_ii|,
// 1e-24) (cuda_backend.cu:855-864).  Strands are taken in length-sorted
// order, longest first, by persistent warps from a work queue, so the
// strands of a warp have similar lengths and the long strands that bound
// the solve start first.
constexpr int kSolveGroup = 6, kSolveGroupsPerWarp = 5;  // float-float kernels: 6 lanes per strand, 5 per warp

// The work items of the solve (Engine::plan_block_solve): places in the
// solve order, marked where the strand has a warp of its own, else the first
// of five; longest expected time first.  Blocks of one warp take them from a
// queue, so the block scheduler spreads few items over as many SMs.
constexpr uint32_t kSolveAlone = 0x80000000u;
constexpr uint32_t kSolveByRule = 0xffffffffu;  // plan_block_solve chooses the split

__global__ void __launch_bounds__(32) k_block_solve(View d, uint32_t items)
{
    follow_previous();
    __shared__ __align__(16) BackRing ring;
    for (;;) {
        uint32_t g = 0;
        if (threadIdx.x == 0) g = atomicAdd(&d.sc->solve_next, 1u);
        g = __shfl_sync(0xffffffffu, g, 0);
        if (g >= items) break;
        const uint32_t item = d.solve_items[g];
        if (item & kSolveAlone) solve_strand_warp(d, item & ~kSolveAlone, ring);
        else solve_strands_five(d, item);
    }
}

// Every strand on a team of three warps, longest first.
__global__ void __launch_bounds__(kTeam) k_block_solve_team(View d)
{
    follow_previous();
    __shared__ __align__(16) TeamShared sh;
    solve_strand_team(d, blockIdx.x, sh);
}

// ---- mixed form: float-float block solve with FP64 refinement -------------
//
// The same block Thomas recurrence as the FP64 solve (per strand, one lane
// per block row, Gauss-Jordan with partial pivoting on the first largest
// |pivot|, relative diagonal shift) evaluated in float-float arithmetic:
// k_ff_factor stores B_n^-1, C_n = B_n^-1 U_n and d'_n and writes the first
// direction; k_ff_residual forms r = -g - A x in FP64 (one thread per row,
// no sequential chain), with the shifts the factorisation used; k_ff_correct
// solves A delta = r with the stored factors and adds delta to the direction
// in FP64.  The float-float factor has about 48 significant bits, so a sweep
// contracts the error by about cond(B) * 2^-48 and one sweep recovers the
// accuracy of the FP64 solve for the condition numbers of these systems
// (block condition numbers up to about 1e10); further sweeps run while the
// largest relative correction of any strand exceeds kRefineRatio.  A pivot
// below 1e-30 or a value outside the FP32 exponent range sets the solve
// failure flag and the host falls back to the FP64 block solve.

constexpr float kRefineRatio = 1.0e-4f;
constexpr int kRefineSweepsMax = 3;

__device__ __forceinline__ void group_range(const View &d, uint32_t warp, int lane, int &r, int &base, uint32_t &begin,
                                            uint32_t &len, uint32_t &maxlen)
{
    const int grp = lane / kSolveGroup;
    r = lane % kSolveGroup;
    base = grp * kSolveGroup;
    const uint32_t k = warp * kSolveGroupsPerWarp + uint32_t(grp);
    const bool member = grp < kSolveGroupsPerWarp && k < d.S;
    begin = 0; len = 0;
    if (member) {
        const uint32_t s = d.sorder[k];
        begin = d.sfirst[s] + d.sfixed[s];
        const uint32_t end = d.sfirst[s] + d.scount[s];
        len = end > begin ? end - begin : 0;
    }
    maxlen = len;
    for (int o = 16; o > 0; o >>= 1) maxlen = max(maxlen, __shfl_xor_sync(0xffffffffu, maxlen, o));
}

__device__ __forceinline__ float2 f2(ff::FF a) { return make_float2(a.hi, a.lo); }
__device__ __forceinline__ ff::FF fromf2(float2 a) { return ff::make(a.x, a.y); }

__device__ __forceinline__ void ff_factor_group(const View &d, uint32_t warp)
{
    const int lane = threadIdx.x & 31;
    int r, base;
    uint32_t begin, len, maxlen;
    group_range(d, warp, lane, r, base, begin, len, maxlen);
    double nd[6], nu[6], nuc[6], ng = 0.0;
    auto fetch = [&](uint32_t t) {
        const bool on = t < len;
        const size_t n = begin + t;
#pragma unroll
        for (int c = 0; c < 6; ++c) nd[c] = on ? d.diag[36 * n + 6 * r + c] : 0.0;
        ng = on ? d.grad[6 * n + r] : 0.0;
        const bool up = on && t + 1 < len;
#pragma unroll
        for (int c = 0; c < 6; ++c) nu[c] = up ? d.upper[36 * n + 6 * r + c] : 0.0;
#pragma unroll
        for (int q = 0; q < 6; ++q) nuc[q] = (on && t > 0) ? d.upper[36 * (n - 1) + 6 * q + r] : 0.0;
    };
    fetch(0);
    ff::FF Crow[6], dprev = ff::make(0.0f);
#pragma unroll
    for (int c = 0; c < 6; ++c) Crow[c] = ff::make(0.0f);
    bool failed = false;
    for (uint32_t t = 0; t < maxlen; ++t) {
        const bool on = t < len && !failed;
        const size_t n = begin + t;
        bool bad = false;
        ff::FF a[6], inv[6], urow[6], ucol[6];
        ff::FF rhs = ff::neg(ff::split(ng, bad));
#pragma unroll
        for (int c = 0; c < 6; ++c) {
            a[c] = ff::split(nd[c], bad);
            inv[c] = ff::make(c == r ? 1.0f : 0.0f);
            ucol[c] = ff::split(nuc[c], bad);
            urow[c] = ff::split(nu[c], bad);
        }
        if (t + 1 < maxlen) fetch(t + 1);
        if (t > 0) {
            // B = D - U_{n-1}^T C_{n-1}, rhs = -g - U_{n-1}^T d'_{n-1}
#pragma unroll
            for (int q = 0; q < 6; ++q) {
#pragma unroll
                for (int c = 0; c < 6; ++c) a[c] = ff::fms(a[c], ucol[q], ff::shfl(Crow[c], base + q));
                rhs = ff::fms(rhs, ucol[q], ff::shfl(dprev, base + q));
            }
        }
        // Relative diagonal shift max(1e-12 max|b_ii|, 1e-24); the value used
        // is stored for the FP64 residual.
        ff::FF diag_r = ff::make(0.0f);
#pragma unroll
        for (int c = 0; c < 6; ++c) if (c == r) diag_r = a[c];
        unsigned smax = 0u;
#pragma unroll
        for (int q = 0; q < 6; ++q) smax = max(smax, __shfl_sync(0xffffffffu, ff::abs_bits(diag_r), base + q));
        const float shift = fmaxf(__fmul_rn(1.0e-12f, __uint_as_float(smax)), 1.0e-24f);
#pragma unroll
        for (int c = 0; c < 6; ++c) if (c == r) a[c] = ff::add(a[c], ff::make(shift));
        if (on && r == 0) d.ff_shift[n] = shift;
        bool ok = !bad;
#pragma unroll
        for (int col = 0; col < 6; ++col) {
            ff::FF mine = ff::make(0.0f);
#pragma unroll
            for (int c = 0; c < 6; ++c) if (c == col) mine = a[c];
            const unsigned mb = ff::abs_bits(mine);
            int pivot = col;
            unsigned best = __shfl_sync(0xffffffffu, mb, base + col);
#pragma unroll
            for (int row = col + 1; row < 6; ++row) {
                const unsigned vrow = __shfl_sync(0xffffffffu, mb, base + row);
                if (vrow > best) { best = vrow; pivot = row; }
            }
            // best < 1e-30 or not finite => failure.
            if (best < 0x0da24260u || best >= 0x7f800000u) ok = false;
            const int partner = r == col ? pivot : (r == pivot ? col : r);
#pragma unroll
            for (int c = col; c < 6; ++c) a[c] = ff::shfl(a[c], base + partner);
#pragma unroll
            for (int c = 0; c < 6; ++c) inv[c] = ff::shfl(inv[c], base + partner);
            ff::FF pv = ff::make(1.0f);
#pragma unroll
            for (int c = 0; c < 6; ++c) if (c == col) pv = a[c];
            const ff::FF ip = ff::rcp(ff::shfl(pv, base + col));
            ff::FF f = ff::make(0.0f);
#pragma unroll
            for (int c = 0; c < 6; ++c) if (c == col) f = a[c];
#pragma unroll
            for (int c = col + 1; c < 6; ++c) {
                const ff::FF p = ff::mul(ff::shfl(a[c], base + col), ip);
                a[c] = (r == col) ? p : ff::fms(a[c], f, p);
            }
#pragma unroll
            for (int c = 0; c < 6; ++c) {
                const ff::FF p = ff::mul(ff::shfl(inv[c], base + col), ip);
                inv[c] = (r == col) ? p : ff::fms(inv[c], f, p);
            }
        }
        if (on && !ok) {
            failed = true;
            if (r == 0) atomicExch(&d.sc->solve_failed, 1);
        }
        // C_n = B^-1 U_n, d'_n = B^-1 rhs (row q of U_n in lane q).
        ff::FF dn = ff::make(0.0f);
#pragma unroll
        for (int c = 0; c < 6; ++c) Crow[c] = ff::make(0.0f);
#pragma unroll
        for (int q = 0; q < 6; ++q) {
#pragma unroll
            for (int c = 0; c < 6; ++c) Crow[c] = ff::fma(Crow[c], inv[q], ff::shfl(urow[c], base + q));
            dn = ff::fma(dn, inv[q], ff::shfl(rhs, base + q));
        }
        dprev = dn;
        if (on && !failed) {
#pragma unroll
            for (int c = 0; c < 6; ++c) {
                d.ff_inv[36 * n + 6 * r + c] = f2(inv[c]);
                d.ff_c[36 * n + 6 * r + c] = f2(Crow[c]);
            }
            d.ff_d[6 * n + r] = f2(dn);
        }
    }
    // Back substitution x_n = d'_n - C_n x_{n+1}.
    ff::FF next = ff::make(0.0f), pc[6], pd = ff::make(0.0f);
    auto fetch_back = [&](uint32_t t) {
        const bool on = t < len && !failed;
        const size_t n = begin + t;
        pd = on ? fromf2(d.ff_d[6 * n + r]) : ff::make(0.0f);
#pragma unroll
        for (int q = 0; q < 6; ++q) pc[q] = on ? fromf2(d.ff_c[36 * n + 6 * r + q]) : ff::make(0.0f);
    };
    if (maxlen) fetch_back(maxlen - 1);
    for (uint32_t t = maxlen; t-- > 0;) {
        const bool on = t < len && !failed;
        const size_t n = begin + t;
        ff::FF value = pd, crow[6];
#pragma unroll
        for (int q = 0; q < 6; ++q) crow[q] = pc[q];
        if (t > 0) fetch_back(t - 1);
        const bool coupled = on && t + 1 < len;
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            const ff::FF xq = ff::shfl(next, base + q);
            if (coupled) value = ff::fms(value, crow[q], xq);
        }
        if (on) d.dir[6 * n + r] = ff::to_double(value);
        next = on ? value : ff::make(0.0f);
    }
}

__global__ void __launch_bounds__(128) k_ff_factor(View d)
{
    follow_previous();
    const uint32_t groups = (d.S + kSolveGroupsPerWarp - 1) / kSolveGroupsPerWarp;
    for (;;) {
        uint32_t g = 0;
        if ((threadIdx.x & 31) == 0) g = atomicAdd(&d.sc->solve_next, 1u);
        g = __shfl_sync(0xffffffffu, g, 0);
        if (g >= groups) break;
        ff_factor_group(d, g);
    }
}

// r = -g - (A + shifts) x in FP64, one thread per row of a free node.
__global__ void __launch_bounds__(kBlock) k_ff_residual(View d)
{
    follow_previous();
    if (blockIdx.x == 0 && threadIdx.x == 0) d.sc->solve_next = 0;  // k_ff_factor has completed
    const uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= 6 * d.N) return;
    const uint32_t n = idx / 6, r = idx % 6;
    if (d.fixed[n]) { d.dprime[idx] = 0.0; return; }
    const double *x = d.dir + 6 * size_t(n);
    const double *D = d.diag + 36 * size_t(n) + 6 * r;
    double res = -d.grad[idx] - double(d.ff_shift[n]) * x[r];
#pragma unroll
    for (int c = 0; c < 6; ++c) res -= D[c] * x[c];
    if (d.elem_right[n] >= 0) {
        const double *U = d.upper + 36 * size_t(n) + 6 * r, *xn = x + 6;
#pragma unroll
        for (int c = 0; c < 6; ++c) res -= U[c] * xn[c];
    }
    if (d.elem_left[n] >= 0 && !d.fixed[n - 1]) {
        const double *U = d.upper + 36 * size_t(n - 1) + r, *xp = x - 6;
#pragma unroll
        for (int c = 0; c < 6; ++c) res -= U[6 * c] * xp[c];
    }
    d.dprime[idx] = res;
}

__device__ __forceinline__ void ff_correct_group(const View &d, uint32_t warp)
{
    const int lane = threadIdx.x & 31;
    int r, base;
    uint32_t begin, len, maxlen;
    group_range(d, warp, lane, r, base, begin, len, maxlen);
    double nres = 0.0, nuc[6];
    float2 ninv[6];
    auto fetch = [&](uint32_t t) {
        const bool on = t < len;
        const size_t n = begin + t;
        nres = on ? d.dprime[6 * n + r] : 0.0;
#pragma unroll
        for (int c = 0; c < 6; ++c) ninv[c] = on ? d.ff_inv[36 * n + 6 * r + c] : make_float2(0.0f, 0.0f);
#pragma unroll
        for (int q = 0; q < 6; ++q) nuc[q] = (on && t > 0) ? d.upper[36 * (n - 1) + 6 * q + r] : 0.0;
    };
    fetch(0);
    ff::FF dprev = ff::make(0.0f);
    for (uint32_t t = 0; t < maxlen; ++t) {
        const bool on = t < len;
        const size_t n = begin + t;
        bool bad = false;
        ff::FF rhs = ff::split(nres, bad), inv[6], ucol[6];
#pragma unroll
        for (int c = 0; c < 6; ++c) { inv[c] = fromf2(ninv[c]); ucol[c] = ff::split(nuc[c], bad); }
        if (t + 1 < maxlen) fetch(t + 1);
#pragma unroll
        for (int q = 0; q < 6; ++q) rhs = ff::fms(rhs, ucol[q], ff::shfl(dprev, base + q));
        ff::FF dn = ff::make(0.0f);
#pragma unroll
        for (int q = 0; q < 6; ++q) dn = ff::fma(dn, inv[q], ff::shfl(rhs, base + q));
        dprev = dn;
        if (on) d.ff_d[6 * n + r] = f2(dn);
    }
    ff::FF next = ff::make(0.0f), pc[6], pd = ff::make(0.0f);
    auto fetch_back = [&](uint32_t t) {
        const bool on = t < len;
        const size_t n = begin + t;
        pd = on ? fromf2(d.ff_d[6 * n + r]) : ff::make(0.0f);
#pragma unroll
        for (int q = 0; q < 6; ++q) pc[q] = on ? fromf2(d.ff_c[36 * n + 6 * r + q]) : ff::make(0.0f);
    };
    if (maxlen) fetch_back(maxlen - 1);
    float dmax = 0.0f, xmax = 0.0f;
    for (uint32_t t = maxlen; t-- > 0;) {
        const bool on = t < len;
        const size_t n = begin + t;
        ff::FF value = pd, crow[6];
#pragma unroll
        for (int q = 0; q < 6; ++q) crow[q] = pc[q];
        if (t > 0) fetch_back(t - 1);
        const bool coupled = on && t + 1 < len;
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            const ff::FF xq = ff::shfl(next, base + q);
            if (coupled) value = ff::fms(value, crow[q], xq);
        }
        if (on) {
            const double x = d.dir[6 * n + r] + ff::to_double(value);
            d.dir[6 * n + r] = x;
            dmax = fmaxf(dmax, fabsf(value.hi));
            xmax = fmaxf(xmax, fabsf(float(x)));
        }
        next = on ? value : ff::make(0.0f);
    }
    // Largest relative correction of the strand (over its rows) for the
    // host's sweep decision.
    for (int o = 16; o > 0; o >>= 1) {
        dmax = fmaxf(dmax, __shfl_xor_sync(0xffffffffu, dmax, o));
        xmax = fmaxf(xmax, __shfl_xor_sync(0xffffffffu, xmax, o));
    }
    if (lane == 0 && dmax > 0.0f) {
        const float ratio = xmax > 0.0f ? dmax / xmax : 3.0e38f;
        atomicMax(&d.sc->refine_bits, __float_as_uint(ratio));
    }
}

__global__ void __launch_bounds__(128) k_ff_correct(View d)
{
    follow_previous();
    const uint32_t groups = (d.S + kSolveGroupsPerWarp - 1) / kSolveGroupsPerWarp;
    for (;;) {
        uint32_t g = 0;
        if ((threadIdx.x & 31) == 0) g = atomicAdd(&d.sc->solve_next, 1u);
        g = __shfl_sync(0xffffffffu, g, 0);
        if (g >= groups) break;
        ff_correct_group(d, g);
    }
}

// Preconditioned steepest descent d = -P g, zero at fixed nodes
// (cuda_backend.cu:632-638).
__global__ void __launch_bounds__(kBlock) k_steepest(View d)
{
    follow_previous();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 6 * d.N) return;
    d.dir[i] = d.fixed[i / 6] ? 0.0 : -d.grad[i] * d.precond[i];
}

__global__ void __launch_bounds__(kBlock) k_scale(View d, double s)
{
    follow_previous();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < 6 * d.N) d.dir[i] *= s;
}

// The larger of two values >= 0, a NaN x ignored (as fmax does), compared as
// bits.
__device__ __forceinline__ double max_nonneg(double best, double x)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(best), v = (unsigned long long)__double_as_longlong(x);
    return v > b && v <= 0x7ff0000000000000ull ? x : best;
}

// Squared translation of a direction, rounded as the contracted dot product
// x x + y y + z z is (the inner sum takes the first product into its
// multiply-add); written out so that no other use of the products changes it.
__device__ __forceinline__ double translation2(const double x[6])
{
    return __fma_rn(x[2], x[2], __fma_rn(x[0], x[0], __dmul_rn(x[1], x[1])));
}

// g.d, |d|^2 and the largest free-node translation of the direction over one
// block's chunk of nodes, into the block's partial.  The root of the largest
// square is the largest root: one square root a block.
__device__ void direction_partial(const View &d, DirRows &rows)
{
    uint32_t nb, ne;
    chunk(d.N, nb, ne);
    double gd = 0.0, dd = 0.0, mx = 0.0;
    for (uint32_t n = nb + threadIdx.x; n < ne; n += kBlock) {
        double x[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            x[k] = d.dir[6 * size_t(n) + k];
            gd += d.grad[6 * size_t(n) + k] * x[k];
            dd += x[k] * x[k];
        }
        if (!d.fixed[n]) mx = max_nonneg(mx, translation2(x));
    }
    const double sums[kDirSums] = {gd, dd};
    block_sums(rows, sums, __double_as_longlong(mx));
    if (threadIdx.x == 0) {
        DirPartial p;
        p.slope = rows.sum[0][0];
        p.dnorm2 = rows.sum[1][0];
        p.max_translation = sqrt(__longlong_as_double(rows.top[0]));
        d.dpartials[blockIdx.x] = p;
    }
}

// True in the last block of the launch to get here, with the other blocks'
// writes visible.
__device__ bool last_block(uint32_t *done)
{
    __shared__ bool last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(done, 1u) == gridDim.x - 1;
        if (last) *done = 0;
    }
    __syncthreads();
    if (last) __threadfence();
    return last;
}

// The partials of all blocks, in block order, to the mailbox and to device
// memory.
__device__ void direction_total(const View &d, DirRows &rows)
{
    double gd = 0, dd = 0;
    long long top = 0;
    for (int b = threadIdx.x; b < kPartials; b += kBlock) {
        const DirPartial *p = d.dpartials + b;
        gd += __ldcg(&p->slope); dd += __ldcg(&p->dnorm2);
        top = OpMax::f(top, __double_as_longlong(__ldcg(&p->max_translation)));
    }
    const double sums[kDirSums] = {gd, dd};
    block_sums(rows, sums, top);
    if (threadIdx.x == 0) {
        const double most = __longlong_as_double(rows.top[0]);
        d.mail->slope = rows.sum[0][0]; d.mail->dir_norm2 = rows.sum[1][0]; d.mail->max_translation = most;
        d.sc->max_translation = most;
    }
}

// The direction as solved: its sums (the last block to finish adds the
// partials), and the flags of the solve.
__global__ void __launch_bounds__(kBlock) k_reduce_dir(View d)
{
    follow_previous();
    __shared__ DirRows rows;
    direction_partial(d, rows);
    if (!last_block(&d.sc->dir_done)) return;
    direction_total(d, rows);
    if (threadIdx.x == 0) {
        Mailbox *m = d.mail;
        m->dir_slope = m->slope; m->dir_max_translation = m->max_translation;
        m->solve_failed = m->dir_solve_failed = d.sc->solve_failed;
        m->refine_bits = d.sc->refine_bits;
        d.sc->solve_failed = 0;
        d.sc->solve_next = 0;
        d.sc->refine_bits = 0;
    }
}

// Publishes the CCD bound and re-arms its counters; the first line-search step
// is formed as the host does: 0.9 x the bound below 1, else 1.
__device__ __forceinline__ void publish_ccd(const View &d)
{
    const double lim = __longlong_as_double((long long)__ldcg(&d.sc->ccd_bits));
    d.mail->ccd_bits = (unsigned long long)__double_as_longlong(lim);
    d.sc->trial_alpha = d.has_collider ? (lim < 1.0 ? __dmul_rn(lim, 0.9) : lim) : 1.0;
    d.mail->pair_count = __ldcg(&d.sc->pair_count);
    d.sc->ccd_bits = 0x3ff0000000000000ULL;  // 1.0
    d.sc->pair_count = 0;
    d.sc->ccd_near = 0;
}

__global__ void k_publish_ccd(View d)
{
    follow_previous();
    if (threadIdx.x == 0 && blockIdx.x == 0) publish_ccd(d);
}

// What lies between the direction and its CCD bound, in one pass over the
// nodes: the trust-radius limit (scaled by trust / largest translation where
// that is exceeded, as the host's k_scale does), the copy of the iterate, and
// the FP32 end points of a full step.  The sums are taken again when the
// limit changed the direction, or with `again` (the host changed it).
// Without a collider the bound (1) is published here.
__global__ void __launch_bounds__(kBlock) k_limit(View d, double trust, int again)
{
    follow_previous();
    __shared__ DirRows rows;
    const double mt = d.sc->max_translation;
    const bool limited = mt > trust;
    const double scale = limited ? trust / mt : 1.0;
    uint32_t nb, ne;
    chunk(d.N, nb, ne);
    for (uint32_t n = nb + threadIdx.x; n < ne; n += kBlock) {
        double2 *q = reinterpret_cast<double2 *>(d.q + 6 * size_t(n)), *base = reinterpret_cast<double2 *>(d.q_base + 6 * size_t(n));
        double2 *dir = reinterpret_cast<double2 *>(d.dir + 6 * size_t(n));
        const double2 qa = q[0], qb = q[1], qc = q[2];
        double2 da = dir[0], db = dir[1];
        base[0] = qa; base[1] = qb; base[2] = qc;
        if (limited) {
            double2 dc = dir[2];
            da.x *= scale; da.y *= scale; db.x *= scale; db.y *= scale; dc.x *= scale; dc.y *= scale;
            dir[0] = da; dir[1] = db; dir[2] = dc;
        }
        d.e32[3 * size_t(n)] = float(qa.x + da.x);
        d.e32[3 * size_t(n) + 1] = float(qa.y + da.y);
        d.e32[3 * size_t(n) + 2] = float(qb.x + db.x);
    }
    if (limited || again) {
        __syncthreads();  // the chunk's scaled directions
        direction_partial(d, rows);
        if (last_block(&d.sc->dir_done)) direction_total(d, rows);
    }
    if (!d.has_collider && blockIdx.x == 0 && threadIdx.x == 0) publish_ccd(d);
}

// Line-search CCD bound (cuda_backend.cu:989-1000); the minimum over all
// elements and candidates is taken with an unsigned atomicMin on the bit
// pattern of the non-negative step.
template<bool MIXED> __global__ void __launch_bounds__(kBlock) k_ccd(View d)
{
    follow_previous();
    const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= d.E) return;
    const uint32_t i = d.ei[e], j = d.ej[e];
    if (d.fixed[i] || !d.econtact[e]) return;
    const V p0 = load3(d.q + 6 * size_t(i)), p1 = load3(d.q + 6 * size_t(j));
    const V d0 = load3(d.dir + 6 * size_t(i)), d1 = load3(d.dir + 6 * size_t(j));
    const V lo = dm::vmin(dm::vmin(p0, p1), dm::vmin(p0 + d0, p1 + d1));
    const V hi = dm::vmax(dm::vmax(p0, p1), dm::vmax(p0 + d0, p1 + d1));
    const double target = d.radius + d.offset + d.min_gap;
    double local = 1.0;
    const dm::F3 f0 = dm::f3(0.f, 0.f, 0.f), f1 = dm::to_local(p1, p0);
    bvh_query_packed(d, lo, hi, d.ccd_pad, [&](uint32_t t) {
        const double speed = fmax(dm::gnorm(d0), dm::gnorm(d1));
        if (speed < 1e-30) return;
        const V a = tri_vertex(d, t, 0), b = tri_vertex(d, t, 1), c = tri_vertex(d, t, 2);
        if (MIXED) {
            // Skip candidates whose first advancement step provably reaches 1.
            float m;
            const float df = dm::segment_triangle_distance_f(f0, f1, dm::to_local(a, p0), dm::to_local(b, p0),
                                                              dm::to_local(c, p0), m);
            if (0.8 * (double(df) - double(m) - target) >= speed * (1.0 + 1e-6)) return;
        }
        double alpha = 0.0;
        // Mixed form: every limit this candidate can still produce is
        // >= 0.9 alpha (alpha only grows), so it stops as soon as that
        // reaches the best limit known (its element's or the global one);
        // the minimum is unchanged.
        double bound = local;
        if (MIXED) bound = fmin(bound, __longlong_as_double(*reinterpret_cast<volatile long long *>(&d.sc->ccd_bits)));
        for (int k = 0; k < 80; ++k) {
            if (MIXED && 0.9 * alpha >= bound) return;
            const double dist = dm::closest_segment_triangle(dm::gadd(p0, dm::gmul(d0, alpha)), dm::gadd(p1, dm::gmul(d1, alpha)), a, b, c).distance;
            const double clear = dist - target;
            if (clear <= 0) { local = fmin(local, fmax(0.0, alpha * 0.9)); return; }
            const double advance = 0.8 * clear / speed;
            if (alpha + advance >= 1) return;
            if (advance < 1e-12) { local = fmin(local, alpha); return; }
            alpha += advance;
        }
        local = fmin(local, alpha);
    });
    if (local < 1.0) atomicMin(&d.sc->ccd_bits, (unsigned long long)__double_as_longlong(local));
}

// CCD bound, load balanced: k_ccd_collect and k_ccd_near list every (element,
// triangle) candidate, in the mixed form (FILTER) without those whose FP32
// lower-bound clearance already lets the first advancement step reach
// alpha = 1; k_advance_pairs runs the exact FP64 conservative advancement
// of cuda_backend.cu:989-1000 per listed pair.  The minimum equals the per-element kernel's
// (k_ccd), which remains for a full pair list.
// The swept element box covers the positions at step 0 and 1.  When all four
// swept end points stay within the slack of the element's leaf cache, the
// cached leaves (collected with the contact padding, which is at least the
// CCD target) hold every leaf the swept box can touch and replace the tree
// walk; most elements have none and are done.  FILTER skips a pair only when
// even the lower bound of 0.8 (dist - target) reaches the speed, so the first
// advancement step of the exact pass would leave the step unlimited anyway.
struct SweptElement {
    QueryBox qb;
    dm::F3 origin, f1;
    float speed_ru;  // an upper bound of the larger end point displacement
};

__device__ __forceinline__ dm::F3 load3f(const float *p) { return dm::f3(p[0], p[1], p[2]); }

__device__ __forceinline__ SweptElement swept_element(const View &d, uint32_t i, uint32_t j)
{
    SweptElement w;
    const dm::F3 p0 = load3f(d.q32 + 3 * size_t(i)), p1 = load3f(d.q32 + 3 * size_t(j));
    const dm::F3 e0 = load3f(d.e32 + 3 * size_t(i)), e1 = load3f(d.e32 + 3 * size_t(j));
    const float lo32[3] = {fminf(fminf(p0.x, p1.x), fminf(e0.x, e1.x)), fminf(fminf(p0.y, p1.y), fminf(e0.y, e1.y)),
                           fminf(fminf(p0.z, p1.z), fminf(e0.z, e1.z))};
    const float hi32[3] = {fmaxf(fmaxf(p0.x, p1.x), fmaxf(e0.x, e1.x)), fmaxf(fmaxf(p0.y, p1.y), fmaxf(e0.y, e1.y)),
                           fmaxf(fmaxf(p0.z, p1.z), fmaxf(e0.z, e1.z))};
    w.qb = make_query_f(lo32, hi32, d.ccd_pad);
    w.origin = p0;
    w.f1 = dm::fsub(p1, p0);
    // Either copy is within 2^-24 of a coordinate's magnitude, a difference of
    // two within 2^-22 of the larger one.
    auto bound = [](dm::F3 p, dm::F3 e) {
        const float mag = fmaxf(fmaxf(fmaxf(fabsf(p.x), fabsf(p.y)), fabsf(p.z)), fmaxf(fmaxf(fabsf(e.x), fabsf(e.y)), fabsf(e.z)));
        const dm::F3 v = dm::fsub(e, p);
        return __fadd_ru(__fmul_ru(sqrtf(dm::fdot(v, v)), 1.00001f), __fmaf_ru(mag, 5.0e-7f, 1.0e-12f));
    };
    w.speed_ru = fmaxf(bound(p0, e0), bound(p1, e1));
    return w;
}

// The FP64 swept box.
__device__ __forceinline__ void swept_box(const View &d, uint32_t i, uint32_t j, V &lo, V &hi)
{
    const V p0 = load3(d.q + 6 * size_t(i)), p1 = load3(d.q + 6 * size_t(j));
    const V e0 = p0 + load3(d.dir + 6 * size_t(i)), e1 = p1 + load3(d.dir + 6 * size_t(j));
    lo = dm::vmin(dm::vmin(p0, p1), dm::vmin(e0, e1));
    hi = dm::vmax(dm::vmax(p0, p1), dm::vmax(e0, e1));
}

template<bool FILTER> __device__ __forceinline__ void list_swept_pair(const View &d, const SweptElement &w, uint32_t e, uint32_t p)
{
    uint32_t t;
    if (FILTER) {
        float m;
        const float df = record_distance_f(d, p, w.origin, dm::f3(0.f, 0.f, 0.f), w.f1, m, t);
        if (__fmul_rd(0.8f, __fsub_rd(__fsub_rd(df, m), d.ccd_pad.up)) >= w.speed_ru) return;
    } else {
        t = __float_as_uint(__ldg(d.tri32 + 3 * size_t(p)).w);
    }
    const unsigned long long slot = append_slot(&d.sc->pair_count);
    if (slot < d.pair_capacity) { d.pair_elem[slot] = e; d.pair_tri[slot] = t; }
}

template<bool FILTER> __global__ void __launch_bounds__(kBlock) k_ccd_collect(View d)
{
    follow_previous();
    const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= d.E) return;
    const uint32_t i = d.ei[e], j = d.ej[e];
    if (d.fixed[i] || !d.econtact[e]) return;
    const uint8_t nl = d.cache_n[e];
    if (nl != kCacheInvalid && d.dhat >= d.min_gap) {
        const float *c = d.cache_x32 + 6 * size_t(e);
        const dm::F3 xi32 = dm::f3(d.q32[3 * size_t(i)], d.q32[3 * size_t(i) + 1], d.q32[3 * size_t(i) + 2]);
        const dm::F3 xj32 = dm::f3(d.q32[3 * size_t(j)], d.q32[3 * size_t(j) + 1], d.q32[3 * size_t(j) + 2]);
        const dm::F3 a0 = load3f(d.e32 + 3 * size_t(i)), a1 = load3f(d.e32 + 3 * size_t(j));
        if (within_cache_slack(c, xi32, xj32) && within_cache_slack(c, a0, a1)) {
            // k_ccd_near tests the cached leaves, one warp per element.
            if (nl > 0) d.near_list[append_slot(&d.sc->ccd_near)] = e;
            return;
        }
    }
    const SweptElement w = swept_element(d, i, j);
    bvh_positions_packed(d, w.qb, d.ccd_pad.exact, [&](V &lo, V &hi) { swept_box(d, i, j, lo, hi); }, [&](uint32_t p) { list_swept_pair<FILTER>(d, w, e, p); });
}

// One warp per element queued by k_ccd_collect: its leaves are tested 32 at a
// time against the swept box and their candidates spread over the warp (the
// pair order does not matter: the bound is a minimum).
template<bool FILTER> __global__ void __launch_bounds__(kBlock) k_ccd_near(View d)
{
    follow_previous();
    __shared__ uint32_t lists[kBlock / 32][kNearList];
    const int lane = threadIdx.x & 31;
    uint32_t *pos = lists[threadIdx.x >> 5];
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t count = d.sc->ccd_near;
    for (uint32_t k = warp; k < count; k += nwarps) {
        const uint32_t e = d.near_list[k];
        uint32_t nleaves = 0;
        const uint32_t *leaves = cached_leaves(d, e, d.cache_n[e], nleaves);
        const uint32_t i = d.ei[e], j = d.ej[e];
        const SweptElement w = swept_element(d, i, j);
        for (uint32_t r0 = 0; r0 < nleaves; r0 += 32) {
            uint32_t first, cnt;
            near_leaf(d, leaves, r0 + lane, nleaves, w.qb, d.ccd_pad.exact, [&](V &lo, V &hi) { swept_box(d, i, j, lo, hi); }, first,
                      cnt);
            const uint32_t here = spread_candidates(first, cnt, pos, lane);
            for (uint32_t c = lane; c < here; c += 32) list_swept_pair<FILTER>(d, w, e, pos[c]);
        }
    }
}

// Conservative advancement of the listed pairs, 32 to a block of five warps as
// in k_contact_exact: in each of at most 80 steps the warps take the parts of
// the distance at the pair's alpha, and warp 0 moves it on.  SWEEP: the
// triangle moves from its old position and the hair stands (the pair's element
// fails unless alpha reaches 1); else the hair moves by its direction and the
// triangle stands (the pair's limit bounds the step).
template<bool SWEEP> __global__ void __launch_bounds__(kPairBlock) k_advance_pairs(View d)
{
    follow_previous();
    __shared__ double sh_d2[kPairWarps][32], sh_alpha[32];
    __shared__ uint32_t sh_active;
    const int part = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t count = uint32_t(min(d.sc->pair_count, (unsigned long long)d.pair_capacity));
    const double target = d.radius + d.offset + d.min_gap;
    for (uint32_t base = 32 * blockIdx.x; base < count; base += 32 * gridDim.x) {
        const uint32_t k = base + lane;
        uint32_t e = 0;
        V p0 = dm::v(0, 0, 0), p1 = p0, a = p0, b = p0, c = p0;  // at alpha 0
        V m0 = p0, m1 = p0, m2 = p0;                             // what alpha moves: p0, p1 or a, b, c
        bool fast = false;
        double speed = 0.0;
        if (k < count) {
            e = d.pair_elem[k];
            const uint32_t t = d.pair_tri[k], i = d.ei[e], j = d.ej[e];
            p0 = load3(d.q + 6 * size_t(i)); p1 = load3(d.q + 6 * size_t(j));
            a = tri_vertex(d, t, 0); b = tri_vertex(d, t, 1); c = tri_vertex(d, t, 2);
            if (SWEEP) {
                const V oa = load3(d.col_old + 3 * size_t(d.tri[3 * t])), ob = load3(d.col_old + 3 * size_t(d.tri[3 * t + 1])),
                        oc = load3(d.col_old + 3 * size_t(d.tri[3 * t + 2]));
                fast = dm::sane_pair(p0, p1, a, b, c) && dm::sane(oa) && dm::sane(ob) && dm::sane(oc);
                m0 = dm::gsub(a, oa); m1 = dm::gsub(b, ob); m2 = dm::gsub(c, oc);
                a = oa; b = ob; c = oc;
            } else {
                m0 = load3(d.dir + 6 * size_t(i)); m1 = load3(d.dir + 6 * size_t(j));
                fast = dm::sane_pair(p0, p1, a, b, c) && dm::sane(m0) && dm::sane(m1);
            }
        }
        double alpha = 0.0;
        if (part == 0) {
            speed = SWEEP ? fmax(dm::gnorm(m0), fmax(dm::gnorm(m1), dm::gnorm(m2))) : fmax(dm::gnorm(m0), dm::gnorm(m1));
            bool on = k < count;
            // Every limit a pair can still produce is >= 0.9 alpha, so it
            // stops as soon as that reaches the smallest limit found so far.
            on = on && !(speed < 1e-30);
            if (!SWEEP) on = on && __longlong_as_double(*reinterpret_cast<volatile long long *>(&d.sc->ccd_bits)) > 0.0;
            const uint32_t active = __ballot_sync(0xffffffffu, on);
            sh_alpha[lane] = 0.0;
            if (lane == 0) sh_active = active;
        }
        __syncthreads();
        for (int it = 0; it < 80; ++it) {
            const uint32_t active = sh_active;
            if (active == 0) break;
            const bool on = active >> lane & 1u;
            double bound = 0.0;
            if (!SWEEP && part == 0) bound = __longlong_as_double(*reinterpret_cast<volatile long long *>(&d.sc->ccd_bits));
            if (on) {
                alpha = sh_alpha[lane];
                dm::PairPart x;
                if (SWEEP)
                    x = part_of(fast, part, p0, p1, dm::gadd(a, dm::gmul(m0, alpha)), dm::gadd(b, dm::gmul(m1, alpha)),
                                dm::gadd(c, dm::gmul(m2, alpha)));
                else
                    x = part_of(fast, part, dm::gadd(p0, dm::gmul(m0, alpha)), dm::gadd(p1, dm::gmul(m1, alpha)), a, b, c);
                sh_d2[part][lane] = x.dist2;
            }
            __syncthreads();
            if (part == 0) {
                bool more = false;
                if (on) {
                    unsigned long long least = 0x7ff0000000000000ull;  // smallest squared distance; NaN never is
#pragma unroll
                    for (int w = 0; w < kPairWarps; ++w) {
                        const unsigned long long x = (unsigned long long)__double_as_longlong(sh_d2[w][lane]);
                        least = x < least ? x : least;
                    }
                    const double dist = least == 0x7ff0000000000000ull ? 1.0e300 : sqrt(__longlong_as_double((long long)least));
                    const double clear = dist - target;
                    double limit = 2.0;  // none
                    bool failed = false;
                    if (clear <= 0) {
                        limit = fmax(0.0, alpha * 0.9);
                        failed = true;
                    } else {
                        const double advance = 0.8 * clear / speed;
                        if (alpha + advance >= 1) {
                        } else if (advance < 1e-12) {
                            limit = alpha;
                            failed = true;
                        } else {
                            alpha += advance;
                            more = it < 79 && (SWEEP || !(0.9 * alpha >= bound));
                            if (it == 79) {
                                limit = alpha;
                                failed = true;
                            }
                        }
                    }
                    if (SWEEP) {
                        if (failed) atomicMin(&d.sc->sweep_fail, e);
                    } else if (limit < 1.0) {
                        atomicMin(&d.sc->ccd_bits, (unsigned long long)__double_as_longlong(limit));
                    }
                    sh_alpha[lane] = alpha;
                }
                const uint32_t next = __ballot_sync(0xffffffffu, more);
                if (lane == 0) sh_active = next;
            }
            __syncthreads();
        }
        __syncthreads();
    }
    if (!SWEEP && last_block(&d.sc->ccd_done) && threadIdx.x == 0) publish_ccd(d);
}

// ---- moving-collider sweep ------------------------------------------------
//
// k_sweep_collect (thread per element): the leaves of the swept BVH (boxes of
// old and new positions) around the standing element, into its cache slots,
// which the substep's first evaluation fills anew.  k_sweep_near (warp per
// element with leaves): exact leaf tests; every candidate, in the mixed form
// without those that sweep_skip_f clears, goes to the pair list.
// k_advance_pairs<true>: the FP64 advancement a pair.  k_sweep_record publishes
// the lowest failing element.  k_sweep, one thread per element for all of it
// (1.3 ms on 67,000 elements, 3.0 ms on 3,200 among contacts in the plain
// form), remains for a full pair list.
__global__ void __launch_bounds__(kBlock) k_sweep_collect(View d)
{
    follow_previous();
    const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= d.E) return;
    const uint32_t i = d.ei[e], j = d.ej[e];
    if (d.fixed[i] || !d.econtact[e]) return;
    const V p0 = load3(d.q + 6 * size_t(i)), p1 = load3(d.q + 6 * size_t(j));
    const uint8_t nl = leaves_to_cache(d, e, dm::vmin(p0, p1), dm::vmax(p0, p1), d.ccd_pad);
    if (nl == kCacheInvalid) {  // the leaf pool is full
        if (sweep_element(d, e, nullptr)) atomicMin(&d.sc->sweep_fail, e);
    } else if (nl > 0) {
        d.near_list[append_slot(&d.sc->ccd_near)] = e;
    }
}

template<bool FILTER> __global__ void __launch_bounds__(kBlock) k_sweep_near(View d)
{
    follow_previous();
    __shared__ uint32_t lists[kBlock / 32][kNearList];
    const int lane = threadIdx.x & 31;
    uint32_t *pos = lists[threadIdx.x >> 5];
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t count = d.sc->ccd_near;
    for (uint32_t k = warp; k < count; k += nwarps) {
        const uint32_t e = d.near_list[k];
        uint32_t nleaves = 0;
        const uint32_t *leaves = cached_leaves(d, e, d.cache_n[e], nleaves);
        const V p0 = load3(d.q + 6 * size_t(d.ei[e])), p1 = load3(d.q + 6 * size_t(d.ej[e]));
        const dm::F3 origin = dm::f3(float(p0.x), float(p0.y), float(p0.z)), end = dm::f3(float(p1.x), float(p1.y), float(p1.z));
        const dm::F3 f1 = dm::fsub(end, origin);
        const float lo32[3] = {fminf(origin.x, end.x), fminf(origin.y, end.y), fminf(origin.z, end.z)};
        const float hi32[3] = {fmaxf(origin.x, end.x), fmaxf(origin.y, end.y), fmaxf(origin.z, end.z)};
        const QueryBox qb = make_query_f(lo32, hi32, d.ccd_pad);
        auto box = [&](V &lo, V &hi) { lo = dm::vmin(p0, p1); hi = dm::vmax(p0, p1); };
        for (uint32_t r0 = 0; r0 < nleaves; r0 += 32) {
            uint32_t first, cnt;
            near_leaf(d, leaves, r0 + lane, nleaves, qb, d.ccd_pad.exact, box, first, cnt);
            const uint32_t here = spread_candidates(first, cnt, pos, lane);
            for (uint32_t c = lane; c < here; c += 32) {
                const uint32_t p = pos[c];
                if (FILTER && sweep_skip_f(d, p, origin, f1, d.ccd_pad.up)) continue;
                const unsigned long long slot = append_slot(&d.sc->pair_count);
                if (slot < d.pair_capacity) {
                    d.pair_elem[slot] = e;
                    d.pair_tri[slot] = __float_as_uint(__ldg(d.tri32 + 3 * size_t(p)).w);
                }
            }
        }
    }
}

// Publishes the lowest failing element of the sweep (with its first failing
// triangle in traversal order) and the length of the pair list, and re-arms.
__global__ void k_sweep_record(View d)
{
    follow_previous();
    if (threadIdx.x || blockIdx.x) return;
    const uint32_t e = d.sc->sweep_fail;
    d.mail->pair_count = d.sc->pair_count;
    d.sc->pair_count = 0;
    d.sc->ccd_near = 0;
    d.sc->sweep_fail = kNone;
    d.mail->sweep_fail = e;
    if (e == kNone) return;
    SweepRecord rec{};
    sweep_element(d, e, &rec);
    *d.sweep = rec;
}

// ---- end of substep -------------------------------------------------------

__global__ void __launch_bounds__(kBlock) k_update_velocity(View d, double inv_dt)
{
    follow_previous();
    const uint32_t n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= d.N || d.fixed[n]) return;
    for (int k = 0; k < 6; ++k) d.v[6 * size_t(n) + k] = (d.q[6 * size_t(n) + k] - d.q_old[6 * size_t(n) + k]) * inv_dt;
}

// The elements between a fixed and a free node take part in friction but not
// in the evaluations' contact pass: their leaves (collected with the others')
// are queued here for k_contact_near and k_contact_exact, and k_friction
// selects their pairs and clears their records.
__device__ __forceinline__ bool friction_root(const View &d, uint32_t e, uint32_t i, uint32_t j)
{
    return d.fixed[i] && !d.fixed[j] && d.econtact[e];
}

__global__ void __launch_bounds__(kBlock) k_friction_collect(View d)
{
    follow_previous();
    const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= d.E) return;
    const uint32_t i = d.ei[e], j = d.ej[e];
    if (!friction_root(d, e, i, j)) return;
    const uint8_t nl = refresh_leaves(d, d.q, e, i, j, false);
    d.surv_n[e] = nl == kCacheInvalid ? kSurvOverflow : 0;
    if (nl != kCacheInvalid && nl > 0) queue_near(d, e, nl);
}

// Coulomb friction impulse (cuda_backend.cu:941-964); each element writes
// its velocity change into its left/right node slots.
template<bool FILTER> __global__ void __launch_bounds__(kBlock) k_friction(View d, double dt)
{
    follow_previous();
    const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e == 0) {  // k_contact_near and k_contact_exact, their only readers, have completed
        d.sc->surv_count = 0;
        d.sc->near_count = 0;
        d.sc->wide_count = 0;
    }
    if (e >= d.E) return;
    const uint32_t i = d.ei[e], j = d.ej[e];
    double di[3] = {0, 0, 0}, dj[3] = {0, 0, 0};
    const bool fi = d.fixed[i], fj = d.fixed[j];
    if (d.econtact[e] && !(fi && fj)) {
        const V p0 = load3(d.q + 6 * size_t(i)), p1 = load3(d.q + 6 * size_t(j));
        uint32_t closest;
        dm::ClosestPair pair;
        if (!fi) {
            // The last gradient evaluation ran the contact pass at this q and
            // this collider state: reuse its closest pair.
            closest = d.c_tri[e];
            pair.t = d.c_t[e]; pair.distance = d.c_dist[e]; pair.bary = load3(d.c_bary + 3 * size_t(e));
        } else {
            closest = select_pair<FILTER>(d, d.q, e, d.surv_n[e], pair);
            d.c_cand[e] = 0; d.c_tri[e] = kNone; d.c_flags[e] = 0; d.c_gap[e] = 0.0;
        }
        const double gap = pair.distance - d.radius - d.offset;
        if (closest != kNone && gap > 0.0 && gap < d.dhat) {
            const double w0 = 1.0 - pair.t, w1 = pair.t;
            const V hair = p0 * w0 + p1 * w1;
            const V body = tri_vertex(d, closest, 0) * pair.bary.x + tri_vertex(d, closest, 1) * pair.bary.y +
                           tri_vertex(d, closest, 2) * pair.bary.z;
            const V ob = load3(d.col_old + 3 * size_t(d.tri[3 * closest])) * pair.bary.x +
                         load3(d.col_old + 3 * size_t(d.tri[3 * closest + 1])) * pair.bary.y +
                         load3(d.col_old + 3 * size_t(d.tri[3 * closest + 2])) * pair.bary.z;
            const V normal = (hair - body) * (1.0 / fmax(pair.distance, 1.0e-15));
            const V v0 = load3(d.v + 6 * size_t(i)), v1 = load3(d.v + 6 * size_t(j));
            const V rel = v0 * w0 + v1 * w1 - (body - ob) * (1.0 / dt);
            const V tangent = rel - normal * dm::dot(normal, rel);
            const double ts = dm::norm(tangent);
            double im = 0.0;
            if (!fi) im += w0 * w0 / fmax(d.mass[i], 1.0e-30);
            if (!fj) im += w1 * w1 / fmax(d.mass[j], 1.0e-30);
            if (!(ts < 1.0e-15) && im > 0.0) {
                const double aa = d.dhat - gap, lg = log(gap / d.dhat);
                const double fn = d.kc * (aa * aa / gap - 2.0 * aa * lg), required = ts / im;
                const double mag = fmin(required, d.friction * fn * dt), smooth = d.smoothing / dt;
                const V imp = tangent * (-mag / fmax(sqrt(ts * ts + smooth * smooth), 1.0e-30));
                if (!fi) { const double s = w0 / fmax(d.mass[i], 1.0e-30); di[0] = imp.x * s; di[1] = imp.y * s; di[2] = imp.z * s; }
                if (!fj) { const double s = w1 / fmax(d.mass[j], 1.0e-30); dj[0] = imp.x * s; dj[1] = imp.y * s; dj[2] = imp.z * s; }
            }
        }
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) { d.as_i_f[3 * size_t(i) + k] = di[k]; d.as_j_f[3 * size_t(j) + k] = dj[k]; }
}

__global__ void __launch_bounds__(kBlock) k_friction_apply(View d)
{
    follow_previous();
    const uint32_t n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= d.N) return;
#pragma unroll
    for (int k = 0; k < 3; ++k) d.v[6 * size_t(n) + k] += d.as_j_f[3 * size_t(n) + k] + d.as_i_f[3 * size_t(n) + k];
}

__global__ void k_init_scalars(View d)
{
    follow_previous();
    if (threadIdx.x || blockIdx.x) return;
    d.sc->ccd_bits = 0x3ff0000000000000ULL;
    d.sc->sweep_fail = kNone;
    d.sc->solve_failed = 0;
    d.sc->pair_count = 0;
    d.sc->surv_count = 0;
    d.sc->solve_next = 0;
    d.sc->refine_bits = 0;
    d.sc->near_count = 0;
    d.sc->wide_count = 0;
    d.sc->ccd_near = 0;
    d.sc->pool_used = 0;
    d.sc->eval_done = 0;
    d.sc->dir_done = 0;
    d.sc->ccd_done = 0;
}

__global__ void __launch_bounds__(kBlock) k_gather(const double *q, const uint32_t *map, uint32_t count, double *out)
{
    follow_previous();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const uint32_t n = map ? map[i] : i;
    out[3 * size_t(i)] = q[6 * size_t(n)];
    out[3 * size_t(i) + 1] = q[6 * size_t(n) + 1];
    out[3 * size_t(i) + 2] = q[6 * size_t(n) + 2];
}

// ---- root targets (src/solver.cpp:416-447) --------------------------------
//
// Target positions and rotation vectors of every node for one set of
// evaluated source points: positions and unit tangents, the tangent-only
// part of each frame step (thread per node), the frame walk along each
// strand (three lanes per strand, longest strands first), then the rotation
// vector of frame * reference^T (thread per node).

constexpr int kRootStrands = 10;  // strands a warp in k_root_frames

struct RootArgs {
    uint32_t N, S, P;
    const double *points;                    // [P][3] evaluated source points
    const uint32_t *bind_l, *bind_r;         // the two source points a node interpolates
    const double *bind_t;
    const uint32_t *node_strand, *sfirst, *scount, *sorder;
    const double *ref;                       // [N][9] reference frames
    double *x, *tangent, *frame, *rot;       // [N][3], [N][3], [N][9], [N][3]
    uint32_t *bad;                           // bit 0: a degenerate tangent, bit 1: a non-finite point
};

__device__ __forceinline__ V root_position(const RootArgs &a, uint32_t n)
{
    return dm::glerp(load3(a.points + 3 * size_t(a.bind_l[n])), load3(a.points + 3 * size_t(a.bind_r[n])), a.bind_t[n]);
}

// Central-difference tangents, one-sided at the strand ends
// (solver.cpp:426-433); a squared length below 1e-24 fails the whole call, and
// so does a point that is not finite.
__global__ void __launch_bounds__(kBlock) k_root_tangents(RootArgs a)
{
    follow_previous();
    const uint32_t n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n < a.P) {
        bool finite = true;
#pragma unroll
        for (int k = 0; k < 3; ++k)
            finite = finite && (uint32_t(__double2hiint(a.points[3 * size_t(n) + k])) & 0x7ff00000u) != 0x7ff00000u;
        if (!finite) atomicOr(a.bad, 2u);
    }
    if (n >= a.N) return;
    const uint32_t s = a.node_strand[n], k = n - a.sfirst[s], count = a.scount[s];
    const V x = root_position(a, n);
    store3(a.x + 3 * size_t(n), x);
    V d;
    if (k == 0) d = dm::gsub(root_position(a, n + 1), x);
    else if (k + 1 == count) d = dm::gsub(x, root_position(a, n - 1));
    else d = dm::gsub(root_position(a, n + 1), root_position(a, n - 1));
    if (dm::gdot(d, d) < 1.0e-24) atomicOr(a.bad, 1u);
    store3(a.tangent + 3 * size_t(n), dm::gunit(d));
}

// Everything of the frame walk that depends on the tangents alone, per node:
// d3 (the tangent normalised once more, as frame_from_tangent does) and the
// minimal rotation from the previous node's tangent, packed into the node's
// frame slot [d3, n, s, c, kind] until k_root_frames replaces it.
__global__ void __launch_bounds__(kBlock) k_root_transport(RootArgs a)
{
    follow_previous();
    const uint32_t n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= a.N) return;
    const V t = load3(a.tangent + 3 * size_t(n));
    double *p = a.frame + 9 * size_t(n);
    store3(p, dm::gunit(t));
    dm::Transport tr{};
    tr.kind = 1;
    if (n != a.sfirst[a.node_strand[n]]) tr = dm::transport_between(load3(a.tangent + 3 * size_t(n - 1)), t);
    store3(p + 3, tr.n);
    p[6] = tr.s; p[7] = tr.c; p[8] = double(tr.kind);
}

// The sequential part (solver.cpp:435-443): each frame's first column is the
// previous one carried by the minimal rotation between consecutive tangents.
// Three lanes a strand, one component each, ten strands a warp, longest
// strands first; a warp a block, so that few strands spread over many SMs.
// What bounds it is the FP64 chain of the longest strands: three normalisations
// a node, each a dot product, a square root and a division; with a component a
// lane a node takes about 130 FP64 instructions (270 with a thread a strand).
// 4,000 strands of 16-160 nodes: 510 us, 2,041 with a thread a strand in
// blocks of 256.
struct Lanes3 {
    int c, base;  // component, first lane of the strand
    __device__ double at(double x, int k) const { return __shfl_sync(0xffffffffu, x, base + k); }
    __device__ double next(double x) const { return at(x, c == 2 ? 0 : c + 1); }
    __device__ double prev(double x) const { return at(x, c == 0 ? 2 : c - 1); }
    __device__ double dot(double a, double b) const
    {
        const double m = dm::xm(a, b);
        return dm::xa(dm::xa(at(m, 0), at(m, 1)), at(m, 2));
    }
    __device__ double cross(double a, double b) const
    {
        return dm::xs(dm::xm(next(a), prev(b)), dm::xm(prev(a), next(b)));
    }
    __device__ double unit(double a) const
    {
        const double n2 = dot(a, a);
        if (!(n2 > 0.0)) return a;  // no shuffle below
        const double n = sqrt(n2);
        return dm::div_by(a, n, dm::recip_any(n));
    }
};

// frame_from_d3 (khs_device_math.cuh) with a component a lane.
__device__ __forceinline__ void frame_lanes(const Lanes3 &l, double d3, double hint, double &d1, double &d2)
{
    d1 = dm::xs(hint, dm::xm(d3, l.dot(hint, d3)));
    const bool flat = l.dot(d1, d1) < 1.0e-16;
    if (__any_sync(0xffffffffu, flat)) {
        const bool along_x = fabs(l.at(d3, 0)) < 0.8;
        const double axis = l.c == (along_x ? 0 : 1) ? 1.0 : 0.0;
        const double other = dm::xs(axis, dm::xm(d3, l.dot(axis, d3)));
        if (flat) d1 = other;
    }
    d1 = l.unit(d1);
    d2 = l.unit(l.cross(d3, d1));
    d1 = l.unit(l.cross(d2, d3));
}

__global__ void __launch_bounds__(32) k_root_frames(RootArgs a)
{
    follow_previous();
    const int lane = threadIdx.x;
    const int slot = min(lane / 3, kRootStrands - 1);  // lanes 30 and 31 shadow the last strand's first two
    Lanes3 l;
    l.c = lane < 3 * kRootStrands ? lane % 3 : lane - 3 * kRootStrands;
    l.base = 3 * slot;
    const uint32_t i = blockIdx.x * kRootStrands + slot;
    const bool member = lane < 3 * kRootStrands && i < a.S;
    const uint32_t s = a.sorder[min(i, a.S - 1)], first = a.sfirst[s], count = a.scount[s];
    const uint32_t most = __reduce_max_sync(0xffffffffu, count);
    double *p = a.frame + 9 * size_t(first);
    double d3 = p[l.c], d1, d2, d3_next = 0.0, n = 0.0, sine = 0.0, cosine = 0.0, kind = 1.0;
    // The next node's tangent and rotation, read while this node's frame is
    // under way; a finished strand goes on with its last slot, unwritten.
    auto fetch = [&](uint32_t k) {
        const double *o = k < count ? p + 9 : p;
        d3_next = o[l.c]; n = o[3 + l.c]; sine = o[6]; cosine = o[7]; kind = o[8];
    };
    fetch(1);
    frame_lanes(l, d3, a.ref[9 * size_t(first) + 3 * l.c], d1, d2);
    for (uint32_t k = 0;;) {
        __syncwarp();  // every lane has read its share of the slot
        if (member && k < count) { p[3 * l.c] = d1; p[3 * l.c + 1] = d2; p[3 * l.c + 2] = d3; }
        if (++k >= most) break;
        if (k < count) p += 9;
        d3 = d3_next;
        // transport_apply of the first column.
        const double nd = l.dot(n, d1);
        double hint = dm::xa(dm::xa(dm::xm(d1, cosine), dm::xm(l.cross(n, d1), sine)), dm::xm(dm::xm(n, nd), dm::xs(1.0, cosine)));
        if (kind == 1.0 || k >= count) hint = d1;
        else if (kind == 2.0) hint = dm::xs(dm::xm(dm::xm(n, 2.0), nd), d1);
        fetch(k + 1);
        frame_lanes(l, d3, hint, d1, d2);
    }
}

__global__ void __launch_bounds__(kBlock) k_root_rotations(RootArgs a)
{
    follow_previous();
    const uint32_t n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= a.N) return;
    const M r = dm::times_transpose(load9(a.frame + 9 * size_t(n)), load9(a.ref + 9 * size_t(n)));
    store3(a.rot + 3 * size_t(n), dm::rotation_vector(r));
}

// ---- device memory --------------------------------------------------------

struct Arena {
    char *base = nullptr;
    size_t size = 0, used = 0;
    template<class T> T *take(size_t count)
    {
        const size_t bytes = (count * sizeof(T) + 255) & ~size_t(255);
        T *p = reinterpret_cast<T *>(base + used);
        used += bytes;
        return p;
    }
};

template<class T> size_t padded(size_t count) { return (count * sizeof(T) + 255) & ~size_t(255); }

}  // namespace

struct Engine::Impl {
    View v{};
    Arena arena;
    cudaStream_t stream = nullptr;
    cudaStream_t side = nullptr;          // contact passes beside the node kernel
    cudaEvent_t fork = nullptr, join = nullptr;
    cudaEvent_t ev_begin = nullptr, ev_end = nullptr;
    Mailbox *mail_host = nullptr;
    SweepRecord *sweep_host = nullptr;
    // Host copies needed by the control flow.
    std::vector<uint32_t> mapping;
    uint32_t original_count = 0;
    double *mapping_gather_out = nullptr;
    uint32_t *mapping_dev = nullptr;
    double *q_snap = nullptr, *v_snap = nullptr;
    double *root_cur_x = nullptr, *root_cur_r = nullptr, *root_pend_x = nullptr, *root_pend_r = nullptr;
    double *col_frame_start = nullptr, *col_pending = nullptr;
    double *anim_root_x = nullptr, *anim_root_r = nullptr, *anim_col = nullptr;
    size_t anim_bytes = 0, ring_bytes = 0;
    double *col_a_copy = nullptr;  // frame-start copy used while stepping
    // Root targets on the device: the two source points each node
    // interpolates and its strand (arena), and the work arrays of one pass
    // (allocated on first use: points [P][3], positions, tangents, frames,
    // rotation vectors, the degenerate-tangent flag).
    uint32_t *bind_l = nullptr, *bind_r = nullptr, *node_strand = nullptr;
    double *bind_t = nullptr;
    char *root_work = nullptr;
    RootArgs root{};
    std::vector<uint8_t> fixed_host;
    uint64_t resident = 0;

    // Per-kernel device-time accounting (CUDA events on this stream).
    struct KernelStat { const char *name; uint64_t launches; double ms; };
    bool profiling = false;
    uint64_t launches = 0;
    // Launch shape of the FP64 block solve: work items, blocks of one warp.
    unsigned solve_items = 0, solve_blocks = 0;
    bool solve_team = false;
    uint32_t sms = 152;
    // Rollback ring: q and v of the last ring_frame.size() animation frames,
    // slot k holding frame ring_frame[k] (-1 = empty), [slots][2][N][6] FP64.
    double *ring = nullptr;
    std::vector<int64_t> ring_frame;
    // Output ring: the original points' positions of the last
    // out_frame.size() animation frames, gathered on the solver's stream after
    // each frame and copied to pinned host memory on copy_stream, so the copy
    // overlaps the next frame ([slots][P][3] FP64 on both sides).
    cudaStream_t copy_stream = nullptr;
    double *out_dev = nullptr, *out_host = nullptr;
    std::vector<cudaEvent_t> out_gathered, out_copied;
    std::vector<int64_t> out_frame;
    size_t out_bytes = 0;
    uint32_t out_next = 0;
    void release_output()
    {
        if (copy_stream) cudaStreamSynchronize(copy_stream);
        for (cudaEvent_t e : out_gathered) cudaEventDestroy(e);
        for (cudaEvent_t e : out_copied) cudaEventDestroy(e);
        out_gathered.clear();
        out_copied.clear();
        if (out_dev) cudaFree(out_dev);
        if (out_host) cudaFreeHost(out_host);
        out_dev = out_host = nullptr;
        resident -= out_bytes;
        out_bytes = 0;
        out_frame.clear();
        out_next = 0;
    }
    std::vector<uint32_t> sorted_len;  // free nodes per strand, in the solve order
    unsigned ff_blocks = 0;     // launch shape of the float-float kernels
    std::vector<KernelStat> kstats;
    std::vector<std::pair<size_t, std::pair<cudaEvent_t, cudaEvent_t>>> pending;
    std::vector<cudaEvent_t> pool;

    cudaEvent_t take_event()
    {
        if (pool.empty()) {
            cudaEvent_t e;
            KHS_CUDA(cudaEventCreate(&e));
            return e;
        }
        cudaEvent_t e = pool.back();
        pool.pop_back();
        return e;
    }
    size_t stat_index(const char *name)
    {
        for (size_t k = 0; k < kstats.size(); ++k)
            if (kstats[k].name == name) return k;
        kstats.push_back({name, 0, 0.0});
        return kstats.size() - 1;
    }
    cudaStream_t ordinary = nullptr;  // stream whose next launch waits in the ordinary way
    void wait_for(cudaStream_t s, cudaEvent_t e)
    {
        KHS_CUDA(cudaStreamWaitEvent(s, e, 0));
        ordinary = s;
    }
    // A launch on stream s (the solver's stream, or the side stream, which
    // is only used while kernels are not timed one by one).
    template<class K, class... A> void launch_on(cudaStream_t s, const char *name, K kernel, unsigned grid, unsigned block,
                                                 A... args)
    {
        if (s == stream) {
            launch(name, kernel, grid, block, args...);
            return;
        }
        ++launches;
        start(s, kernel, grid, block, args...);
    }
    // A kernel that may come up while the previous one on its stream drains
    // (follow_previous), unless another stream's work comes between.
    template<class K, class... A> void start(cudaStream_t s, K kernel, unsigned grid, unsigned block, A... args)
    {
        cudaLaunchAttribute early{};
        early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        early.val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t config{};
        config.gridDim = dim3(grid);
        config.blockDim = dim3(block);
        config.stream = s;
        config.attrs = &early;
        config.numAttrs = s == ordinary ? 0 : 1;
        if (s == ordinary) ordinary = nullptr;
        KHS_CUDA(cudaLaunchKernelEx(&config, kernel, args...));
    }
    template<class K, class... A> void launch(const char *name, K kernel, unsigned grid, unsigned block, A... args)
    {
        ++launches;
        if (!profiling) {
            start(stream, kernel, grid, block, args...);
            return;
        }
        cudaEvent_t a = take_event(), b = take_event();
        KHS_CUDA(cudaEventRecord(a, stream));
        kernel<<<grid, block, 0, stream>>>(args...);
        KHS_CUDA(cudaEventRecord(b, stream));
        pending.push_back({stat_index(name), {a, b}});
    }
    void resolve()
    {
        for (auto &p : pending) {
            float ms = 0.0f;
            KHS_CUDA(cudaEventElapsedTime(&ms, p.second.first, p.second.second));
            kstats[p.first].launches += 1;
            kstats[p.first].ms += ms;
            pool.push_back(p.second.first);
            pool.push_back(p.second.second);
        }
        pending.clear();
    }

    ~Impl()
    {
        for (auto &p : pending) { pool.push_back(p.second.first); pool.push_back(p.second.second); }
        for (cudaEvent_t e : pool) cudaEventDestroy(e);
        if (arena.base) cudaFree(arena.base);
        if (ring) cudaFree(ring);
        if (anim_root_x) cudaFree(anim_root_x);
        if (root_work) cudaFree(root_work);
        release_output();
        if (copy_stream) cudaStreamDestroy(copy_stream);
        if (mail_host) cudaFreeHost(mail_host);
        if (sweep_host) cudaFreeHost(sweep_host);
        if (ev_begin) cudaEventDestroy(ev_begin);
        if (ev_end) cudaEventDestroy(ev_end);
        if (side) cudaStreamDestroy(side);
        if (fork) cudaEventDestroy(fork);
        if (join) cudaEventDestroy(join);
        if (stream) cudaStreamDestroy(stream);
    }
    void sync()
    {
        KHS_CUDA(cudaStreamSynchronize(stream));
        if (!pending.empty()) resolve();
    }
    void check() { KHS_CUDA(cudaGetLastError()); }
};

Engine::Engine() : d_(new Impl) {}
Engine::~Engine() = default;

void Engine::initialize(const Model &m, const KhsSolverDesc &desc, const KhsHairMaterial &material,
                        const std::vector<Vec> &root_pos, const std::vector<Vec> &root_rot)
{
    Impl &I = *d_;
    KHS_CUDA(cudaSetDevice(0));
    KHS_CUDA(cudaStreamCreateWithFlags(&I.stream, cudaStreamNonBlocking));
    KHS_CUDA(cudaStreamCreateWithFlags(&I.side, cudaStreamNonBlocking));
    KHS_CUDA(cudaEventCreateWithFlags(&I.fork, cudaEventDisableTiming));
    KHS_CUDA(cudaEventCreateWithFlags(&I.join, cudaEventDisableTiming));
    KHS_CUDA(cudaEventCreate(&I.ev_begin));
    KHS_CUDA(cudaEventCreate(&I.ev_end));
    KHS_CUDA(cudaHostAlloc(reinterpret_cast<void **>(&I.mail_host), sizeof(Mailbox), cudaHostAllocMapped));
    KHS_CUDA(cudaHostAlloc(reinterpret_cast<void **>(&I.sweep_host), sizeof(SweepRecord), cudaHostAllocMapped));
    std::memset(I.mail_host, 0, sizeof(Mailbox));
    std::memset(I.sweep_host, 0, sizeof(SweepRecord));
    desc_ = desc;
    material_ = material;
    const size_t N = m.nodes(), E = m.elements(), S = m.strands(), Vn = m.collider.size(), T = m.tri.size() / 3,
                 B = m.bvh.size(), L = m.bvh.leaves.size(), O = m.mapping.size();
    // Arena sizing.
    size_t bytes = 0;
    bytes += 13 * padded<double>(6 * N);     // q q_old v q_base grad dir precond dprime as_i_g as_j_g q_snap v_snap inertia
    bytes += 5 * padded<double>(36 * N);     // diag upper cprime as_i_h as_j_h
    bytes += 2 * padded<double>(9 * N) + padded<double>(9 * N);  // rot jl ref
    bytes += 4 * padded<double>(N);          // node_energy kinetic mass rmass
    bytes += 2 * padded<double>(3 * N);      // as_i_f as_j_f
    bytes += padded<uint8_t>(N) + 2 * padded<int32_t>(N);
    bytes += 4 * padded<double>(3 * N);      // root cur/pending x r
    bytes += 3 * padded<uint32_t>(N) + padded<double>(N);  // root bindings, node strand
    bytes += 3 * padded<uint32_t>(E) + padded<uint8_t>(E) + 2 * padded<double>(E) + 2 * padded<double>(3 * E);
    bytes += 3 * padded<double>(E) + 2 * padded<uint32_t>(E) + padded<uint8_t>(E) + padded<double>(kPush * E);
    bytes += 5 * padded<uint32_t>(S);
    bytes += padded<uint32_t>(3 * T) + 5 * padded<double>(3 * Vn) + padded<float>(3 * Vn);
    bytes += 2 * padded<float4>(2 * B);
    // Pairs of the contact pass: the mixed form keeps one or two candidates of
    // an element near the surface, the plain form all of them, hundreds at a
    // mesh pole; a full pool falls back to the search by one thread.
    const size_t surv_capacity = std::max<size_t>(size_t(1) << 18, 8 * E);
    const size_t pair_capacity = std::min<size_t>(std::max<size_t>(size_t(1) << 20, 8 * E), size_t(16) << 20);
    bytes += 2 * padded<double>(E) + padded<double>(3 * E) + 2 * padded<uint32_t>(pair_capacity);
    bytes += padded<uint32_t>(size_t(kCacheLeaves) * E) + padded<uint8_t>(E);
    const size_t leaf_pool = std::min<size_t>(std::max<size_t>(size_t(1) << 20, 4 * E), size_t(16) << 20);
    bytes += padded<uint32_t>(leaf_pool);
    bytes += 2 * padded<float>(3 * N) + padded<float>(6 * E);
    bytes += padded<uint32_t>(E);
    bytes += 2 * padded<float2>(36 * N) + padded<float2>(6 * N) + padded<float>(N);
    bytes += 2 * padded<float4>(3 * T) + 2 * padded<uint32_t>(surv_capacity) + 2 * padded<uint32_t>(E) +
             padded<double>(5 * surv_capacity);
    bytes += 4 * padded<double>(3 * B) + 4 * padded<uint32_t>(B) + padded<int32_t>(B) + 2 * padded<uint32_t>(B) +
             padded<uint32_t>(L) + padded<uint32_t>(T);
    bytes += padded<Partial>(kPartials) + padded<DirPartial>(kPartials) + padded<Scalars>(1);
    bytes += padded<uint32_t>(O) + padded<double>(3 * std::max(N, O));
    KHS_CUDA(cudaMalloc(reinterpret_cast<void **>(&I.arena.base), bytes));
    KHS_CUDA(cudaMemsetAsync(I.arena.base, 0, bytes, I.stream));
    I.arena.size = bytes;
    I.resident = bytes;
    Arena &a = I.arena;
    View &v = I.v;
    v.N = uint32_t(N); v.E = uint32_t(E); v.S = uint32_t(S); v.V = uint32_t(Vn); v.T = uint32_t(T); v.B = uint32_t(B);
    v.L = uint32_t(L);
    v.q = a.take<double>(6 * N); v.q_old = a.take<double>(6 * N); v.v = a.take<double>(6 * N);
    v.q_base = a.take<double>(6 * N); v.grad = a.take<double>(6 * N); v.dir = a.take<double>(6 * N);
    v.precond = a.take<double>(6 * N); v.dprime = a.take<double>(6 * N); v.inertia = a.take<double>(6 * N);
    v.q32 = a.take<float>(3 * N); v.e32 = a.take<float>(3 * N);
    v.as_i_g = a.take<double>(6 * N); v.as_j_g = a.take<double>(6 * N);
    I.q_snap = a.take<double>(6 * N); I.v_snap = a.take<double>(6 * N);
    v.diag = a.take<double>(36 * N); v.upper = a.take<double>(36 * N); v.cprime = a.take<double>(36 * N);
    v.as_i_h = a.take<double>(36 * N); v.as_j_h = a.take<double>(36 * N);
    v.rot = a.take<double>(9 * N); v.jl = a.take<double>(9 * N);
    double *ref = a.take<double>(9 * N);
    v.node_energy = a.take<double>(N); v.node_kinetic = a.take<double>(N);
    double *mass = a.take<double>(N), *rmass = a.take<double>(N);
    v.as_i_f = a.take<double>(3 * N); v.as_j_f = a.take<double>(3 * N);
    uint8_t *fixed = a.take<uint8_t>(N);
    int32_t *eleft = a.take<int32_t>(N), *eright = a.take<int32_t>(N);
    I.root_cur_x = a.take<double>(3 * N); I.root_cur_r = a.take<double>(3 * N);
    I.root_pend_x = a.take<double>(3 * N); I.root_pend_r = a.take<double>(3 * N);
    I.bind_l = a.take<uint32_t>(N); I.bind_r = a.take<uint32_t>(N); I.node_strand = a.take<uint32_t>(N);
    I.bind_t = a.take<double>(N);
    uint32_t *ei = a.take<uint32_t>(E), *ej = a.take<uint32_t>(E), *es = a.take<uint32_t>(E);
    uint8_t *ec = a.take<uint8_t>(E);
    double *L0 = a.take<double>(E), *invL = a.take<double>(E), *g0 = a.take<double>(3 * E), *k0 = a.take<double>(3 * E);
    v.e_el = a.take<double>(E); v.e_co = a.take<double>(E); v.c_gap = a.take<double>(E);
    v.push = a.take<double>(kPush * E);
    v.c_cand = a.take<uint32_t>(E); v.c_tri = a.take<uint32_t>(E); v.c_flags = a.take<uint8_t>(E);
    uint32_t *sf = a.take<uint32_t>(S), *sc = a.take<uint32_t>(S), *sx = a.take<uint32_t>(S), *so = a.take<uint32_t>(S);
    v.solve_items = a.take<uint32_t>(S);
    uint32_t *tri = a.take<uint32_t>(3 * T);
    v.col_cur = a.take<double>(3 * Vn); v.col_old = a.take<double>(3 * Vn);
    v.col32 = a.take<float>(3 * Vn);
    I.col_frame_start = a.take<double>(3 * Vn); I.col_pending = a.take<double>(3 * Vn); I.col_a_copy = a.take<double>(3 * Vn);
    v.blo = a.take<double>(3 * B); v.bhi = a.take<double>(3 * B);
    v.swept_lo = a.take<double>(3 * B); v.swept_hi = a.take<double>(3 * B);
    v.bnode = B ? a.take<float4>(2 * B) : nullptr;
    v.swept_node = B ? a.take<float4>(2 * B) : nullptr;
    v.c_t = a.take<double>(E); v.c_dist = a.take<double>(E); v.c_bary = a.take<double>(3 * E);
    v.pair_elem = a.take<uint32_t>(pair_capacity); v.pair_tri = a.take<uint32_t>(pair_capacity);
    v.pair_capacity = uint32_t(pair_capacity);
    v.cache_leaf = a.take<uint32_t>(size_t(kCacheLeaves) * E); v.cache_n = a.take<uint8_t>(E);
    v.leaf_pool = a.take<uint32_t>(leaf_pool); v.leaf_pool_capacity = uint32_t(leaf_pool);
    v.cache_x32 = a.take<float>(6 * E);
    v.tri32 = a.take<float4>(3 * T); v.tri32_old = a.take<float4>(3 * T);
    v.ff_inv = a.take<float2>(36 * N); v.ff_c = a.take<float2>(36 * N); v.ff_d = a.take<float2>(6 * N);
    v.ff_shift = a.take<float>(N);
    v.surv_elem = a.take<uint32_t>(surv_capacity); v.surv_tri = a.take<uint32_t>(surv_capacity);
    v.surv_off = a.take<uint32_t>(E); v.surv_n = a.take<uint32_t>(E); v.surv_res = a.take<double>(5 * surv_capacity);
    v.surv_capacity = uint32_t(surv_capacity);
    v.near_list = a.take<uint32_t>(E);
    if (E) KHS_CUDA(cudaMemsetAsync(v.cache_n, kCacheInvalid, E, I.stream));
    uint32_t *bfirst = a.take<uint32_t>(B), *bcount = a.take<uint32_t>(B);
    v.brefit = a.take<uint32_t>(B);
    int32_t *bparent = a.take<int32_t>(B);
    uint32_t *bleft = a.take<uint32_t>(B), *bright = a.take<uint32_t>(B), *bleaves = a.take<uint32_t>(L);
    uint32_t *border = a.take<uint32_t>(T);
    v.partials = a.take<Partial>(kPartials);
    v.dpartials = a.take<DirPartial>(kPartials);
    v.sc = a.take<Scalars>(1);
    I.mapping_dev = a.take<uint32_t>(O);
    I.mapping_gather_out = a.take<double>(3 * std::max(N, O));
    if (a.used > a.size) throw std::runtime_error("device arena overflow");

    // Host staging.
    auto up = [&](void *dst, const void *src, size_t bytes2) {
        if (bytes2) KHS_CUDA(cudaMemcpyAsync(dst, src, bytes2, cudaMemcpyHostToDevice, I.stream));
    };
    std::vector<double> hq(6 * N, 0.0), href(9 * N);
    std::vector<int32_t> hl(N, -1), hr(N, -1);
    for (size_t n = 0; n < N; ++n) {
        hq[6 * n] = m.x[n].x; hq[6 * n + 1] = m.x[n].y; hq[6 * n + 2] = m.x[n].z;
        std::memcpy(&href[9 * n], m.frame[n].m, 9 * sizeof(double));
    }
    for (size_t e = 0; e < E; ++e) { hr[m.elem_i[e]] = int32_t(e); hl[m.elem_j[e]] = int32_t(e); }
    std::vector<double> hg0(3 * E), hk0(3 * E);
    for (size_t e = 0; e < E; ++e) {
        hg0[3 * e] = m.rest_shear[e].x; hg0[3 * e + 1] = m.rest_shear[e].y; hg0[3 * e + 2] = m.rest_shear[e].z;
        hk0[3 * e] = m.rest_curvature[e].x; hk0[3 * e + 1] = m.rest_curvature[e].y; hk0[3 * e + 2] = m.rest_curvature[e].z;
    }
    std::vector<uint32_t> order(S);
    std::iota(order.begin(), order.end(), 0u);
    std::stable_sort(order.begin(), order.end(), [&](uint32_t l, uint32_t r) {
        return m.strand_count[l] - m.strand_fixed[l] > m.strand_count[r] - m.strand_fixed[r];
    });
    I.sorted_len.resize(S);
    for (size_t k = 0; k < S; ++k) I.sorted_len[k] = m.strand_count[order[k]] - m.strand_fixed[order[k]];
    std::vector<double> hcol(3 * Vn);
    for (size_t k = 0; k < Vn; ++k) { hcol[3 * k] = m.collider[k].x; hcol[3 * k + 1] = m.collider[k].y; hcol[3 * k + 2] = m.collider[k].z; }
    std::vector<double> hrx(3 * N), hrr(3 * N);
    for (size_t n = 0; n < N; ++n) {
        hrx[3 * n] = root_pos[n].x; hrx[3 * n + 1] = root_pos[n].y; hrx[3 * n + 2] = root_pos[n].z;
        hrr[3 * n] = root_rot[n].x; hrr[3 * n + 1] = root_rot[n].y; hrr[3 * n + 2] = root_rot[n].z;
    }
    up(v.q, hq.data(), 6 * N * 8); up(v.q_old, hq.data(), 6 * N * 8); up(I.q_snap, hq.data(), 6 * N * 8);
    up(v.q_base, hq.data(), 6 * N * 8);
    up(ref, href.data(), 9 * N * 8);
    up(mass, m.mass.data(), N * 8); up(rmass, m.rotational_mass.data(), N * 8);
    up(fixed, m.fixed.data(), N);
    up(eleft, hl.data(), N * 4); up(eright, hr.data(), N * 4);
    up(I.root_cur_x, hrx.data(), 3 * N * 8); up(I.root_cur_r, hrr.data(), 3 * N * 8);
    up(I.root_pend_x, hrx.data(), 3 * N * 8); up(I.root_pend_r, hrr.data(), 3 * N * 8);
    std::vector<uint32_t> hbl(N), hbr(N);
    std::vector<double> hbt(N);
    for (size_t n = 0; n < N; ++n) { hbl[n] = m.binding[n].left; hbr[n] = m.binding[n].right; hbt[n] = m.binding[n].t; }
    up(I.bind_l, hbl.data(), N * 4); up(I.bind_r, hbr.data(), N * 4); up(I.bind_t, hbt.data(), N * 8);
    up(I.node_strand, m.node_strand.data(), N * 4);
    I.root.N = uint32_t(N); I.root.S = uint32_t(S);
    I.root.bind_l = I.bind_l; I.root.bind_r = I.bind_r; I.root.bind_t = I.bind_t; I.root.node_strand = I.node_strand;
    I.root.sfirst = sf; I.root.scount = sc; I.root.sorder = so; I.root.ref = ref;
    up(ei, m.elem_i.data(), E * 4); up(ej, m.elem_j.data(), E * 4); up(es, m.elem_strand.data(), E * 4);
    up(ec, m.elem_contact.data(), E);
    std::vector<double> hinv(E);
    for (size_t e = 0; e < E; ++e) hinv[e] = 1.0 / m.rest_length[e];
    up(invL, hinv.data(), E * 8);
    up(L0, m.rest_length.data(), E * 8); up(g0, hg0.data(), 3 * E * 8); up(k0, hk0.data(), 3 * E * 8);
    up(sf, m.strand_first.data(), S * 4); up(sc, m.strand_count.data(), S * 4); up(sx, m.strand_fixed.data(), S * 4);
    up(so, order.data(), S * 4);
    up(tri, m.tri.data(), 3 * T * 4);
    up(v.col_cur, hcol.data(), 3 * Vn * 8); up(v.col_old, hcol.data(), 3 * Vn * 8);
    std::vector<float> hcol32(hcol.begin(), hcol.end());
    up(v.col32, hcol32.data(), 3 * Vn * 4);
    up(I.col_frame_start, hcol.data(), 3 * Vn * 8); up(I.col_pending, hcol.data(), 3 * Vn * 8);
    if (B) {
        up(v.blo, m.bvh.lower.data(), 3 * B * 8); up(v.bhi, m.bvh.upper.data(), 3 * B * 8);
        std::vector<float> lo32(3 * B), hi32(3 * B);
        for (size_t k = 0; k < 3 * B; ++k) {
            lo32[k] = std::nextafter(float(m.bvh.lower[k]), -std::numeric_limits<float>::infinity());
            hi32[k] = std::nextafter(float(m.bvh.upper[k]), std::numeric_limits<float>::infinity());
        }
        std::vector<float4> packed(2 * B);
        for (size_t k = 0; k < B; ++k) {
            const uint32_t leaf = m.bvh.count[k] ? (m.bvh.first[k] << 4) | m.bvh.count[k] : 0u;
            uint32_t esc = m.bvh.escape[k];
            float e_f, l_f;
            std::memcpy(&e_f, &esc, 4);
            std::memcpy(&l_f, &leaf, 4);
            packed[2 * k] = make_float4(lo32[3 * k], lo32[3 * k + 1], lo32[3 * k + 2], e_f);
            packed[2 * k + 1] = make_float4(hi32[3 * k], hi32[3 * k + 1], hi32[3 * k + 2], l_f);
        }
        up(v.bnode, packed.data(), 2 * B * sizeof(float4));
        up(v.swept_node, packed.data(), 2 * B * sizeof(float4));  // its .w words are never written again
        up(bfirst, m.bvh.first.data(), B * 4); up(bcount, m.bvh.count.data(), B * 4);
        up(bparent, m.bvh.parent.data(), B * 4); up(bleft, m.bvh.left_child.data(), B * 4);
        up(bright, m.bvh.right_child.data(), B * 4); up(bleaves, m.bvh.leaves.data(), L * 4);
        up(border, m.bvh.order.data(), T * 4);
    }
    up(I.mapping_dev, m.mapping.data(), O * 4);
    v.ref = ref; v.mass = mass; v.rmass = rmass; v.fixed = fixed; v.elem_left = eleft; v.elem_right = eright;
    v.ei = ei; v.ej = ej; v.estrand = es; v.econtact = ec; v.L0 = L0; v.invL = invL; v.gamma0 = g0; v.kappa0 = k0;
    v.sfirst = sf; v.scount = sc; v.sfixed = sx; v.sorder = so; v.tri = tri;
    v.bfirst = bfirst; v.bcount = bcount; v.border = border; v.bleaves = bleaves; v.bparent = bparent;
    v.bleft = bleft; v.bright = bright;
    KHS_CUDA(cudaHostGetDevicePointer(reinterpret_cast<void **>(&v.mail), I.mail_host, 0));
    KHS_CUDA(cudaHostGetDevicePointer(reinterpret_cast<void **>(&v.sweep), I.sweep_host, 0));
    v.has_collider = T > 0 ? 1 : 0;
    I.launch("k_init_scalars", k_init_scalars, 1, 1, v);
    if (T) I.launch("k_refit", k_refit, grid_for(size_t(kLeafTriangles) * v.L), kBlock, v);
    KHS_CUDA(cudaGetLastError());
    I.original_count = uint32_t(O);
    I.fixed_host = m.fixed;
    max_rest_length_ = 0.0;
    for (double L : m.rest_length) max_rest_length_ = std::fmax(max_rest_length_, L);
    update_runtime(desc, material, m.mass, m.rotational_mass);
    plan_block_solve(kSolveByRule, 0);
    I.sync();
    clear_failure();
    step_stats_ = {};
    step_stats_.struct_size = sizeof(step_stats_);
    gpu_stats_ = {};
    gpu_stats_.struct_size = sizeof(gpu_stats_);
    gpu_stats_.resident_bytes = I.resident;
    initialized_ = true;
}

void Engine::update_runtime(const KhsSolverDesc &desc, const KhsHairMaterial &material, const std::vector<double> &mass,
                            const std::vector<double> &rotational_mass)
{
    Impl &I = *d_;
    desc_ = desc;
    material_ = material;
    View &v = I.v;
    if (initialized_ || !mass.empty()) {
        KHS_CUDA(cudaMemcpyAsync(const_cast<double *>(v.mass), mass.data(), mass.size() * 8, cudaMemcpyHostToDevice, I.stream));
        KHS_CUDA(cudaMemcpyAsync(const_cast<double *>(v.rmass), rotational_mass.data(), rotational_mass.size() * 8,
                                 cudaMemcpyHostToDevice, I.stream));
        I.sync();
    }
    v.radius = material.radius; v.offset = material.collider_offset; v.dhat = material.barrier_distance;
    v.kc = material.contact_stiffness; v.friction = material.friction; v.smoothing = material.friction_smoothing;
    v.damping = material.mass_damping; v.min_gap = desc.minimum_gap;
    auto padding = [](double x) {
        float near = float(x), inf = std::numeric_limits<float>::infinity();
        return View::Padding{x, double(near) < x ? std::nextafter(near, inf) : near, double(near) > x ? std::nextafter(near, -inf) : near};
    };
    v.contact_pad = padding(v.radius + v.offset + v.dhat);
    v.ccd_pad = padding(v.radius + v.offset + v.min_gap);
    v.gx = desc.gravity.x; v.gy = desc.gravity.y; v.gz = desc.gravity.z;
    v.young = material.young_modulus; v.poisson = material.poisson_ratio; v.shear_corr = material.shear_correction;
    v.w = dm::strain_weights(material.radius, material.young_modulus, material.poisson_ratio, material.shear_correction);
    trust_radius_ = std::fmax(0.25 * max_rest_length_, 8.0 * (material.radius + material.collider_offset + material.barrier_distance));
}

KhsResult Engine::run_root_pass(const KhsVec3 *points, uint32_t count)
{
    Impl &I = *d_;
    const size_t N = I.v.N;
    if (!points || count != I.original_count) return fail(KHS_ERROR_INVALID_ARGUMENT, "the root target point count does not match the source curves");
    if (!I.root_work) {
        const size_t bytes = padded<double>(3 * size_t(count)) + 3 * padded<double>(3 * N) + padded<double>(9 * N) +
                             padded<uint32_t>(1);
        char *base = nullptr;
        if (cudaMalloc(reinterpret_cast<void **>(&base), bytes) != cudaSuccess) {
            cudaGetLastError();
            return fail(KHS_ERROR_OUT_OF_MEMORY, "cannot allocate the device root-target arrays");
        }
        I.root_work = base;
        I.resident += bytes;
        gpu_stats_.resident_bytes = I.resident;
        size_t off = 0;
        auto take = [&](size_t doubles) { double *p = reinterpret_cast<double *>(base + off); off += padded<double>(doubles); return p; };
        I.root.points = take(3 * size_t(count));
        I.root.x = take(3 * N); I.root.tangent = take(3 * N); I.root.rot = take(3 * N); I.root.frame = take(9 * N);
        I.root.bad = reinterpret_cast<uint32_t *>(base + off);
    }
    KHS_CUDA(cudaMemcpyAsync(const_cast<double *>(I.root.points), points, size_t(count) * 24, cudaMemcpyHostToDevice, I.stream));
    I.root.P = count;
    KHS_CUDA(cudaMemsetAsync(I.root.bad, 0, sizeof(uint32_t), I.stream));
    I.launch("k_root_tangents", k_root_tangents, grid_for(std::max<size_t>(N, count)), kBlock, I.root);
    I.launch("k_root_transport", k_root_transport, grid_for(N), kBlock, I.root);
    I.launch("k_root_frames", k_root_frames, grid_for(I.v.S, kRootStrands), 32, I.root);
    I.launch("k_root_rotations", k_root_rotations, grid_for(N), kBlock, I.root);
    I.check();
    uint32_t bad = 0;
    KHS_CUDA(cudaMemcpyAsync(&bad, I.root.bad, sizeof(bad), cudaMemcpyDeviceToHost, I.stream));
    I.sync();
    if (bad & 2u) {
        error_ = kRootPointsNotFinite;  // rejected like other bad arguments: no failed phase
        return KHS_ERROR_INVALID_HAIR;
    }
    if (bad) return fail(KHS_ERROR_INVALID_HAIR, "cannot compute root directions from the root targets");
    return KHS_OK;
}

KhsResult Engine::set_pending_root_points(const KhsVec3 *points, uint32_t count)
{
    Impl &I = *d_;
    const KhsResult r = run_root_pass(points, count);
    if (r != KHS_OK) return r;
    const size_t bytes = 3 * size_t(I.v.N) * 8;
    KHS_CUDA(cudaMemcpyAsync(I.root_pend_x, I.root.x, bytes, cudaMemcpyDeviceToDevice, I.stream));
    KHS_CUDA(cudaMemcpyAsync(I.root_pend_r, I.root.rot, bytes, cudaMemcpyDeviceToDevice, I.stream));
    return KHS_OK;
}

KhsResult Engine::root_targets_to_host(const KhsVec3 *points, uint32_t count, KhsVec3 *positions, KhsVec3 *rotations)
{
    Impl &I = *d_;
    const KhsResult r = run_root_pass(points, count);
    if (r != KHS_OK) return r;
    const size_t bytes = 3 * size_t(I.v.N) * 8;
    KHS_CUDA(cudaMemcpyAsync(positions, I.root.x, bytes, cudaMemcpyDeviceToHost, I.stream));
    KHS_CUDA(cudaMemcpyAsync(rotations, I.root.rot, bytes, cudaMemcpyDeviceToHost, I.stream));
    I.sync();
    return KHS_OK;
}

void Engine::set_pending_collider(const std::vector<Vec> &vertices)
{
    Impl &I = *d_;
    KHS_CUDA(cudaMemcpyAsync(I.col_pending, vertices.data(), vertices.size() * sizeof(Vec), cudaMemcpyHostToDevice, I.stream));
    I.sync();
}

KhsResult Engine::allocate_animation(uint32_t frames)
{
    Impl &I = *d_;
    if (!initialized_ || frames < 1) return fail(KHS_ERROR_INVALID_ARGUMENT, "invalid animation frame count");
    if (I.anim_root_x) { cudaFree(I.anim_root_x); I.anim_root_x = nullptr; I.resident -= I.anim_bytes; }
    const size_t N = I.v.N, Vn = I.v.V;
    const size_t root_bytes = size_t(frames) * 3 * N * 8, col_bytes = size_t(frames) * 3 * Vn * 8;
    const size_t total = 2 * padded<char>(root_bytes) + padded<char>(col_bytes);
    char *base = nullptr;
    if (cudaMalloc(reinterpret_cast<void **>(&base), total) != cudaSuccess) {
        cudaGetLastError();
        return fail(KHS_ERROR_OUT_OF_MEMORY, "cannot allocate device animation storage");
    }
    I.anim_root_x = reinterpret_cast<double *>(base);
    I.anim_root_r = reinterpret_cast<double *>(base + padded<char>(root_bytes));
    I.anim_col = reinterpret_cast<double *>(base + 2 * padded<char>(root_bytes));
    I.anim_bytes = total;
    I.resident += total;
    animation_frames_ = frames;
    animation_ready_ = false;
    root_frame_set_.assign(frames, false);
    collider_frame_set_.assign(frames, Vn == 0);
    gpu_stats_.animation_frame_count = frames;
    gpu_stats_.resident_bytes = I.resident;
    return KHS_OK;
}

KhsResult Engine::set_root_animation_frame(uint32_t frame, const KhsVec3 *points, uint32_t count)
{
    Impl &I = *d_;
    const size_t N = I.v.N;
    // Targets first, then the frame index, in the reference's order
    // (solver.cpp:802-824 computes before the backend checks the frame).
    const KhsResult r = run_root_pass(points, count);
    if (r != KHS_OK) return r;
    if (frame >= animation_frames_) return fail(KHS_ERROR_INVALID_ARGUMENT, "invalid root animation frame");
    KHS_CUDA(cudaMemcpyAsync(I.anim_root_x + size_t(frame) * 3 * N, I.root.x, 3 * N * 8, cudaMemcpyDeviceToDevice, I.stream));
    KHS_CUDA(cudaMemcpyAsync(I.anim_root_r + size_t(frame) * 3 * N, I.root.rot, 3 * N * 8, cudaMemcpyDeviceToDevice, I.stream));
    root_frame_set_[frame] = true;
    return KHS_OK;
}

KhsResult Engine::set_collider_animation_frame(uint32_t frame, const KhsVec3 *vertices, uint32_t count)
{
    Impl &I = *d_;
    if (frame >= animation_frames_ || count != I.v.V) return fail(KHS_ERROR_INVALID_COLLIDER, "invalid collider animation frame");
    if (count) {
        KHS_CUDA(cudaMemcpyAsync(I.anim_col + size_t(frame) * 3 * I.v.V, vertices, size_t(count) * 24, cudaMemcpyHostToDevice, I.stream));
        I.sync();
    }
    collider_frame_set_[frame] = true;
    return KHS_OK;
}

KhsResult Engine::finalize_animation()
{
    if (animation_frames_ < 1 || std::find(root_frame_set_.begin(), root_frame_set_.end(), false) != root_frame_set_.end() ||
        std::find(collider_frame_set_.begin(), collider_frame_set_.end(), false) != collider_frame_set_.end())
        return fail(KHS_ERROR_INVALID_STATE, "animation has missing frames");
    animation_ready_ = true;
    current_frame_ = 0;
    return KHS_OK;
}

KhsResult Engine::fail(KhsResult r, const std::string &message)
{
    error_ = message;
    step_stats_.phase = KHS_PHASE_FAILED;
    progress_phase_.store(KHS_PHASE_FAILED);
    return r;
}

void Engine::clear_failure()
{
    failure_ = {};
    failure_.struct_size = sizeof(failure_);
    failure_.strand_index = kNone;
    failure_.element_index = kNone;
    failure_.collider_triangle_index = kNone;
}

void Engine::set_failure_context(uint32_t kind, uint32_t frame, uint32_t sub, uint32_t attempted, uint32_t maximum,
                                 uint32_t attempts)
{
    failure_.kind = kind; failure_.frame_index = frame; failure_.substep = sub;
    failure_.requested_substeps = desc_.substeps; failure_.attempted_substeps = attempted;
    failure_.maximum_substeps = maximum; failure_.adaptive_attempt_count = attempts;
}

KhsProgress Engine::progress() const
{
    KhsProgress p{};
    p.struct_size = sizeof(p);
    p.phase = progress_phase_.load(); p.frame_index = progress_frame_.load(); p.frame_count = progress_frame_count_.load();
    p.substep = progress_substep_.load(); p.substep_count = progress_substep_count_.load();
    p.nonlinear_iteration = progress_iteration_.load(); p.nonlinear_iteration_limit = desc_.newton_iterations;
    p.cancelled = cancel_.load() ? 1u : 0u;
    p.frame_elapsed_seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - frame_clock_).count();
    return p;
}

EvalStats Engine::evaluate(bool gradient, double dt, double alpha, const double *alpha_dev)
{
    Impl &I = *d_;
    const View &v = I.v;
    const bool trial = alpha >= 0.0 || alpha_dev;
    const double a = alpha >= 0.0 ? alpha : 0.0;
    if (v.has_collider) {
        // The contact passes read only q and its FP32 copy: once k_positions
        // has written them, the passes run on a second stream beside the node
        // and element kernels (on one stream while kernels are timed one by
        // one).  The same kernels see the same inputs either way.
        I.launch("k_positions", k_positions, grid_for(v.N), kBlock, v, trial ? 1 : 0, a, alpha_dev);
        const bool side = !I.profiling;
        const cudaStream_t cs = side ? I.side : I.stream;
        if (side) {
            KHS_CUDA(cudaEventRecord(I.fork, I.stream));
            I.wait_for(I.side, I.fork);
        }
        const double *q = v.q;
        if (rebuild_cache_) KHS_CUDA(cudaMemsetAsync(&v.sc->pool_used, 0, sizeof(v.sc->pool_used), cs));
        I.launch_on(cs, rebuild_cache_ ? "k_contact_filter_rebuild" : trial ? "k_contact_filter_trial" : "k_contact_filter",
                    k_contact_filter, grid_for(v.E), kBlock, v, q, rebuild_cache_ ? 1 : 0);
        I.launch_on(cs, "k_contact_near", mode_ ? k_contact_near<true> : k_contact_near<false>, near_grid(v.E), kBlock, v);
        I.launch_on(cs, "k_contact_exact", k_contact_exact, kPairGrid, kPairBlock, v, q);
        I.launch_on(cs, "k_contact_select", mode_ ? k_contact_select<true> : k_contact_select<false>,
                    grid_for(v.E, kSelectBlock), kSelectBlock, v, q, gradient ? 1 : 0);
        if (side) KHS_CUDA(cudaEventRecord(I.join, I.side));
    }
    I.launch(gradient ? "k_node_eval_grad" : "k_node_eval_energy", k_node_eval, grid_for(v.N, kEvalBlock), kEvalBlock, v,
             gradient ? 1 : 0, trial ? 1 : 0, a, dt, alpha_dev, v.has_collider);
    rebuild_cache_ = false;
    // Brought up early, the element kernel's blocks would take the registers that
    // the contact passes need (1,000 strands: 186.5 ms a frame, so 181.1).
    if (v.has_collider) I.ordinary = I.stream;
    if (gradient && v.E <= kEndElements * 2 * I.sms) I.launch("k_elem_eval_grad", k_elem_ends, grid_for(v.E, kEndElements), kEndBlock, v);
    else I.launch(gradient ? "k_elem_eval_grad" : "k_elem_eval_energy", k_elem_eval, grid_for(v.E, kEvalBlock), kEvalBlock, v, gradient ? 1 : 0);
    if (v.has_collider && !I.profiling) I.wait_for(I.stream, I.join);
    if (gradient) I.launch("k_node_sum", k_node_sum, grid_for(21 * size_t(v.N)), kBlock, v);
    I.launch("k_reduce_eval", k_reduce_eval, kPartials, kBlock, v, gradient ? 1 : 0);
    I.check();
    I.sync();
    const Mailbox &mb = *I.mail_host;
    EvalStats s;
    s.objective = mb.objective; s.elastic = mb.elastic; s.contact = mb.contact; s.kinetic = mb.kinetic;
    s.minimum_gap = mb.minimum_gap; s.grad_norm2 = mb.grad_norm2; s.candidates = mb.candidates; s.active = mb.active;
    s.feasible = mb.feasible;
    return s;
}

bool Engine::limit_direction(double max_translation)
{
    Impl &I = *d_;
    if (max_translation > trust_radius_) {
        I.launch("k_scale", k_scale, grid_for(6 * size_t(I.v.N)), kBlock, I.v, trust_radius_ / max_translation);
        return true;
    }
    return false;
}

bool Engine::make_steepest()
{
    Impl &I = *d_;
    I.launch("k_precond", k_precond, grid_for(I.v.N), kBlock, I.v, last_dt_);
    I.launch("k_steepest", k_steepest, grid_for(6 * size_t(I.v.N)), kBlock, I.v);
    I.launch("k_reduce_dir", k_reduce_dir, kPartials, kBlock, I.v);
    I.check();
    I.sync();
    return limit_direction(I.mail_host->max_translation);
}

// Work items of the FP64 block solve: the `alone` longest strands on a warp
// each, the rest five to a warp, longest expected time first; by rule, or
// every strand on a team of three warps.  None of it changes the result
// (khs_block_solve.cuh).
//
// The rule's model, in cycles measured on GB300 (160-node strands on random
// blocks): a node of a strand alone takes 4,950 with one warp on a
// sub-partition and 6,400 beside a second one; a node of five strands 14,700
// and 20,200; the machine is full at two warps on each of its 608
// sub-partitions, where a node of either kind costs 3,200 and 2,020 of a
// sub-partition's time.  The expected time of a split is its longest chain
// or, if larger, the total work plus half of the shortest item (the uneven
// end of the queue).  Against a sweep of the split on GB300 it picks the best
// or is within 4% of it: 100 strands of 16-160 nodes all alone (384 us a
// solve, all by fives 992); 2,000 all alone (491, 1,159); the body scene's
// 6,757 strands of 8-200 nodes with a quarter alone (575, all alone 654, all
// by fives 1,650; 831 with the timed shapes this replaces).
//
// Teams are taken while the work on one warp a strand is at most 1.1 times
// the longest chain, us a solve against a warp each: the body scene with 700 of
// its strands 376 and 458, with 3,000 476 and 530 (work 0.6 of the chain);
// 1,000 strands of 20-120 nodes 291 and 343, of 16-160 nodes 380 and 457, 1,800
// of these 467 and 490 (1.05); against the best split beyond the line, 2,200
// of 16-160 nodes 513 and 495 (1.3), 2,000 of 8-24 nodes 84 and 87 (1.4), 4,000
// 162 and 161 (2.8), all of the body scene 674 and 568 (1.4).
void Engine::plan_block_solve(uint32_t alone, uint32_t blocks_per_sm)
{
    Impl &I = *d_;
    const std::vector<uint32_t> &len = I.sorted_len;
    const uint32_t S = uint32_t(len.size());
    int sms = 0;
    KHS_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, kDevice));
    I.sms = uint32_t(sms);
    constexpr double kAlone[2] = {4950.0, 6400.0}, kFive[2] = {14700.0, 20200.0}, kAloneWork = 3200.0, kFiveWork = 2020.0;
    I.solve_team = false;
    if (alone == kSolveByRule) {
        std::vector<double> sum(S + 1, 0.0);
        for (uint32_t k = 0; k < S; ++k) sum[k + 1] = sum[k] + len[k];
        const double parts = 4.0 * sms;
        I.solve_team = S && sum[S] * kAloneWork <= 1.1 * parts * len[0] * kAlone[0];
        double best = std::numeric_limits<double>::infinity();
        for (uint32_t step = 0; step <= 20; ++step) {
            const uint32_t w = uint32_t(uint64_t(S) * step / 20);
            const double items = w + (S - w + kStrandsPerWarp - 1) / kStrandsPerWarp;
            const double crowd = std::min(1.0, std::max(0.0, items / parts - 1.0));
            auto node = [&](const double cost[2]) { return cost[0] + crowd * (cost[1] - cost[0]); };
            double chain = 0.0, shortest = std::numeric_limits<double>::infinity();
            if (w) { chain = len[0] * node(kAlone); shortest = len[w - 1] * kAlone[1]; }
            if (w < S) {
                chain = std::max(chain, len[w] * node(kFive));
                shortest = std::min(shortest, len[w + (S - w - 1) / kStrandsPerWarp * kStrandsPerWarp] * kFive[1]);
            }
            const double work = (sum[w] * kAloneWork + (sum[S] - sum[w]) * kFiveWork) / parts;
            const double time = std::max(chain, items > 2.0 * parts ? work + 0.5 * shortest : 0.0);
            if (time <= best) { best = time; alone = w; }
        }
    }
    struct Item { double cost; uint32_t code; };
    std::vector<Item> items;
    for (uint32_t k = 0; k < alone; ++k) items.push_back({len[k] * kAlone[1], k | kSolveAlone});
    for (uint32_t k = alone; k < S; k += kStrandsPerWarp) items.push_back({len[k] * kFive[1], k});
    std::stable_sort(items.begin(), items.end(), [](const Item &a, const Item &b) { return a.cost > b.cost; });
    std::vector<uint32_t> codes;
    for (const Item &i : items) codes.push_back(i.code);
    KHS_CUDA(cudaMemcpyAsync(const_cast<uint32_t *>(I.v.solve_items), codes.data(), codes.size() * 4, cudaMemcpyHostToDevice,
                             I.stream));
    I.sync();
    I.solve_items = unsigned(items.size());
    I.solve_blocks = std::min(I.solve_items, 4 * (blocks_per_sm ? blocks_per_sm : 2u) * unsigned(sms));
    const unsigned ff_groups = unsigned((S + kSolveGroupsPerWarp - 1) / kSolveGroupsPerWarp);
    I.ff_blocks = std::min(std::max(1u, (ff_groups + 3) / 4), 2u * unsigned(sms));
}

// 5: the long_strands longest on a warp each, the rest five to a warp; 2 and
// 1: every strand on a warp of its own, or with long_strands as 5 does.
KhsResult Engine::set_block_solve_schedule(uint32_t strands_per_warp, uint32_t blocks_per_sm, uint32_t long_strands)
{
    const uint32_t S = d_->v.S;
    if (strands_per_warp == 0) {
        plan_block_solve(kSolveByRule, 0);
        return KHS_OK;
    }
    if ((strands_per_warp != 5 && strands_per_warp != 2 && strands_per_warp != 1) || blocks_per_sm < 1 || blocks_per_sm > 8 ||
        (long_strands && ((strands_per_warp != 5 && strands_per_warp != 1) || long_strands >= S)))
        return KHS_ERROR_INVALID_ARGUMENT;
    plan_block_solve(strands_per_warp == 5 || long_strands ? long_strands : S, blocks_per_sm);
    return KHS_OK;
}

// The quads + singles + doubles longest strands on a warp each, the rest five
// to a warp.
KhsResult Engine::set_block_solve_tiers(uint32_t quads, uint32_t singles, uint32_t doubles, uint32_t blocks_per_sm)
{
    if (blocks_per_sm < 1 || blocks_per_sm > 8 || uint64_t(quads) + singles + doubles > d_->v.S)
        return KHS_ERROR_INVALID_ARGUMENT;
    plan_block_solve(quads + singles + doubles, blocks_per_sm);
    return KHS_OK;
}

void Engine::launch_block_solve()
{
    Impl &I = *d_;
    if (I.solve_team) I.launch("k_block_solve", k_block_solve_team, I.v.S, kTeam, I.v);
    else I.launch("k_block_solve", k_block_solve, I.solve_blocks, 32, I.v, uint32_t(I.solve_items));
}

bool Engine::make_direction(KhsxSubstepRecord &rec, double grad_norm2)
{
    Impl &I = *d_;
    (void)grad_norm2;
    const Mailbox &mb = *I.mail_host;
    bool fp64 = mode_ != KHSX_MODE_MIXED_FF;
    if (!fp64) {
        I.launch("k_ff_factor", k_ff_factor, I.ff_blocks, 128, I.v);
        uint32_t sweeps = 0;
        for (;;) {
            I.launch("k_ff_residual", k_ff_residual, grid_for(6 * size_t(I.v.N)), kBlock, I.v);
            I.launch("k_ff_correct", k_ff_correct, I.ff_blocks, 128, I.v);
            ++sweeps;
            I.launch("k_reduce_dir", k_reduce_dir, kPartials, kBlock, I.v);
            I.check();
            I.sync();
            if (mb.solve_failed) break;
            float ratio;
            std::memcpy(&ratio, &mb.refine_bits, sizeof(ratio));
            if (!(ratio > kRefineRatio) || sweeps >= uint32_t(kRefineSweepsMax)) break;
        }
        rec.refinement_sweeps += sweeps;
        if (mb.solve_failed) {
            ++rec.fp64_fallbacks;
            fp64 = true;
        }
    }
    if (fp64) {
        launch_block_solve();
        I.launch("k_reduce_dir", k_reduce_dir, kPartials, kBlock, I.v);
        I.check();
        I.sync();
    }
    const bool used = !mb.solve_failed && mb.slope < 0 && std::isfinite(mb.slope);
    if (!used) {
        ++rec.steepest_fallbacks;
        if (make_steepest()) ++rec.trust_scalings;
        return false;
    }
    if (limit_direction(mb.max_translation)) ++rec.trust_scalings;
    return true;
}

// The line-search CCD bound of the current direction.
void Engine::launch_ccd_bound()
{
    Impl &I = *d_;
    const View &v = I.v;
    I.launch("k_ccd_collect", mode_ ? k_ccd_collect<true> : k_ccd_collect<false>, grid_for(v.E), kBlock, v);
    I.launch("k_ccd_near", mode_ ? k_ccd_near<true> : k_ccd_near<false>, 152u * 8u, kBlock, v);
    I.launch("k_ccd_pairs", k_advance_pairs<false>, kPairGrid, kPairBlock, v);
}

KhsResult Engine::optimize_substep(double dt, KhsxSubstepRecord &rec)
{
    Impl &I = *d_;
    last_dt_ = dt;
    const View &v = I.v;
    EvalStats current = evaluate(true, dt, -1.0);
    if (!current.feasible) return fail(KHS_ERROR_NOT_CONVERGED, "state is outside the barrier feasible region");
    const double initial = std::sqrt(current.grad_norm2);
    step_stats_.initial_residual_norm = std::fmax(step_stats_.initial_residual_norm, initial);
    const double dof = 6.0 * double(v.N);
    for (uint32_t it = 0; it <= desc_.newton_iterations; ++it) {
        progress_iteration_.store(it);
        if (cancel_.load()) return fail(KHS_ERROR_INVALID_STATE, "solve cancelled");
        const double residual = std::sqrt(current.grad_norm2);
        const double relative = residual / std::fmax(initial, 1e-30);
        step_stats_.final_residual_norm = residual;
        step_stats_.relative_residual_norm = relative;
        step_stats_.minimum_gap = std::fmin(step_stats_.minimum_gap, current.minimum_gap);
        step_stats_.contact_candidate_count += current.candidates;
        step_stats_.active_contact_count += current.active;
        step_stats_.kinetic_energy = current.kinetic;
        step_stats_.elastic_energy = current.elastic;
        step_stats_.contact_energy = current.contact;
        step_stats_.friction_energy = 0.0;
        rec.final_residual_norm = residual;
        rec.minimum_gap = std::fmin(rec.minimum_gap, current.minimum_gap);
        rec.contact_candidates += current.candidates;
        rec.active_contacts += current.active;
        if (residual <= std::fmax(desc_.absolute_tolerance, 1.0e-5 * std::sqrt(dof)) ||
            relative <= std::fmax(desc_.relative_tolerance, 1.0e-4)) {
            I.launch("k_update_velocity", k_update_velocity, grid_for(v.N), kBlock, v, 1.0 / dt);
            return KHS_OK;
        }
        if (it == desc_.newton_iterations) break;
        progress_phase_.store(KHS_PHASE_LINEAR_SOLVE);
        // FP64 solve: the direction, its CCD bound and the first line-search
        // trial (at the step publish_ccd leaves in device memory) are enqueued
        // together, with one host synchronisation instead of three.  The
        // device runs the same kernels in the same order as step by step.
        // The trust-radius limit is applied on the device (k_limit, the host's
        // scale when it applies, else nothing).  When the direction is
        // not used as is (steepest fallback, CCD work-list overflow, step
        // below the minimum) the trial is discarded: the iterate is restored
        // and evaluated again, and the iteration goes on step by step.
        bool block_direction;
        bool pipelined = false;
        EvalStats first{};
        double first_alpha = 1.0, first_slope = 0.0;
        if (mode_ != KHSX_MODE_MIXED_FF) {
            launch_block_solve();
            I.launch("k_reduce_dir", k_reduce_dir, kPartials, kBlock, v);
            I.launch("k_limit", k_limit, kPartials, kBlock, v, trust_radius_, 0);
            if (v.has_collider) launch_ccd_bound();
            first = evaluate(true, dt, -1.0, &v.sc->trial_alpha);
            const Mailbox &mb = *I.mail_host;
            const bool used = !mb.dir_solve_failed && mb.dir_slope < 0 && std::isfinite(mb.dir_slope);
            const double max_translation = mb.dir_max_translation;
            first_slope = mb.slope;  // of the (possibly limited) direction, from the CCD pass
            if (v.has_collider) {
                unsigned long long bits = mb.ccd_bits;
                double lim;
                std::memcpy(&lim, &bits, sizeof(lim));
                first_alpha = lim;
                if (first_alpha < 1.0) first_alpha *= 0.9;
            }
            const bool overflow = v.has_collider && mb.pair_count > v.pair_capacity;
            // The direction was limited to the trust radius on the device.
            const bool scaled = max_translation > trust_radius_;
            pipelined = used && !overflow && first_alpha >= desc_.minimum_line_search_step;
            block_direction = used;
            if (used && scaled) ++rec.trust_scalings;
            if (!pipelined) {
                KHS_CUDA(cudaMemcpyAsync(v.q, v.q_base, 6 * size_t(v.N) * 8, cudaMemcpyDeviceToDevice, I.stream));
                evaluate(true, dt, -1.0);
                if (!used) {
                    ++rec.steepest_fallbacks;
                    if (make_steepest()) ++rec.trust_scalings;
                }
            }
        } else {
            block_direction = make_direction(rec, current.grad_norm2);
            KHS_CUDA(cudaMemcpyAsync(v.q_base, v.q, 6 * size_t(v.N) * 8, cudaMemcpyDeviceToDevice, I.stream));
        }
        ++step_stats_.linear_solves;
        bool accepted = false;
        // The first trial of the Gauss-Newton direction also evaluates the
        // gradient, the Hessian blocks and the rotation Jacobians (its
        // energy is computed by the same operations as an energy-only
        // evaluation).  When it is accepted -- most iterations -- that
        // evaluation is the next iterate's, and the separate evaluation at
        // the accepted state is skipped: same values, one evaluation fewer.
        bool graded_trial = false;     // a trial evaluated the gradient at its own state
        bool accepted_graded = false;  // ... and it was the accepted one
        EvalStats graded{};
        double alpha = 1.0;
        for (int attempt = 0; attempt < 2; ++attempt) {
            const bool reuse = pipelined && attempt == 0;  // bound and first trial already evaluated
            double slope;
            if (reuse) {
                slope = first_slope;
                alpha = first_alpha;
            } else {
                // Slope of the (possibly scaled) direction, and the CCD bound.
                I.launch("k_limit", k_limit, kPartials, kBlock, v, std::numeric_limits<double>::infinity(), 1);
                if (v.has_collider) {
                    progress_phase_.store(KHS_PHASE_CCD);
                    launch_ccd_bound();
                }
                I.check();
                I.sync();
                if (v.has_collider && I.mail_host->pair_count > v.pair_capacity) {
                    // Work list overflow: redo the bound with the per-element kernel.
                    I.launch("k_ccd", mode_ ? k_ccd<true> : k_ccd<false>, grid_for(v.E), kBlock, v);
                    I.launch("k_publish_ccd", k_publish_ccd, 1, 1, v);
                    I.check();
                    I.sync();
                }
                slope = I.mail_host->slope;
                alpha = 1.0;
                if (v.has_collider) {
                    unsigned long long bits = I.mail_host->ccd_bits;
                    double lim;
                    std::memcpy(&lim, &bits, sizeof(lim));
                    alpha = lim;
                    if (alpha < 1.0) alpha *= 0.9;
                }
            }
            if (v.has_collider) step_stats_.ccd_step_limit = std::fmin(step_stats_.ccd_step_limit, alpha);
            accepted = false;
            progress_phase_.store(KHS_PHASE_LINE_SEARCH);
            if (alpha >= desc_.minimum_line_search_step)
                for (uint32_t s = 0; s < desc_.line_search_iterations; ++s) {
                    const bool with_gradient = attempt == 0 && s == 0;
                    const EvalStats trial = reuse && s == 0 ? first : evaluate(with_gradient, dt, alpha);
                    graded_trial = graded_trial || with_gradient;
                    ++step_stats_.line_search_evaluations;
                    ++rec.line_search_evaluations;
                    if (trial.feasible && std::isfinite(trial.objective) &&
                        trial.objective <= current.objective + 1e-4 * alpha * slope) {
                        accepted = true;
                        accepted_graded = with_gradient;
                        if (with_gradient) graded = trial;
                        break;
                    }
                    alpha *= 0.5;
                    if (alpha < desc_.minimum_line_search_step) break;
                }
            if (accepted) break;
            if (!block_direction) break;
            KHS_CUDA(cudaMemcpyAsync(v.q, v.q_base, 6 * size_t(v.N) * 8, cudaMemcpyDeviceToDevice, I.stream));
            // The trials left their own gradient, blocks, rotations and FP32
            // positions behind; the steepest direction (gradient) and the
            // mixed form's CCD filter (FP32 positions) need the iterate's.
            if (graded_trial) evaluate(true, dt, -1.0);
            ++rec.steepest_fallbacks;
            if (make_steepest()) ++rec.trust_scalings;
            block_direction = false;
        }
        if (!accepted) {
            KHS_CUDA(cudaMemcpyAsync(v.q, v.q_base, 6 * size_t(v.N) * 8, cudaMemcpyDeviceToDevice, I.stream));
            I.sync();
            return fail(KHS_ERROR_NOT_CONVERGED, "Gauss-Newton line search failed");
        }
        current = accepted_graded ? graded : evaluate(true, dt, -1.0);
        const double dnorm = std::sqrt(I.mail_host->dir_norm2);
        step_stats_.increment_norm = alpha * dnorm;
        step_stats_.accepted_step_length = alpha;
        ++step_stats_.newton_iterations;
        ++rec.newton_iterations;
        progress_phase_.store(KHS_PHASE_ASSEMBLING);
        if (step_stats_.increment_norm / std::sqrt(dof) <= 2.0 * desc_.increment_tolerance) {
            I.launch("k_update_velocity", k_update_velocity, grid_for(v.N), kBlock, v, 1.0 / dt);
            return KHS_OK;
        }
    }
    I.launch("k_update_velocity", k_update_velocity, grid_for(v.N), kBlock, v, 1.0 / dt);
    return KHS_OK;
}

KhsResult Engine::run_frame(double frame_dt, const double *root_a, const double *rot_a, const double *root_b,
                            const double *rot_b, const double *col_a, const double *col_b, uint32_t frame,
                            uint32_t frame_count)
{
    Impl &I = *d_;
    View &v = I.v;
    if (!(frame_dt > 0 && std::isfinite(frame_dt))) return fail(KHS_ERROR_INVALID_ARGUMENT, "invalid time step");
    cancel_.store(false);
    clear_failure();
    frame_clock_ = std::chrono::steady_clock::now();
    progress_frame_.store(frame); progress_frame_count_.store(frame_count); progress_iteration_.store(0);
    const size_t q_bytes = 6 * size_t(v.N) * 8, c_bytes = 3 * size_t(v.V) * 8;
    KHS_CUDA(cudaEventRecord(I.ev_begin, I.stream));
    KHS_CUDA(cudaMemcpyAsync(I.q_snap, v.q, q_bytes, cudaMemcpyDeviceToDevice, I.stream));
    KHS_CUDA(cudaMemcpyAsync(I.v_snap, v.v, q_bytes, cudaMemcpyDeviceToDevice, I.stream));
    // Keep the frame's start collider: for khsStep it aliases the
    // frame-start buffer that is rewritten on success.
    if (v.V) {
        KHS_CUDA(cudaMemcpyAsync(I.col_a_copy, col_a, c_bytes, cudaMemcpyDeviceToDevice, I.stream));
        if (col_a != I.col_frame_start)
            KHS_CUDA(cudaMemcpyAsync(I.col_frame_start, col_a, c_bytes, cudaMemcpyDeviceToDevice, I.stream));
    }
    uint32_t substeps = desc_.substeps;
    const uint32_t maximum = v.has_collider ? desc_.maximum_substeps : desc_.substeps;
    uint32_t attempts = 0;
    for (;;) {
        ++attempts;
        KHS_CUDA(cudaMemcpyAsync(v.q, I.q_snap, q_bytes, cudaMemcpyDeviceToDevice, I.stream));
        KHS_CUDA(cudaMemcpyAsync(v.v, I.v_snap, q_bytes, cudaMemcpyDeviceToDevice, I.stream));
        clear_failure();
        error_.clear();
        records_.clear();
        progress_phase_.store(KHS_PHASE_ASSEMBLING);
        progress_substep_count_.store(substeps);
        progress_iteration_.store(0);
        step_stats_ = {};
        step_stats_.struct_size = sizeof(step_stats_);
        step_stats_.substeps = substeps;
        step_stats_.minimum_gap = std::numeric_limits<double>::infinity();
        step_stats_.ccd_step_limit = 1.0;
        if (v.V) KHS_CUDA(cudaMemcpyAsync(v.col_cur, I.col_a_copy, c_bytes, cudaMemcpyDeviceToDevice, I.stream));
        const double dt = frame_dt / substeps;
        bool crossed = false;
        KhsResult result = KHS_OK;
        for (uint32_t sub = 1; sub <= substeps; ++sub) {
            if (substep_limit_ && sub > substep_limit_) break;
            progress_substep_.store(sub);
            progress_iteration_.store(0);
            KhsxSubstepRecord rec{};
            rec.struct_size = sizeof(rec);
            rec.substep = sub;
            rec.minimum_gap = std::numeric_limits<double>::infinity();
            const double f = double(sub) / substeps;
            const SubstepTargets targets{root_a, rot_a, root_b, rot_b, I.col_a_copy, col_b, f, dt};
            I.launch("k_begin_substep", k_begin_substep, grid_for(std::max(v.N, v.has_collider ? v.V : 0u)), kBlock, v, targets);
            if (v.has_collider) {
                I.launch("k_refit", k_refit, grid_for(size_t(kLeafTriangles) * v.L), kBlock, v);
                View vs = v;  // walks the swept tree
                vs.bnode = v.swept_node; vs.blo = v.swept_lo; vs.bhi = v.swept_hi;
                progress_phase_.store(KHS_PHASE_CCD);
                KHS_CUDA(cudaMemsetAsync(&v.sc->pool_used, 0, sizeof(v.sc->pool_used), I.stream));
                I.launch("k_sweep_collect", k_sweep_collect, grid_for(v.E), kBlock, vs);
                I.launch("k_sweep_near", mode_ ? k_sweep_near<true> : k_sweep_near<false>, 152u * 8u, kBlock, vs);
                I.launch("k_sweep_pairs", k_advance_pairs<true>, kPairGrid, kPairBlock, vs);
                I.launch("k_sweep_record", k_sweep_record, 1, 1, vs);
                I.check();
                I.sync();
                if (I.mail_host->pair_count > v.pair_capacity) {
                    // Pair list overflow: every element by one thread.
                    I.launch("k_sweep", k_sweep, grid_for(v.E), kBlock, vs);
                    I.launch("k_sweep_record", k_sweep_record, 1, 1, vs);
                    I.check();
                    I.sync();
                }
                if (I.mail_host->sweep_fail != kNone) {
                    const SweepRecord &sr = *I.sweep_host;
                    set_failure_context(KHS_FAILURE_MOVING_COLLIDER_SWEEP, frame, sub, substeps, maximum, attempts);
                    if (sr.claimed) {
                        failure_.strand_index = sr.strand; failure_.element_index = sr.element;
                        failure_.collider_triangle_index = sr.triangle;
                        failure_.distance = sr.distance; failure_.required_distance = sr.required;
                        failure_.clearance = sr.clearance; failure_.collider_substep_displacement = sr.displacement;
                        failure_.collider_frame_displacement = sr.displacement * substeps;
                        failure_.hair_start = {sr.hair_start[0], sr.hair_start[1], sr.hair_start[2]};
                        failure_.hair_end = {sr.hair_end[0], sr.hair_end[1], sr.hair_end[2]};
                        failure_.collider_point = {sr.collider_point[0], sr.collider_point[1], sr.collider_point[2]};
                    }
                    crossed = true;
                    break;
                }
                rebuild_cache_ = true;
            }
            progress_phase_.store(KHS_PHASE_ASSEMBLING);
            result = optimize_substep(dt, rec);
            records_.push_back(rec);
            if (result != KHS_OK) {
                if (!cancel_.load()) {
                    const uint32_t kind = error_.find("outside the barrier") != std::string::npos ? KHS_FAILURE_BARRIER_INFEASIBLE
                                                                                                   : KHS_FAILURE_NONLINEAR_SOLVE;
                    set_failure_context(kind, frame, sub, substeps, maximum, attempts);
                }
                break;
            }
            if (v.has_collider && material_.friction > 0.0) {
                I.launch("k_friction_collect", k_friction_collect, grid_for(v.E), kBlock, v);
                I.launch("k_contact_near", mode_ ? k_contact_near<true> : k_contact_near<false>, near_grid(v.E), kBlock, v);
                I.launch("k_contact_exact", k_contact_exact, kPairGrid, kPairBlock, v, v.q);
                I.launch("k_friction", mode_ ? k_friction<true> : k_friction<false>, grid_for(v.E), kBlock, v, dt);
                I.launch("k_friction_apply", k_friction_apply, grid_for(v.N), kBlock, v);
            }
            ++step_stats_.converged_substeps;
        }
        if (!crossed && result == KHS_OK) break;
        KHS_CUDA(cudaMemcpyAsync(v.q, I.q_snap, q_bytes, cudaMemcpyDeviceToDevice, I.stream));
        KHS_CUDA(cudaMemcpyAsync(v.v, I.v_snap, q_bytes, cudaMemcpyDeviceToDevice, I.stream));
        I.sync();
        if (cancel_.load()) return result;
        if (substeps >= maximum) {
            if (crossed) return fail(KHS_ERROR_NOT_CONVERGED, "animated collider crossed hair after adaptive substepping");
            return result;
        }
        substeps = std::min(maximum, substeps * 2);
    }
    if (!animation_ready_) {
        KHS_CUDA(cudaMemcpyAsync(I.root_cur_x, I.root_pend_x, 3 * size_t(v.N) * 8, cudaMemcpyDeviceToDevice, I.stream));
        KHS_CUDA(cudaMemcpyAsync(I.root_cur_r, I.root_pend_r, 3 * size_t(v.N) * 8, cudaMemcpyDeviceToDevice, I.stream));
        if (v.V) KHS_CUDA(cudaMemcpyAsync(I.col_frame_start, I.col_pending, c_bytes, cudaMemcpyDeviceToDevice, I.stream));
    }
    clear_failure();
    step_stats_.phase = KHS_PHASE_FINISHED;
    progress_phase_.store(KHS_PHASE_FINISHED);
    KHS_CUDA(cudaEventRecord(I.ev_end, I.stream));
    KHS_CUDA(cudaEventSynchronize(I.ev_end));
    float ms = 0;
    KHS_CUDA(cudaEventElapsedTime(&ms, I.ev_begin, I.ev_end));
    gpu_stats_.last_frame_milliseconds = ms;
    error_.clear();
    return KHS_OK;
}

KhsResult Engine::step(double frame_dt)
{
    Impl &I = *d_;
    return run_frame(frame_dt, I.root_cur_x, I.root_cur_r, I.root_pend_x, I.root_pend_r, I.col_frame_start, I.col_pending, 0, 0);
}

KhsResult Engine::step_animation_frame(uint32_t frame, double frame_dt)
{
    Impl &I = *d_;
    if (!animation_ready_ || frame >= animation_frames_) return fail(KHS_ERROR_INVALID_ARGUMENT, "invalid animation frame index");
    if (frame == 0) {
        current_frame_ = 0;
        push_output(0);
        return KHS_OK;
    }
    if (frame != current_frame_ + 1) return fail(KHS_ERROR_INVALID_STATE, "animation frames must be stepped in order");
    const size_t N3 = 3 * size_t(I.v.N), V3 = 3 * size_t(I.v.V);
    const uint32_t a = frame - 1, b = frame;
    const KhsResult r = run_frame(frame_dt, I.anim_root_x + a * N3, I.anim_root_r + a * N3, I.anim_root_x + b * N3,
                                  I.anim_root_r + b * N3, I.v.V ? I.anim_col + a * V3 : nullptr,
                                  I.v.V ? I.anim_col + b * V3 : nullptr, frame, animation_frames_);
    if (r == KHS_OK) {
        current_frame_ = frame;
        push_ring(frame);
        push_output(frame);
    }
    return r;
}

void Engine::push_output(uint32_t frame)
{
    Impl &I = *d_;
    if (!I.out_dev || !I.original_count) return;
    const uint32_t k = I.out_next;
    I.out_next = uint32_t((k + 1) % I.out_frame.size());
    for (int64_t &held : I.out_frame)
        if (held == int64_t(frame)) held = -1;  // an older pass over this frame (before a rollback)
    const size_t per = 3 * size_t(I.original_count);
    double *dst = I.out_dev + k * per;
    // The slot's previous copy must have finished before the gather
    // overwrites it; an event never recorded does not wait.
    I.wait_for(I.stream, I.out_copied[k]);
    I.launch("k_gather", k_gather, grid_for(I.original_count), kBlock, I.v.q, I.mapping_dev, I.original_count, dst);
    KHS_CUDA(cudaEventRecord(I.out_gathered[k], I.stream));
    KHS_CUDA(cudaStreamWaitEvent(I.copy_stream, I.out_gathered[k], 0));
    KHS_CUDA(cudaMemcpyAsync(I.out_host + k * per, dst, per * 8, cudaMemcpyDeviceToHost, I.copy_stream));
    KHS_CUDA(cudaEventRecord(I.out_copied[k], I.copy_stream));
    I.out_frame[k] = int64_t(frame);
}

// Outputs of frames after `frame` belong to a trajectory that a rollback or
// a checkpoint restore has left.
void Engine::drop_outputs_after(uint32_t frame)
{
    for (int64_t &held : d_->out_frame)
        if (held > int64_t(frame)) held = -1;
}

KhsResult Engine::set_output_ring(uint32_t slots)
{
    Impl &I = *d_;
    if (slots > 1024) return fail(KHS_ERROR_INVALID_ARGUMENT, "output ring holds at most 1024 frames");
    I.sync();
    I.release_output();
    if (!slots) return KHS_OK;
    const size_t bytes = size_t(slots) * 3 * size_t(I.original_count) * 8;
    if (!I.copy_stream) KHS_CUDA(cudaStreamCreateWithFlags(&I.copy_stream, cudaStreamNonBlocking));
    if (cudaMalloc(reinterpret_cast<void **>(&I.out_dev), std::max<size_t>(bytes, 256)) != cudaSuccess ||
        cudaHostAlloc(reinterpret_cast<void **>(&I.out_host), std::max<size_t>(bytes, 256), cudaHostAllocDefault) != cudaSuccess) {
        cudaGetLastError();
        if (I.out_dev) cudaFree(I.out_dev);
        I.out_dev = I.out_host = nullptr;
        return fail(KHS_ERROR_OUT_OF_MEMORY, "cannot allocate the output ring");
    }
    I.out_bytes = bytes;
    I.resident += bytes;
    gpu_stats_.resident_bytes = I.resident;
    I.out_gathered.resize(slots);
    I.out_copied.resize(slots);
    for (uint32_t k = 0; k < slots; ++k) {
        KHS_CUDA(cudaEventCreateWithFlags(&I.out_gathered[k], cudaEventDisableTiming));
        KHS_CUDA(cudaEventCreateWithFlags(&I.out_copied[k], cudaEventDisableTiming));
    }
    I.out_frame.assign(slots, -1);
    I.out_next = 0;
    return KHS_OK;
}

KhsResult Engine::output_frame(uint32_t frame, KhsVec3 *out, uint32_t capacity, const KhsVec3 **view)
{
    Impl &I = *d_;
    if (!I.out_dev) return fail(KHS_ERROR_INVALID_STATE, "the output ring is off");
    size_t k = I.out_frame.size();
    for (size_t s = 0; s < I.out_frame.size(); ++s)
        if (I.out_frame[s] == int64_t(frame)) k = s;
    if (k == I.out_frame.size()) return fail(KHS_ERROR_INVALID_ARGUMENT, "the frame is not in the output ring");
    if (out && capacity < I.original_count) return fail(KHS_ERROR_INVALID_ARGUMENT, "output buffer smaller than the point count");
    KHS_CUDA(cudaEventSynchronize(I.out_copied[k]));
    const double *src = I.out_host + k * 3 * size_t(I.original_count);
    if (view) *view = reinterpret_cast<const KhsVec3 *>(src);
    if (out) std::memcpy(out, src, size_t(I.original_count) * 24);
    return KHS_OK;
}

void Engine::push_ring(uint32_t frame)
{
    Impl &I = *d_;
    if (!I.ring) return;
    const size_t slots = I.ring_frame.size(), qn = 6 * size_t(I.v.N);
    const size_t k = frame % slots;
    KHS_CUDA(cudaMemcpyAsync(I.ring + 2 * qn * k, I.v.q, qn * 8, cudaMemcpyDeviceToDevice, I.stream));
    KHS_CUDA(cudaMemcpyAsync(I.ring + 2 * qn * k + qn, I.v.v, qn * 8, cudaMemcpyDeviceToDevice, I.stream));
    I.ring_frame[k] = int64_t(frame);
}

KhsResult Engine::set_rollback_ring(uint32_t slots)
{
    Impl &I = *d_;
    if (slots > 1024) return fail(KHS_ERROR_INVALID_ARGUMENT, "rollback ring holds at most 1024 frames");
    I.sync();
    if (I.ring) { cudaFree(I.ring); I.ring = nullptr; I.resident -= I.ring_bytes; I.ring_bytes = 0; }
    I.ring_frame.clear();
    if (!slots) return KHS_OK;
    const size_t bytes = size_t(slots) * 2 * 6 * size_t(I.v.N) * 8;
    if (cudaMalloc(reinterpret_cast<void **>(&I.ring), bytes) != cudaSuccess) {
        I.ring = nullptr;
        cudaGetLastError();
        return fail(KHS_ERROR_OUT_OF_MEMORY, "cannot allocate the rollback ring");
    }
    I.ring_bytes = bytes;
    I.resident += bytes;
    I.ring_frame.assign(slots, -1);
    gpu_stats_.resident_bytes = I.resident;
    if (animation_ready_) push_ring(current_frame_);
    return KHS_OK;
}

KhsResult Engine::rollback_to_frame(uint32_t frame)
{
    Impl &I = *d_;
    if (!animation_ready_) return fail(KHS_ERROR_INVALID_STATE, "finalize the animation before rolling back");
    const size_t slots = I.ring_frame.size();
    if (!I.ring || !slots || I.ring_frame[frame % slots] != int64_t(frame))
        return fail(KHS_ERROR_INVALID_ARGUMENT, "frame is not held by the rollback ring");
    const size_t qn = 6 * size_t(I.v.N), k = frame % slots, qb = qn * 8;
    KHS_CUDA(cudaMemcpyAsync(I.v.q, I.ring + 2 * qn * k, qb, cudaMemcpyDeviceToDevice, I.stream));
    KHS_CUDA(cudaMemcpyAsync(I.v.v, I.ring + 2 * qn * k + qn, qb, cudaMemcpyDeviceToDevice, I.stream));
    KHS_CUDA(cudaMemcpyAsync(I.v.q_old, I.v.q, qb, cudaMemcpyDeviceToDevice, I.stream));
    KHS_CUDA(cudaMemcpyAsync(I.q_snap, I.v.q, qb, cudaMemcpyDeviceToDevice, I.stream));
    KHS_CUDA(cudaMemcpyAsync(I.v_snap, I.v.v, qb, cudaMemcpyDeviceToDevice, I.stream));
    I.sync();
    // Frames after the restored one are no longer on this trajectory.
    for (size_t j = 0; j < slots; ++j)
        if (I.ring_frame[j] > int64_t(frame)) I.ring_frame[j] = -1;
    drop_outputs_after(frame);
    current_frame_ = frame;
    cancel_.store(false);
    progress_frame_.store(frame);
    progress_substep_.store(0); progress_substep_count_.store(0); progress_iteration_.store(0);
    progress_phase_.store(KHS_PHASE_FINISHED);
    step_stats_ = {};
    step_stats_.struct_size = sizeof(step_stats_);
    step_stats_.phase = KHS_PHASE_FINISHED;
    clear_failure();
    error_.clear();
    return KHS_OK;
}

namespace {
struct CheckpointHeader {
    uint64_t magic;
    uint32_t abi_version;
    uint32_t animation_frame;
    uint64_t dof_count;
};
}  // namespace

uint64_t Engine::checkpoint_size() const
{
    if (!initialized_ || !animation_ready_) return 0;
    return sizeof(CheckpointHeader) + 2 * uint64_t(6) * d_->v.N * sizeof(double);
}

KhsResult Engine::save_checkpoint(void *data, uint64_t capacity)
{
    Impl &I = *d_;
    const uint64_t required = checkpoint_size();
    if (!data || !required || capacity < required) return fail(KHS_ERROR_INVALID_ARGUMENT, "invalid checkpoint output buffer");
    CheckpointHeader h{kCheckpointMagic, KHS_ABI_VERSION, current_frame_, uint64_t(6) * I.v.N};
    auto *out = static_cast<unsigned char *>(data);
    std::memcpy(out, &h, sizeof(h));
    const size_t qb = 6 * size_t(I.v.N) * 8;
    KHS_CUDA(cudaMemcpyAsync(out + sizeof(h), I.v.q, qb, cudaMemcpyDeviceToHost, I.stream));
    KHS_CUDA(cudaMemcpyAsync(out + sizeof(h) + qb, I.v.v, qb, cudaMemcpyDeviceToHost, I.stream));
    I.sync();
    error_.clear();
    return KHS_OK;
}

KhsResult Engine::restore_checkpoint(const void *data, uint64_t size)
{
    Impl &I = *d_;
    const uint64_t required = checkpoint_size();
    if (!data || !required || size != required) return fail(KHS_ERROR_INVALID_ARGUMENT, "invalid checkpoint size");
    CheckpointHeader h{};
    std::memcpy(&h, data, sizeof(h));
    if (h.magic != kCheckpointMagic || h.abi_version != KHS_ABI_VERSION || h.dof_count != uint64_t(6) * I.v.N ||
        h.animation_frame >= animation_frames_)
        return fail(KHS_ERROR_INVALID_ARGUMENT, "checkpoint does not match this solver");
    const auto *in = static_cast<const unsigned char *>(data);
    const size_t qb = 6 * size_t(I.v.N) * 8;
    KHS_CUDA(cudaMemcpyAsync(I.v.q, in + sizeof(h), qb, cudaMemcpyHostToDevice, I.stream));
    KHS_CUDA(cudaMemcpyAsync(I.v.v, in + sizeof(h) + qb, qb, cudaMemcpyHostToDevice, I.stream));
    KHS_CUDA(cudaMemcpyAsync(I.v.q_old, I.v.q, qb, cudaMemcpyDeviceToDevice, I.stream));
    KHS_CUDA(cudaMemcpyAsync(I.q_snap, I.v.q, qb, cudaMemcpyDeviceToDevice, I.stream));
    KHS_CUDA(cudaMemcpyAsync(I.v_snap, I.v.v, qb, cudaMemcpyDeviceToDevice, I.stream));
    // The rollback ring must describe the restored trajectory: frames after
    // the checkpoint's are forgotten, and the checkpoint's own frame is
    // replaced by the restored state (the slot may hold another trajectory).
    for (size_t j = 0; j < I.ring_frame.size(); ++j)
        if (I.ring_frame[j] > int64_t(h.animation_frame)) I.ring_frame[j] = -1;
    push_ring(h.animation_frame);
    I.sync();
    current_frame_ = h.animation_frame;
    drop_outputs_after(h.animation_frame);
    cancel_.store(false);
    progress_frame_.store(h.animation_frame);
    progress_substep_.store(0); progress_substep_count_.store(0); progress_iteration_.store(0);
    progress_phase_.store(KHS_PHASE_FINISHED);
    step_stats_ = {};
    step_stats_.struct_size = sizeof(step_stats_);
    step_stats_.phase = KHS_PHASE_FINISHED;
    clear_failure();
    error_.clear();
    return KHS_OK;
}

KhsResult Engine::copy_original_positions(KhsVec3 *out, uint32_t capacity) const
{
    Impl &I = *d_;
    if (!out || capacity < I.original_count) return KHS_ERROR_INVALID_ARGUMENT;
    if (!I.original_count) return KHS_OK;
    I.launch("k_gather", k_gather, grid_for(I.original_count), kBlock, I.v.q, I.mapping_dev, I.original_count, I.mapping_gather_out);
    KHS_CUDA(cudaGetLastError());
    KHS_CUDA(cudaMemcpyAsync(out, I.mapping_gather_out, size_t(I.original_count) * 24, cudaMemcpyDeviceToHost, I.stream));
    I.sync();
    return KHS_OK;
}

KhsResult Engine::copy_internal_positions(KhsVec3 *out, uint32_t capacity) const
{
    Impl &I = *d_;
    if (!out || capacity < I.v.N) return KHS_ERROR_INVALID_ARGUMENT;
    I.launch("k_gather", k_gather, grid_for(I.v.N), kBlock, I.v.q, nullptr, I.v.N, I.mapping_gather_out);
    KHS_CUDA(cudaGetLastError());
    KHS_CUDA(cudaMemcpyAsync(out, I.mapping_gather_out, size_t(I.v.N) * 24, cudaMemcpyDeviceToHost, I.stream));
    I.sync();
    return KHS_OK;
}

KhsResult Engine::copy_state(double *q, double *v, uint64_t capacity) const
{
    Impl &I = *d_;
    const size_t dof = 6 * size_t(I.v.N);
    if (capacity < dof) return KHS_ERROR_INVALID_ARGUMENT;
    if (q) KHS_CUDA(cudaMemcpyAsync(q, I.v.q, dof * 8, cudaMemcpyDeviceToHost, I.stream));
    if (v) KHS_CUDA(cudaMemcpyAsync(v, I.v.v, dof * 8, cudaMemcpyDeviceToHost, I.stream));
    I.sync();
    return KHS_OK;
}

KhsResult Engine::query_contacts(const double *q, uint64_t dof, KhsxContactRecord *out, uint32_t capacity)
{
    Impl &I = *d_;
    if (!q || dof < 6 * uint64_t(I.v.N) || !out || capacity < I.v.E) return KHS_ERROR_INVALID_ARGUMENT;
    KHS_CUDA(cudaMemcpyAsync(I.v.q_base, q, 6 * size_t(I.v.N) * 8, cudaMemcpyHostToDevice, I.stream));
    I.launch("k_contact_query", mode_ ? k_contact<true> : k_contact<false>, grid_for(I.v.E), kBlock, I.v,
             static_cast<const double *>(I.v.q_base));
    KHS_CUDA(cudaGetLastError());
    return copy_contact_records(out, capacity);
}

namespace {

constexpr int kMaxScratchDevices = 64;
std::mutex g_no_alloc_mutex;
void *g_no_alloc_ptr[kMaxScratchDevices] = {};

// Device address of g_no_alloc_scratch on device `device`, looked up once per
// device with that device current (the first call may load the module).
cudaError_t no_alloc_scratch(int device, void **ptr)
{
    if (device < 0 || device >= kMaxScratchDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(g_no_alloc_mutex);
    if (!g_no_alloc_ptr[device]) {
        int previous = 0;
        cudaError_t err = cudaGetDevice(&previous);
        if (err != cudaSuccess) return err;
        if (previous != device && (err = cudaSetDevice(device)) != cudaSuccess) return err;
        void *p = nullptr;
        err = cudaGetSymbolAddress(&p, g_no_alloc_scratch);
        if (previous != device) {
            const cudaError_t back = cudaSetDevice(previous);
            if (err == cudaSuccess) err = back;
        }
        if (err != cudaSuccess) return err;
        if (!p) return cudaErrorInvalidSymbol;
        g_no_alloc_ptr[device] = p;
    }
    *ptr = g_no_alloc_ptr[device];
    return cudaSuccess;
}

}  // namespace

KhsResult Engine::query_contacts_no_alloc(const double *q, uint64_t dof, KhsxContactRecord *out, uint32_t capacity)
{
    Impl &I = *d_;
    const View &v = I.v;
    if (!q || dof < 6 * uint64_t(v.N) || !out || capacity < v.E) return KHS_ERROR_INVALID_ARGUMENT;
    const uint64_t q_bytes = 6 * uint64_t(v.N) * sizeof(double);
    const uint64_t rec_offset = (q_bytes + 255) / 256 * 256;
    if (rec_offset + uint64_t(v.E) * sizeof(KhsxContactRecord) > KHSX_NO_ALLOC_SCRATCH_BYTES) return KHS_ERROR_INVALID_ARGUMENT;
    if (v.E == 0) return KHS_OK;
    void *base = nullptr;
    if (no_alloc_scratch(kDevice, &base) != cudaSuccess) return KHS_ERROR_INTERNAL;
    double *q_dev = static_cast<double *>(base);
    KhsxContactRecord *rec = reinterpret_cast<KhsxContactRecord *>(static_cast<unsigned char *>(base) + rec_offset);
    if (cudaMemcpyAsync(q_dev, q, q_bytes, cudaMemcpyHostToDevice, I.stream) != cudaSuccess) return KHS_ERROR_INTERNAL;
    if (mode_) k_contact_query_records<true><<<grid_for(v.E), kBlock, 0, I.stream>>>(v, q_dev, rec);
    else k_contact_query_records<false><<<grid_for(v.E), kBlock, 0, I.stream>>>(v, q_dev, rec);
    ++I.launches;
    if (cudaGetLastError() != cudaSuccess) return KHS_ERROR_INTERNAL;
    if (cudaMemcpyAsync(out, rec, size_t(v.E) * sizeof(KhsxContactRecord), cudaMemcpyDeviceToHost, I.stream) != cudaSuccess)
        return KHS_ERROR_INTERNAL;
    return cudaStreamSynchronize(I.stream) == cudaSuccess ? KHS_OK : KHS_ERROR_INTERNAL;
}

KhsResult Engine::copy_contact_records(KhsxContactRecord *out, uint32_t capacity) const
{
    Impl &I = *d_;
    const size_t E = I.v.E;
    if (!out || capacity < E) return KHS_ERROR_INVALID_ARGUMENT;
    std::vector<uint32_t> cand(E), tri(E);
    std::vector<uint8_t> flags(E);
    std::vector<double> gap(E);
    if (E) {
        KHS_CUDA(cudaMemcpyAsync(cand.data(), I.v.c_cand, E * 4, cudaMemcpyDeviceToHost, I.stream));
        KHS_CUDA(cudaMemcpyAsync(tri.data(), I.v.c_tri, E * 4, cudaMemcpyDeviceToHost, I.stream));
        KHS_CUDA(cudaMemcpyAsync(flags.data(), I.v.c_flags, E, cudaMemcpyDeviceToHost, I.stream));
        KHS_CUDA(cudaMemcpyAsync(gap.data(), I.v.c_gap, E * 8, cudaMemcpyDeviceToHost, I.stream));
        I.sync();
    }
    for (size_t e = 0; e < E; ++e) {
        const bool closest = flags[e] & kFlagClosest;
        out[e] = KhsxContactRecord{cand[e], closest ? tri[e] : kNone, (flags[e] & kFlagActive) ? 1u : 0u, 0u,
                                   closest ? gap[e] : std::numeric_limits<double>::infinity()};
    }
    return KHS_OK;
}

void Engine::set_profiling(bool on)
{
    Impl &I = *d_;
    I.sync();
    I.profiling = on;
}

std::vector<KernelTiming> Engine::kernel_timings() const
{
    Impl &I = *d_;
    I.sync();
    std::vector<KernelTiming> out;
    for (const auto &k : I.kstats) out.push_back({k.name, k.launches, k.ms});
    return out;
}

void Engine::reset_kernel_timings()
{
    Impl &I = *d_;
    I.sync();
    I.kstats.clear();
}

uint64_t Engine::kernel_launches() const { return d_->launches; }

bool query_device(KhsGpuInfo &info, std::string &error)
{
    std::memset(&info, 0, sizeof(info));
    info.struct_size = sizeof(info);
    int count = 0;
    const cudaError_t r = cudaGetDeviceCount(&count);
    if (r != cudaSuccess || count < 1) {
        error = r == cudaSuccess ? "no CUDA GPU found" : cudaGetErrorString(r);
        cudaGetLastError();
        return false;
    }
    cudaDeviceProp prop{};
    if (cudaGetDeviceProperties(&prop, 0) != cudaSuccess) { error = "cannot query the CUDA device"; return false; }
    info.available = 1;
    info.device_ordinal = 0;
    info.compute_capability_major = uint32_t(prop.major);
    info.compute_capability_minor = uint32_t(prop.minor);
    info.total_vram_bytes = prop.totalGlobalMem;
    std::strncpy(info.device_name, prop.name, sizeof(info.device_name) - 1);
    return true;
}

}  // namespace khs
