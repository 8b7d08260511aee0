/*
 * traverse.cuh -- device-side voxtrees searches over the pool of
 * pool_layout.h.
 *
 * Exactness.  Every float operation the reference performs is performed
 * here, in the same order, with the IEEE round-to-nearest intrinsics
 * (__fadd_rn, __fsub_rn, __fmul_rn, __fdiv_rn), which the compiler never
 * contracts into FMAs.  Comparisons keep the reference's NaN behaviour.  The
 * result is the reference's leaf, voxel and intersection point, bit for bit.
 *
 * Recursion becomes an explicit per-thread stack of pending tasks {record
 * offset, ray origin} (see trace_ray).  Over images of the SHAPE_* kinds below
 * rays and balls take cheaper searches with the same results (trace_mirrored,
 * trace_ball_nested); over any other image, and for the rays and boxes those
 * leave, the general ones run.
 *
 * Checked build (-DVOX_CUDA_CHECKED, libvoxtrees_cuda_checked.so): every
 * load from the tree image and the light tree first proves its index inside
 * the uploaded arrays; an index outside marks the tree's status word with
 * VOX_STATUS_RANGE and ends that search as an error instead of reading.  It
 * stands in for a memory checker on the search kernels; the normal build
 * relies on the upload-time validation of the image instead.
 */
#ifndef VOX_TRAVERSE_CUH
#define VOX_TRAVERSE_CUH

#include <cstdint>
#include <cuda_runtime.h>

#include "image_shape.h"
#include "pool_layout.h"
#include "../../include/voxtrees_cuda.h"

namespace vox {

struct DevTree {
    const uint4 *pool;
    const uint32_t *rec_of_id;   // pre-order id -> record offset
    uint32_t root;               // record offset of the root, VOXP_EMPTY if none
    uint32_t n_nodes;
    float vx, vy, vz;            // vox_voxel at upload time
    uint32_t max_steps;          // nodes + voxels: no search takes more loop steps
    uint32_t n_units;            // 16-byte units in the image (pool)
    uint32_t shape;              // SHAPE_* bits of the image (image_shape in voxtrees_cuda.cu)
    uint32_t *fault;             // the tree's status word (checked build only)
};

struct Counts {
    uint32_t nodes, inner, voxels;
};

// Status word bits: a search ran out of stack or steps; (checked build) an
// index outside the uploaded arrays.
constexpr uint32_t VOX_STATUS_STACK = 1u, VOX_STATUS_RANGE = 2u;

#ifdef VOX_CUDA_CHECKED
constexpr bool CHECKED = true;
#else
constexpr bool CHECKED = false;
#endif

// Units [at, at + span) lie in an array of n units; without the checked
// build always true (and compiled away).  Marks `fault` when not.
__device__ __forceinline__ bool in_range(uint64_t at, uint32_t span, uint64_t n, uint32_t *fault)
{
    if (!CHECKED) return true;
    if (at + span <= n) return true;
    if (fault) atomicOr(fault, VOX_STATUS_RANGE);
    return false;
}

__device__ __forceinline__ float ubf(uint32_t u) { return __uint_as_float(u); }

__device__ __forceinline__ uint4 ld16(const uint4 *p) { return __ldg(p); }

/* geom.c:13-31 + :69-99 (hit_box).  Returns the entry point of the ray into
 * the closed box [lo, hi] in r.  An axis on which the origin already lies
 * inside the slab yields a distance of +-0 or NaN in the reference, which can
 * never be the winning positive distance, so only clamped axes divide. */
__device__ __forceinline__ bool hit_box(float lx, float ly, float lz, float hx, float hy, float hz,
                                        float ox, float oy, float oz, float dx, float dy, float dz,
                                        float &rx, float &ry, float &rz)
{
    bool cx = true, cy = true, cz = true;
    rx = ox; ry = oy; rz = oz;
    if (ox < lx) rx = lx; else if (ox > hx) rx = hx; else cx = false;
    if (oy < ly) ry = ly; else if (oy > hy) ry = hy; else cy = false;
    if (oz < lz) rz = lz; else if (oz > hz) rz = hz; else cz = false;
    if (!(cx | cy | cz)) return true;

    int plane = -1;
    float maxd = -1.0f;
    if (cx) { float t = __fdiv_rn(__fsub_rn(rx, ox), dx); if (t > maxd) { plane = 0; maxd = t; } }
    if (cy) { float t = __fdiv_rn(__fsub_rn(ry, oy), dy); if (t > maxd) { plane = 1; maxd = t; } }
    if (cz) { float t = __fdiv_rn(__fsub_rn(rz, oz), dz); if (t > maxd) { plane = 2; maxd = t; } }
    if (maxd <= 0.0f) return false;

    if (plane != 0) {
        float t = __fadd_rn(ox, __fmul_rn(maxd, dx));
        if (t < lx || t > hx) return false;
        rx = t;
    }
    if (plane != 1) {
        float t = __fadd_rn(oy, __fmul_rn(maxd, dy));
        if (t < ly || t > hy) return false;
        ry = t;
    }
    if (plane != 2) {
        float t = __fadd_rn(oz, __fmul_rn(maxd, dz));
        if (t < lz || t > hz) return false;
        rz = t;
    }
    return true;
}

/* geom.c:125-131 vox_abs_metric: ((|dx| + |dy|) + |dz|). */
__device__ __forceinline__ float l1(float ax, float ay, float az, float bx, float by, float bz)
{
    return __fadd_rn(__fadd_rn(fabsf(__fsub_rn(ax, bx)), fabsf(__fsub_rn(ay, by))),
                     fabsf(__fsub_rn(az, bz)));
}

/* geom.c:101-123 hit_plane_within_box for axis p.  Every comparison is made
 * and combined, with no early exit: the answer is the reference's (its point
 * is used only when the answer is true), and the lanes of a warp take no
 * branch here.  Measured: per-frame BEST launches 15% faster than with the
 * reference's early returns, the persistent batch kernel 2.6%. */
__device__ __forceinline__ bool hit_plane(int p, float ox, float oy, float oz, float dx, float dy, float dz,
                                          float cp, float lx, float ly, float lz, float hx, float hy, float hz,
                                          float &rx, float &ry, float &rz)
{
    float op = p == 0 ? ox : (p == 1 ? oy : oz);
    float dp = p == 0 ? dx : (p == 1 ? dy : dz);
    float k = __fsub_rn(cp, op);
    bool ok = !(k == 0.0f || ((dp < 0.0f) != (k < 0.0f)));
    k = __fdiv_rn(k, dp);
    rx = __fadd_rn(ox, __fmul_rn(k, dx));
    ry = __fadd_rn(oy, __fmul_rn(k, dy));
    rz = __fadd_rn(oz, __fmul_rn(k, dz));
    // NaN coordinates pass, as the reference's `<` / `>` tests let them
    ok &= !(rx < lx) & !(rx > hx) & !(ry < ly) & !(ry > hy) & !(rz < lz) & !(rz > hz);
    return ok;
}

struct RayHit {
    float x, y, z;
    uint32_t leaf;    // pre-order id
    uint32_t slot;    // winning voxel, 0xFF for dense
    uint32_t rec;     // record offset of the leaf
};

/* vox_ray_tree_intersection (search.c:8-153) as a resumable search.
 *
 * RaySearch holds everything one search carries between loop iterations
 * except its stack of pending tasks, which the caller keeps beside it (a
 * separate local array, so the search state itself stays in registers), and
 * ray_step() runs one iteration.  Every iteration makes one 16..48-byte load
 * (a node record, or one voxel of the leaf being scanned) and one box test,
 * so the lanes of a warp stay in step whatever mix of nodes and voxels they
 * are on, and a lane whose search ended could start another between any
 * two iterations.  The box test of a node is
 * search.c:22-23; of a voxel, the leaf loop's test at :55.  When an inner
 * node's box is entered, its plane crossings (:105-148) are computed at once:
 * the children behind the crossings are pushed in visiting order and the
 * search continues in the entry octant (:86-97).  Computing the crossings
 * before the entry octant has been searched changes nothing: they depend only
 * on the node and the ray, and they are used only if that octant finds
 * nothing.  The first hit ends the search, as the first non-NULL return ends
 * the recursion.
 *
 * The stack holds pending tasks {record offset, ray origin}; it never needs
 * more than 3 entries per inner level, which the upload-time depth check
 * guarantees for CAP.  A search that would overflow it, or that takes more
 * iterations than the tree has nodes and voxels (a damaged pool), ends with
 * STEP_ERROR. */
enum : int { STEP_MORE = 0, STEP_HIT = 1, STEP_MISS = 2, STEP_ERROR = 3 };

struct RaySearch {
    int sp;                    // entries on the caller's stack
    uint32_t cur;              // node mode: record offset; voxel mode: first voxel
    float ox, oy, oz;          // origin of the next box test
    float dx, dy, dz;
    bool scan;                 // scanning the voxels of a leaf
    uint32_t vi, vn, vrec, vid;
    float best, bx, by, bz;
    int win;
    uint32_t steps;
};

__device__ __forceinline__ void ray_begin(RaySearch &s, uint32_t start, float ox, float oy, float oz,
                                          float dx, float dy, float dz)
{
    s.sp = 0;
    s.cur = start;
    s.ox = ox; s.oy = oy; s.oz = oz;
    s.dx = dx; s.dy = dy; s.dz = dz;
    s.scan = false;
    s.vi = 0; s.vn = 0; s.vrec = 0; s.vid = 0;
    s.best = 0.0f; s.bx = 0.0f; s.by = 0.0f; s.bz = 0.0f;
    s.win = -1;
    s.steps = 0;
}

/* search.c:105-148: the crossings of the ray (from the entry point e of an
 * inner node) with the node's three dividing planes that lie in its box,
 * sorted by L1 distance from e with the reference's selection sort
 * (:115-134, immediate swaps on '<'); each crossing flips one octant bit of
 * the entry octant `sub` (:137).  Pushes the crossing children so that they
 * pop in visiting order (NULL children are skipped: they return NULL at
 * once).  Returns false when the stack would overflow. */
template <int CAP>
__device__ __forceinline__ bool push_crossings(RaySearch &s, uint4 (&stack)[CAP], float ex, float ey, float ez,
                                               float lx, float ly, float lz, float hx, float hy, float hz,
                                               float cx, float cy, float cz, uint32_t sub, uint32_t mask,
                                               uint32_t link)
{
    const float dx = s.dx, dy = s.dy, dz = s.dz;
    float qx0, qy0, qz0, qx1, qy1, qz1, qx2, qy2, qz2;
    bool v0 = hit_plane(0, ex, ey, ez, dx, dy, dz, cx, lx, ly, lz, hx, hy, hz, qx0, qy0, qz0);
    bool v1 = hit_plane(1, ex, ey, ez, dx, dy, dz, cy, lx, ly, lz, hx, hy, hz, qx1, qy1, qz1);
    bool v2 = hit_plane(2, ex, ey, ez, dx, dy, dz, cz, lx, ly, lz, hx, hy, hz, qx2, qy2, qz2);
    int pc = (int)v0 + (int)v1 + (int)v2;
    // compacted slots a, b, c = first, second, third valid crossing
    float ax = v0 ? qx0 : (v1 ? qx1 : qx2);
    float ay = v0 ? qy0 : (v1 ? qy1 : qy2);
    float az = v0 ? qz0 : (v1 ? qz1 : qz2);
    int ai = v0 ? 0 : (v1 ? 1 : 2);
    bool ab1 = v0 && v1;
    float bxp = ab1 ? qx1 : qx2, byp = ab1 ? qy1 : qy2, bzp = ab1 ? qz1 : qz2;
    int bi = ab1 ? 1 : 2;
    float cxp = qx2, cyp = qy2, czp = qz2;
    int ci = 2;
    float ma = l1(ex, ey, ez, ax, ay, az);
    float mb = l1(ex, ey, ez, bxp, byp, bzp);
    float mc = l1(ex, ey, ez, cxp, cyp, czp);
    if (pc > 1 && mb < ma) {
        float t0 = ax; ax = bxp; bxp = t0; t0 = ay; ay = byp; byp = t0; t0 = az; az = bzp; bzp = t0;
        t0 = ma; ma = mb; mb = t0; int ti = ai; ai = bi; bi = ti;
    }
    if (pc > 2 && mc < ma) {
        float t0 = ax; ax = cxp; cxp = t0; t0 = ay; ay = cyp; cyp = t0; t0 = az; az = czp; czp = t0;
        t0 = ma; ma = mc; mc = t0; int ti = ai; ai = ci; ci = ti;
    }
    if (pc > 2 && mc < mb) {
        float t0 = bxp; bxp = cxp; cxp = t0; t0 = byp; byp = cyp; cyp = t0; t0 = bzp; bzp = czp; czp = t0;
        t0 = mb; mb = mc; mc = t0; int ti = bi; bi = ci; ci = ti;
    }
    uint32_t s1 = sub ^ (1u << ai), s2 = s1 ^ (1u << bi), s3 = s2 ^ (1u << ci);
    bool w1 = pc > 0 && ((mask >> s1) & 1u);
    bool w2 = pc > 1 && ((mask >> s2) & 1u);
    bool w3 = pc > 2 && ((mask >> s3) & 1u);
    int npush = (int)w1 + (int)w2 + (int)w3;
    if (s.sp + npush > CAP) return false;
    if (w3) stack[s.sp++] = make_uint4(link + VOXP_REC_UNITS * (uint32_t)__popc(mask & ((1u << s3) - 1u)),
                                       __float_as_uint(cxp), __float_as_uint(cyp), __float_as_uint(czp));
    if (w2) stack[s.sp++] = make_uint4(link + VOXP_REC_UNITS * (uint32_t)__popc(mask & ((1u << s2) - 1u)),
                                       __float_as_uint(bxp), __float_as_uint(byp), __float_as_uint(bzp));
    if (w1) stack[s.sp++] = make_uint4(link + VOXP_REC_UNITS * (uint32_t)__popc(mask & ((1u << s1) - 1u)),
                                       __float_as_uint(ax), __float_as_uint(ay), __float_as_uint(az));
    return true;
}

template <int CAP, bool COUNT>
__device__ __forceinline__ int ray_step(const DevTree &t, RaySearch &s, uint4 (&stack)[CAP], RayHit &hit,
                                        Counts &cnt)
{
    // Each node and each voxel is tested at most once per search, so more
    // steps than the tree holds means a damaged pool: stop with an error.
    if (++s.steps > t.max_steps) return STEP_ERROR;
    const uint4 *pool = t.pool;
    const float dx = s.dx, dy = s.dy, dz = s.dz;
    if (!in_range(s.scan ? (uint64_t)s.cur + s.vi : s.cur, s.scan ? 1u : VOXP_REC_UNITS, t.n_units, t.fault))
        return STEP_ERROR;
    uint4 u0 = ld16(pool + (s.scan ? s.cur + s.vi : s.cur));
    uint4 u1 = make_uint4(0u, 0u, 0u, 0u), u2 = make_uint4(0u, 0u, 0u, 0u);
    if (!s.scan) {
        u1 = ld16(pool + s.cur + 1);
        u2 = ld16(pool + s.cur + 2);
    }
    float lx = ubf(u0.x), ly = ubf(u0.y), lz = ubf(u0.z), hx, hy, hz;
    if (s.scan) {   // voxel box [dot, dot + vox_voxel] (search.c:53-54)
        hx = __fadd_rn(lx, t.vx); hy = __fadd_rn(ly, t.vy); hz = __fadd_rn(lz, t.vz);
        if (COUNT) cnt.voxels++;
    } else {
        hx = ubf(u0.w); hy = ubf(u1.x); hz = ubf(u1.y);
        if (COUNT) cnt.nodes++;
    }
    float ex, ey, ez;
    bool in = hit_box(lx, ly, lz, hx, hy, hz, s.ox, s.oy, s.oz, dx, dy, dz, ex, ey, ez);
    bool resume = false;

    if (s.scan) {
        // leaf loop body, search.c:55-78: nearest voxel by L1 distance from
        // the leaf's entry point, first one at distance 0 wins at once
        bool stop = false;
        if (in) {
            float dist = l1(s.ox, s.oy, s.oz, ex, ey, ez);
            if (dist == 0.0f) {
                s.bx = ex; s.by = ey; s.bz = ez; s.win = (int)s.vi; stop = true;
            } else if (dist < s.best) {
                s.best = dist; s.bx = ex; s.by = ey; s.bz = ez; s.win = (int)s.vi;
            }
        }
        s.vi++;
        if (stop || s.vi == s.vn) {
            if (s.win >= 0) {
                hit.x = s.bx; hit.y = s.by; hit.z = s.bz;
                hit.leaf = s.vid; hit.slot = (uint32_t)s.win; hit.rec = s.vrec;
                return STEP_HIT;
            }
            s.scan = false;
            resume = true;
        }
    } else if (!in) {
        resume = true;
    } else {
        uint32_t meta = u1.z, link = u1.w, kind = meta & 3u;
        if (kind == VOXP_KIND_DENSE) {                      // search.c:31-37
            hit.x = ex; hit.y = ey; hit.z = ez;
            hit.leaf = link; hit.slot = 0xFFu; hit.rec = s.cur;
            return STEP_HIT;
        }
        if (kind == VOXP_KIND_LEAF) {                       // search.c:39-50
            s.vn = meta >> 2;
            if (s.vn == 0) {
                resume = true;
            } else {
                s.scan = true; s.vrec = s.cur; s.vid = u2.x; s.cur = link; s.vi = 0;
                s.best = __int_as_float(0x7f800000); s.win = -1;
                s.ox = ex; s.oy = ey; s.oz = ez;
            }
        } else {                                            // inner node
            if (COUNT) cnt.inner++;
            float cx = ubf(u2.x), cy = ubf(u2.y), cz = ubf(u2.z);
            // geom.c:53-65 get_corrected_subspace_idx
            uint32_t sub = ((cx == ex) ? (dx < 0.0f) : (cx > ex))
                         | (((cy == ey) ? (dy < 0.0f) : (cy > ey)) << 1)
                         | (((cz == ez) ? (dz < 0.0f) : (cz > ez)) << 2);
            uint32_t mask = (meta >> 8) & 0xFFu;
            if (!push_crossings<CAP>(s, stack, ex, ey, ez, lx, ly, lz, hx, hy, hz, cx, cy, cz, sub, mask, link))
                return STEP_ERROR;
            if ((mask >> sub) & 1u) {                       // search.c:92-93
                s.cur = link + VOXP_REC_UNITS * (uint32_t)__popc(mask & ((1u << sub) - 1u));
                s.ox = ex; s.oy = ey; s.oz = ez;
            } else {
                resume = true;
            }
        }
    }
    if (resume) {
        if (s.sp == 0) return STEP_MISS;
        uint4 e = stack[--s.sp];
        s.cur = e.x;
        s.ox = ubf(e.y); s.oy = ubf(e.z); s.oz = ubf(e.w);
    }
    return STEP_MORE;
}

/* The same search for ordinary rays: mirrored coordinates.
 *
 * What bounds the search is instruction issue (no memory level is near its
 * limit), and most of the instructions were the IEEE divisions of the box
 * test and the plane crossings, the two-sided comparisons and the sort of the
 * crossings.  For a ray whose direction has no component near zero and whose
 * numbers are of ordinary size (mirror_ok), in a tree whose boxes are
 * ordered (SHAPE_ORDERED), the same results come from fewer operations:
 *
 *  - Every axis on which the ray goes backwards is negated, in the ray and in
 *    every box and centre as it is loaded (the near and far faces swap).
 *    Round-to-nearest arithmetic is symmetric under negation, so every
 *    number is the reference's up to that sign, and now all directions are
 *    positive: coordinates only grow along the ray.  A point the ray reaches
 *    from inside a box is never below the box's near faces (e + q*d with
 *    q, d > 0 rounds to at least e), so only the far faces need a comparison;
 *    a plane crossing lies ahead exactly when the centre is above the entry
 *    point; an origin beyond a far face fails the far comparison of the point
 *    tested anyway.
 *  - (near - o) / d is positive exactly on the axes the reference clamps
 *    forward, so the largest of the three quotients is its `maxd` and no
 *    clamping is made; equal quotients go to the first axis as there.
 *  - The quotients are Markstein's (IBM J. Res. Dev. 34, 1990): with y =
 *    RN(1/d), q0 = RN(a*y), r = fma(-d, q0, a) (exact), the quotient is
 *    RN(q0 + r*y) -- the correctly rounded a/d for every pair of significands
 *    (checked exhaustively against __fdiv_rn) while nothing leaves the normal
 *    range, which the bounds below ensure for every quotient.
 *  - Crossings that are not there count as infinitely far, and the order the
 *    reference's selection sort gives is read off three comparisons (ties
 *    included), each child stored at its own place on the stack.
 *
 *  - A zero on a negated axis is +0 once turned back (turned_back): a sum that
 *    cancels is +0 with the axis negated or not, and the other zeros there are
 *    faces and origins, of which none is -0 (image_shape.h, mirror_ok).
 *
 * A search that meets a quotient too small for the bounds reports STEP_AGAIN and
 * is made again by the general search below.
 *
 * Measured against the general search alone (256^3 noise tree; in brackets
 * with the packed arithmetic and the smaller changes since):
 * a 1080p orbit frame 80.6 -> 51.5 us back to back (52.4), ADAPTIVE 112 -> 74
 * us (75); 32 such frames in the batch kernel 1,995 -> 1,366 us (1,260); 24
 * mixed frames over four trees 1,203 -> 850 us (762); a near 4K FAST frame of
 * the 512^3 tree 1,496 -> 1,145 us (1,030); 4M incoherent rays 710 -> 569 us
 * (474). */
constexpr int STEP_AGAIN = 4;
constexpr float DIR_MIN = 2.384185791015625e-7f, DIR_MAX = 262144.0f;   // 2^-22, 2^18
// Every coordinate of such a search is a multiple of 2^-102: the image's numbers
// and the ray's origin are zero or at least SHAPE_LEAST = 2^-79, and so is every
// q*d that is added to one, as a search goes on only from quotients q of at
// least QUOT_MIN = 2^-57 (of a crossing that is known by its distance: a smaller
// q takes a point no more than 3 * 2 * q * DIR_MAX < DIST_MIN away, roundings
// included).  So a numerator a is zero or at least 2^-102, the quotient a/d at
// least 2^-120 and r above, a multiple of 2^(-102-47), exact: every quotient is
// right, those that lose a comparison too.  (With numerators unbounded below,
// searches over voxels of 2^-145 lost crossings by a wrong last bit.)  A smaller
// voxel than SHAPE_VOXEL would have many of its searches made again.
constexpr float QUOT_MIN = 6.938893903907228e-18f;     // 2^-57
constexpr float DIST_MIN = 1.4551915228366852e-11f;    // 2^-36

__device__ __forceinline__ float quot(float a, float d, float y)
{
    float q = __fmul_rn(a, y);
    return __fmaf_rn(__fmaf_rn(-d, q, a), y, q);
}

// Two floats in a register pair and their packed round-to-nearest arithmetic
// (one instruction for both; each half rounds as the scalar operation): the
// mirrored search does its x and y together.  The directions are held
// negated, since a difference can subtract a product and the remainder of a
// quotient wants -d.  A packed product that a packed sum takes is written as an
// fma with -0, which rounds alike: ptxas 13.0 joins mul.rn.f32x2 and
// sub.rn.f32x2 into one fma and rounds once (seen in results), and the -0 is
// computed so that it cannot see through it.  Measured beside the scalar form:
// 32 frames in the batch kernel 1,363 -> 1,309 us, the near 4K FAST frame 1,097
// -> 1,067 us, ADAPTIVE 80.8 -> 79.0 us.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pair(float a, float b)
{
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void halves(f32x2 v, float &a, float &b)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c)
{
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 quot2(f32x2 a, f32x2 nd, f32x2 y)   // nd = -d
{
    f32x2 q = mul2(a, y);
    return fma2(fma2(nd, q, a), y, q);
}

// -0 twice, where ptxas does not see what it holds: as an operand in constant
// memory it costs the batch kernel no registers (32 frames 1,324 -> 1,314 us, the
// mixed batch 815 -> 809); the other kernels do better with one computed per ray
// (near 4K FAST frame 1,056 against 1,063 us).
static __constant__ f32x2 c_mzero = 0x8000000080000000ull;

// Whether the mirrored search may make this search.
__device__ __forceinline__ bool mirror_ok(const DevTree &t, float ox, float oy, float oz, float dx, float dy, float dz)
{
    const float lo = fminf(fminf(fabsf(dx), fabsf(dy)), fabsf(dz)), hi = fmaxf(fmaxf(fabsf(dx), fabsf(dy)), fabsf(dz));
    const float o = fmaxf(fmaxf(fabsf(ox), fabsf(oy)), fabsf(oz));
    const auto bits = [](float v) { return 2u * __float_as_uint(v) - 1u; };   // of the magnitude; zero's are the largest
    const uint32_t least = min(min(bits(ox), bits(oy)), bits(oz));
    // (the sum is not finite where a NaN hid from the extremes)
    const uint32_t mzero = 0x80000000u;
    return (t.shape & SHAPE_ORDERED) && lo >= DIR_MIN && hi <= DIR_MAX && o <= SHAPE_LIMIT &&
           fabsf(dx + dy + dz) < 4e6f && fabsf(ox + oy + oz) < 4e18f && least >= 2u * __float_as_uint(SHAPE_LEAST) - 1u &&
           __float_as_uint(ox) != mzero && __float_as_uint(oy) != mzero && __float_as_uint(oz) != mzero;
}

// A coordinate of a hit turned back; a zero becomes +0 on a negated axis, here
// or, in the batch kernels (LATE), by late_zero after the search.  (There this
// form, as any other in the loop, takes 32 orbit frames from 1,255 to 1,287 us;
// after the search they take 1,257, but a 1080p frame of its own 58.9 instead
// of 58.0.  Searching again every ray that ended on such a zero made a frame
// from inside a tree about the origin, where crossings of the planes at zero
// cancel, 27.6 us instead of 9.4, a floor with its top at zero 257 instead of 134.)
template <bool LATE>
__device__ __forceinline__ float turned_back(bool negated, float v)
{
    if (LATE) return negated ? -v : v;
    return __fsub_rn(negated ? 0.0f : v, negated ? v : 0.0f);
}
// -0 to +0 where the direction is negative: adding +0 does, adding -0 changes nothing.
__device__ __forceinline__ float late_zero(float v, float d)
{
    return __fadd_rn(v, __uint_as_float(~__float_as_uint(d) & 0x80000000u));
}

template <int CAP, bool MZERO_CONST, bool LATE>
__device__ __forceinline__ int trace_mirrored(const DevTree &t, uint32_t start, float ox, float oy, float oz,
                                              float dx, float dy, float dz, uint4 (&stack)[CAP], RayHit &hit)
{
    const uint4 *pool = t.pool;
    const bool nx = dx < 0.0f, ny = dy < 0.0f, nz = dz < 0.0f;   // negated axes
    const uint32_t neg = (uint32_t)nx | ((uint32_t)ny << 1) | ((uint32_t)nz << 2);
    ox = nx ? -ox : ox; oy = ny ? -oy : oy; oz = nz ? -oz : oz;
    dx = fabsf(dx); dy = fabsf(dy); dz = fabsf(dz);
    const float yz = __frcp_rn(dz);
    const float mz = MZERO_CONST ? 0.0f : __fmul_rn(-dx, 0.0f);   // -0
    const f32x2 mzero = MZERO_CONST ? c_mzero : pair(mz, mz), ndxy = pair(-dx, -dy), yxy = pair(__frcp_rn(dx), __frcp_rn(dy));
    int sp = 0;
    uint32_t cur = start;      // a record, or while scanning a leaf the voxel to test
    uint32_t vend = 0;         // one past the leaf's last voxel; 0: cur is a record
    uint32_t vrec = 0, win = 0;
    float best = 0.0f, bx = 0.0f, by = 0.0f, bz = 0.0f;
    for (uint32_t steps = 0; steps < t.max_steps; steps++) {
        const bool scan = vend != 0u;
        if (!in_range(cur, scan ? 1u : VOXP_REC_UNITS, t.n_units, t.fault)) return STEP_ERROR;
        const uint4 u0 = ld16(pool + cur);
        uint4 u1 = make_uint4(0u, 0u, 0u, 0u), u2 = make_uint4(0u, 0u, 0u, 0u);
        if (!scan) {
            u1 = ld16(pool + cur + 1);
            u2 = ld16(pool + cur + 2);
        }
        float lx = ubf(u0.x), ly = ubf(u0.y), lz = ubf(u0.z), hx = ubf(u0.w), hy = ubf(u1.x), hz = ubf(u1.y);
        if (scan) {   // voxel box [dot, dot + vox_voxel] (search.c:53-54)
            hx = __fadd_rn(lx, t.vx); hy = __fadd_rn(ly, t.vy); hz = __fadd_rn(lz, t.vz);
        }
        float x;
        x = nx ? -hx : lx; hx = nx ? -lx : hx; lx = x;
        x = ny ? -hy : ly; hy = ny ? -ly : hy; ly = x;
        x = nz ? -hz : lz; hz = nz ? -lz : hz; lz = x;

        // geom.c:69-99 hit_box: m is the largest forward distance to a near
        // face, -0 when there is none (the origin itself is then the point:
        // o + -0 * d is o)
        float qx, qy;
        halves(quot2(sub2(pair(lx, ly), pair(ox, oy)), ndxy, yxy), qx, qy);
        const float qz = quot(__fsub_rn(lz, oz), dz, yz);
        float m = fmaxf(fmaxf(qx, qy), qz);
        const bool fwd = m > 0.0f;
        if (fwd && m < QUOT_MIN) return STEP_AGAIN;
        m = fwd ? m : -0.0f;
        const bool p0 = fwd && qx == m, p1 = fwd && qy == m && !p0, p2 = fwd && !p0 && !p1;
        float ex, ey, ez = __fadd_rn(oz, __fmul_rn(m, dz));
        halves(sub2(pair(ox, oy), fma2(pair(m, m), ndxy, mzero)), ex, ey);
        ex = p0 ? lx : ex; ey = p1 ? ly : ey; ez = p2 ? lz : ez;
        const bool in = ex >= lx && ex <= hx && ey >= ly && ey <= hy && ez >= lz && ez <= hz;
        bool resume = !in;

        if (scan) {
            // leaf loop body, search.c:55-78
            bool stop = false;
            if (in) {
                float dist = __fadd_rn(__fadd_rn(__fsub_rn(ex, ox), __fsub_rn(ey, oy)), __fsub_rn(ez, oz));
                stop = dist == 0.0f;
                if (dist < best) {
                    best = dist; bx = ex; by = ey; bz = ez; win = cur;
                }
            }
            cur++;
            resume = false;
            if (stop || cur == vend) {
                if (win) {
                    hit.x = turned_back<LATE>(nx, bx); hit.y = turned_back<LATE>(ny, by); hit.z = turned_back<LATE>(nz, bz);
                    const uint4 r1 = ld16(pool + vrec + 1), r2 = ld16(pool + vrec + 2);
                    hit.leaf = r2.x; hit.slot = win - r1.w; hit.rec = vrec;
                    return STEP_HIT;
                }
                vend = 0;
                resume = true;
            }
        } else if (in) {
            const uint32_t meta = u1.z, link = u1.w, kind = meta & 3u;
            if (kind == VOXP_KIND_DENSE) {                      // search.c:31-37
                hit.x = turned_back<LATE>(nx, ex); hit.y = turned_back<LATE>(ny, ey); hit.z = turned_back<LATE>(nz, ez);
                hit.leaf = link; hit.slot = 0xFFu; hit.rec = cur;
                return STEP_HIT;
            }
            if (kind == VOXP_KIND_LEAF) {                       // search.c:39-50
                const uint32_t vn = meta >> 2;
                if (vn == 0) {
                    resume = true;
                } else {
                    vrec = cur; cur = link; vend = link + vn; win = 0;
                    best = __int_as_float(0x7f800000);
                    ox = ex; oy = ey; oz = ez;
                }
            } else {                                            // search.c:86-148
                const float cx = nx ? -ubf(u2.x) : ubf(u2.x), cy = ny ? -ubf(u2.y) : ubf(u2.y),
                            cz = nz ? -ubf(u2.z) : ubf(u2.z);
                const bool a0 = cx > ex, a1 = cy > ey, a2 = cz > ez;
                // geom.c:53-65 get_corrected_subspace_idx: an equal centre takes the side the ray goes to
                const uint32_t sub = ((uint32_t)a0 | ((uint32_t)a1 << 1) | ((uint32_t)a2 << 2)) ^ neg;
                const uint32_t mask = (meta >> 8) & 0xFFu;
                float k0, k1;
                const f32x2 exy = pair(ex, ey);
                halves(quot2(sub2(pair(cx, cy), exy), ndxy, yxy), k0, k1);
                const float k2 = quot(__fsub_rn(cz, ez), dz, yz);
                const f32x2 c0 = sub2(exy, fma2(pair(k0, k0), ndxy, mzero)), c1 = sub2(exy, fma2(pair(k1, k1), ndxy, mzero)),
                            c2 = sub2(exy, fma2(pair(k2, k2), ndxy, mzero));
                float x0, y0, x1, y1, x2, y2;
                halves(c0, x0, y0);
                halves(c1, x1, y1);
                halves(c2, x2, y2);
                const float z0 = __fadd_rn(ez, __fmul_rn(k0, dz)), z1 = __fadd_rn(ez, __fmul_rn(k1, dz)),
                            z2 = __fadd_rn(ez, __fmul_rn(k2, dz));
                const bool v0 = a0 && x0 <= hx && y0 <= hy && z0 <= hz, v1 = a1 && x1 <= hx && y1 <= hy && z1 <= hz,
                           v2 = a2 && x2 <= hx && y2 <= hy && z2 <= hz;
                const float inf = __int_as_float(0x7f800000);
                // L1 distances from the entry point (search.c:115-134), every term positive
                float d0, d1, d2, t0, t1, t2;
                halves(sub2(c0, exy), d0, t0);
                halves(sub2(c1, exy), d1, t1);
                halves(sub2(c2, exy), d2, t2);
                d0 = __fadd_rn(__fadd_rn(d0, t0), __fsub_rn(z0, ez));
                d1 = __fadd_rn(__fadd_rn(d1, t1), __fsub_rn(z1, ez));
                d2 = __fadd_rn(__fadd_rn(d2, t2), __fsub_rn(z2, ez));
                d0 = v0 ? d0 : inf; d1 = v1 ? d1 : inf; d2 = v2 ? d2 : inf;
                if (fminf(fminf(d0, d1), d2) < DIST_MIN) return STEP_AGAIN;
                // oij: crossing i comes before crossing j.  The selection sort with immediate
                // swaps keeps equal distances in axis order, except that crossing 2 before an
                // equal pair 0, 1 turns it round
                const bool o20 = d2 < d0, o21 = d2 < d1, o10 = d1 < d0 || (d1 == d0 && o20);
                // the octant behind each crossing (:137): the bits of the crossings up to it flipped
                const uint32_t s0 = sub ^ 1u ^ (o10 ? 2u : 0u) ^ (o20 ? 4u : 0u);
                const uint32_t s1 = sub ^ 2u ^ (o10 ? 0u : 1u) ^ (o21 ? 4u : 0u);
                const uint32_t s2 = sub ^ 4u ^ (o20 ? 0u : 1u) ^ (o21 ? 0u : 2u);
                // the children's bits, at the bottom, and above them the siblings that follow:
                // one shift gives both whether a child is there and, counted back from the
                // block's end, its record (32 orbit frames in the batch kernel 1,305 -> 1,277
                // us, against the siblings before it masked and counted)
                const uint32_t r0 = mask >> s0, r1 = mask >> s1, r2 = mask >> s2, r3 = mask >> sub;
                const uint32_t end = link + VOXP_REC_UNITS * (uint32_t)__popc(mask);
                const bool w0 = v0 && (r0 & 1u), w1 = v1 && (r1 & 1u), w2 = v2 && (r2 & 1u);
                const int n = (int)w0 + (int)w1 + (int)w2;
                if (sp > CAP - 3) return STEP_ERROR;   // (never in a tree whose depth the class holds)
                // each child above those visited after it
                if (w0)
                    stack[sp + (int)(w1 && !o10) + (int)(w2 && !o20)] =
                        make_uint4(end - VOXP_REC_UNITS * (uint32_t)__popc(r0),
                                   __float_as_uint(x0), __float_as_uint(y0), __float_as_uint(z0));
                if (w1)
                    stack[sp + (int)(w0 && o10) + (int)(w2 && !o21)] =
                        make_uint4(end - VOXP_REC_UNITS * (uint32_t)__popc(r1),
                                   __float_as_uint(x1), __float_as_uint(y1), __float_as_uint(z1));
                if (w2)
                    stack[sp + (int)(w0 && o20) + (int)(w1 && o21)] =
                        make_uint4(end - VOXP_REC_UNITS * (uint32_t)__popc(r2),
                                   __float_as_uint(x2), __float_as_uint(y2), __float_as_uint(z2));
                sp += n;
                if (r3 & 1u) {                                  // search.c:92-93
                    cur = end - VOXP_REC_UNITS * (uint32_t)__popc(r3);
                    ox = ex; oy = ey; oz = ez;
                } else {
                    resume = true;
                }
            }
        }
        if (resume) {
            if (sp == 0) return STEP_MISS;
            const uint4 e = stack[--sp];
            cur = e.x;
            ox = ubf(e.y); oy = ubf(e.z); oz = ubf(e.w);
        }
    }
    return STEP_ERROR;   // damaged pool
}

/* The general search from the node whose record is at `start`: any numbers. */
template <int CAP, bool COUNT>
__device__ __forceinline__ bool trace_general(const DevTree &t, uint32_t start,
                                              float ox0, float oy0, float oz0,
                                              float dx, float dy, float dz, uint4 (&stack)[CAP],
                                              RayHit &hit, Counts &cnt, bool &overflow)
{
    RaySearch s;
    ray_begin(s, start, ox0, oy0, oz0, dx, dy, dz);
    for (;;) {
        int r = ray_step<CAP, COUNT>(t, s, stack, hit, cnt);
        if (r != STEP_MORE) {
            if (r == STEP_ERROR) overflow = true;
            return r == STEP_HIT;
        }
    }
}

// The general search as a call of its own, on the caller's stack: it takes no
// registers from the loop above.
struct GeneralResult {
    RayHit hit;
    uint32_t found, overflow;
};
template <int CAP>
__device__ __noinline__ GeneralResult trace_general_call(const uint4 *pool, uint32_t start, float ox, float oy, float oz,
                                                         float dx, float dy, float dz, float vx, float vy, float vz,
                                                         uint32_t max_steps, uint32_t n_units, uint32_t *fault,
                                                         uint4 (&stack)[CAP])
{
    DevTree t;
    t.pool = pool;
    t.vx = vx; t.vy = vy; t.vz = vz;
    t.max_steps = max_steps;
    t.n_units = n_units;
    t.fault = fault;
    GeneralResult g;
    Counts c{0, 0, 0};
    bool overflow = false;
    g.hit = RayHit{0.0f, 0.0f, 0.0f, 0u, 0u, 0u};
    g.found = trace_general<CAP, false>(t, start, ox, oy, oz, dx, dy, dz, stack, g.hit, c, overflow);
    g.overflow = overflow;
    return g;
}

/* The whole search from the node whose record is at `start`.  Returns true
 * on a hit; `overflow` is set (and the search ends as a miss) on STEP_ERROR.
 * Counting searches count the reference's work: the general search, as those
 * of a kernel built for images that the mirrored one leaves (GENERAL). */
template <int CAP, bool COUNT, bool MZERO_CONST = false, bool GENERAL = false, bool LATE = MZERO_CONST>
__device__ __forceinline__ bool trace_ray(const DevTree &t, uint32_t start,
                                          float ox0, float oy0, float oz0,
                                          float dx, float dy, float dz,
                                          RayHit &hit, Counts &cnt, bool &overflow)
{
    uint4 stack[CAP];
    if (COUNT || GENERAL) return trace_general<CAP, COUNT>(t, start, ox0, oy0, oz0, dx, dy, dz, stack, hit, cnt, overflow);
    int r = STEP_AGAIN;
    if (mirror_ok(t, ox0, oy0, oz0, dx, dy, dz))
        r = trace_mirrored<CAP, MZERO_CONST, LATE>(t, start, ox0, oy0, oz0, dx, dy, dz, stack, hit);
    if (r == STEP_AGAIN) {
        GeneralResult g = trace_general_call<CAP>(t.pool, start, ox0, oy0, oz0, dx, dy, dz, t.vx, t.vy, t.vz,
                                                  t.max_steps, t.n_units, t.fault, stack);
        hit = g.hit;
        if (g.overflow) overflow = true;
        return g.found;
    }
    if (r == STEP_ERROR) overflow = true;
    if (LATE) {
        hit.x = late_zero(hit.x, dx); hit.y = late_zero(hit.y, dy); hit.z = late_zero(hit.z, dz);
    }
    return r == STEP_HIT;
}

/* geom.c:149-154 box_ball_interp with vox_sqr_metric (geom.c:133-139):
 * clamp the centre into the box, ((dx*dx + dy*dy) + dz*dz) < r*r. */
__device__ __forceinline__ bool ball_box(float lx, float ly, float lz, float hx, float hy, float hz,
                                         float cx, float cy, float cz, float rr)
{
    float fx = cx < lx ? lx : (cx > hx ? hx : cx);
    float fy = cy < ly ? ly : (cy > hy ? hy : cy);
    float fz = cz < lz ? lz : (cz > hz ? hz : cz);
    float ex = __fsub_rn(fx, cx), ey = __fsub_rn(fy, cy), ez = __fsub_rn(fz, cz);
    float s = __fadd_rn(__fadd_rn(__fmul_rn(ex, ex), __fmul_rn(ey, ey)), __fmul_rn(ez, ez));
    return s < rr;
}

/* vox_tree_ball_collidep (search.c:155-183): any voxel box meeting the open
 * ball; children in octant order, first hit ends the search. */
template <int CAP, bool COUNT>
__device__ __forceinline__ bool trace_ball(const DevTree &t, float cx, float cy, float cz, float r,
                                           Counts &cnt, bool &overflow)
{
    if (t.root == VOXP_EMPTY) return false;
    uint32_t stack[CAP];
    int sp = 0;
    uint32_t cur = t.root;
    const uint4 *pool = t.pool;
    float rr = __fmul_rn(r, r);
    uint32_t steps = 0;
    for (;;) {
        if (++steps > t.max_steps) { overflow = true; return false; }   // damaged pool
        if (!in_range(cur, 2, t.n_units, t.fault)) { overflow = true; return false; }
        uint4 a = ld16(pool + cur);
        uint4 b = ld16(pool + cur + 1);
        if (COUNT) cnt.nodes++;
        if (ball_box(ubf(a.x), ubf(a.y), ubf(a.z), ubf(a.w), ubf(b.x), ubf(b.y), cx, cy, cz, rr)) {
            uint32_t kind = b.z & 3u, link = b.w;
            if (kind == VOXP_KIND_DENSE) return true;
            if (kind == VOXP_KIND_LEAF) {
                uint32_t n = b.z >> 2;
                if (!in_range(link, n, t.n_units, t.fault)) { overflow = true; return false; }
                for (uint32_t i = 0; i < n; i++) {
                    uint4 v = ld16(pool + link + i);
                    if (COUNT) cnt.voxels++;
                    float vx = ubf(v.x), vy = ubf(v.y), vz = ubf(v.z);
                    if (ball_box(vx, vy, vz, __fadd_rn(vx, t.vx), __fadd_rn(vy, t.vy),
                                 __fadd_rn(vz, t.vz), cx, cy, cz, rr))
                        return true;
                }
            } else {
                if (COUNT) cnt.inner++;
                uint32_t mask = (b.z >> 8) & 0xFFu;
                int k = __popc(mask);
                if (k > 0) {
                    if (sp + k - 1 > CAP) { overflow = true; return false; }
                    // children in octant order = consecutive records; push in
                    // reverse so octant order is the pop order.
                    for (int i = k - 1; i >= 1; i--) stack[sp++] = link + VOXP_REC_UNITS * (uint32_t)i;
                    cur = link;
                    continue;
                }
            }
        }
        if (sp == 0) return false;
        cur = stack[--sp];
    }
}

/* The same answer in a tree of ordered, nested boxes, where it depends on no
 * order: a ball hits when any voxel's or dense leaf's own test passes.
 *
 * In round-to-nearest arithmetic the test is monotone -- a box inside
 * another is no nearer on any axis, nor, squared and summed in the same
 * order, in all -- so the tests of the nodes above a voxel that passes pass
 * too, and pruning by them (search.c:160) changes nothing.  By the same
 * monotony a child needs no test when on one axis the ball stays its radius
 * away from all that lies on the child's side of the dividing plane: the
 * child's own distance there is at least the radius, its square at least the
 * radius's square (ball_side).
 *
 * What bounds the search is instruction issue at few active lanes (7 of 32 in
 * 73% of the slots for 1M balls) and the loads waited for beside it.  A ball
 * small beside the upper nodes can meet one or two of their eight children,
 * so leaving the others out takes a search from 45 box tests to 13 on
 * average (balls of radius 0.5-8 in the 256^3 tree), and the child where the
 * centre lies goes first, where a voxel is likeliest.  One record a step
 * keeps the lanes of a warp alike; testing all of a node's children in one
 * step, handing idle lanes new balls, and accepting nodes of which the ball
 * holds a whole face were each slower (see launch_balls). */
// The octants (a bit each, as in a child mask) a ball can meet on one axis:
// none below the dividing plane when it stays r above the highest face a
// voxel there can have, none above when it stays r below the plane.  `low` is
// the axis's octants below the plane (geom.c:44-51: their bit is set).
__device__ __forceinline__ uint32_t ball_side(float c, float plane, float v, float r, uint32_t low)
{
    uint32_t m = 0xFFu;
    if (__fsub_rn(c, __fadd_rn(plane, v)) >= r) m = ~low;
    if (__fsub_rn(plane, c) >= r) m = low;
    return m;
}

template <int CAP>
__device__ __forceinline__ bool trace_ball_nested(const DevTree &t, float cx, float cy, float cz, float r, bool &overflow)
{
    if (t.root == VOXP_EMPTY || !(cx == cx && cy == cy && cz == cz && r == r)) return false;   // NaN is near nothing
    const uint4 *pool = t.pool;
    const float rr = __fmul_rn(r, r);
    r = fabsf(r);
    uint32_t stack[CAP];
    int sp = 0;
    uint32_t cur = t.root;
    for (uint32_t steps = 0; steps < t.max_steps; steps++) {
        if (!in_range(cur, VOXP_REC_UNITS, t.n_units, t.fault)) break;
        const uint4 a = ld16(pool + cur), b = ld16(pool + cur + 1), c = ld16(pool + cur + 2);
        const float ex = fmaxf(fmaxf(__fsub_rn(ubf(a.x), cx), __fsub_rn(cx, ubf(a.w))), 0.0f),
                    ey = fmaxf(fmaxf(__fsub_rn(ubf(a.y), cy), __fsub_rn(cy, ubf(b.x))), 0.0f),
                    ez = fmaxf(fmaxf(__fsub_rn(ubf(a.z), cz), __fsub_rn(cz, ubf(b.y))), 0.0f);
        const float s = __fadd_rn(__fadd_rn(__fmul_rn(ex, ex), __fmul_rn(ey, ey)), __fmul_rn(ez, ez));
        bool pop = true;
        if (s < rr) {
            const uint32_t kind = b.z & 3u, link = b.w;
            if (kind == VOXP_KIND_DENSE) return true;
            if (kind == VOXP_KIND_LEAF) {
                const uint32_t n = b.z >> 2;
                if (!in_range(link, n, t.n_units, t.fault)) break;
                for (uint32_t j = 0; j < n; j++) {
                    const uint4 v = ld16(pool + link + j);
                    const float vx = ubf(v.x), vy = ubf(v.y), vz = ubf(v.z);
                    if (ball_box(vx, vy, vz, __fadd_rn(vx, t.vx), __fadd_rn(vy, t.vy), __fadd_rn(vz, t.vz), cx, cy, cz, rr))
                        return true;
                }
            } else {
                const uint32_t mask = (b.z >> 8) & 0xFFu;
                uint32_t left = mask & ball_side(cx, ubf(c.x), t.vx, r, 0xAAu) & ball_side(cy, ubf(c.y), t.vy, r, 0xCCu) &
                                ball_side(cz, ubf(c.z), t.vz, r, 0xF0u);
                if (left) {
                    // the octant of the centre first, else the first one
                    const uint32_t home = 1u << ((uint32_t)(ubf(c.x) > cx) | ((uint32_t)(ubf(c.y) > cy) << 1) |
                                                 ((uint32_t)(ubf(c.z) > cz) << 2));
                    const uint32_t first = left & home ? home : left & (0u - left);
                    left ^= first;
                    cur = link + VOXP_REC_UNITS * (uint32_t)__popc(mask & (first - 1u));
                    pop = false;
                    if (sp + __popc(left) > CAP) break;
                    while (left) {
                        const uint32_t low = left & (0u - left);
                        left ^= low;
                        stack[sp++] = link + VOXP_REC_UNITS * (uint32_t)__popc(mask & (low - 1u));
                    }
                }
            }
        }
        if (pop) {
            if (sp == 0) return false;
            cur = stack[--sp];
        }
    }
    overflow = true;   // damaged pool
    return false;
}

/* simple-camera.c:21-31 (+ vect-ops.c:7-15, :28-36) and doom-camera.c:24-57. */
__device__ __forceinline__ void screen2world(const vox_cuda_camera &cam, int sx, int sy,
                                             float &rx, float &ry, float &rz)
{
    float v0 = __fsub_rn(__fmul_rn(cam.mul, (float)sx), cam.xsub);
    float v2 = __fsub_rn(cam.ysub, __fmul_rn(cam.mul, (float)sy));
    if (cam.kind == VOX_CUDA_CAMERA_DOOM) {
        const float v1 = 1.0f;
        v2 = __fadd_rn(v2, cam.k);
        rx = __fsub_rn(__fmul_rn(v0, cam.cosphi), __fmul_rn(v1, cam.sinphi));
        ry = __fadd_rn(__fmul_rn(v1, cam.cosphi), __fmul_rn(v0, cam.sinphi));
        rz = v2;
        return;
    }
    const float v1 = 1.0f;
    float qw = cam.rotation[0], qi = cam.rotation[1], qj = cam.rotation[2], qk = cam.rotation[3];
    // t = 2 * (q.xyz x v)
    float t0 = __fsub_rn(__fmul_rn(qj, v2), __fmul_rn(qk, v1));
    float t1 = __fadd_rn(__fmul_rn(-qi, v2), __fmul_rn(qk, v0));
    float t2 = __fsub_rn(__fmul_rn(qi, v1), __fmul_rn(qj, v0));
    t0 = __fmul_rn(t0, 2.0f); t1 = __fmul_rn(t1, 2.0f); t2 = __fmul_rn(t2, 2.0f);
    // u = q.xyz x t
    float u0 = __fsub_rn(__fmul_rn(qj, t2), __fmul_rn(qk, t1));
    float u1 = __fadd_rn(__fmul_rn(-qi, t2), __fmul_rn(qk, t0));
    float u2 = __fsub_rn(__fmul_rn(qi, t1), __fmul_rn(qj, t0));
    rx = __fadd_rn(__fadd_rn(v0, __fmul_rn(qw, t0)), u0);
    ry = __fadd_rn(__fadd_rn(v1, __fmul_rn(qw, t1)), u1);
    rz = __fadd_rn(__fadd_rn(v2, __fmul_rn(qw, t2)), u2);
}

/* renderer.c:27-39 get_color without a light manager; SDL_MapRGB on an
 * ARGB8888 surface packs an opaque grey. */
__device__ __forceinline__ uint32_t texel_color(const uint8_t *__restrict__ tex, const DevTree &t,
                                                float x, float y, float z)
{
    int ix = abs(__float2int_rz(__fdiv_rn(x, t.vx))) & 31;
    int iy = abs(__float2int_rz(__fdiv_rn(y, t.vy))) & 31;
    int iz = abs(__float2int_rz(__fdiv_rn(z, t.vz))) & 31;
    uint32_t c = __ldg(tex + ix * 1024 + iy * 32 + iz);
    return 0xFF000000u | (c << 16) | (c << 8) | c;
}

/* Lights of a light manager on the device (layout: lights_internal.h).
 * nodes == nullptr: no bound lights, ambient only. */
struct DevLights {
    const float4 *nodes;     // 2 per M-tree node
    const float4 *spheres;   // 2 per light sphere
    float ar, ag, ab;        // ambient light
    uint32_t on;             // 0: draw without lights (grey texels)
    uint32_t n_nodes, n_spheres;
};

constexpr int LIGHT_STACK = 64;   // (children - 1) per level; the upload refuses deeper trees

/* geom.c:133-139 vox_sqr_metric: ((dx*dx + dy*dy) + dz*dz). */
__device__ __forceinline__ float sqr_dist(float ax, float ay, float az, float bx, float by, float bz)
{
    float x = __fsub_rn(ax, bx), y = __fsub_rn(ay, by), z = __fsub_rn(az, bz);
    return __fadd_rn(__fadd_rn(__fmul_rn(x, x), __fmul_rn(y, y)), __fmul_rn(z, z));
}

/* lights.c:91-102 get_color_callback: the light of one sphere containing p. */
__device__ __forceinline__ void add_light(const float4 &sa, const float4 &sb, float px, float py, float pz,
                                          float &r, float &g, float &b)
{
    float dist = fminf(sb.w, __fsqrt_rn(sqr_dist(sa.x, sa.y, sa.z, px, py, pz)));
    float add = __fsub_rn(1.0f, __fdiv_rn(dist, sb.w));
    r = __fadd_rn(r, __fmul_rn(add, sb.x));
    g = __fadd_rn(g, __fmul_rn(add, sb.y));
    b = __fadd_rn(b, __fmul_rn(add, sb.z));
}

/* renderer.c:40-49 with lights.c:104-116 (vox_get_light) and
 * mtree.c:463-493 (vox_mtree_spheres_containing_f): ambient light plus the
 * spheres containing the hit, in the M-tree's depth-first order (a
 * one-sphere leaf whose bounding sphere holds the hit counts its sphere
 * without a second test), then min(light, 1) * texel per channel, truncated
 * to 8 bits.  `overflow` is set if the search stack would overflow. */
__device__ __forceinline__ uint32_t lit_color(const DevLights &L, uint32_t c, float px, float py, float pz,
                                              bool &overflow, uint32_t *fault)
{
    float r = L.ar, g = L.ag, b = L.ab;
    if (L.nodes) {
        uint32_t stack[LIGHT_STACK];
        int sp = 0;
        uint32_t cur = 0;
        for (;;) {
            if (!in_range(cur, 1, L.n_nodes, fault)) { overflow = true; break; }
            float4 na = L.nodes[2 * cur];
            float4 nb = L.nodes[2 * cur + 1];
            uint32_t leaf = __float_as_uint(nb.x), num = __float_as_uint(nb.y), first = __float_as_uint(nb.z);
            bool next_from_stack = true;
            if (sqr_dist(na.x, na.y, na.z, px, py, pz) < na.w) {
                if (leaf) {
                    if (!in_range(first, num, L.n_spheres, fault)) { overflow = true; break; }
                    if (num == 1) {
                        add_light(L.spheres[2 * first], L.spheres[2 * first + 1], px, py, pz, r, g, b);
                    } else {
                        for (uint32_t i = 0; i < num; i++) {
                            float4 sa = L.spheres[2 * (first + i)];
                            if (sqr_dist(sa.x, sa.y, sa.z, px, py, pz) < sa.w)
                                add_light(sa, L.spheres[2 * (first + i) + 1], px, py, pz, r, g, b);
                        }
                    }
                } else if (num > 0) {
                    if (sp + (int)num - 1 > LIGHT_STACK) { overflow = true; break; }
                    for (uint32_t i = num - 1; i >= 1; i--) stack[sp++] = first + i;
                    cur = first;
                    next_from_stack = false;
                }
            }
            if (next_from_stack) {
                if (sp == 0) break;
                cur = stack[--sp];
            }
        }
    }
    uint32_t R = __float2uint_rz(__fmul_rn(fminf(r, 1.0f), (float)c));
    uint32_t G = __float2uint_rz(__fmul_rn(fminf(g, 1.0f), (float)c));
    uint32_t B = __float2uint_rz(__fmul_rn(fminf(b, 1.0f), (float)c));
    return 0xFF000000u | ((R & 0xFFu) << 16) | ((G & 0xFFu) << 8) | (B & 0xFFu);
}

/* renderer.c:27-52 get_color: the texel of the hit point, grey without a
 * light manager (SDL_MapRGB on ARGB8888), lit with one. */
__device__ __forceinline__ uint32_t hit_color(const uint8_t *__restrict__ tex, const DevTree &t, const DevLights &L,
                                              float x, float y, float z, bool &overflow)
{
    int ix = abs(__float2int_rz(__fdiv_rn(x, t.vx))) & 31;
    int iy = abs(__float2int_rz(__fdiv_rn(y, t.vy))) & 31;
    int iz = abs(__float2int_rz(__fdiv_rn(z, t.vz))) & 31;
    uint32_t c = __ldg(tex + ix * 1024 + iy * 32 + iz);
    if (!L.on) return 0xFF000000u | (c << 16) | (c << 8) | c;
    return lit_color(L, c, x, y, z, overflow, t.fault);
}

}  // namespace vox

#endif
