/*
 * build.cu -- voxtrees octrees built on the GPU, straight into the device
 * image of pool_layout.h: the tree that vox_make_tree builds from a voxel set
 * (tree.c:249-338) and the raw-volume reader of datareader.c:11-85.
 *
 * The tree must be the reference's node for node and voxel for voxel, and two
 * steps of its construction are sequential by definition:
 *
 *  - the subdivision centre is the mean of the node's voxels, summed in float
 *    in the set's current order (find_center, tree.c:125-136), so its
 *    rounding depends on that order;
 *  - the set is split by eight in-place swapping passes, one per octant
 *    (sort_set, tree.c:166-183), which leave the voxels of later octants
 *    permuted; the next level's sums and the leaves' voxel order see that
 *    permutation.
 *
 * Both are computed here in parallel and exactly.
 *
 *  Swapping pass.  In one pass over a range, the claimed voxels (those of
 *  the pass's octant) go to the front in their order.  The others behave as
 *  a queue: an unclaimed voxel joins its tail and each claimed voxel moves
 *  the head to the tail.  So the voxel that ends at position t (t at or past
 *  the claimed count) is found by walking back: if position t held a claimed
 *  voxel, the voxel that ends there is the one that stood at C(t), the
 *  number of claimed positions before t, and so on until an unclaimed
 *  position is reached.  Inside a run of claimed positions every step
 *  subtracts the same number (the unclaimed positions before the run), so a
 *  whole run is crossed in one step.  A prefix count gives C, and the list of
 *  unclaimed positions gives each run's start.
 *
 *  Float sum.  Within one binade, adding d >= 0 to acc = A * 2^e (A an
 *  integer in [2^23, 2^24)) gives (A + q + delta) * 2^e with q = floor(d/2^e)
 *  and delta in {0, 1}, which depends on the fraction of d/2^e and, for an
 *  exact half (rounded to even), on the parity of A + q.  A run of additions
 *  is therefore a map from the parity of A to (increment, new parity): a
 *  two-state machine, and such maps compose associatively.  Most sums need
 *  none of it: no addition rounds while the sum stays below 2^24 times a power
 *  of two that divides every term, and then any order gives it (PlainSum).
 *  For the others, chunks of 1024 voxels get their maps, in parallel, for the
 *  two binades the sum is expected in there (from the chunks' plain sums); a
 *  warp then scans 32 chunks' maps at a time, and adds a chunk voxel by voxel
 *  only where the sum leaves its binade inside the chunk (a dozen times per
 *  node) or no map was made for it.  The root of the 256^3 set: 423 us walking
 *  its 1,332 chunks one by one, and 147 for maps of 16 binades, became 70 and
 *  26 (raw volume with a first frame 4,790 -> 3,830 us).
 *
 * The rest (bounding boxes, the density test, leaf decisions, children) is
 * per node or per voxel.  The tree is built a level at a time.  Then subtree
 * sizes (bottom up), pre-order ids and image offsets (top down) place every
 * node where the host flattener (flatten.cpp) puts it, and one pass writes the
 * records and the leaves' voxel runs: the image equals the host build followed
 * by vox_cuda_tree_upload, byte for byte.
 */
#include <cuda_runtime.h>

#include <algorithm>
#include <cerrno>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <new>
#include <vector>

#include <fcntl.h>
#include <sys/stat.h>
#include <unistd.h>

#include "internal.h"
#include "abi_guard.h"
#include "build_sizes.h"
#include "host_wait.h"

#define EXPORT extern "C" __attribute__((visibility("default")))

namespace {

using namespace build_sizes;

constexpr uint32_t NONE = 0xFFFFFFFFu;
constexpr int RAW_THREADS = 256;
constexpr uint32_t RAW_ITEMS = 16;                       // consecutive samples a thread reads
constexpr uint32_t RAW_TILE = RAW_THREADS * RAW_ITEMS;   // samples a block reads
constexpr int CHUNK_THREADS = 128;   // 8 consecutive voxels per thread
constexpr uint32_t SAT = 1u << 25;   // map increments saturate here (any >= 2^24 is unusable)
constexpr int MAX_LEVELS = 90;       // deeper trees exceed the traversal stack anyway
static_assert(LEAF == VOX_MAX_DOTS, "leaves");

enum : uint8_t { K_INNER = 0, K_LEAF = 1, K_DENSE = 2, K_OVER = 3 };
enum : int { S_INNER = 0, S_LEAF = 1, S_DENSE = 2, S_DOTS = 3, S_OVER = 4, NSTATS = 5 };   // a level's counts

// error bits reported by kernels
constexpr uint32_t ERR_WALK = 1u;       // a swapping-pass walk did not end as it must
constexpr uint32_t ERR_BIG_LEAF = 2u;   // a leaf holds 2^30 voxels or more (record limit)
constexpr uint32_t ERR_LAYOUT = 4u;     // a record or voxel run fell outside the image

// The kernels of a build follow one another on one stream, many of them a few
// microseconds long.  Each is launched while the one before runs (programmatic
// dependent launch) and starts with this: it waits for the kernel before to be
// complete and its memory visible, then lets the next one be launched.  (What
// comes before the call may read what kernels before the last one wrote.)  Of
// every launch some block has to wait, else the one after could pass it.  256^3
// raw volume with a first frame: 1,720 us, 1,930 with plain launches.
__device__ __forceinline__ void after_previous()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;");
}

// The kernels of a level's size classes need nothing of one another: only the
// first waits before its work, the others after theirs (so that none is
// complete before its predecessors), and each level's few large nodes run
// beside its many small ones.
__device__ __forceinline__ void class_begin(bool first)
{
    if (first) asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;");
}
__device__ __forceinline__ void class_end(bool first)
{
    if (!first) asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <class... K, class... A>
void launch_after_with(size_t shared, void (*kern)(K...), unsigned grid, unsigned block, cudaStream_t s, A... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = shared;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kern, K(args)...);   // errors: cudaGetLastError
    count_launch();
}

template <class... K, class... A>
void launch_after(void (*kern)(K...), unsigned grid, unsigned block, cudaStream_t s, A... args)
{
    launch_after_with(0, kern, grid, block, s, args...);
}

inline unsigned grid_for(uint64_t n, unsigned threads) { return (unsigned)((n + threads - 1) / threads); }

// ------------------------------------------------------------------ scans

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t x)
{
    int lane = threadIdx.x & 31;
    for (int off = 1; off < 32; off <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, off);
        if (lane >= off) x += y;
    }
    return x;
}

// Exclusive scan of n values in place, and their total (one block).
__global__ void __launch_bounds__(1024) k_scan_tiles(uint32_t *a, uint32_t n, uint32_t *total)
{
    __shared__ uint32_t ws[32];
    __shared__ uint32_t carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (uint32_t base = 0; base < n; base += 1024) {
        uint32_t i = base + threadIdx.x;
        uint32_t x = i < n ? a[i] : 0;
        uint32_t incl = warp_incl_scan(x);
        if ((threadIdx.x & 31) == 31) ws[threadIdx.x >> 5] = incl;
        __syncthreads();
        if (threadIdx.x < 32) {
            uint32_t w = ws[threadIdx.x];
            ws[threadIdx.x] = warp_incl_scan(w) - w;
        }
        __syncthreads();
        uint32_t c = carry;
        uint32_t excl = c + ws[threadIdx.x >> 5] + incl - x;
        if (i < n) a[i] = excl;
        __syncthreads();
        if (threadIdx.x == 1023) carry = excl + x;
        __syncthreads();
    }
    if (threadIdx.x == 0) *total = carry;
}

// ------------------------------------------------------------ level arrays

// The nodes of one level, in no particular order (the children of a node are
// consecutive, in octant order).  The voxels of a level's leaves stay where
// they are in the order of their level: the orders of successive levels
// alternate between two buffers, and a later level writes only where its own
// nodes lie.
struct Level {
    uint32_t m = 0;
    void *mem = nullptr;
    uint32_t *start, *n, *cnt, *first_child, *sub_nodes, *id, *ustart, *rec;
    unsigned long long *sub_units;
    float *box, *centre;
    int *ehi;
    uint8_t *kind, *mask;
};

template <typename T>
T *carve(char *&p, size_t count)
{
    T *r = reinterpret_cast<T *>(p);
    p += (count * sizeof(T) + 255) & ~size_t(255);
    return r;
}

cudaError_t level_alloc(Level &L, uint32_t m, cudaStream_t s)
{
    size_t mm = m ? m : 1;
    size_t bytes = 0;
    auto add = [&](size_t b) { bytes += (b + 255) & ~size_t(255); };
    add(4 * mm); add(4 * mm); add(32 * mm); add(4 * mm); add(4 * mm); add(4 * mm); add(4 * mm);
    add(4 * mm); add(8 * mm); add(24 * mm); add(12 * mm); add(12 * mm); add(mm); add(mm);
    cudaError_t e = pool_alloc(&L.mem, bytes, s);
    if (e != cudaSuccess) { L.mem = nullptr; return e; }
    char *p = static_cast<char *>(L.mem);
    L.m = m;
    L.start = carve<uint32_t>(p, mm);
    L.n = carve<uint32_t>(p, mm);
    L.cnt = carve<uint32_t>(p, 8 * mm);
    L.first_child = carve<uint32_t>(p, mm);
    L.sub_nodes = carve<uint32_t>(p, mm);
    L.id = carve<uint32_t>(p, mm);
    L.ustart = carve<uint32_t>(p, mm);
    L.rec = carve<uint32_t>(p, mm);
    L.sub_units = carve<unsigned long long>(p, mm);
    L.box = carve<float>(p, 6 * mm);
    L.centre = carve<float>(p, 3 * mm);
    L.ehi = carve<int>(p, 3 * mm);
    L.kind = carve<uint8_t>(p, mm);
    L.mask = carve<uint8_t>(p, mm);
    return cudaSuccess;
}

// -------------------------------------------------------- per-level kernels

// The nodes of a level that take more than one thread, by size class, in no
// particular order (above VOX_MAX_DOTS, TINY, SMALL, LOW, MID and HIGH voxels).
// A tiled node's slot, its first tile and its first sub come from one counter,
// so that first tiles and subs ascend with slots.
struct NodeLists {
    uint32_t *tiny, *small, *low, *mid, *high;
    uint4 *tiled;                 // a slot: its node, first tile, first sub and voxels, in one load
    uint32_t *ntiny, *nsmall, *nlow, *nmid, *nhigh;
    unsigned long long *ntiled;   // slots from bit 48 on, tiles from bit 24, subs (all below 2^24: N < 2^31)
    __device__ void add_large(uint32_t k, uint32_t n) const
    {
        if (n > HIGH) {
            const unsigned long long at = atomicAdd(ntiled, (1ull << 48) | ((unsigned long long)parts(n, tile_shift(n)) << 24) |
                                                                parts(n, SUB_SHIFT));
            tiled[at >> 48] = make_uint4(k, (uint32_t)(at >> 24) & 0xFFFFFFu, (uint32_t)at & 0xFFFFFFu, n);
        } else if (n > MID) {
            high[atomicAdd(nhigh, 1u)] = k;
        } else if (n > LOW) {
            mid[atomicAdd(nmid, 1u)] = k;
        } else if (n > SMALL) {
            low[atomicAdd(nlow, 1u)] = k;
        } else if (n > TINY) {
            small[atomicAdd(nsmall, 1u)] = k;
        }
    }
    __device__ uint32_t slots() const { return (uint32_t)(*ntiled >> 48); }
};

// What a level counts: kinds (S_*), the next level's nodes and the largest.
struct Tally {
    unsigned long long *stats;
    uint32_t *children, *largest, *err;
};

constexpr uint32_t NO_POS = 0xFFFFFFFFu;

// The slot whose part (tile or sub, by `first`) this is: the last that starts at
// or before it.
template <class F>
__device__ __forceinline__ uint32_t slot_of(const uint4 *tiled, uint32_t slots, uint32_t part, F first)
{
    uint32_t lo = 0, hi = slots;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (first(tiled[mid]) <= part) lo = mid;
        else hi = mid;
    }
    return lo;
}

// A block's tile of a tiled node: the node, its voxels, first tile and first
// sub, the tile's size and its positions in the node; false for a block
// without one.  (From the slot alone: with loads by node and by slot on the way
// the 256^3 raw volume took 1,352 us, 1,345 with this.)
struct TileRange {
    uint32_t k, n, ft, fs, shift, b, e;
    __device__ __forceinline__ bool find(const NodeLists &lists)
    {
        const unsigned long long count = *lists.ntiled;
        if (blockIdx.x >= ((uint32_t)(count >> 24) & 0xFFFFFFu)) return false;
        const uint4 s = lists.tiled[slot_of(lists.tiled, (uint32_t)(count >> 48), blockIdx.x, [](const uint4 &x) { return x.y; })];
        k = s.x; ft = s.y; fs = s.z; n = s.w;
        shift = tile_shift(n);
        b = (blockIdx.x - ft) << shift;
        e = min(n, b + (1u << shift));
        return true;
    }
    __device__ __forceinline__ uint64_t words() const { return (uint64_t)fs * (SUB / 32); }   // the node's first word
};

// Tiled nodes are summed by chunks of CHUNK voxels, counted through the subs:
// the range of chunk c; false for a chunk past its node's end.
constexpr uint32_t SUB_CHUNKS = SUB / CHUNK;
struct ChunkRange {
    uint32_t k;
    uint64_t b, e;
    __device__ bool find(const NodeLists &lists, const Level &L, uint32_t c)
    {
        const unsigned long long count = *lists.ntiled;
        if (c / SUB_CHUNKS >= ((uint32_t)count & 0xFFFFFFu)) return false;
        const uint4 s = lists.tiled[slot_of(lists.tiled, (uint32_t)(count >> 48), c / SUB_CHUNKS, [](const uint4 &x) { return x.z; })];
        k = s.x;
        const uint32_t at = (c - s.z * SUB_CHUNKS) * CHUNK, n = s.w;
        if (at >= n) return false;
        b = (uint64_t)L.start[k] + at;
        e = min(b + CHUNK, (uint64_t)L.start[k] + n);
        return true;
    }
};

// First-occurrence extremes: the serial scan of tree.c:138-155 keeps the first
// of equal values (which matters only for -0 against +0), so ties go to the
// lower position.
__device__ __forceinline__ void take_min(float &v, uint32_t &i, float v2, uint32_t i2)
{
    if (v2 < v || (v2 == v && i2 < i)) { v = v2; i = i2; }
}
__device__ __forceinline__ void take_max(float &v, uint32_t &i, float v2, uint32_t i2)
{
    if (v2 > v || (v2 == v && i2 < i)) { v = v2; i = i2; }
}

struct Extremes {
    float mn[3], mx[3];
    uint32_t mni[3], mxi[3];
    __device__ void init()
    {
        for (int a = 0; a < 3; a++) {
            mn[a] = INFINITY; mx[a] = -INFINITY; mni[a] = NONE; mxi[a] = NONE;
        }
    }
    __device__ void add(const float *p, uint32_t t)
    {
        for (int a = 0; a < 3; a++) {
            take_min(mn[a], mni[a], p[a], t);
            take_max(mx[a], mxi[a], p[a], t);
        }
    }
    __device__ void merge(const Extremes &o)
    {
        for (int a = 0; a < 3; a++) {
            take_min(mn[a], mni[a], o.mn[a], o.mni[a]);
            take_max(mx[a], mxi[a], o.mx[a], o.mxi[a]);
        }
    }
    __device__ void warp_merge()
    {
        for (int off = 16; off; off >>= 1) {
            Extremes o;
            for (int a = 0; a < 3; a++) {
                o.mn[a] = __shfl_xor_sync(0xffffffffu, mn[a], off);
                o.mx[a] = __shfl_xor_sync(0xffffffffu, mx[a], off);
                o.mni[a] = __shfl_xor_sync(0xffffffffu, mni[a], off);
                o.mxi[a] = __shfl_xor_sync(0xffffffffu, mxi[a], off);
            }
            merge(o);
        }
    }
};

// Partial extremes of one chunk of a tiled node.
__global__ void __launch_bounds__(CHUNK_THREADS) k_chunk_box(const float *P, Level L, NodeLists lists, float *cv,
                                                            uint32_t *ci)
{
    after_previous();
    __shared__ Extremes part[CHUNK_THREADS / 32];
    const uint32_t c = blockIdx.x;
    ChunkRange r;
    if (!r.find(lists, L, c)) return;
    Extremes x;
    x.init();
    for (uint64_t t = r.b + threadIdx.x; t < r.e; t += CHUNK_THREADS) x.add(P + 3 * t, (uint32_t)t);
    x.warp_merge();
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = x;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < CHUNK_THREADS / 32; w++) x.merge(part[w]);
        for (int a = 0; a < 3; a++) {
            cv[6 * c + a] = x.mn[a]; ci[6 * c + a] = x.mni[a];
            cv[6 * c + 3 + a] = x.mx[a]; ci[6 * c + 3 + a] = x.mxi[a];
        }
    }
}

// The scan of tree.c:138-155 starts with the first voxel's coordinate, and
// nothing is less or greater than a NaN: one there is the node's bound on both
// sides.  (A later NaN is no extreme.)
__device__ __forceinline__ void first_nan(float first, float &mn, float &mx)
{
    if (first != first) mn = mx = first;
}

// The box of node k (calc_bounding_box, tree.c:138-155) and what it is by its
// density (geom.c:157-167) and size, before it is split (tree.c:249-275).
__device__ uint8_t write_box(const Level &L, uint32_t k, uint32_t nk, const float *mn, const float *mx, const float *v)
{
    float hi[3];
    for (int a = 0; a < 3; a++) {
        hi[a] = __fadd_rn(mx[a], v[a]);
        L.box[6 * (size_t)k + a] = mn[a];
        L.box[6 * (size_t)k + 3 + a] = hi[a];
    }
    const float bbv = __fmul_rn(__fmul_rn(__fsub_rn(hi[0], mn[0]), __fsub_rn(hi[1], mn[1])), __fsub_rn(hi[2], mn[2]));
    const float vv = __fmul_rn(__fmul_rn(v[0], v[1]), v[2]);
    const uint8_t kind = fabsf(__fsub_rn(__fmul_rn(__uint2float_rn(nk), vv), bbv)) < vv ? K_DENSE
                       : (nk <= VOX_MAX_DOTS ? K_LEAF : K_INNER);
    L.kind[k] = kind;
    L.mask[k] = 0;
    return kind;
}

// Tiled nodes: a block per node over its chunks' partial extremes; and the top
// binade its coordinate sums can reach.
constexpr int NODE_THREADS = 256;
__global__ void __launch_bounds__(NODE_THREADS) k_box_tiled(const float *P, Level L, NodeLists lists, const float *cv,
                                                            const uint32_t *ci, float vx, float vy, float vz, Tally tally)
{
    after_previous();
    __shared__ Extremes part[NODE_THREADS / 32];
    if (blockIdx.x >= lists.slots()) return;
    const uint4 slot = lists.tiled[blockIdx.x];
    const uint32_t k = slot.x, nk = slot.w, nch = (nk + CHUNK - 1) / CHUNK, c0 = slot.z * SUB_CHUNKS;
    Extremes x;
    x.init();
    for (uint32_t j = threadIdx.x; j < nch; j += NODE_THREADS) {
        Extremes o;
        const size_t c = c0 + j;
        for (int a = 0; a < 3; a++) {
            o.mn[a] = cv[6 * c + a]; o.mni[a] = ci[6 * c + a];
            o.mx[a] = cv[6 * c + 3 + a]; o.mxi[a] = ci[6 * c + 3 + a];
        }
        x.merge(o);
    }
    x.warp_merge();
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = x;
    __syncthreads();
    if (threadIdx.x) return;
    for (int w = 1; w < NODE_THREADS / 32; w++) x.merge(part[w]);
    for (int a = 0; a < 3; a++) first_nan(P[3 * (uint64_t)L.start[k] + a], x.mn[a], x.mx[a]);
    const float v[3] = {vx, vy, vz};
    if (write_box(L, k, nk, x.mn, x.mx, v) == K_DENSE) atomicAdd(&tally.stats[S_DENSE], 1ull);
    for (int a = 0; a < 3; a++) {
        // The float sum of nk values in [0, extent] stays below 2 * nk * extent
        // for any nk this builder accepts (each addition rounds up by at most
        // 2^-24 relative); were it ever higher, its chunks would just be added
        // one voxel at a time.
        double bound = 2.0 * (double)nk * (double)__fsub_rn(L.box[6 * (size_t)k + 3 + a], x.mn[a]);
        int ehi = -100000;
        if (bound > 0.0 && bound < 1e38) {
            int ex;
            frexp(bound, &ex);
            ehi = ex - 24;           // bound in [2^(ex-1), 2^ex): its ulp exponent
            if (ehi < -149) ehi = -149;
        }
        L.ehi[3 * (size_t)k + a] = ehi;
    }
}

// ---- sums that no addition rounds
//
// When every d of a node is a multiple of some power of two g and their sum is
// below 2^24 g, each partial sum, in any order, is a multiple of g below 2^24 g:
// a float, so no addition rounds and the serial sum is the sum.  (A sum made in
// floats in another order that comes out below 2^24 g proves it: rounding is
// monotone, so no partial sum can have reached 2^24 g.)  On unit voxels g is 1
// and this covers all but the largest nodes.

// The exponent of the largest power of two that divides d (d > 0).
__device__ __forceinline__ int grid_exp(float d)
{
    const uint32_t b = __float_as_uint(d), e = max(b >> 23, 1u), m = (b & 0x7FFFFFu) | (b >> 23 ? 0x800000u : 0u);
    return (int)e - 150 + __ffs((int)m) - 1;
}

struct PlainSum {
    float sum[3];
    int g[3];       // exponent of the common power of two
    __device__ void init()
    {
        for (int a = 0; a < 3; a++) { sum[a] = 0.0f; g[a] = 1000; }
    }
    __device__ void add(int a, float d)
    {
        sum[a] = __fadd_rn(sum[a], d);
        if (d > 0.0f) g[a] = min(g[a], grid_exp(d));
    }
    __device__ void merge(int a, float x, int e)
    {
        sum[a] = __fadd_rn(sum[a], x);
        g[a] = min(g[a], e);
    }
    __device__ void warp_merge()
    {
        for (int off = 16; off; off >>= 1)
            for (int a = 0; a < 3; a++)
                merge(a, __shfl_xor_sync(0xffffffffu, sum[a], off), __shfl_xor_sync(0xffffffffu, g[a], off));
    }
    // sum[a] is the serial float sum
    __device__ bool exact(int a) const
    {
        const int e = g[a] + 24;
        return sum[a] == 0.0f || (e >= -126 && (e > 127 || sum[a] < __int_as_float((e + 127) << 23)));
    }
};

// ---- the two-state machine of a float sum within one binade

struct Tr {
    uint32_t w0, w1;   // for parity p: increment (bits 0-30) and new parity (bit 31)
};

__device__ __forceinline__ Tr tr_id() { return {0u, 0x80000000u}; }

__device__ __forceinline__ Tr tr_cat(Tr f, Tr g)   // f, then g
{
    uint32_t g0 = (f.w0 >> 31) ? g.w1 : g.w0;
    uint32_t g1 = (f.w1 >> 31) ? g.w1 : g.w0;
    Tr r;
    r.w0 = min((f.w0 & 0x7FFFFFFFu) + (g0 & 0x7FFFFFFFu), SAT) | (g0 & 0x80000000u);
    r.w1 = min((f.w1 & 0x7FFFFFFFu) + (g1 & 0x7FFFFFFFu), SAT) | (g1 & 0x80000000u);
    return r;
}

// Adding d >= 0 to A * 2^e, A in [2^23, 2^24), with round to nearest even.
__device__ __forceinline__ Tr tr_elem(float d, int e)
{
    // d / 2^e by a power-of-two multiply: exact, except that an x below the
    // normal range may round, which leaves it far below one half all the same.
    // Binades whose 2^-e is not a normal float never get a usable map.
    if (e < -126 || e > 126) return {SAT, SAT | 0x80000000u};
    float x = __fmul_rn(d, __int_as_float((127 - e) << 23));
    if (!(x < 33554432.0f)) return {SAT, SAT | 0x80000000u};
    float qf = floorf(x);
    float f = __fsub_rn(x, qf);
    uint32_t q = (uint32_t)qf;
    uint32_t up = f > 0.5f, tie = f == 0.5f;
    uint32_t par0 = q & 1u, par1 = par0 ^ 1u;    // parity of A + q for A even / odd
    uint32_t d0 = up | (tie & par0), d1 = up | (tie & par1);
    return {(q + d0) | ((par0 ^ d0) << 31), (q + d1) | ((par1 ^ d1) << 31)};
}

__device__ __forceinline__ Tr tr_shfl_down(Tr t, int off)
{
    return {__shfl_down_sync(0xffffffffu, t.w0, off), __shfl_down_sync(0xffffffffu, t.w1, off)};
}

// Sums and common powers of two of one chunk of a tiled node, per axis.
__global__ void __launch_bounds__(CHUNK_THREADS) k_chunk_sums(const float *P, Level L, NodeLists lists, float *csum,
                                                              int *cgrid)
{
    after_previous();
    __shared__ PlainSum part[CHUNK_THREADS / 32];
    const uint32_t c = blockIdx.x;
    ChunkRange r;
    if (!r.find(lists, L, c)) return;
    PlainSum x;
    x.init();
    for (uint64_t t = r.b + threadIdx.x; t < r.e; t += CHUNK_THREADS)
        for (int a = 0; a < 3; a++) x.add(a, __fsub_rn(P[3 * t + a], L.box[6 * (size_t)r.k + a]));
    x.warp_merge();
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = x;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < CHUNK_THREADS / 32; w++)
            for (int a = 0; a < 3; a++) x.merge(a, part[w].sum[a], part[w].g[a]);
        for (int a = 0; a < 3; a++) {
            csum[3 * c + a] = x.sum[a];
            cgrid[3 * c + a] = x.g[a];
        }
    }
}

__device__ __forceinline__ float centre_of(float acc, uint32_t nk, float mn, float v)
{
    float mean = __fadd_rn(__fdiv_rn(acc, __uint2float_rn(nk)), mn);
    return __fmul_rn(ceilf(__fdiv_rn(mean, v)), v);
}

// Centres of the big nodes whose sums no addition rounds, a block per node;
// for the other axes, where the first addition may round (the first chunk that
// takes the sum to 2^24 of the common power of two, and the sum before it,
// which is still a plain one), and the first of the binades (biased exponent) that each
// chunk gets a map for: the one that 63/64 of the sum before the chunk lies in,
// so that with the next one the sum's own binade is among them unless its
// roundings added up to more than that.  0: the axis needs no maps.  With
// window > 2 (sums so long that they do) the binades below the node's top.
__global__ void __launch_bounds__(NODE_THREADS) k_centre_plain(Level L, NodeLists lists, const float *csum,
                                                               const int *cgrid, uint8_t *cbase,
                                                               int window, uint2 *starts, float vx, float vy, float vz)
{
    after_previous();
    __shared__ PlainSum part[NODE_THREADS / 32];
    __shared__ float wsum[NODE_THREADS / 32], carry;
    if (blockIdx.x >= lists.slots()) return;
    const uint4 slot = lists.tiled[blockIdx.x];
    const uint32_t k = slot.x, nk = slot.w, nch = (nk + CHUNK - 1) / CHUNK, c0 = slot.z * SUB_CHUNKS;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    PlainSum x;
    x.init();
    for (uint32_t j = threadIdx.x; j < nch; j += NODE_THREADS)
        for (int a = 0; a < 3; a++) x.merge(a, csum[3 * (c0 + j) + a], cgrid[3 * (c0 + j) + a]);
    x.warp_merge();
    if (lane == 0) part[warp] = x;
    __syncthreads();
    x = part[0];
    for (int w = 1; w < NODE_THREADS / 32; w++)
        for (int a = 0; a < 3; a++) x.merge(a, part[w].sum[a], part[w].g[a]);
    const float v[3] = {vx, vy, vz};
    for (int a = 0; a < 3; a++) {
        if (x.exact(a)) {
            if (threadIdx.x == 0) L.centre[3 * k + a] = centre_of(x.sum[a], nk, L.box[6 * k + a], v[a]);
            for (uint32_t j = threadIdx.x; j < nch; j += NODE_THREADS) cbase[3 * (c0 + j) + a] = 0;
            continue;
        }
        const int top = max(1, min(254, L.ehi[3 * k + a] + 150 - (window - 1)));
        const float limit = ldexpf(1.0f, x.g[a] + 24);   // (below it float sums are exact)
        if (threadIdx.x == 0) starts[3 * blockIdx.x + a] = make_uint2(0u, 0u);
        __syncthreads();   // the axis before may still set it
        if (threadIdx.x == 0) carry = 0.0f;
        for (uint32_t j0 = 0; j0 < nch; j0 += NODE_THREADS) {
            const uint32_t j = j0 + threadIdx.x;
            const float d = j < nch ? csum[3 * (c0 + j) + a] : 0.0f;
            float s = d;
            for (int off = 1; off < 32; off <<= 1) {
                const float y = __shfl_up_sync(0xffffffffu, s, off);
                if (lane >= (uint32_t)off) s += y;
            }
            if (lane == 31) wsum[warp] = s;
            __syncthreads();
            float before = __shfl_up_sync(0xffffffffu, s, 1);
            before = lane ? before : 0.0f;
            for (uint32_t w = 0; w < warp; w++) before += wsum[w];
            before += carry;
            if (j < nch) {
                const uint32_t e = __float_as_uint(before * (63.0f / 64.0f)) >> 23;
                cbase[3 * (c0 + j) + a] = (uint8_t)(window > 2 ? (uint32_t)top : max(1u, min(e, 253u)));
                if (before < limit && before + d >= limit)
                    starts[3 * blockIdx.x + a] = make_uint2(j, __float_as_uint(before));
            }
            __syncthreads();
            if (threadIdx.x == NODE_THREADS - 1) carry = before + d;
        }
    }
}

__device__ __forceinline__ size_t map_index(uint64_t maxc, int window, int a, uint32_t c, int bi)
{
    return ((size_t)a * maxc + c) * window + bi;
}

// Maps of one chunk of a big node for the `window` binades from its base on,
// per axis that needs them.
__global__ void __launch_bounds__(CHUNK_THREADS) k_chunk_maps(const float *P, Level L, NodeLists lists,
                                                             const uint8_t *cbase, int window, uint2 *maps,
                                                             uint64_t maxc)
{
    after_previous();
    __shared__ Tr part[NBIN][3][CHUNK_THREADS / 32];
    const uint32_t c = blockIdx.x;
    ChunkRange r;
    if (!r.find(lists, L, c)) return;
    const int base[3] = {cbase[3 * c], cbase[3 * c + 1], cbase[3 * c + 2]};
    if (!(base[0] | base[1] | base[2])) return;
    const uint64_t t0 = r.b + (uint64_t)threadIdx.x * 8, e = r.e;
    float d[8][3];
    uint32_t cnt = t0 < e ? (uint32_t)(e - t0 < 8 ? e - t0 : 8) : 0u;
    for (int q = 0; q < 8; q++)
        for (int a = 0; a < 3; a++)
            d[q][a] = (uint32_t)q < cnt ? __fsub_rn(P[3 * (t0 + q) + a], L.box[6 * (size_t)r.k + a]) : 0.0f;
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int bi = 0; bi < window; bi++)
        for (int a = 0; a < 3; a++) {
            if (!base[a]) continue;
            Tr t = tr_id();
            for (int q = 0; q < 8; q++)
                if ((uint32_t)q < cnt) t = tr_cat(t, tr_elem(d[q][a], base[a] + bi - 150));
            for (int off = 1; off < 32; off <<= 1) {
                Tr u = tr_shfl_down(t, off);
                if ((lane & (2 * off - 1)) == 0) t = tr_cat(t, u);
            }
            if (lane == 0) part[bi][a][warp] = t;
        }
    __syncthreads();
    if (threadIdx.x < (uint32_t)window * 3) {
        int bi = threadIdx.x / 3, a = threadIdx.x % 3;
        if (!base[a]) return;
        Tr t = part[bi][a][0];
        for (int w = 1; w < CHUNK_THREADS / 32; w++) t = tr_cat(t, part[bi][a][w]);
        maps[map_index(maxc, window, a, c, bi)] = make_uint2(t.w0, t.w1);
    }
}

// acc plus the d of positions [b, e) in order, by one warp (every lane returns
// the same sum): 128 voxels a step, 4 consecutive ones per lane.  A scan of the
// lanes' maps of the binade acc is in adds all of them up to the first lane
// in which the sum leaves it; that lane's four are added one at a time, and
// the scan goes on behind it in the new binade.
__device__ float warp_sum(const float *P, uint64_t b, uint64_t e, int a, float mn, float acc)
{
    const uint32_t lane = threadIdx.x & 31;
    float nx[4];
    for (int j = 0; j < 4; j++) {
        uint64_t t = b + 4 * (uint64_t)lane + j;
        nx[j] = t < e ? P[3 * t + a] : mn;
    }
    for (uint64_t s = b; s < e; s += 128) {
        float d[4];
        for (int j = 0; j < 4; j++) d[j] = __fsub_rn(nx[j], mn);   // past e: +0, which changes no sum
        for (int j = 0; j < 4; j++) {                              // the next step's voxels, in flight meanwhile
            uint64_t t = s + 128 + 4 * (uint64_t)lane + j;
            nx[j] = t < e ? P[3 * t + a] : mn;
        }
        for (uint32_t done = 0; done < 32;) {                      // lanes below `done` are added
            uint32_t f = done;                                     // the next lane to add one at a time
            const uint32_t bits = __float_as_uint(acc), E = bits >> 23, A = (bits & 0x7FFFFFu) | 0x800000u;
            if (acc == 0.0f) {
                const bool some = lane >= done && !(d[0] == 0.0f && d[1] == 0.0f && d[2] == 0.0f && d[3] == 0.0f);
                const uint32_t any = __ballot_sync(0xffffffffu, some);
                f = any ? (uint32_t)__ffs((int)any) - 1u : 32u;
            } else if (E >= 1u && E < 255u) {
                const int ee = (int)E - 150;
                Tr t = tr_id();
                if (lane >= done)
                    t = tr_cat(tr_cat(tr_elem(d[0], ee), tr_elem(d[1], ee)), tr_cat(tr_elem(d[2], ee), tr_elem(d[3], ee)));
                for (int off = 1; off < 32; off <<= 1) {
                    const Tr u = {__shfl_up_sync(0xffffffffu, t.w0, off), __shfl_up_sync(0xffffffffu, t.w1, off)};
                    if (lane >= (uint32_t)off) t = tr_cat(u, t);
                }
                const uint32_t An = A + (((A & 1u) ? t.w1 : t.w0) & 0x7FFFFFFFu);
                const uint32_t leaves = __ballot_sync(0xffffffffu, An >= (1u << 24));
                f = leaves ? (uint32_t)__ffs((int)leaves) - 1u : 32u;
                const uint32_t Af = __shfl_sync(0xffffffffu, An, f ? f - 1u : 0u);
                if (f) acc = __uint_as_float((E << 23) | (Af & 0x7FFFFFu));
            }
            if (f < 32)
                for (int j = 0; j < 4; j++) acc = __fadd_rn(__shfl_sync(0xffffffffu, d[j], f), acc);
            done = f + 1;
        }
    }
    return acc;
}

// Centres of the other big nodes: a warp per (node, axis) walks the node's
// chunks from where additions may round, 32 at a time: a scan of their maps of
// the binade the sum is in gives the sum after each, up to the first chunk in
// which it leaves the binade (or which has no map of it); that chunk is added
// by its voxels.  The next 32 chunks' bases and sums, and with two maps a
// chunk the maps, are loaded meanwhile: the walk is one warp's chain.
constexpr int CENTRE_WARPS = 4;

struct ChunkMaps {
    int base;
    bool some;       // the chunk's sum is not zero
    uint4 two;       // its maps (window 2)
    __device__ __forceinline__ void load(const uint2 *maps, const uint8_t *cbase, const float *csum, int window,
                                         uint64_t maxc, int a, uint32_t c, bool in)
    {
        base = 0;
        some = false;
        two = make_uint4(0u, 0u, 0u, 0u);
        if (!in) return;
        base = cbase[3 * c + a];
        some = csum[3 * c + a] != 0.0f;
        if (window == 2) two = *reinterpret_cast<const uint4 *>(maps + map_index(maxc, 2, a, c, 0));
    }
};

__global__ void __launch_bounds__(CENTRE_WARPS * 32) k_centre_big(const float *P, Level L, NodeLists lists,
                                                                  const uint2 *maps,
                                                                  const uint8_t *cbase, const float *csum, int window,
                                                                  const uint2 *starts, uint64_t maxc, float vx, float vy,
                                                                  float vz)
{
    after_previous();
    uint32_t w = (uint32_t)(((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const uint32_t lane = threadIdx.x & 31;
    uint32_t j = w / 3;
    int a = (int)(w % 3);
    if (j >= lists.slots()) return;
    const uint4 slot = lists.tiled[j];
    const uint32_t k = slot.x, c0 = slot.z * SUB_CHUNKS;
    if (L.kind[k] != K_INNER || !cbase[3 * c0 + a]) return;
    const uint32_t nk = slot.w, nch = (nk + CHUNK - 1) / CHUNK;
    const uint64_t s = L.start[k], end = s + nk;
    const uint2 first = starts[3 * j + a];
    float mn = L.box[6 * k + a], acc = __uint_as_float(first.y);
    uint32_t g = first.x;
    ChunkMaps now, next;
    now.load(maps, cbase, csum, window, maxc, a, c0 + g + lane, g + lane < nch);
    for (; g < nch; g += 32) {
        next.load(maps, cbase, csum, window, maxc, a, c0 + g + 32 + lane, g + 32 + lane < nch);
        const uint32_t cnt = min(32u, nch - g);
        for (uint32_t done = 0; done < cnt;) {            // chunks before g + done are added
            uint32_t f = done;                            // the next chunk to add by its voxels
            const uint32_t bits = __float_as_uint(acc), E = bits >> 23, A = (bits & 0x7FFFFFu) | 0x800000u;
            if (acc == 0.0f) {                            // chunks of zeros change nothing
                const uint32_t some = __ballot_sync(0xffffffffu, lane >= done && now.some);
                f = some ? (uint32_t)__ffs((int)some) - 1u : cnt;
            } else if (E >= 1u && E < 255u) {
                const int bi = (int)E - now.base;
                Tr t = tr_id();
                if (lane >= done && lane < cnt) {
                    t = {SAT, SAT | 0x80000000u};
                    if (bi >= 0 && bi < window) {
                        uint2 m = bi ? make_uint2(now.two.z, now.two.w) : make_uint2(now.two.x, now.two.y);
                        if (window != 2) m = maps[map_index(maxc, window, a, c0 + g + lane, bi)];
                        t = {m.x, m.y};
                    }
                }
                for (int off = 1; off < 32; off <<= 1) {
                    const Tr u = {__shfl_up_sync(0xffffffffu, t.w0, off), __shfl_up_sync(0xffffffffu, t.w1, off)};
                    if (lane >= (uint32_t)off) t = tr_cat(u, t);
                }
                const uint32_t An = A + (((A & 1u) ? t.w1 : t.w0) & 0x7FFFFFFFu);
                const uint32_t leaves = __ballot_sync(0xffffffffu, An >= (1u << 24));
                f = leaves ? (uint32_t)__ffs((int)leaves) - 1u : cnt;
                const uint32_t Af = __shfl_sync(0xffffffffu, An, f ? f - 1u : 0u);
                if (f) acc = __uint_as_float((E << 23) | (Af & 0x7FFFFFu));
            }
            if (f < cnt) {
                const uint64_t b = s + (uint64_t)(g + f) * CHUNK;
                acc = warp_sum(P, b, min(b + CHUNK, end), a, mn, acc);
            }
            done = f + 1;
        }
        now = next;
    }
    float v[3] = {vx, vy, vz};
    if (lane == 0) L.centre[3 * k + a] = centre_of(acc, nk, mn, v[a]);
}

// ---- the swapping passes (sort_set, tree.c:166-183)
//
// A pass needs, at any position, whether its voxel is claimed, how many
// claimed ones stand before it and where the last unclaimed one before it
// stands: a bit per position, and per 32-bit word of them the count and that
// position so far (Marks).  Claimed voxels leave for good, straight to their
// place in the next level's order; only the others move on to the next pass.

// The source of position t (local to the node), which is claimed with c
// claimed positions before it, in a pass whose range starts at `from`: the
// walk back described at the top of the file.  claimed(s, c) says whether
// position s is claimed and gives that count; unclaimed_before(s) gives the
// last unclaimed position before s.  Few walks have more than a step or two
// inside one run, so the first are made one at a time, without looking for
// the run's start (256^3 raw volume with a first frame 1,402 -> 1,376 us with
// 6 of them; 1,397 with 2, 1,357 with 12 or 24, 1,366 with 64).
constexpr uint32_t PLAIN_STEPS = 12;
template <class F, class G>
__device__ __forceinline__ uint32_t walk_back(uint32_t t, uint32_t from, uint32_t limit, uint32_t c, F claimed,
                                              G unclaimed_before, uint32_t *err)
{
    uint32_t s = t;
    for (uint32_t steps = 0;; steps++) {
        uint32_t to = from + c;                            // one step: unclaimed positions before s back
        if (steps >= PLAIN_STEPS && to < s) {              // to before the run's start
            const uint32_t u = s - to, last = unclaimed_before(s);
            if (last < s) to = s - ((s - last - 1) / u + 1) * u;
            else to = s;
        }
        if (to >= s || to < from || steps > limit) {       // impossible for a consistent pass
            atomicOr(err, ERR_WALK);
            return t;
        }
        s = to;
        if (!claimed(s, c)) return s;
    }
}

// Scan of up to 32 * PER words' claimed counts and last unclaimed positions
// by one warp, in place: before[w] and last[w] become those of the words
// before w (from `run` and `prev` on, which advance).
// (Word w's count is before[STRIDE * w].)
template <int PER, int STRIDE>
__device__ __forceinline__ void scan_words(uint32_t *before, uint32_t *last, uint32_t nw, uint32_t &run, uint32_t &prev)
{
    const uint32_t lane = threadIdx.x & 31;
    uint32_t c[PER], l[PER], sum = 0, top = 0;   // top: last position + 1, 0 for none
    for (int j = 0; j < PER; j++) {
        const uint32_t w = lane * PER + j;
        c[j] = w < nw ? before[STRIDE * w] : 0u;
        l[j] = w < nw ? last[w] + 1u : 0u;
        sum += c[j];
        top = max(top, l[j]);
    }
    uint32_t ps = sum, pt = top;
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t a = __shfl_up_sync(0xffffffffu, ps, off), b = __shfl_up_sync(0xffffffffu, pt, off);
        if (lane >= (uint32_t)off) { ps += a; pt = max(pt, b); }
    }
    const uint32_t all = __shfl_sync(0xffffffffu, ps, 31), high = __shfl_sync(0xffffffffu, pt, 31);
    uint32_t r = run + ps - sum, t = __shfl_up_sync(0xffffffffu, pt, 1);
    t = max(lane ? t : 0u, prev + 1u);
    for (int j = 0; j < PER; j++) {
        const uint32_t w = lane * PER + j;
        if (w < nw) { before[STRIDE * w] = r; last[w] = t - 1u; }
        r += c[j];
        t = max(t, l[j]);
    }
    run += all;
    prev = max(prev + 1u, high) - 1u;
}

__device__ __forceinline__ uint32_t lanes_below(uint32_t i) { return (1u << i) - 1u; }

// The last unclaimed position before bit i of word w, whose claimed bits are
// m; positions before `from` are none.  NO_POS when the word has none.
__device__ __forceinline__ uint32_t last_in_word(uint32_t w, uint32_t i, uint32_t m, uint32_t from)
{
    uint32_t u = ~m & lanes_below(i);
    if (w == from >> 5) u &= ~lanes_below(from & 31);
    return u ? (w << 5) + 31u - (uint32_t)__clz((int)u) : NO_POS;
}

// Octants are listed by pass: a pass leaves the places of its octant's voxels,
// in their order, in the buffer that it writes.  The seventh has the eighth's
// there too: nothing but octant 7 is left, and its own pass would move nothing.
// So the octant of a position, given where each octant ends, tells the buffer.
__device__ __forceinline__ uint32_t final_buffer(const uint32_t *ends, uint32_t t)
{
    uint32_t o = 0;
    for (int j = 0; j < 7; j++) o += t >= ends[j];
    return o == 7 ? 1u : (o & 1u) ^ 1u;
}

// Voxel i of one order to place `to` of the next.
__device__ __forceinline__ void place(const float *P, float *Pn, uint64_t to, uint64_t i)
{
    Pn[3 * to] = P[3 * i];
    Pn[3 * to + 1] = P[3 * i + 1];
    Pn[3 * to + 2] = P[3 * i + 2];
}

// Octant of voxel p about centre c (get_subspace_idx, geom.c:44-51).
__device__ __forceinline__ uint32_t octant(const float *c, const float *p)
{
    return (uint32_t)(c[0] > p[0]) | ((uint32_t)(c[1] > p[1]) << 1) | ((uint32_t)(c[2] > p[2]) << 2);
}

// What a warp has counted of the nodes it made, added to the level's tally
// when it leaves.
struct WarpTally {
    uint32_t inner = 0, dense = 0, over = 0, top = 0;
    unsigned long long over_dots = 0;
    // One split node, from its octants' counts (lane o < 8 holds octant o's):
    // an overflowed leaf when one octant took the whole set (tree.c:281-305).
    // Returns its child mask.
    __device__ uint32_t split(const Level &L, uint32_t k, uint32_t n, uint32_t cnt, uint32_t *err)
    {
        const uint32_t lane = threadIdx.x & 31;
        if (lane < 8) L.cnt[8 * (size_t)k + lane] = cnt;
        const uint32_t mask = __ballot_sync(0xffffffffu, lane < 8 && cnt), most = __reduce_max_sync(0xffffffffu, lane < 8 ? cnt : 0u);
        if (most == n) {
            over++;
            over_dots += n;
            if (lane == 0) {
                L.kind[k] = K_OVER;
                if (n >= (1u << 30)) atomicOr(err, ERR_BIG_LEAF);
            }
            return 0u;
        }
        inner++;
        top = max(top, most);
        if (lane == 0) L.mask[k] = (uint8_t)mask;
        return mask;
    }
    __device__ void flush(const Tally &t) const
    {
        if (threadIdx.x & 31) return;
        if (inner) {
            atomicAdd(&t.stats[S_INNER], (unsigned long long)inner);
            atomicMax(t.largest, top);
        }
        if (dense) atomicAdd(&t.stats[S_DENSE], (unsigned long long)dense);
        if (over) {
            atomicAdd(&t.stats[S_LEAF], (unsigned long long)over);
            atomicAdd(&t.stats[S_OVER], (unsigned long long)over);
            atomicAdd(&t.stats[S_DOTS], over_dots);
        }
    }
};

// A float's bits in an order that unsigned comparison follows, and back.
__device__ __forceinline__ uint32_t ordered(float f)
{
    const uint32_t b = __float_as_uint(f);
    return b ^ ((uint32_t)((int)b >> 31) | 0x80000000u);
}
__device__ __forceinline__ float unordered(uint32_t u)
{
    return __uint_as_float(u ^ ((u >> 31) ? 0x80000000u : 0xFFFFFFFFu));
}

// Nodes of VOX_MAX_DOTS+1..MOST voxels, up to 32 of them to a warp at a time.
// Each node's box, density, centre and octants are the warp's work, in
// registers; then every lane makes the passes over one node of its own,
// as the reference makes them (swap each claimed voxel to the front), in a
// column of shared memory; then the warp moves each node's voxels and takes
// the children's places in the next level, all with one atomic.
//
// What bounds the parallel form of a pass is instruction issue (945 of them a
// voxel and level in the block kernel below); the serial one takes five steps
// of ten instructions a voxel, and there are enough nodes for the lanes.  The
// two levels of the 256^3 set where most nodes have 8 to 128 voxels took
// 291 us with a warp on every pass, 160 like this.
constexpr int LANE_WARPS = 4;
template <uint32_t MOST>
__device__ __forceinline__ void nodes_lanes(const Level &L, const uint32_t *list, const uint32_t *count, const float *P,
                                            float *Pn, float vx, float vy, float vz, const Tally &tally)
{
    static_assert(MOST % 32 == 0 && MOST <= 128, "octants are counted in bytes");
    constexpr uint32_t FULL = 0xffffffffu, J = MOST / 32;
    __shared__ uint16_t columns[LANE_WARPS][MOST][32];   // per voxel of 32 nodes {octant, place in the node}
    uint16_t (*col)[32] = columns[threadIdx.x >> 5];
    const uint32_t lane = threadIdx.x & 31, total = *count;
    const uint32_t warps = gridDim.x * LANE_WARPS, per = min(32u, max(1u, (total + warps - 1) / warps));
    const float v[3] = {vx, vy, vz};
    WarpTally mine;
    for (uint32_t b = (blockIdx.x * LANE_WARPS + (threadIdx.x >> 5)) * per; b < total; b += warps * per) {
        const uint32_t here = min(per, total - b);
        uint32_t my = NONE, my_n = 0, c03 = 0, c47 = 0;   // this lane's node, its octants' counts (a byte each)
        uint64_t my_s = 0;
        if (lane < here) {
            my = list[b + lane];
            my_n = L.n[my];
            my_s = L.start[my];
        }
        bool split = false;
        for (uint32_t q = 0; q < here; q++) {
            const uint32_t k = __shfl_sync(FULL, my, q), n = __shfl_sync(FULL, my_n, q);
            const uint64_t s0 = __shfl_sync(FULL, my_s, q);
            float p[J][3], mn[3], mx[3];
            for (uint32_t j = 0; j < J; j++)
                for (int a = 0; a < 3; a++) p[j][a] = j * 32 + lane < n ? P[3 * (s0 + j * 32 + lane) + a] : 0.0f;
            for (int a = 0; a < 3; a++) {
                float lo = INFINITY, hi = -INFINITY;      // NaN is never an extreme
                for (uint32_t j = 0; j < J; j++)
                    if (j * 32 + lane < n) { lo = fminf(lo, p[j][a]); hi = fmaxf(hi, p[j][a]); }
                mn[a] = unordered(__reduce_min_sync(FULL, ordered(lo)));
                mx[a] = unordered(__reduce_max_sync(FULL, ordered(hi)));
                if (mn[a] == 0.0f || mx[a] == 0.0f) {     // the first of equal extremes: -0 equals +0
                    bool found = false;
                    float zero = 0.0f;
                    for (uint32_t j = 0; j < J; j++) {
                        const uint32_t m = __ballot_sync(FULL, j * 32 + lane < n && p[j][a] == 0.0f);
                        const float z = __shfl_sync(FULL, p[j][a], m ? __ffs((int)m) - 1 : 0);
                        if (m && !found) { zero = z; found = true; }
                    }
                    if (mn[a] == 0.0f) mn[a] = zero;
                    if (mx[a] == 0.0f) mx[a] = zero;
                }
                first_nan(__shfl_sync(FULL, p[0][a], 0), mn[a], mx[a]);
            }
            uint32_t kind = 0;
            if (lane == 0) kind = write_box(L, k, n, mn, mx, v);
            kind = __shfl_sync(FULL, kind, 0);
            if (kind != K_INNER) {
                mine.dense++;                             // above VOX_MAX_DOTS voxels it is no leaf
                continue;
            }
            if (lane == q) split = true;
            float c[3];
            PlainSum x;
            x.init();
            for (uint32_t j = 0; j < J; j++)
                if (j * 32 + lane < n)
                    for (int a = 0; a < 3; a++) x.add(a, __fsub_rn(p[j][a], mn[a]));
            for (int a = 0; a < 3; a++) {
                x.g[a] = __reduce_min_sync(FULL, x.g[a]);
                for (int off = 16; off; off >>= 1) x.sum[a] = __fadd_rn(x.sum[a], __shfl_xor_sync(FULL, x.sum[a], off));
            }
            for (int a = 0; a < 3; a++) {
                const float acc = x.exact(a) ? x.sum[a] : warp_sum(P, s0, s0 + n, a, mn[a], 0.0f);
                c[a] = centre_of(acc, n, mn[a], v[a]);
                if (lane == 0) L.centre[3 * (size_t)k + a] = c[a];
            }
            uint32_t n03 = 0, n47 = 0;
            for (uint32_t j = 0; j < J; j++)
                if (j * 32 + lane < n) {
                    const uint32_t o = octant(c, p[j]);
                    col[j * 32 + lane][q] = (uint16_t)((o << 13) | (j * 32 + lane));
                    if (o < 4) n03 += 1u << (8 * o);
                    else n47 += 1u << (8 * (o - 4));
                }
            n03 = __reduce_add_sync(FULL, n03);
            n47 = __reduce_add_sync(FULL, n47);
            if (lane == q) { c03 = n03; c47 = n47; }
        }
        __syncwarp();
        if (split) {                                      // sort_set, tree.c:166-183, on the lane's own node
            uint32_t at = 0;
            for (uint32_t o = 0; o < 7; o++) {            // (the last has nothing to move)
                const uint32_t end = at + (((o < 4 ? c03 : c47) >> (8 * (o & 3))) & 0xFFu);
                uint32_t i = at;
                uint16_t x = at < end ? col[i][lane] : 0;
                while (at < end) {                        // until the octant's last voxel is placed
                    const uint16_t next = i + 1 < my_n ? col[i + 1][lane] : 0;
                    if ((uint32_t)(x >> 13) == o) {
                        col[i][lane] = col[at][lane];
                        col[at][lane] = x;
                        at++;
                    }
                    x = next;
                    if (++i > my_n) {                     // impossible: the counts are of these voxels
                        atomicOr(tally.err, ERR_WALK);
                        break;
                    }
                }
            }
        }
        __syncwarp();
        uint32_t kids = 0;
        for (uint32_t q = 0; q < here; q++) {
            if (!__shfl_sync(FULL, (int)split, q)) continue;
            const uint32_t k = __shfl_sync(FULL, my, q), n = __shfl_sync(FULL, my_n, q), n03 = __shfl_sync(FULL, c03, q),
                           n47 = __shfl_sync(FULL, c47, q);
            const uint64_t s0 = __shfl_sync(FULL, my_s, q);
            for (uint32_t t = lane; t < n; t += 32) place(P, Pn, s0 + t, s0 + (col[t][q] & 8191u));
            const uint32_t mask = mine.split(L, k, n, ((lane < 4 ? n03 : n47) >> (8 * (lane & 3))) & 0xFFu, tally.err);
            if (lane == q) kids = (uint32_t)__popc(mask);
        }
        const uint32_t incl = warp_incl_scan(kids);
        uint32_t first = 0;
        if (lane == 31 && incl) first = atomicAdd(tally.children, incl);
        first = __shfl_sync(FULL, first, 31) + incl - kids;
        if (kids) L.first_child[my] = first;
        __syncwarp();
    }
    mine.flush(tally);
}

template <uint32_t MOST>
__global__ void __launch_bounds__(LANE_WARPS * 32) k_nodes_lanes(Level L, const uint32_t *list, const uint32_t *count,
                                                                 const float *P, float *Pn, float vx, float vy, float vz,
                                                                 Tally tally, bool first)
{
    class_begin(first);
    nodes_lanes<MOST>(L, list, count, P, Pn, vx, vy, vz, tally);
    class_end(first);
}

// Nodes of at most MOST voxels: a block of THREADS each, as above, a voxel in
// 16 bits {octant, place in the node}, or above 8,192 voxels in 24.  (A level
// of 64 nodes of 21,000 tile by tile is eighteen launches, 210 us; by a block
// each the raw volume's 1,600 us become 1,566, a build of 13.8 M voxels 13.0 ms
// 11.5.)
template <uint32_t MOST, bool WIDE = (MOST > 8192)>
struct NodeBuffer {                      // two orders of a node's voxels
    uint16_t v[2][MOST];
    __device__ void set(uint32_t i, uint32_t o) { v[0][i] = (uint16_t)((o << 13) | i); }
    __device__ uint32_t oct(uint32_t b, uint32_t t) const { return v[b][t] >> 13; }
    __device__ uint32_t place(uint32_t b, uint32_t t) const { return v[b][t] & 8191u; }
    __device__ void move(uint32_t b, uint32_t t, uint32_t s) { v[b ^ 1][t] = v[b][s]; }
};
template <uint32_t MOST>
struct NodeBuffer<MOST, true> {
    uint16_t v[2][MOST];
    uint8_t q[2][MOST];
    __device__ void set(uint32_t i, uint32_t o) { v[0][i] = (uint16_t)i; q[0][i] = (uint8_t)o; }
    __device__ uint32_t oct(uint32_t b, uint32_t t) const { return q[b][t]; }
    __device__ uint32_t place(uint32_t b, uint32_t t) const { return v[b][t]; }
    __device__ void move(uint32_t b, uint32_t t, uint32_t s) { v[b ^ 1][t] = v[b][s]; q[b ^ 1][t] = q[b][s]; }
};
template <uint32_t MOST>
struct NodeShared {
    NodeBuffer<MOST> buf;
    uint2 word[2][MOST / 32];            // the marks of a pass and of the next: claimed bits, claimed count before
    uint32_t last[2][MOST / 32];         // and the last unclaimed position before
};
template <int THREADS, uint32_t MOST>
__device__ __forceinline__ void nodes_block(const Level &L, const uint32_t *list, const uint32_t *count, const float *P,
                                            float *Pn, float vx, float vy, float vz, const Tally &tally)
{
    static_assert(MOST <= 65536 && MOST % 1024 == 0, "16 bits of place; whole words a lane in scan_words");
    constexpr int WARPS = THREADS / 32;
    static_assert(WARPS >= 3 && WARPS <= 32, "an axis a warp");
    extern __shared__ __align__(16) unsigned char dynamic[];
    NodeShared<MOST> &w = *reinterpret_cast<NodeShared<MOST> *>(dynamic);
    __shared__ uint32_t total, s_kind, ends[8];
    __shared__ Extremes epart[WARPS];
    __shared__ PlainSum spart[WARPS];
    __shared__ float centre[3];
    if (blockIdx.x >= *count) return;
    const uint32_t k = list[blockIdx.x], n = L.n[k], lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t s0 = L.start[k];
    const float v[3] = {vx, vy, vz};
    {
        Extremes e;
        e.init();
        for (uint32_t j = threadIdx.x; j < n; j += THREADS) e.add(P + 3 * (s0 + j), j);
        e.warp_merge();
        if (lane == 0) epart[warp] = e;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int i = 1; i < WARPS; i++) e.merge(epart[i]);
            for (int a = 0; a < 3; a++) first_nan(P[3 * s0 + a], e.mn[a], e.mx[a]);
            s_kind = write_box(L, k, n, e.mn, e.mx, v);
            epart[0] = e;
            if (s_kind == K_DENSE) atomicAdd(&tally.stats[S_DENSE], 1ull);
        }
        __syncthreads();
        if (s_kind != K_INNER) return;
    }
    const float mn[3] = {epart[0].mn[0], epart[0].mn[1], epart[0].mn[2]};
    {
        PlainSum x;
        x.init();
        for (uint32_t j = threadIdx.x; j < n; j += THREADS)
            for (int a = 0; a < 3; a++) x.add(a, __fsub_rn(P[3 * (s0 + j) + a], mn[a]));
        x.warp_merge();
        if (lane == 0) spart[warp] = x;
        __syncthreads();
        if (warp < 3) {             // an axis a warp
            const int a = (int)warp;
            float sum = lane < WARPS ? spart[lane].sum[a] : 0.0f;
            for (int off = 16; off; off >>= 1) sum = __fadd_rn(sum, __shfl_xor_sync(0xffffffffu, sum, off));
            x.sum[a] = sum;
            x.g[a] = __reduce_min_sync(0xffffffffu, lane < WARPS ? spart[lane].g[a] : 1000);
            const float acc = x.exact(a) ? sum : warp_sum(P, s0, s0 + n, a, mn[a], 0.0f);
            if (lane == 0) L.centre[3 * (size_t)k + a] = centre[a] = centre_of(acc, n, mn[a], v[a]);
        }
        __syncthreads();
    }
    const uint32_t nw = (n + 31) / 32;
    auto mark = [&](uint32_t b, uint32_t i, bool cl, bool un) {   // word i's claimed and unclaimed flags
        const uint32_t m = __ballot_sync(0xffffffffu, cl), u = __ballot_sync(0xffffffffu, un);
        if (lane == 0) {
            w.word[b][i] = make_uint2(m, (uint32_t)__popc(m));
            w.last[b][i] = u ? (i << 5) + 31u - (uint32_t)__clz((int)u) : NO_POS;
        }
    };
    for (uint32_t i = warp; i < nw; i += WARPS) {
        const uint32_t t = (i << 5) + lane;
        uint32_t q = 8;
        if (t < n) {
            const float p[3] = {P[3 * (s0 + t)], P[3 * (s0 + t) + 1], P[3 * (s0 + t) + 2]};
            q = octant(centre, p);
            w.buf.set(t, q);
        }
        mark(0, i, q == 0, t < n && q != 0);
    }
    if (threadIdx.x < 8) ends[threadIdx.x] = n;
    uint32_t from = 0, cnt = 0;     // lane o of warp 0 holds octant o's count
    for (uint32_t o = 0; o < 7 && from < n; o++) {
        const uint32_t in = o & 1, *const last = w.last[in];
        const uint2 *const word = w.word[in];
        __syncthreads();
        if (warp == 0) {
            constexpr uint32_t PER = MOST / 1024 < 8 ? MOST / 1024 : 8;
            uint32_t run = 0, prev = NO_POS;
            for (uint32_t i = from >> 5; i < nw; i += 32 * PER)
                scan_words<PER, 2>(&w.word[in][i].y, w.last[in] + i, min(nw - i, 32 * PER), run, prev);
            if (lane == 0) {
                total = run;
                ends[o] = from + run;
            }
            if (lane == o) cnt = run;
        }
        __syncthreads();
        const uint32_t rest = from + total;
        auto claimed = [&](uint32_t s, uint32_t &c) {
            const uint2 m = word[s >> 5];
            c = m.y + (uint32_t)__popc(m.x & lanes_below(s & 31));
            return ((m.x >> (s & 31)) & 1u) != 0u;
        };
        auto unclaimed_before = [&](uint32_t s) {
            const uint32_t l = last_in_word(s >> 5, s & 31, word[s >> 5].x, from);
            return l != NO_POS ? l : last[s >> 5];
        };
        for (uint32_t i = (from >> 5) + warp; i < nw; i += WARPS) {
            const uint32_t t = (i << 5) + lane;
            const bool left = t >= rest && t < n;
            uint32_t q = 8;
            if (t >= from && t < n) {
                uint32_t c, s = t;
                if (claimed(t, c)) {
                    w.buf.move(in, from + c, t);
                    if (left) s = walk_back(t, from, MOST, c, claimed, unclaimed_before, tally.err);
                }
                if (left) {
                    w.buf.move(in, t, s);
                    q = w.buf.oct(in, s);
                }
            }
            if (o < 6) mark(in ^ 1, i, q == o + 1, left && q != o + 1);
        }
        from = rest;
    }
    if (warp == 0 && lane == 7) cnt = n - from;
    __syncthreads();
    // the voxels, all at once (a pass at a time, an eighth of the lanes had a
    // load to wait for; here and tile by tile together, with the eighth pass
    // gone and marks made as voxels move, a 256^3 raw volume 1,496 -> 1,402 us)
    for (uint32_t t0 = threadIdx.x; t0 < n; t0 += 4 * THREADS) {
        float p[4][3];
#pragma unroll
        for (uint32_t j = 0; j < 4; j++) {
            const uint32_t t = t0 + j * THREADS;
            if (t >= n) break;
            const uint64_t i = s0 + w.buf.place(final_buffer(ends, t), t);
            for (int a = 0; a < 3; a++) p[j][a] = P[3 * i + a];
        }
#pragma unroll
        for (uint32_t j = 0; j < 4; j++) {
            const uint32_t t = t0 + j * THREADS;
            if (t >= n) break;
            for (int a = 0; a < 3; a++) Pn[3 * (s0 + t) + a] = p[j][a];
        }
    }
    if (warp == 0) {
        WarpTally mine;
        const uint32_t m = mine.split(L, k, n, cnt, tally.err);
        if (lane == 0 && m) L.first_child[k] = atomicAdd(tally.children, (uint32_t)__popc(m));
        mine.flush(tally);
    }
}

template <int THREADS, uint32_t MOST>
__global__ void __launch_bounds__(THREADS) k_nodes_block(Level L, const uint32_t *list, const uint32_t *count,
                                                         const float *P, float *Pn, float vx, float vy, float vz,
                                                         Tally tally, bool first)
{
    class_begin(first);
    nodes_block<THREADS, MOST>(L, list, count, P, Pn, vx, vy, vz, tally);
    class_end(first);
}

// Larger nodes, tile by tile: a launch a pass, a block a tile of one node.
// The marks of a pass are made by the launch before it (the first ones by
// k_tile_marks): per word as above, counted from the tile's start, and per
// tile the claimed count and the last unclaimed position.  Every block scans
// its node's tiles for itself (at most MAX_TILES).
//
// What bounds a pass is the chain of dependent loads of each word's walk, so
// a warp has few words to go through, and enough for a block's scan to be worth
// it: the 256^3 set's raw build takes 1,349 us with 4 words a warp and 512
// threads, 1,363 with 256 threads, 1,390 with 1,024; with 8 words a warp 1,380
// (256 threads), with 2 1,405 (1,024 threads).
constexpr int PASS_THREADS = 512;

struct Marks {
    uint4 *word;                        // per word of a node, from its first sub on: claimed bits, count before, last before
    uint2 *tile;                        // per tile: claimed count, last unclaimed position + 1 (0: none)
};

// Marks of one SUB of positions from their claimed flags, word by word.  (run
// and prev, what comes before, are warp 0's.)
struct SubMarks {
    uint32_t mask[SUB / 32], before[SUB / 32], last[SUB / 32];
    __device__ void flush(const Marks &m, uint64_t word0, uint32_t nw, uint32_t &run, uint32_t &prev)
    {
        __syncthreads();
        if (threadIdx.x < 32) {
            scan_words<SUB / 32 / 32, 1>(before, last, nw, run, prev);
            __syncwarp();
            for (uint32_t w = threadIdx.x; w < nw; w += 32)
                m.word[word0 + w] = make_uint4(mask[w], before[w], last[w], 0u);
        }
        __syncthreads();
    }
};

// Octants, and the marks of octant 0 over the given order.
__global__ void __launch_bounds__(PASS_THREADS) k_tile_marks(Level L, NodeLists lists, const float *P, uint8_t *oct,
                                                             Marks out)
{
    after_previous();
    __shared__ SubMarks sub;
    TileRange range;
    if (!range.find(lists)) return;
    const uint32_t k = range.k, b = range.b, e = range.e, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (L.kind[k] != K_INNER) return;
    const uint64_t start = L.start[k];
    const float centre[3] = {L.centre[3 * (size_t)k], L.centre[3 * (size_t)k + 1], L.centre[3 * (size_t)k + 2]};
    if (b == 0 && threadIdx.x < 8) L.cnt[8 * (size_t)k + threadIdx.x] = 0;
    uint64_t word0 = range.words() + b / 32;
    uint32_t run = 0, prev = NO_POS;
    for (uint32_t sb = b; sb < e; sb += SUB, word0 += SUB / 32) {
        const uint32_t nw = (min(e - sb, SUB) + 31) / 32;
        for (uint32_t w = warp; w < nw; w += PASS_THREADS / 32) {
            const uint32_t t = sb + (w << 5) + lane;
            const bool in = t < e;
            uint32_t q = 0xFF;
            if (in) {
                q = octant(centre, P + 3 * (start + t));
                oct[start + t] = (uint8_t)q;
            }
            const bool cl = q == 0;
            const uint32_t m = __ballot_sync(0xffffffffu, cl), u = __ballot_sync(0xffffffffu, in && !cl);
            if (lane == 0) {
                sub.mask[w] = m;
                sub.before[w] = (uint32_t)__popc(m);
                sub.last[w] = u ? sb + (w << 5) + 31u - (uint32_t)__clz((int)u) : NO_POS;
            }
        }
        sub.flush(out, word0, nw, run, prev);
    }
    if (threadIdx.x == 0) out.tile[blockIdx.x] = make_uint2(run, prev + 1u);
}

// Pass o over every tiled node.
__global__ void __launch_bounds__(PASS_THREADS) k_tile_pass(Level L, NodeLists lists, uint32_t o, Marks in, Marks out,
                                                            const uint32_t *in_idx, const uint8_t *in_oct,
                                                            uint32_t *out_idx, uint8_t *out_oct, uint32_t *err)
{
    __shared__ SubMarks sub;
    __shared__ uint32_t tbefore[MAX_TILES], tlast[MAX_TILES];
    __shared__ uint32_t wsum[PASS_THREADS / 32], wtop[PASS_THREADS / 32];
    TileRange range;
    if (!range.find(lists)) return;
    const uint32_t k = range.k, n = range.n, ft = range.ft, shift = range.shift, b = range.b, e = range.e,
                   lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t words = range.words();
    const uint64_t start = L.start[k];
    const bool inner = L.kind[k] == K_INNER;
    after_previous();                          // the marks and counts of the pass before
    if (!inner) return;
    uint32_t from = 0;
    for (uint32_t q = 0; q < o; q++) from += L.cnt[8 * (size_t)k + q];
    if (e <= from) return;                     // all of it placed by earlier passes
    const uint32_t t0 = from >> shift, nt = parts(n, shift) - t0;   // the tiles still in play
    // what comes before each of them: a run of tiles a thread, scanned over the block
    constexpr uint32_t PER = MAX_TILES / PASS_THREADS;
    const uint32_t i0 = threadIdx.x * PER;
    uint2 t[PER];
    uint32_t sum = 0, top = 0;
    for (uint32_t j = 0; j < PER; j++) {
        t[j] = i0 + j < nt ? in.tile[ft + t0 + i0 + j] : make_uint2(0u, 0u);
        sum += t[j].x;
        top = max(top, t[j].y);
    }
    uint32_t ps = sum, pt = top;
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t x = __shfl_up_sync(0xffffffffu, ps, off), y = __shfl_up_sync(0xffffffffu, pt, off);
        if (lane >= (uint32_t)off) { ps += x; pt = max(pt, y); }
    }
    if (lane == 31) { wsum[warp] = ps; wtop[warp] = pt; }
    __syncthreads();
    uint32_t total = 0, before = ps - sum, above = __shfl_up_sync(0xffffffffu, pt, 1);
    if (lane == 0) above = 0;
    for (uint32_t w = 0; w < PASS_THREADS / 32; w++) {
        if (w < warp) { before += wsum[w]; above = max(above, wtop[w]); }
        total += wsum[w];
    }
    for (uint32_t j = 0; j < PER; j++) {
        if (i0 + j < nt) { tbefore[i0 + j] = before; tlast[i0 + j] = above - 1u; }
        before += t[j].x;
        above = max(above, t[j].y);
    }
    const uint32_t rest = from + total;
    if (e == n && threadIdx.x == 0) {          // read by later launches only
        L.cnt[8 * (size_t)k + o] = total;
        if (o == 6) L.cnt[8 * (size_t)k + 7] = n - rest;
    }
    __syncthreads();
    auto claimed = [&](uint32_t s, uint32_t &c) {
        const uint4 word = in.word[words + (s >> 5)];
        c = tbefore[(s >> shift) - t0] + word.y + (uint32_t)__popc(word.x & lanes_below(s & 31));
        return ((word.x >> (s & 31)) & 1u) != 0u;
    };
    auto unclaimed_before = [&](uint32_t s) {
        const uint4 word = in.word[words + (s >> 5)];
        uint32_t l = last_in_word(s >> 5, s & 31, word.x, from);
        if (l == NO_POS) l = word.z;
        return l != NO_POS ? l : tlast[(s >> shift) - t0];
    };
    uint32_t run = 0, prev = NO_POS;
    for (uint32_t sb = b; sb < e; sb += SUB) {
        const uint32_t nw = (min(e - sb, SUB) + 31) / 32;
        for (uint32_t w = warp; w < nw; w += PASS_THREADS / 32) {
            const uint32_t t = sb + (w << 5) + lane;
            const bool left = t >= rest && t < e;
            uint8_t q = 0xFF;
            if (t >= from && t < e) {
                q = in_oct[start + t];
                const uint32_t own = o == 0 ? (uint32_t)start + t : in_idx[start + t];
                uint32_t c, src = own;
                const bool taken = claimed(t, c);
                if (taken && left) {
                    const uint32_t s = walk_back(t, from, 1u << 22, c, claimed, unclaimed_before, err);
                    q = in_oct[start + s];
                    src = o == 0 ? (uint32_t)start + s : in_idx[start + s];
                }
                if (taken) out_idx[start + from + c] = own;
                if (left) {
                    out_idx[start + t] = src;
                    out_oct[start + t] = q;
                }
            }
            const bool cl = left && q == o + 1;
            const uint32_t m = __ballot_sync(0xffffffffu, cl), u = __ballot_sync(0xffffffffu, left && !cl);
            if (lane == 0) {
                sub.mask[w] = m;
                sub.before[w] = (uint32_t)__popc(m);
                sub.last[w] = u ? sb + (w << 5) + 31u - (uint32_t)__clz((int)u) : NO_POS;
            }
        }
        sub.flush(out, words + (sb >> 5), nw, run, prev);
    }
    if (threadIdx.x == 0) out.tile[blockIdx.x] = make_uint2(run, prev + 1u);
}

// The voxels of tiled nodes in their order after the passes, a block a tile.
__global__ void __launch_bounds__(PASS_THREADS) k_tile_gather(Level L, NodeLists lists, const uint32_t *idx0,
                                                              const uint32_t *idx1, const float *P, float *Pn)
{
    after_previous();
    TileRange range;
    if (!range.find(lists)) return;
    const uint32_t k = range.k, b = range.b, e = range.e;
    if (L.kind[k] != K_INNER) return;
    const uint64_t start = L.start[k];
    uint32_t ends[7], sum = 0;
    for (int o = 0; o < 7; o++) ends[o] = sum += L.cnt[8 * (size_t)k + o];
    constexpr uint32_t PER = SUB / PASS_THREADS;
    for (uint32_t t0 = b + threadIdx.x; t0 < e; t0 += SUB) {
        uint32_t i[PER];
        float p[PER][3];
#pragma unroll
        for (uint32_t j = 0; j < PER; j++) {
            const uint32_t t = min(t0 + j * PASS_THREADS, e - 1);
            i[j] = (final_buffer(ends, t) ? idx1 : idx0)[start + t];
        }
#pragma unroll
        for (uint32_t j = 0; j < PER; j++)
            for (int a = 0; a < 3; a++) p[j][a] = P[3 * (uint64_t)i[j] + a];
#pragma unroll
        for (uint32_t j = 0; j < PER; j++) {
            const uint32_t t = t0 + j * PASS_THREADS;
            if (t < e)
                for (int a = 0; a < 3; a++) Pn[3 * (start + t) + a] = p[j][a];
        }
    }
}

// Tiled nodes after their passes, a warp each.
__global__ void k_finish_tiled(Level L, NodeLists lists, Tally tally)
{
    after_previous();
    const uint32_t slot = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (slot >= lists.slots()) return;
    const uint32_t k = lists.tiled[slot].x;
    if (L.kind[k] != K_INNER) return;
    WarpTally mine;
    const uint32_t m = mine.split(L, k, lists.tiled[slot].w, lane < 8 ? L.cnt[8 * (size_t)k + lane] : 0u, tally.err);
    if (lane == 0 && m) L.first_child[k] = atomicAdd(tally.children, (uint32_t)__popc(m));
    mine.flush(tally);
}

// The set into the first level's order; *odd is set when a coordinate is not
// finite, above LIMIT in magnitude or below LEAST and not zero.
constexpr float LIMIT = 1.4411518807585587e17f;    // 2^57
constexpr float LEAST = 2.7755575615628914e-17f;   // 2^-55
__device__ __forceinline__ bool ordinary_coordinate(float v)
{
    return v == 0.0f || (fabsf(v) >= LEAST && fabsf(v) <= LIMIT);
}
__global__ void __launch_bounds__(256) k_copy_set(const float *__restrict__ set, float *__restrict__ P, uint64_t n,
                                                  uint32_t *odd)
{
    after_previous();
    const uint64_t i0 = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    bool fine = true;
    if (i0 + 4 <= n && (reinterpret_cast<uintptr_t>(set) & 15u) == 0) {
        const float4 v = *reinterpret_cast<const float4 *>(set + i0);
        fine = ordinary_coordinate(v.x) && ordinary_coordinate(v.y) && ordinary_coordinate(v.z) && ordinary_coordinate(v.w);
        *reinterpret_cast<float4 *>(P + i0) = v;
    } else {
        for (uint64_t i = i0; i < n && i < i0 + 4; i++) {
            const float v = set[i];
            fine = fine && ordinary_coordinate(v);
            P[i] = v;
        }
    }
    if (__any_sync(0xffffffffu, !fine) && (threadIdx.x & 31) == 0) *odd = 1u;
}

// A new node of n voxels from position s0 on (n 0: none; every thread of the
// warp calls): made here when it has at most VOX_MAX_DOTS voxels (a leaf, or
// dense), else put on the list of its class.
__device__ __forceinline__ void new_node(const Level &L, uint32_t k, uint32_t s0, uint32_t n, const float *P, const float *v,
                                         const NodeLists &lists, uint32_t &leaves, uint32_t &dense, uint32_t &dots)
{
    constexpr uint32_t FULL = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31;
    if (n) {
        L.start[k] = s0;
        L.n[k] = n;
    }
    if (n && n <= VOX_MAX_DOTS) {
        const float *p = P + 3 * (uint64_t)s0;
        float mn[3] = {p[0], p[1], p[2]}, mx[3] = {p[0], p[1], p[2]};
        for (uint32_t i = 1; i < n; i++)
            for (int a = 0; a < 3; a++) {
                const float x = p[3 * i + a];
                if (x < mn[a]) mn[a] = x;
                else if (x > mx[a]) mx[a] = x;
            }
        if (write_box(L, k, n, mn, mx, v) == K_DENSE) {
            dense++;
        } else {
            leaves++;
            dots += n;
        }
    }
    if (n > TINY) lists.add_large(k, n);
    const bool tiny = n > VOX_MAX_DOTS && n <= TINY;
    const uint32_t m = __ballot_sync(FULL, tiny);
    uint32_t at = 0;
    if (lane == 0 && m) at = atomicAdd(lists.ntiny, (uint32_t)__popc(m));
    at = __shfl_sync(FULL, at, 0) + (uint32_t)__popc(m & ((1u << lane) - 1u));
    if (tiny) lists.tiny[at] = k;
}

// The next level's nodes: a thread per octant of every node of this one.
constexpr int CHILD_THREADS = 256;
__global__ void __launch_bounds__(CHILD_THREADS) k_children(Level L, Level Nx, NodeLists lists, const float *P, float vx,
                                                            float vy, float vz, unsigned long long *stats)
{
    after_previous();
    __shared__ uint32_t sums[3];
    if (threadIdx.x < 3) sums[threadIdx.x] = 0;
    __syncthreads();
    const uint64_t t = (uint64_t)blockIdx.x * CHILD_THREADS + threadIdx.x;
    const uint32_t o = threadIdx.x & 7;
    const size_t k = t >> 3;
    const uint32_t mask = k < L.m ? L.mask[k] : 0u;
    const uint32_t n = mask ? L.cnt[8 * k + o] : 0u;
    uint32_t incl = n;              // over the node's eight octants
    for (int off = 1; off < 8; off <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, off, 8);
        if (o >= (uint32_t)off) incl += y;
    }
    const float v[3] = {vx, vy, vz};
    uint32_t leaves = 0, dense = 0, dots = 0, child = 0, s0 = 0;
    if (n) {
        child = L.first_child[k] + (uint32_t)__popc(mask & ((1u << o) - 1u));
        s0 = L.start[k] + incl - n;
    }
    new_node(Nx, child, s0, n, P, v, lists, leaves, dense, dots);
    leaves = __reduce_add_sync(0xffffffffu, leaves);
    dense = __reduce_add_sync(0xffffffffu, dense);
    dots = __reduce_add_sync(0xffffffffu, dots);
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&sums[0], leaves);
        atomicAdd(&sums[1], dense);
        atomicAdd(&sums[2], dots);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (sums[0]) atomicAdd(&stats[S_LEAF], (unsigned long long)sums[0]);
        if (sums[1]) atomicAdd(&stats[S_DENSE], (unsigned long long)sums[1]);
        if (sums[2]) atomicAdd(&stats[S_DOTS], (unsigned long long)sums[2]);
    }
}

// The root (one warp).
__global__ void k_root_node(Level L, uint32_t n, NodeLists lists, const float *P, float vx, float vy, float vz,
                            unsigned long long *stats)
{
    after_previous();
    const float v[3] = {vx, vy, vz};
    uint32_t leaves = 0, dense = 0, dots = 0;
    new_node(L, 0, 0, threadIdx.x == 0 ? n : 0u, P, v, lists, leaves, dense, dots);
    if (threadIdx.x == 0) {
        stats[S_LEAF] = leaves;
        stats[S_DENSE] = dense;
        stats[S_DOTS] = dots;
        L.id[0] = 0;
        L.rec[0] = 0;
        L.ustart[0] = VOXP_REC_UNITS;
    }
}

// ------------------------------------------------------------------ layout

// Units a node appends to the image (its child block or voxel run), nodes and
// units of its subtree (flatten.cpp's placement).
__global__ void k_up(Level L, Level Nx, bool has_next)
{
    after_previous();
    uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= L.m) return;
    uint8_t kind = L.kind[k];
    uint32_t nch = (uint32_t)__popc(L.mask[k]);
    unsigned long long app = kind == K_INNER ? 3ull * nch : (kind == K_DENSE ? 0ull : L.n[k]);
    uint32_t sn = 1;
    unsigned long long su = app;
    if (kind == K_INNER && has_next) {
        uint32_t f = L.first_child[k];
        for (uint32_t j = 0; j < nch; j++) {
            sn += Nx.sub_nodes[f + j];
            su += Nx.sub_units[f + j];
        }
    }
    L.sub_nodes[k] = sn;
    L.sub_units[k] = su;
}

// Node records (pool_layout.h), the pre-order id map, the voxel runs of leaves
// of at most VOX_MAX_DOTS voxels; and pre-order ids and image offsets of the
// children, for the next level's launch.
__global__ void k_emit(Level L, Level Nx, const float *P, uint4 *pool, uint32_t *rec_of_id, uint64_t units, uint64_t nodes,
                       uint32_t *err, uint32_t *dots_of_id)
{
    after_previous();
    uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= L.m) return;
    uint8_t kind = L.kind[k];
    uint32_t id = L.id[k], rec = L.rec[k], cnt = L.n[k], us = L.ustart[k], meta, link;
    if ((uint64_t)rec + VOXP_REC_UNITS > units || id >= nodes) {   // cannot happen for a consistent layout
        atomicOr(err, ERR_LAYOUT);
        return;
    }
    if (dots_of_id) dots_of_id[id] = cnt;   // the node's dots_num (tree.c:262)
    uint4 extra = make_uint4(0u, 0u, 0u, 0u);
    if (kind == K_DENSE) {
        meta = VOXP_KIND_DENSE;
        link = id;
    } else if (kind == K_INNER) {
        const uint32_t mask = L.mask[k], nch = (uint32_t)__popc(mask), f = L.first_child[k];
        meta = VOXP_KIND_INNER | (mask << 8);
        link = us;
        const float *c = L.centre + 3 * (size_t)k;
        extra = make_uint4(__float_as_uint(c[0]), __float_as_uint(c[1]), __float_as_uint(c[2]), 0u);
        uint32_t cid = id + 1, cu = us + VOXP_REC_UNITS * nch;
        for (uint32_t j = 0; j < nch; j++) {
            Nx.id[f + j] = cid;
            Nx.ustart[f + j] = cu;
            Nx.rec[f + j] = us + VOXP_REC_UNITS * j;
            cid += Nx.sub_nodes[f + j];
            cu += (uint32_t)Nx.sub_units[f + j];
        }
    } else {
        meta = VOXP_KIND_LEAF | (cnt << 2);
        link = us;
        extra = make_uint4(id, cnt, 0u, 0u);
        if ((uint64_t)us + cnt > units) {
            atomicOr(err, ERR_LAYOUT);
        } else if (kind == K_LEAF) {
            const float *p = P + 3 * (uint64_t)L.start[k];
            for (uint32_t i = 0; i < cnt; i++)
                pool[us + i] = make_uint4(__float_as_uint(p[3 * i]), __float_as_uint(p[3 * i + 1]),
                                          __float_as_uint(p[3 * i + 2]), 0u);
        }
    }
    const float *b = L.box + 6 * (size_t)k;
    pool[rec] = make_uint4(__float_as_uint(b[0]), __float_as_uint(b[1]), __float_as_uint(b[2]), __float_as_uint(b[3]));
    pool[rec + 1] = make_uint4(__float_as_uint(b[4]), __float_as_uint(b[5]), meta, link);
    pool[rec + 2] = extra;
    rec_of_id[id] = rec;
}

// Voxel runs of a level's overflowed leaves, a warp per node.
__global__ void k_emit_over(Level L, const float *P, uint4 *pool, uint64_t units, uint32_t *err)
{
    after_previous();
    uint32_t k = (uint32_t)(((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    int lane = threadIdx.x & 31;
    if (k >= L.m || L.kind[k] != K_OVER) return;
    uint64_t s = L.start[k];
    uint32_t u = L.ustart[k], nk = L.n[k];
    if ((uint64_t)u + nk > units) {
        if (lane == 0) atomicOr(err, ERR_LAYOUT);
        return;
    }
    for (uint32_t i = lane; i < nk; i += 32) {
        const float *p = P + 3 * (s + i);
        pool[u + i] = make_uint4(__float_as_uint(p[0]), __float_as_uint(p[1]), __float_as_uint(p[2]), 0u);
    }
}

// The set's final order (tree.c sorts it in place): a level's leaves, a warp
// per node.
__global__ void k_final_order(Level L, const float *P, float *order)
{
    after_previous();
    uint32_t k = (uint32_t)(((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    int lane = threadIdx.x & 31;
    if (k >= L.m || L.kind[k] == K_INNER) return;
    const uint64_t b = 3 * (uint64_t)L.start[k], e = b + 3 * (uint64_t)L.n[k];
    for (uint64_t i = b + lane; i < e; i += 32) order[i] = P[i];
}

// --------------------------------------------------------- host's page

// What comes back to the host while it builds, in page-locked memory: kernels
// write it there, and `step` last.
struct Back {
    uint32_t next[2], root_nodes, err, odd, unshaped, step;
    float box[6];
    unsigned long long units, stats[NSTATS * MAX_LEVELS];
};
static_assert(sizeof(Back) <= THREAD_PAGE, "the counts of every level fit the thread's page");

// A level is split: the next one's nodes and the largest of them, and the
// level's counters zeroed.  The host sees them as soon as they are stored; with
// a copy, a wait for the stream and a memset a level the 256^3 raw volume with
// a first frame took 1,570 us, with this 1,496.
__global__ void k_level_done(uint32_t *scal, Back *back, uint32_t step)
{
    after_previous();
    back->next[0] = scal[2];
    back->next[1] = scal[3];
    for (int i = 0; i < 9; i++) scal[i] = 0;
    __threadfence_system();
    *static_cast<volatile uint32_t *>(&back->step) = step;
}

// The tree is split: every level's counts, and the image's size.
__global__ void __launch_bounds__(128) k_all_done(Level root, const unsigned long long *stats, const uint32_t *err, Back *back, uint32_t step)
{
    after_previous();
    for (int i = threadIdx.x; i < NSTATS * MAX_LEVELS; i += 128) back->stats[i] = stats[i];
    if (threadIdx.x < 6) back->box[threadIdx.x] = root.box[threadIdx.x];
    if (threadIdx.x == 0) {
        back->root_nodes = root.sub_nodes[0];
        back->units = root.sub_units[0];
        back->err = err[0];
        back->odd = err[1];
    }
    __threadfence_system();
    __syncthreads();
    if (threadIdx.x == 0) *static_cast<volatile uint32_t *>(&back->step) = step;
}

// ------------------------------------------------------------ raw reader

// Which samples are solid (datareader.c:51-77): 16 consecutive ones a thread,
// read 16 bytes at a time (samples of SS little-endian bytes; the buffer starts
// on a 256-byte boundary), as a bit mask.  Single-byte loads, 32 bytes a warp,
// took 40 us to count and 107 to place a 256^3 volume of bytes, these 13 and 25.
struct RawTest {
    const uint8_t *samples, *mask;
    uint64_t V;
    uint32_t lo, hi;
};

template <int SS>
__device__ __forceinline__ uint32_t raw_solid(const RawTest &r, uint64_t v0)
{
    uint32_t w[4 * SS];
    if (v0 + RAW_ITEMS <= r.V) {
        const uint4 *p = reinterpret_cast<const uint4 *>(r.samples + v0 * SS);
        for (int i = 0; i < SS; i++) {
            const uint4 u = p[i];
            w[4 * i] = u.x; w[4 * i + 1] = u.y; w[4 * i + 2] = u.z; w[4 * i + 3] = u.w;
        }
    } else {
        for (int i = 0; i < 4 * SS; i++) {
            w[i] = 0;
            for (int b = 0; b < 4; b++)
                if (v0 * SS + 4 * i + b < r.V * SS) w[i] |= (uint32_t)r.samples[v0 * SS + 4 * i + b] << (8 * b);
        }
    }
    uint32_t m = 0;
    for (int j = 0; j < (int)RAW_ITEMS; j++) {
        uint32_t x = 0;
        for (int l = 0; l < SS; l++) x |= ((w[(j * SS + l) / 4] >> (8 * ((j * SS + l) % 4))) & 0xFFu) << (8 * l);
        const bool solid = r.mask ? ((r.mask[x >> 3] >> (x & 7)) & 1u) != 0u : x >= r.lo && x <= r.hi;
        m |= (uint32_t)(solid && v0 + j < r.V) << j;
    }
    return m;
}

template <int SS>
__global__ void __launch_bounds__(RAW_THREADS) k_raw_count(RawTest r, uint32_t *tile)
{
    __shared__ uint32_t ws[RAW_THREADS / 32];
    const uint64_t v0 = ((uint64_t)blockIdx.x * RAW_THREADS + threadIdx.x) * RAW_ITEMS;
    const uint32_t n = __reduce_add_sync(0xffffffffu, v0 < r.V ? (uint32_t)__popc(raw_solid<SS>(r, v0)) : 0u);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = n;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0;
        for (int w = 0; w < RAW_THREADS / 32; w++) t += ws[w];
        tile[blockIdx.x] = t;
    }
}

// The solid samples' voxels in order, from the tiles' scanned counts:
// array[counter][a] = index * vox_voxel[a] (datareader.c:73-77).
template <int SS>
__global__ void __launch_bounds__(RAW_THREADS) k_raw_place(RawTest r, const uint32_t *tile, uint32_t d1, uint32_t d2,
                                                           float vx, float vy, float vz, float *P)
{
    __shared__ uint32_t ws[RAW_THREADS / 32];
    const uint64_t v0 = ((uint64_t)blockIdx.x * RAW_THREADS + threadIdx.x) * RAW_ITEMS;
    uint32_t m = v0 < r.V ? raw_solid<SS>(r, v0) : 0u;
    const uint32_t n = (uint32_t)__popc(m), incl = warp_incl_scan(n);
    if ((threadIdx.x & 31) == 31) ws[threadIdx.x >> 5] = incl;
    __syncthreads();
    uint64_t at = (uint64_t)tile[blockIdx.x] + incl - n;
    for (uint32_t w = 0; w < (threadIdx.x >> 5); w++) at += ws[w];
    for (; m; m &= m - 1, at++) {
        const uint32_t v = (uint32_t)v0 + (uint32_t)__ffs((int)m) - 1u;   // below 2^32 (check_raw_args)
        const uint32_t row = v / d2, k = v - row * d2, i = row / d1, j = row - i * d1;
        P[3 * at] = __fmul_rn(__uint2float_rn(i), vx);
        P[3 * at + 1] = __fmul_rn(__uint2float_rn(j), vy);
        P[3 * at + 2] = __fmul_rn(__uint2float_rn(k), vz);
    }
}

// ---------------------------------------------------------------- host side

struct Dev {
    cudaStream_t s;
    std::vector<void *> owned;
    explicit Dev(cudaStream_t st) : s(st) {}
    template <typename T>
    cudaError_t get(T **p, size_t count)
    {
        void *q = nullptr;
        cudaError_t e = pool_alloc(&q, count * sizeof(T) + 16, s);
        if (e == cudaSuccess) owned.push_back(q);
        *p = static_cast<T *>(q);
        return e;
    }
    ~Dev()
    {
        for (void *p : owned) cudaFreeAsync(p, s);
        cudaStreamSynchronize(s);   // after an error, copies from the caller's memory may be in flight
    }
};

int fail(cudaError_t e) { return e == cudaErrorMemoryAllocation ? VOX_CUDA_ENOMEM : VOX_CUDA_ECUDA; }

#define TRY(x)                                   \
    do {                                         \
        cudaError_t e_ = (x);                    \
        if (e_ != cudaSuccess) return fail(e_);  \
    } while (0)

// Builds the tree of the N voxels at d_set (device, 3N floats, not modified)
// into t.  Synchronous on s.  With `x`, also hands back what a host tree
// needs beyond the image (see HostTreeExtras).
int build_tree(vox_cuda_tree *t, const float *d_set, uint64_t N, cudaStream_t s, HostTreeExtras *x = nullptr)
{
    const float vx = vox_voxel[0], vy = vox_voxel[1], vz = vox_voxel[2];
    ImageStats st{};
    st.voxel[0] = vx; st.voxel[1] = vy; st.voxel[2] = vz;
    if (N == 0) return adopt_image(t, nullptr, 0, nullptr, 0, nullptr, st);
    if (N > MAX_VOXELS) return VOX_CUDA_ETOOBIG;

    Dev d(s);
    std::vector<Level> levels;
    levels.reserve(MAX_LEVELS + 1);   // throws here or not at all
    struct LevelFree {
        std::vector<Level> &v;
        cudaStream_t s;
        ~LevelFree()
        {
            for (auto &L : v)
                if (L.mem) cudaFreeAsync(L.mem, s);
        }
    } level_free{levels, s};

    float *P[2];
    uint32_t *scal, *cidx = nullptr, *idx[2] = {nullptr, nullptr};
    uint8_t *oct[2] = {nullptr, nullptr}, *cbase = nullptr;
    float *cv = nullptr, *csum = nullptr;
    int *cgrid = nullptr;
    uint2 *maps = nullptr, *starts = nullptr;
    unsigned long long *stats;
    TRY(d.get(&P[0], 3 * N));
    TRY(d.get(&P[1], 3 * N));
    TRY(d.get(&stats, NSTATS * (MAX_LEVELS + 1)));
    // scal: the level's tiny, small, children, largest child, low, mid, tiled nodes
    // with their tiles and subs (6-7), high (8); 10 error bits, 11 whether a
    // coordinate is out of the ordinary
    TRY(d.get(&scal, 12));
    uint32_t *err = scal + 10;
    NodeLists lists{};
    lists.ntiny = scal;
    lists.nsmall = scal + 1;
    lists.nlow = scal + 4;
    lists.nmid = scal + 5;
    lists.nhigh = scal + 8;
    lists.ntiled = reinterpret_cast<unsigned long long *>(scal + 6);
    const Sizes sz(N);
    const int window = (int)sz.window;
    TRY(d.get(&lists.tiny, sz.tiny));
    TRY(d.get(&lists.small, sz.small));
    TRY(d.get(&lists.low, sz.low));
    TRY(d.get(&lists.mid, sz.mid));
    TRY(d.get(&lists.high, sz.high));
    Marks marks[2] = {};
    if (sz.tiled) {
        for (int i = 0; i < 2; i++) {
            TRY(d.get(&idx[i], N));
            TRY(d.get(&oct[i], N));
            TRY(d.get(&marks[i].word, sz.subs * (SUB / 32)));
            TRY(d.get(&marks[i].tile, sz.tiles));
        }
        TRY(d.get(&lists.tiled, sz.tiled));
        TRY(d.get(&cv, 6 * sz.chunks));
        TRY(d.get(&cidx, 6 * sz.chunks));
        TRY(d.get(&csum, 3 * sz.chunks));
        TRY(d.get(&cgrid, 3 * sz.chunks));
        TRY(d.get(&cbase, 3 * sz.chunks));
        TRY(d.get(&maps, sz.chunks * window * 3));
        TRY(d.get(&starts, 3 * sz.tiled));
    }
    TRY(cudaMemsetAsync(scal, 0, 12 * 4, s));
    TRY(cudaMemsetAsync(stats, 0, NSTATS * (MAX_LEVELS + 1) * sizeof(unsigned long long), s));
    launch_after(k_copy_set, grid_for(3 * N, 1024), 256, s, d_set, P[0], 3 * N, scal + 11);

    int dev = 0, nsm = 0;
    TRY(cudaGetDevice(&dev));
    TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    Back *back = static_cast<Back *>(thread_page());
    if (!back) return VOX_CUDA_ENOMEM;
    void *back_dev = nullptr;
    TRY(cudaHostGetDevicePointer(&back_dev, back, 0));
    Back *back_d = static_cast<Back *>(back_dev);
    back->step = 0;
    uint32_t step = 0;
    unsigned schedule = 0;
    TRY(wait_schedule(&schedule));

    Level root;
    TRY(level_alloc(root, 1, s));
    levels.push_back(root);
    launch_after(k_root_node, 1, 32, s, root, (uint32_t)N, lists, P[0], vx, vy, vz, stats);

    uint32_t largest = (uint32_t)N;   // the largest node of the level
    for (int lv = 0;; lv++) {
        if (lv >= MAX_LEVELS) return VOX_CUDA_EDEPTH;
        Level L = levels[lv];
        const uint32_t m = L.m;
        const float *Pc = P[lv & 1];
        float *Pn = P[(lv & 1) ^ 1];
        const Tally tally{stats + NSTATS * lv, scal + 2, scal + 3, err};
        if (largest > HIGH) {
            // boxes, centres and the swapping passes of the largest nodes
            const uint64_t most = std::min<uint64_t>(m, sz.tiled);   // of the level's nodes
            const unsigned nt = (unsigned)most, nc = (unsigned)sz.subs_of(most) * SUB_CHUNKS, np = (unsigned)sz.tiles_of(most);
            launch_after(k_chunk_box, nc, CHUNK_THREADS, s, Pc, L, lists, cv, cidx);
            launch_after(k_box_tiled, nt, NODE_THREADS, s, Pc, L, lists, cv, cidx, vx, vy, vz, tally);
            launch_after(k_chunk_sums, nc, CHUNK_THREADS, s, Pc, L, lists, csum, cgrid);
            launch_after(k_centre_plain, nt, NODE_THREADS, s, L, lists, csum, cgrid, cbase, window, starts, vx, vy, vz);
            launch_after(k_chunk_maps, nc, CHUNK_THREADS, s, Pc, L, lists, cbase, window, maps, sz.chunks);
            launch_after(k_centre_big, grid_for(most * 3 * 32, CENTRE_WARPS * 32), CENTRE_WARPS * 32, s, Pc, L, lists, maps, cbase, csum, window, starts, sz.chunks, vx, vy, vz);
            launch_after(k_tile_marks, np, PASS_THREADS, s, L, lists, Pc, oct[0], marks[0]);
            for (uint32_t o = 0; o < 7; o++) {
                const int in = o & 1, out = in ^ 1;
                launch_after(k_tile_pass, np, PASS_THREADS, s, L, lists, o, marks[in], marks[out], idx[in], oct[in], idx[out], oct[out], err);
            }
            launch_after(k_tile_gather, np, PASS_THREADS, s, L, lists, idx[0], idx[1], Pc, Pn);
            launch_after(k_finish_tiled, grid_for(most * 32, 256), 256, s, L, lists, tally);
        }
        bool first = true;   // of the size classes that are made whole
        if (largest > MID) {
            TRY(cudaFuncSetAttribute(k_nodes_block<1024, HIGH>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)sizeof(NodeShared<HIGH>)));
            launch_after_with(sizeof(NodeShared<HIGH>), k_nodes_block<1024, HIGH>, (unsigned)std::min<uint64_t>(m, sz.high),
                              1024, s, L, lists.high, lists.nhigh, Pc, Pn, vx, vy, vz, tally, first);
            first = false;
        }
        if (largest > LOW) {
            launch_after_with(sizeof(NodeShared<MID>), k_nodes_block<512, MID>, (unsigned)std::min<uint64_t>(m, sz.mid), 512, s,
                              L, lists.mid, lists.nmid, Pc, Pn, vx, vy, vz, tally, first);
            first = false;
        }
        if (largest > SMALL) {
            launch_after_with(sizeof(NodeShared<LOW>), k_nodes_block<96, LOW>, (unsigned)std::min<uint64_t>(m, sz.low), 96, s,
                              L, lists.low, lists.nlow, Pc, Pn, vx, vy, vz, tally, first);
            first = false;
        }
        if (largest > TINY) {
            const unsigned blocks = grid_for(std::min<uint64_t>(m, sz.small), LANE_WARPS);
            launch_after(k_nodes_lanes<SMALL>, std::min(blocks, (unsigned)(nsm * 5)), LANE_WARPS * 32, s, L, lists.small,
                         lists.nsmall, Pc, Pn, vx, vy, vz, tally, first);
            first = false;
        }
        if (largest > VOX_MAX_DOTS) {
            const unsigned blocks = grid_for(std::min<uint64_t>(m, sz.tiny), LANE_WARPS);
            launch_after(k_nodes_lanes<TINY>, std::min(blocks, (unsigned)(nsm * 8)), LANE_WARPS * 32, s, L, lists.tiny,
                         lists.ntiny, Pc, Pn, vx, vy, vz, tally, first);
        }
        launch_after(k_level_done, 1, 1, s, scal, back_d, ++step);
        TRY(cudaGetLastError());
        TRY(wait_for_word(&back->step, step, schedule, s));
        const uint32_t mn = back->next[0];
        largest = back->next[1];
        if (mn == 0) break;
        Level Nx;
        TRY(level_alloc(Nx, mn, s));
        levels.push_back(Nx);
        launch_after(k_children, grid_for((uint64_t)m * 8, CHILD_THREADS), CHILD_THREADS, s, L, Nx, lists, Pn, vx, vy, vz, stats + NSTATS * (lv + 1));
    }

    // bottom up: subtree sizes
    int nl = (int)levels.size();
    for (int lv = nl - 1; lv >= 0; lv--) {
        Level L = levels[lv];
        Level Nx = lv + 1 < nl ? levels[lv + 1] : L;
        launch_after(k_up, grid_for(L.m, 256), 256, s, L, Nx, lv + 1 < nl);
    }
    launch_after(k_all_done, 1, 128, s, levels[0], stats, err, back_d, ++step);
    TRY(cudaGetLastError());
    TRY(wait_for_word(&back->step, step, schedule, s));
    if (back->err & ERR_WALK) return VOX_CUDA_ECUDA;
    if (back->err & ERR_BIG_LEAF) return VOX_CUDA_ETOOBIG;
    uint64_t units = VOXP_REC_UNITS + back->units;
    if (units > VOXP_MAX_UNITS) return VOX_CUDA_ETOOBIG;
    uint64_t nodes = back->root_nodes;

    uint4 *pool = nullptr;
    uint32_t *map = nullptr, *dots = nullptr;
    float *order = nullptr;
    size_t pool_bytes = units * 16, map_bytes = nodes * 4;
    if (x) TRY(d.get(&dots, nodes));
    if (x && x->order) TRY(d.get(&order, 3 * N));
    // the tree's own memory, given back unless the tree takes it
    struct Image {
        cudaStream_t s;
        void *p[3] = {nullptr, nullptr, nullptr};
        ~Image()
        {
            for (void *q : p)
                if (q) cudaFreeAsync(q, s);
        }
    } image{s};
    TRY(pool_alloc(&image.p[0], pool_bytes, s));
    TRY(pool_alloc(&image.p[1], map_bytes, s));
    TRY(pool_alloc(&image.p[2], 4, s));
    pool = static_cast<uint4 *>(image.p[0]);
    map = static_cast<uint32_t *>(image.p[1]);
    uint32_t *status = static_cast<uint32_t *>(image.p[2]);
    TRY(cudaMemsetAsync(status, 0, 4, s));
    // top down: ids, offsets and the image
    for (int lv = 0; lv < nl; lv++) {
        const Level &L = levels[lv], &Nx = levels[std::min(lv + 1, nl - 1)];
        const float *Pc = P[lv & 1];
        launch_after(k_emit, grid_for(L.m, 256), 256, s, L, Nx, Pc, pool, map, units, nodes, err, dots);
        if (back->stats[NSTATS * lv + S_OVER]) {
            launch_after(k_emit_over, grid_for((uint64_t)L.m * 32, 256), 256, s, L, Pc, pool, units, err);
        }
        if (order) {
            launch_after(k_final_order, grid_for((uint64_t)L.m * 32, 256), 256, s, L, Pc, order);
        }
    }
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(&back->err, err, 4, cudaMemcpyDeviceToHost, s);
    // A tree made here of ordinary voxels has every property the searches may
    // rely on: boxes are least boxes of their voxels (min <= max as the voxel
    // size is positive), children's voxels lie on their side of the dividing
    // planes, no centre passes 2^60, and every number is a multiple of 2^-78
    // (sums of the voxels' own, which are of LEAST's ulp, and of the voxel
    // size's).  Any other is looked over.
    const auto ordinary = [](float v) { return v >= vox::SHAPE_VOXEL && v <= LIMIT; };
    back->unshaped = 0;
    if (back->odd || !ordinary(vx) || !ordinary(vy) || !ordinary(vz)) {
        if (e == cudaSuccess) e = image_shape(pool, map, nodes, st.voxel, &back_d->unshaped, s);
    }
    if (x) {
        x->dots_of_id.resize(nodes);
        if (e == cudaSuccess && x->order)
            e = cudaMemcpyAsync(x->order, order, 12 * N, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(x->dots_of_id.data(), dots, nodes * 4, cudaMemcpyDeviceToHost, s);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess || back->err) return e != cudaSuccess ? fail(e) : VOX_CUDA_ECUDA;
    st.unshaped = back->unshaped;
    st.nodes = nodes;
    st.units = units;
    for (int lv = 0; lv < nl; lv++) {
        const unsigned long long *h = &back->stats[NSTATS * lv];
        st.inner += h[S_INNER];
        st.leaf += h[S_LEAF];
        st.dense += h[S_DENSE];
        st.dots += h[S_DOTS];
        if (h[S_INNER]) st.depth = (uint64_t)lv + 1;
    }
    for (int i = 0; i < 6; i++) st.bbox[i] = back->box[i];
    int rc = adopt_image(t, pool, pool_bytes, map, map_bytes, status, st);
    if (rc == VOX_CUDA_OK)
        for (void *&q : image.p) q = nullptr;
    return rc;
}

struct Stream {
    cudaStream_t s = nullptr;
    Stream() { cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking); }
    ~Stream()
    {
        if (s) cudaStreamDestroy(s);
    }
};

// A new tree handle built by f(t, stream).
template <class F>
int new_tree(vox_cuda_tree **out, F f)
{
    if (!out) return VOX_CUDA_EINVAL;
    *out = nullptr;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return VOX_CUDA_ENODEV;
    Stream st;
    if (!st.s) return VOX_CUDA_ECUDA;
    struct Owned {
        vox_cuda_tree *t;
        ~Owned() { if (t) vox_cuda_tree_free(t); }   // on an error, also one that f throws
    } own{new (std::nothrow) vox_cuda_tree(dev)};
    if (!own.t) return VOX_CUDA_ENOMEM;
    if (int rc = f(own.t, st.s)) return rc;
    *out = own.t;
    own.t = nullptr;
    return VOX_CUDA_OK;
}

int raw_build(vox_cuda_tree *t, const void *samples, const unsigned dim[3], unsigned samplesize,
              const vox_cuda_raw_test *test, cudaStream_t s)
{
    uint64_t V = (uint64_t)dim[0] * dim[1] * dim[2];
    uint64_t bytes = V * samplesize;
    uint64_t mask_bytes = test->mask ? ((1ull << (8 * samplesize)) + 7) / 8 : 0;
    float *P = nullptr;
    uint8_t *d_samples = nullptr, *d_mask = nullptr;
    uint32_t *tile = nullptr, *total = nullptr;
    int rc = VOX_CUDA_OK;
    {
        Dev d(s);
        if (d.get(&d_samples, bytes ? bytes : 1) != cudaSuccess || d.get(&tile, V / RAW_TILE + 2) != cudaSuccess ||
            d.get(&total, 1) != cudaSuccess || (mask_bytes && d.get(&d_mask, mask_bytes) != cudaSuccess))
            return VOX_CUDA_ENOMEM;
        if (bytes && cudaMemcpyAsync(d_samples, samples, bytes, cudaMemcpyHostToDevice, s) != cudaSuccess)
            return VOX_CUDA_ECUDA;
        if (mask_bytes && cudaMemcpyAsync(d_mask, test->mask, mask_bytes, cudaMemcpyHostToDevice, s) != cudaSuccess)
            return VOX_CUDA_ECUDA;
        const RawTest raw{d_samples, d_mask, V, test->lo, test->hi};
        void (*const count[])(RawTest, uint32_t *) = {k_raw_count<1>, k_raw_count<2>, k_raw_count<3>, k_raw_count<4>};
        void (*const place[])(RawTest, const uint32_t *, uint32_t, uint32_t, float, float, float, float *) = {
            k_raw_place<1>, k_raw_place<2>, k_raw_place<3>, k_raw_place<4>};
        // count the solid voxels first: the set is allocated to size
        uint32_t nt = (uint32_t)((V + RAW_TILE - 1) / RAW_TILE);
        uint32_t h_total = 0, *page = static_cast<uint32_t *>(thread_page());
        if (!page) return VOX_CUDA_ENOMEM;
        if (nt) {
            count[samplesize - 1]<<<nt, RAW_THREADS, 0, s>>>(raw, tile);
            count_launch();
            k_scan_tiles<<<1, 1024, 0, s>>>(tile, nt, total);
            count_launch();
            if (cudaMemcpyAsync(page, total, 4, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
                cudaStreamSynchronize(s) != cudaSuccess)
                return VOX_CUDA_ECUDA;
            h_total = *page;
        }
        if (h_total) {
            if (pool_alloc(reinterpret_cast<void **>(&P), 12ull * h_total, s) != cudaSuccess) return VOX_CUDA_ENOMEM;
            place[samplesize - 1]<<<nt, RAW_THREADS, 0, s>>>(raw, tile, dim[1], dim[2], vox_voxel[0], vox_voxel[1],
                                                             vox_voxel[2], P);
            count_launch();
            if (cudaGetLastError() != cudaSuccess) rc = VOX_CUDA_ECUDA;
        }
        if (rc == VOX_CUDA_OK) rc = build_tree(t, P, h_total, s);
    }
    if (P) cudaFreeAsync(P, s);
    cudaStreamSynchronize(s);
    return rc;
}

int check_raw_args(const unsigned dim[3], unsigned samplesize, const vox_cuda_raw_test *test)
{
    if (!dim || !test || samplesize < 1 || samplesize > 4) return VOX_CUDA_EINVAL;
    if (test->mask && samplesize > 2) return VOX_CUDA_EINVAL;
    uint64_t V = (uint64_t)dim[0] * dim[1] * dim[2];
    if (V > 0xFFFFFFFFull) return VOX_CUDA_ETOOBIG;   // the reference counts samples in an unsigned int
    return VOX_CUDA_OK;
}

}  // namespace

// ======================================================================== API

int build_for_host_tree(const float *set, size_t n, vox_cuda_tree **out, HostTreeExtras *x)
{
    if (n == 0 || n > MAX_VOXELS || !set) return VOX_CUDA_EINVAL;
    return new_tree(out, [&](vox_cuda_tree *t, cudaStream_t s) {
        float *d = nullptr;
        if (pool_alloc(reinterpret_cast<void **>(&d), 12ull * n, s) != cudaSuccess) return (int)VOX_CUDA_ENOMEM;
        int rc = VOX_CUDA_OK;
        if (cudaMemcpyAsync(d, set, 12ull * n, cudaMemcpyHostToDevice, s) != cudaSuccess) rc = VOX_CUDA_ECUDA;
        if (rc == VOX_CUDA_OK) rc = build_tree(t, d, n, s, x);
        cudaFreeAsync(d, s);
        cudaStreamSynchronize(s);
        return rc;
    });
}

EXPORT int vox_cuda_tree_build_device(const float *d_set, size_t n, vox_cuda_tree **out)
try {
    if (n && !d_set) return VOX_CUDA_EINVAL;
    return new_tree(out, [&](vox_cuda_tree *t, cudaStream_t s) {
        // the set may still be on its way, in any stream of the caller's: the
        // build's own stream waits for none of them
        if (n && wait_for_device() != cudaSuccess) return (int)VOX_CUDA_ECUDA;
        return build_tree(t, d_set, n, s);
    });
} VOX_ABI_FAIL_INT

EXPORT int vox_cuda_tree_build(const float *set, size_t n, vox_cuda_tree **out)
try {
    if (n && !set) return VOX_CUDA_EINVAL;
    return new_tree(out, [&](vox_cuda_tree *t, cudaStream_t s) {
        if (n > MAX_VOXELS) return (int)VOX_CUDA_ETOOBIG;
        float *d = nullptr;
        if (n && pool_alloc(reinterpret_cast<void **>(&d), 12ull * n, s) != cudaSuccess) return (int)VOX_CUDA_ENOMEM;
        int rc = VOX_CUDA_OK;
        if (n && cudaMemcpyAsync(d, set, 12ull * n, cudaMemcpyHostToDevice, s) != cudaSuccess) rc = VOX_CUDA_ECUDA;
        if (rc == VOX_CUDA_OK) rc = build_tree(t, d, n, s);
        if (d) cudaFreeAsync(d, s);
        cudaStreamSynchronize(s);
        return rc;
    });
} VOX_ABI_FAIL_INT

EXPORT int vox_cuda_tree_build_raw(const void *samples, const unsigned dim[3], unsigned samplesize,
                                   const vox_cuda_raw_test *test, vox_cuda_tree **out)
try {
    int rc = check_raw_args(dim, samplesize, test);
    if (rc) return rc;
    if (!samples && (uint64_t)dim[0] * dim[1] * dim[2] != 0) return VOX_CUDA_EINVAL;
    return new_tree(out, [&](vox_cuda_tree *t, cudaStream_t s) {
        return raw_build(t, samples, dim, samplesize, test, s);
    });
} VOX_ABI_FAIL_INT

EXPORT int vox_cuda_read_raw_data(const char *filename, const unsigned dim[3], unsigned samplesize,
                                  const vox_cuda_raw_test *test, vox_cuda_tree **out, const char **error)
try {
    if (out) *out = nullptr;
    int rc = check_raw_args(dim, samplesize, test);
    if (rc || !filename || !out) {
        if (error) *error = "Invalid argument";
        return rc ? rc : VOX_CUDA_EINVAL;
    }
    int fd = open(filename, O_RDONLY);
    if (fd == -1) {
        if (error) *error = strerror(errno);
        return VOX_CUDA_EINVAL;
    }
    struct stat sb;
    if (fstat(fd, &sb) == -1) {
        if (error) *error = strerror(errno);
        close(fd);
        return VOX_CUDA_EINVAL;
    }
    uint64_t bytes = (uint64_t)dim[0] * dim[1] * dim[2] * samplesize;
    if ((uint64_t)sb.st_size != bytes) {   // datareader.c:40-43
        if (error) *error = "Wrong size of dataset";
        close(fd);
        return VOX_CUDA_EINVAL;
    }
    void *buf = nullptr;
    if (bytes && cudaMallocHost(&buf, bytes) != cudaSuccess) {
        close(fd);
        if (error) *error = "Cannot allocate memory";
        return VOX_CUDA_ENOMEM;
    }
    uint64_t got = 0;
    while (got < bytes) {
        ssize_t r = read(fd, static_cast<char *>(buf) + got, (size_t)std::min<uint64_t>(bytes - got, 1u << 30));
        if (r <= 0) {
            if (error) *error = r == 0 ? "Unexpected end of file" : strerror(errno);
            close(fd);
            cudaFreeHost(buf);
            return VOX_CUDA_EINVAL;
        }
        got += (uint64_t)r;
    }
    close(fd);
    rc = vox_cuda_tree_build_raw(buf, dim, samplesize, test, out);
    if (buf) cudaFreeHost(buf);
    if (rc && error) *error = vox_cuda_strerror(rc);
    return rc;
} VOX_ABI_FAIL_INT
