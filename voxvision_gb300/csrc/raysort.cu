/*
 * raysort.cu -- the order in which a large ray batch is traced.
 *
 * Every ray of a batch is an independent search, so the order in which they
 * are traced changes no result, only how alike the 32 searches of a warp are.
 * Rays given in random order (origins anywhere, directions anywhere) put 32
 * unrelated searches in every warp.  Tracing them grouped by the octant of
 * their direction, then by the cell of the point where they enter the tree's
 * box on an 8x8x8 grid over it (Morton order), makes the searches of a warp
 * start at the same part of the tree and walk it the same way: 1M random
 * rays over the 256^3 tree take 163 us, sorting included, against 223 in the
 * given order.  Ball batches can be grouped the same way by the cell of their
 * centre on a 16x16x16 grid over the tree's box (launch_balls says when).
 *
 * The order is a counting sort on those 12-bit keys: per block of up to
 * 65,536 items (fewer for smaller batches, so that every SM gets blocks) a
 * histogram in shared memory, the position of each (key, block) pair from a
 * prefix over blocks and keys, then each item's slot in `order`; the search
 * kernel reads the j-th item of the order from where it was given and writes
 * its result there.  Items of one (key, block) pair land in any order among
 * themselves; that, too, changes no result.
 * (Copying the rays into order instead makes a batch slower: each ray's six
 * floats become scattered partial-sector stores.  Finer keys are slower too:
 * of the entry point's cell on a 16^3 grid 2.84-2.87 ms, of the direction's
 * dominant axis as well 2.99, against 2.77-2.78, for 16M rays with the general
 * search.)
 */
#include <cuda_runtime.h>

#include <cstdint>

#include "internal.h"

namespace {

constexpr int KEY_BITS = 12;
constexpr uint32_t NKEYS = 1u << KEY_BITS;
constexpr int SORT_THREADS = 1024;

// Items one block keys and places: 65,536 for large batches, for smaller ones
// as many as give two blocks to each of 152 SMs (4M rays: 528 us searched and
// all, 531 in 256 blocks, 535 in 152), 8,192 at least, which keeps the
// per-block histograms small beside the items.
size_t items_per_block(size_t n)
{
    size_t per = (n + 303) / 304;
    per = per < 8192 ? 8192 : (per > 65536 ? 65536 : per);
    return per;
}

struct KeyFrame {
    float lo[3], inv[3];   // cell = floor((p - lo) * inv), clamped to the grid
    float blo[3], bhi[3];  // the tree's box, where the rays' entry points are found
};

// Morton index of point i's cell on a (2^bits)^3 grid.
template <int BITS>
__device__ __forceinline__ uint32_t morton_cell(const float *pt, size_t i, const KeyFrame &f)
{
    constexpr float TOP = (float)((1 << BITS) - 1);
    uint32_t cell[3];
    for (int a = 0; a < 3; a++) {
        float q = (pt[3 * i + a] - f.lo[a]) * f.inv[a];
        cell[a] = q >= TOP ? (uint32_t)TOP : (q > 0.0f ? (uint32_t)q : 0u);   // NaN -> 0
    }
    uint32_t m = 0;
    for (int b = 0; b < BITS; b++)
        for (int a = 0; a < 3; a++) m |= ((cell[a] >> b) & 1u) << (3 * b + a);
    return m;
}

// Direction octant, then the cell, on an 8^3 grid over the tree's box, of
// where the ray enters that box (rays that miss it: the last key).  Rays of
// one key start their searches at the same part of the tree and walk it the
// same way; keyed on the origin's cell instead, a warp's rays of one octant
// still entered the box anywhere (16M rays, general search: 3.94 ms against 2.80).
__device__ __forceinline__ uint32_t ray_key(const float *o, const float *d, size_t i, const KeyFrame &f)
{
    uint32_t oct = (d[3 * i] < 0.0f) | ((d[3 * i + 1] < 0.0f) << 1) | ((d[3 * i + 2] < 0.0f) << 2);
    float t0 = 0.0f, t1 = 3.0e38f;
    for (int a = 0; a < 3; a++) {
        const float inv = 1.0f / d[3 * i + a];
        float ta = (f.blo[a] - o[3 * i + a]) * inv, tb = (f.bhi[a] - o[3 * i + a]) * inv;
        if (ta > tb) { float x = ta; ta = tb; tb = x; }
        t0 = fmaxf(t0, ta);      // NaN (a zero direction inside the slab) keeps the bound
        t1 = fminf(t1, tb);
    }
    if (!(t0 <= t1)) return (oct << 9) | 0x1FFu;
    float p[3];
    for (int a = 0; a < 3; a++) p[a] = o[3 * i + a] + t0 * d[3 * i + a];
    return (oct << 9) | morton_cell<3>(p, 0, f);
}

// Keys of a block's items and the block's histogram (block-major): rays
// (d given) by ray_key, balls (d NULL) by the cell of their centre on a
// 16^3 grid over the tree's box.
__global__ void __launch_bounds__(SORT_THREADS) k_keys(const float *__restrict__ o, const float *__restrict__ d, size_t n,
                                                        size_t per, KeyFrame f, uint16_t *__restrict__ keys,
                                                        uint32_t *__restrict__ hist)
{
    __shared__ uint32_t h[NKEYS];
    for (uint32_t k = threadIdx.x; k < NKEYS; k += SORT_THREADS) h[k] = 0;
    __syncthreads();
    size_t b0 = (size_t)blockIdx.x * per, b1 = b0 + per < n ? b0 + per : n;
    for (size_t i = b0 + threadIdx.x; i < b1; i += SORT_THREADS) {
        uint32_t k = d ? ray_key(o, d, i, f) : morton_cell<4>(o, i, f);
        keys[i] = (uint16_t)k;
        atomicAdd(&h[k], 1u);
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < NKEYS; k += SORT_THREADS) hist[(size_t)blockIdx.x * NKEYS + k] = h[k];
}

// For every key: its count before each block (in place) and its total; a block
// takes 32 keys, a lane each, and its warps a run of the blocks each.
__global__ void __launch_bounds__(1024) k_key_blocks(uint32_t *hist, uint32_t nblocks, uint32_t *total)
{
    __shared__ uint32_t part[32][32];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, k = blockIdx.x * 32 + lane;
    const uint32_t per = (nblocks + 31) / 32, b0 = min(warp * per, nblocks), b1 = min(b0 + per, nblocks);
    uint32_t sum = 0;
    for (uint32_t b = b0; b < b1; b++) sum += hist[(size_t)b * NKEYS + k];
    part[warp][lane] = sum;
    __syncthreads();
    uint32_t run = 0;
    for (uint32_t w = 0; w < warp; w++) run += part[w][lane];
    if (warp == 31) total[k] = run + sum;
    for (uint32_t b = b0; b < b1; b++) {
        const uint32_t c = hist[(size_t)b * NKEYS + k];
        hist[(size_t)b * NKEYS + k] = run;
        run += c;
    }
}

// Each item's slot in the traced order: the keys' starts (an exclusive scan of
// the totals, made by every block for itself), the counts of the blocks
// before, then a place each.
__global__ void __launch_bounds__(SORT_THREADS) k_place(const uint16_t *__restrict__ keys, size_t n, size_t per,
                                                         const uint32_t *__restrict__ hist,
                                                         const uint32_t *__restrict__ total, uint32_t *__restrict__ order)
{
    __shared__ uint32_t base[NKEYS];
    __shared__ uint32_t part[32];
    constexpr uint32_t PER = NKEYS / SORT_THREADS;
    static_assert(PER == 4, "a thread scans one 16-byte piece of the totals");
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint4 v = reinterpret_cast<const uint4 *>(total)[threadIdx.x];
    const uint4 h = reinterpret_cast<const uint4 *>(hist + (size_t)blockIdx.x * NKEYS)[threadIdx.x];
    const uint32_t sum = v.x + v.y + v.z + v.w;
    uint32_t x = sum;
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, off);
        if (lane >= (uint32_t)off) x += y;
    }
    if (lane == 31) part[warp] = x;
    __syncthreads();
    if (warp == 0) {
        const uint32_t p = part[lane];
        uint32_t q = p;
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, q, off);
            if (lane >= (uint32_t)off) q += y;
        }
        part[lane] = q - p;
    }
    __syncthreads();
    const uint32_t first = part[warp] + x - sum;
    reinterpret_cast<uint4 *>(base)[threadIdx.x] =
        make_uint4(first + h.x, first + v.x + h.y, first + v.x + v.y + h.z, first + v.x + v.y + v.z + h.w);
    __syncthreads();
    size_t b0 = (size_t)blockIdx.x * per, b1 = b0 + per < n ? b0 + per : n;
    for (size_t i = b0 + threadIdx.x; i < b1; i += SORT_THREADS) order[atomicAdd(&base[keys[i]], 1u)] = (uint32_t)i;
}

}  // namespace

static size_t up256(size_t x) { return (x + 255) & ~size_t(255); }

size_t ray_order_bytes(size_t n)
{
    size_t nb = (n + items_per_block(n) - 1) / items_per_block(n);
    return up256(n * 2) + up256(n * 4) + nb * NKEYS * 4 + NKEYS * 4 + 256;
}

// The order of n rays (d given) or balls (d NULL) in `scratch`.
static cudaError_t sort_order(const vox_cuda_tree *t, const float *o, const float *d, size_t n, void *scratch,
                              uint32_t **order, cudaStream_t s)
{
    const size_t per = items_per_block(n), nb = (n + per - 1) / per;
    char *p = static_cast<char *>(scratch);
    uint16_t *keys = reinterpret_cast<uint16_t *>(p);
    p += up256(n * 2);
    *order = reinterpret_cast<uint32_t *>(p);
    p += up256(n * 4);
    uint32_t *hist = reinterpret_cast<uint32_t *>(p);
    uint32_t *total = hist + nb * NKEYS;
    // cells over the tree's box: 8 per axis for rays' entry points, 16 for
    // balls' centres
    const float cells = d ? 8.0f : 16.0f;
    KeyFrame f;
    for (int a = 0; a < 3; a++) {
        f.blo[a] = t->bbox[a];
        f.bhi[a] = t->bbox[3 + a];
        f.lo[a] = t->bbox[a];
        f.inv[a] = cells / fmaxf(t->bbox[3 + a] - t->bbox[a], 1e-30f);
    }
    k_keys<<<(unsigned)nb, SORT_THREADS, 0, s>>>(o, d, n, per, f, keys, hist);
    k_key_blocks<<<NKEYS / 32, 1024, 0, s>>>(hist, (uint32_t)nb, total);
    k_place<<<(unsigned)nb, SORT_THREADS, 0, s>>>(keys, n, per, hist, total, *order);
    for (int i = 0; i < 3; i++) count_launch();
    return cudaGetLastError();
}

cudaError_t ray_order(const vox_cuda_tree *t, const float *o, const float *d, size_t n, void *scratch,
                      uint32_t **order, cudaStream_t s)
{
    return sort_order(t, o, d, n, scratch, order, s);
}

cudaError_t ball_order(const vox_cuda_tree *t, const float *centres, size_t n, void *scratch, uint32_t **order,
                       cudaStream_t s)
{
    return sort_order(t, centres, nullptr, n, scratch, order, s);
}
