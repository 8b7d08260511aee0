/* image_shape.h -- what is known of every box of a tree's image, and the check
 * of one record of it, for the host (small images) and the device.
 *
 * SHAPE_ORDERED: every number of a node's box, a centre or a voxel is zero or
 * SHAPE_LEAST to SHAPE_LIMIT in magnitude, min <= max on every axis and no max
 * is -0, and the voxel size is SHAPE_VOXEL to SHAPE_LIMIT.  Trees that vox_make_tree or the GPU
 * build make from ordinary voxels have it; a caller's own tree need not.
 *
 * SHAPE_NESTED: every child's box and every leaf's voxel lie inside their
 * node's box, and a child on the lower side of a dividing plane reaches at
 * most one voxel past it, one on the upper side not below it.
 */
#ifndef VOX_IMAGE_SHAPE_H
#define VOX_IMAGE_SHAPE_H

#include <cstdint>
#include <cstring>

#include "pool_layout.h"

#ifdef __CUDACC__
#define VOX_SHAPE_HD __host__ __device__ __forceinline__
#else
#define VOX_SHAPE_HD inline
#endif

namespace vox {

constexpr uint32_t SHAPE_ORDERED = 1u, SHAPE_NESTED = 2u;
constexpr float SHAPE_LIMIT = 1.152921504606847e18f;     // 2^60
constexpr float SHAPE_LEAST = 1.6543612251060553e-24f;   // 2^-79
constexpr float SHAPE_VOXEL = 1.4901161193847656e-8f;    // 2^-26

VOX_SHAPE_HD float shape_float(uint32_t u)
{
#ifdef __CUDA_ARCH__
    return __uint_as_float(u);
#else
    float f;
    std::memcpy(&f, &u, 4);
    return f;
#endif
}

// (false for NaN)
VOX_SHAPE_HD bool shape_fine(float v)
{
    const float m = v < 0.0f ? -v : v;
    return v == 0.0f || (m >= SHAPE_LEAST && m <= SHAPE_LIMIT);
}

struct ImageShape {
    float vox[3];
    bool ok, nested;   // what holds so far
    VOX_SHAPE_HD ImageShape(float vx, float vy, float vz) : vox{vx, vy, vz}, ok(true), nested(true)
    {
        for (int k = 0; k < 3; k++) ok = ok && vox[k] >= SHAPE_VOXEL && vox[k] <= SHAPE_LIMIT;
    }
    // a voxel of a leaf whose box is [lo, hi]
    template <class U>
    VOX_SHAPE_HD void voxel(const U &v, const float *lo, const float *hi)
    {
        const float p[3] = {shape_float(v.x), shape_float(v.y), shape_float(v.z)};
        for (int k = 0; k < 3; k++) {
            ok = ok && shape_fine(p[k]);
            nested = nested && p[k] >= lo[k] && p[k] + vox[k] <= hi[k];   // (a sum alone: nothing to contract)
        }
    }
    // The record at `rec`; of a leaf the voxels too, unless there are more than
    // `most` (then their number is returned, else 0).
    template <class U>
    VOX_SHAPE_HD uint32_t record(const U *pool, uint32_t rec, uint32_t most)
    {
        const U a = pool[rec], b = pool[rec + 1], c = pool[rec + 2];
        const float lo[3] = {shape_float(a.x), shape_float(a.y), shape_float(a.z)},
                    hi[3] = {shape_float(a.w), shape_float(b.x), shape_float(b.y)};
        for (int k = 0; k < 3; k++) ok = ok && shape_fine(lo[k]) && shape_fine(hi[k]) && lo[k] <= hi[k];
        ok = ok && a.w != 0x80000000u && b.x != 0x80000000u && b.y != 0x80000000u;
        const uint32_t kind = b.z & 3u;
        if (kind == VOXP_KIND_INNER) {
            const float plane[3] = {shape_float(c.x), shape_float(c.y), shape_float(c.z)};
            uint32_t at = b.w;
            for (uint32_t oct = 0; oct < 8; oct++) {
                if (!((b.z >> (8 + oct)) & 1u)) continue;
                const U v = pool[at], u = pool[at + 1];
                at += VOXP_REC_UNITS;
                const float p[3] = {shape_float(v.x), shape_float(v.y), shape_float(v.z)},
                            q[3] = {shape_float(v.w), shape_float(u.x), shape_float(u.y)};
                for (int k = 0; k < 3; k++)
                    nested = nested && p[k] >= lo[k] && q[k] <= hi[k] &&
                             ((oct >> k) & 1u ? q[k] <= plane[k] + vox[k] : p[k] >= plane[k]);
            }
            for (int k = 0; k < 3; k++) ok = ok && shape_fine(plane[k]);
        } else if (kind == VOXP_KIND_LEAF) {
            const uint32_t n = b.z >> 2;
            if (n > most) return n;
            for (uint32_t i = 0; i < n; i++) voxel(pool[b.w + i], lo, hi);
        }
        return 0;
    }
    VOX_SHAPE_HD uint32_t missing() const { return (ok ? 0u : SHAPE_ORDERED) | (nested ? 0u : SHAPE_NESTED); }
};

}  // namespace vox

#endif
