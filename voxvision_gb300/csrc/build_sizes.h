/* build_sizes.h -- how build.cu divides a set of voxels, and what memory that
 * takes beside the levels' nodes: host code, with no need of CUDA. */
#ifndef VOX_BUILD_SIZES_H
#define VOX_BUILD_SIZES_H

#include <algorithm>
#include <cstdint>

#ifdef __CUDACC__
#define VOX_HD __host__ __device__
#else
#define VOX_HD
#endif

namespace build_sizes {

constexpr uint32_t LEAF = 7;         // VOX_MAX_DOTS: nodes with at most this many are leaves
constexpr uint32_t TINY = 32;        // nodes with at most this many voxels, and
constexpr uint32_t SMALL = 128;      // with at most this many, are split by a lane each,
constexpr uint32_t LOW = 1024;       // with at most this many by a block of 96 threads,
constexpr uint32_t MID = 8192;       // with at most this many by a block of 512, and
constexpr uint32_t HIGH = 32768;     // with at most this many by a block of 1024, larger ones tile by tile
constexpr uint32_t CHUNK = 1024;     // voxels per chunk
constexpr uint32_t SUB = 2048;       // positions marked at a time; a tile is a multiple of it
constexpr uint32_t SUB_SHIFT = 11;
constexpr uint32_t MAX_TILES = 2048; // tiles of one node
constexpr uint32_t NBIN = 16;        // binades with a precomputed map per chunk
constexpr uint64_t MAX_VOXELS = 0x7FFFFFFFull;
static_assert(SUB == 1u << SUB_SHIFT && SUB % CHUNK == 0, "whole chunks to a sub, whole subs to a tile");

// Positions per tile of a node of n voxels: 1 << this.  A node's own size
// decides, so that all its tiles together are little more than the node; with
// one tile size for the set, every node above HIGH had a whole tile of the
// root's to itself, and the scratch of a large set grew with its square.
VOX_HD inline uint32_t tile_shift(uint32_t n)
{
    uint32_t s = SUB_SHIFT;
    while (((uint64_t)MAX_TILES << s) < n) s++;
    return s;
}

VOX_HD inline uint32_t parts(uint32_t n, uint32_t shift) { return (uint32_t)(((uint64_t)n + (1u << shift) - 1) >> shift); }

// The most that any level of a set of N voxels has of each: nodes per class
// and, of the tiled nodes, tiles, subs and chunks.
struct Sizes {
    uint64_t N, tiny, small, low, mid, high, tiled, tiles, subs, chunks;
    uint32_t window;   // maps per chunk: past 2^24 additions a sum's roundings can add up to a sizeable part of it
    explicit Sizes(uint64_t n)
        : N(n), tiny(n / (LEAF + 1) + 1), small(n / (TINY + 1) + 1), low(n / SMALL + 1), mid(n / LOW + 1),
          high(n / MID + 1), tiled(n / HIGH), tiles(tiles_of(tiled)), subs(subs_of(tiled)), chunks(subs * (SUB / CHUNK)),
          window(n > (1u << 24) ? NBIN : 2)
    {
    }
    // of m tiled nodes
    uint64_t subs_of(uint64_t m) const { return m ? N / SUB + m : 0; }
    uint64_t tiles_of(uint64_t m) const { return std::min(m * MAX_TILES, subs_of(m)); }

    // bytes of the lists, and of what tiled nodes take
    uint64_t lists() const { return 4 * (tiny + small + low + mid + high); }
    uint64_t orders() const { return tiled ? 2 * N * (4 + 1) : 0; }                 // places and octants, twice
    uint64_t marks() const { return 2 * (subs * (SUB / 32) * 16 + tiles * 8); }
    uint64_t sums() const { return chunks * (24 + 24 + 12 + 12 + 3 + (uint64_t)window * 3 * 8) + tiled * (16 + 3 * 8); }
    // beside the two orders of the voxels themselves (24 bytes a voxel)
    uint64_t scratch() const { return lists() + orders() + marks() + sums(); }
};

}  // namespace build_sizes

#endif
