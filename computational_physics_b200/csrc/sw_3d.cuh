// Geometry of the 3D engine and the layouts its kernels and the host share (sw_3d.cu).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

namespace swb {

constexpr uint32_t k3Pitch = 32;          // block-local index: ((zl * k3Rows) + yl) * k3Pitch + xl
constexpr uint32_t k3Rows = 16, k3Layers = 16;
constexpr uint32_t k3Layer = k3Rows * k3Pitch;
constexpr uint32_t k3MaxThreads = 512;    // a warp per piece, at most 16 pieces
constexpr uint32_t k3MergeThreads = 256;
constexpr uint32_t k3FlipThreads = 512;   // four quads of a 32 x 16 x 16 block per thread
constexpr uint32_t k3Window = 256;        // listed unions of a piece worked off at a time
constexpr uint32_t k3Links = 256;         // linked labels a piece remembers
constexpr uint32_t k3ShareBlocks = 148;   // up to a block per SM: spread3, draw_share3

struct Geo3 {
    uint32_t L0, L1, L2;        // extent
    uint32_t TX, TY, TZ;        // tile
    uint32_t TBX, TBY, TBZ;     // tiles per block
    uint32_t BX, BY, BZ;        // block in sites
    uint32_t n0, n1, n2;        // tiles per direction
    uint32_t nbx, nby, nbz;     // blocks per direction
    uint32_t py, pcy;           // tile rows per piece; pieces per tile layer
};

// What follows from the tiles per block.
inline void fit3(Geo3 &g)
{
    g.BX = g.TBX * g.TX; g.BY = g.TBY * g.TY; g.BZ = g.TBZ * g.TZ;
    g.nbx = (g.L0 + g.BX - 1) / g.BX;
    g.nby = (g.L1 + g.BY - 1) / g.BY;
    g.nbz = (g.L2 + g.BZ - 1) / g.BZ;
    g.py = std::min(std::max(1u, 32 / (g.TY * g.TZ)), g.TBY);
    g.pcy = (g.TBY + g.py - 1) / g.py;
}

// Blocks of up to 32 x 16 x 16 sites, whole tiles.  Larger blocks have fewer face sites (15.6 % of the
// sites against 21.9 % with 32 x 8 x 16), which the merge pays for.
inline Geo3 make_geo3(uint32_t L0, uint32_t L1, uint32_t L2, uint32_t TX, uint32_t TY, uint32_t TZ)
{
    Geo3 g{};
    g.L0 = L0; g.L1 = L1; g.L2 = L2; g.TX = TX; g.TY = TY; g.TZ = TZ;
    g.n0 = (L0 + TX - 1) / TX;
    g.n1 = (L1 + TY - 1) / TY;
    g.n2 = (L2 + TZ - 1) / TZ;
    g.TBX = std::min(32 / TX, g.n0);
    g.TBY = std::min(k3Rows / TY, g.n1);
    g.TBZ = std::min(k3Layers / TZ, g.n2);
    fit3(g);
    return g;
}

// Passes of draws of a piece: its tiles' lanes, a warp at a time.
__host__ __device__ inline uint32_t passes3(const Geo3 &g, uint32_t W) { return (g.py * (32 / g.TX) * W + 31) / 32; }

// Smaller blocks for a small lattice whose blocks leave half of the SMs idle and would draw in more passes than
// a CTA has warps: tile 8 x 1 x 3 with W 32 on 38 x 12 x 60 59 -> 27 us a sweep (8 blocks of 400 passes become 64),
// 8 x 1 x 1 with W 32 on 64^3 70 -> 41, 16 x 2 x 1 on 2 x 16 x 18 30 -> 18.  The default tile's blocks have 16 passes and stay.
inline void spread3(Geo3 &g, uint32_t W)
{
    while (passes3(g, W) * g.pcy * g.TBZ > k3MaxThreads / 32 && 2 * g.nbx * g.nby * g.nbz <= k3ShareBlocks &&
           g.TBY * g.TBZ > 1) {
        if (g.TBZ > 1 && (g.BZ >= g.BY || g.TBY == 1))
            g.TBZ = (g.TBZ + 1) / 2;
        else
            g.TBY = (g.TBY + 1) / 2;
        fit3(g);
    }
}

// Face bitmaps of a block: a bit per row (zl * k3Rows + yl) for +x, a word per layer for +y, a word per
// row for +z.
constexpr uint32_t k3FaceX = k3Rows * k3Layers / 32, k3FaceY = k3Layers, k3FaceZ = k3Rows;
constexpr uint32_t k3FaceWords = k3FaceX + k3FaceY + k3FaceZ;
constexpr uint32_t k3FaceSites = k3Rows * k3Layers + 32 * (k3Layers + k3Rows);
// A block's merge slots: the number of active face bonds, then the root each of their unions linked.
constexpr uint32_t k3Slots = k3FaceSites + 1;

__host__ __device__ inline uint32_t pieces3(const Geo3 &g) { return g.pcy * g.TBZ; }

// Updates of a tile's lanes per sweep: the requests of its rows for x, y, z, then the face request.
struct Draws3 {
    uint32_t ur, y, z, face, total;  // updates per row request; first update of each part
};
template <int W>
__host__ __device__ inline Draws3 draws3(uint32_t TX, uint32_t TY, uint32_t TZ)
{
    Draws3 d{};
    d.ur = (TX + W - 1) / W;
    d.y = TY * TZ * d.ur;
    d.z = d.y + (TY - 1) * TZ * d.ur;
    d.face = d.z + TY * (TZ - 1) * d.ur;
    d.total = d.face + (TX * TZ + TY * TZ + TX * TY + W - 1) / W;
    return d;
}

struct Assign3Smem {
    uint32_t raw, scan, work, links, sums, pairs, total;  // byte offsets (parent is at 0)
    uint32_t wcap, rows;                                  // words of a piece's work area; rows of a piece
};

template <int W>
__host__ __device__ inline Assign3Smem assign3_smem(const Geo3 &g)
{
    Assign3Smem s{};
    const uint32_t np = pieces3(g), nd = passes3(g, W) * draws3<W>(g.TX, g.TY, g.TZ).total;
    s.rows = g.py * g.TY * g.TZ;
    s.wcap = nd > 2 * s.rows ? nd : 2 * s.rows;
    s.wcap = s.wcap > k3Window / 2 ? s.wcap : k3Window / 2;
    s.wcap += s.wcap & 1u;  // a row's marks are 8 bytes, and the pieces' areas follow each other
    s.raw = g.BZ * k3Layer * 4;                        // [row] {x, y, z bonds, -}, shared by the block
    s.scan = s.raw + g.BZ * k3Rows * 16;               // [piece][row] scan words (below)
    s.work = s.scan + np * s.rows * 32;                // [piece] ballots, then marks, then listed unions
    s.links = s.work + np * s.wcap * 4;                // [piece] linked labels, uint16
    s.sums = s.links + np * k3Links * 2;               // energy and magnetisation sums, deep flag
    s.pairs = (s.sums + 16 + 7) & ~7u;
    s.total = s.pairs + 40;
    return s;
}

constexpr uint32_t k3SmemMax = 100 * 1024;  // above any block's need (checked at creation)

}  // namespace swb
