// A whole sweep of a small lattice in one kernel: a thread-block cluster holds the lattice, each CTA the
// labels of its rows in shared memory, from the draws to the flip.
//
// What bounds the three- or four-kernel sweep of a small lattice is latency: launches, and chains of
// dependent loads of labels through L2.  Here CTA r owns tile rows [r tr, (r + 1) tr) over the full width,
// so a site's place (rank, row * pitch + x) orders as its site index does; the pieces (32 columns of a tile
// row, one warp each, as in sw_strip.cuh) are drawn, scanned and joined inside the CTA, the last row of
// each CTA is united with the next CTA's first row through distributed shared memory, linked roots are
// resolved and every site flips from shared memory: one launch, two cluster barriers and a last one
// that keeps the shared memory alive.  128^2 12.4 us a sweep (17.5 in three kernels), 256^2 13.8
// (19.5); of 256^2's, in clocks: loads 1500, draws 1000, bonds 300, scan 1850, unions 4000, the exchange between
// CTAs up to 14000 (a walk along the chain of their roots, some 900 a remote step), resolve 2500, flip 2300.
#pragma once

#include <cooperative_groups.h>

#include "sw_strip.cuh"

namespace swb {

constexpr uint32_t kWholeSites = 32768;   // parents per CTA, at most (128 KiB)
constexpr uint32_t kWholeCtas = 16;       // CTAs of a cluster, at most
constexpr uint32_t kWholeThreads = 1024;  // a warp per piece
constexpr uint32_t kWholeList = 64;       // unions of a piece listed at a time (a 32 x 8 piece has about 40)

struct Whole {
    Geo g;              // TBX = n0: a tile row of the lattice
    uint32_t pitch;     // strips * 32
    uint32_t strips;
    uint32_t tr;        // tile rows per CTA
    uint32_t ctas;      // cluster size
};

struct WholeSmem {
    uint32_t raw, spin, scan, work, counts, edge, sums, pairs, total;  // byte offsets (parent is at 0)
    uint32_t slots, wcap, rows;                                        // rows per CTA
};

__host__ __device__ inline WholeSmem whole_smem(const Whole &w, uint32_t W)
{
    WholeSmem s{};
    const uint32_t tps = 32 / w.g.TX, pieces = w.strips * w.tr;
    s.rows = w.tr * w.g.TY;
    s.slots = draw_slots(w.g, W);
    const uint32_t nd = (tps * W + 31) / 32 * s.slots;
    s.wcap = nd > kWholeList ? nd : kWholeList;
    s.raw = s.rows * w.pitch * 4;                 // [strip][row] {x, y bonds}
    s.spin = s.raw + w.strips * s.rows * 8;       // [strip][row] spin words
    s.scan = (s.spin + w.strips * s.rows * 4 + 15) & ~15u;  // [strip][row] scan words
    s.work = s.scan + w.strips * s.rows * 16;     // [piece] ballots, then marks, then listed unions and their links
    s.counts = s.work + pieces * s.wcap * 4;      // [piece] listed unions
    s.edge = s.counts + pieces * 4;               // [2][pitch] roots of the first and the last row's sites
    s.sums = s.edge + 2 * w.pitch * 4;            // energy and magnetisation sums, deep flag
    s.pairs = (s.sums + 16 + 7) & ~7u;
    s.total = s.pairs + 40;
    return s;
}

constexpr uint32_t kWholeSmemMax = 200 * 1024;

// Sets the kernels' attributes on the current device and tells whether the cluster fits it; one sweep
// (sw_whole.cu).
cudaError_t allow_whole(const Whole &w, uint32_t W, bool *fits);
int launch_whole(const Whole &w, uint32_t W, uint8_t *spins, uint32_t *rng_state, uint8_t *rng_sel, uint32_t *rng_iter,
                 uint32_t thr, const MeasureArgs &meas, unsigned int *fault, cudaStream_t st);

// A cluster for the lattice, or ctas = 0 where the phase kernels are faster: the fewest CTAs (a power of
// two, each with a tile row) that leave each at most 16 pieces, and at most 32 with the largest
// cluster.  More CTAs lengthen the chains of roots from row to row, fewer the work of each.  us a sweep
// with 1 / 2 / 4 / 8 / 16 CTAs, phase kernels: 64^2 9.5 / 11.4 / 11.5 / 11.9 / 11.9, 17; 128^2 19.8 / 14.2 /
// 12.4 / 12.9 / 14.7, 17.5; 256 x 128 35.7 / 22.5 / 14.5 / 13.3 / 13.8, 18; 256^2 - / 38.7 / 22.7 / 14.9 / 13.8, 19.5;
// 512 x 256 (32 pieces a CTA) 17.0, 20.1; 512^2 (64) 24.4, 20.6.
inline Whole make_whole(uint32_t L0, uint32_t L1, uint32_t TX, uint32_t TY)
{
    Whole w{};
    w.g = make_geo(L0, L1, TX, TY);
    w.g.TBX = w.g.n0;
    w.strips = (L0 + 31) / 32;
    w.pitch = w.strips * 32;
    for (uint32_t c = 1; c <= kWholeCtas && c <= w.g.n1; c *= 2) {
        w.tr = (w.g.n1 + c - 1) / c;
        const uint64_t pieces = (uint64_t)w.tr * w.strips;
        if ((uint64_t)w.tr * TY * w.pitch <= kWholeSites && pieces <= kWholeThreads / 32) {
            w.ctas = c;
            if (pieces <= 16)
                break;
        }
    }
    if (w.ctas)
        w.tr = (w.g.n1 + w.ctas - 1) / w.ctas;
    return w;
}

// Nodes across the cluster: rank << 16 | offset.  An entry below 2^16 is an offset in its own CTA (its own
// for a root), any other is (rank + 1) << 16 | offset.
struct ClusterNodes {
    uint32_t *parent;  // this CTA's
    uint32_t rank;
    __device__ __forceinline__ uint32_t *at(uint32_t node) const
    {
        return cooperative_groups::this_cluster().map_shared_rank(parent, node >> 16) + (node & 0xFFFFu);
    }
    // the node that node's entry points at
    __device__ __forceinline__ uint32_t next(uint32_t node) const
    {
        return target(node, *(volatile uint32_t *)at(node));
    }
    __device__ __forceinline__ static uint32_t target(uint32_t node, uint32_t v)
    {
        return v < 0x10000u ? (node & 0xFFFF0000u) | v : v - 0x10000u;
    }
    __device__ __forceinline__ static uint32_t entry(uint32_t node, uint32_t to)
    {
        return (node >> 16) == (to >> 16) ? to & 0xFFFFu : to + 0x10000u;
    }
    // Unites two trees: the walk goes on from whichever node has the later parent (a lower place is a
    // smaller site index), so neither side has to reach its root; a root is linked below the other
    // side's parent.
    __device__ __forceinline__ void unite(uint32_t a, uint32_t b, unsigned int *fault) const
    {
        uint32_t pa = next(a), pb = next(b);
        for (uint32_t n = 0; pa != pb; ++n) {
            if (n >= kChainCap) {
                atomicOr(fault, kFaultChain);
                return;
            }
            if (pa < pb) {
                uint32_t t = a;
                a = b;
                b = t;
                t = pa;
                pa = pb;
                pb = t;
            }
            if (a == pa) {
                const uint32_t old = atomicCAS(at(a), a & 0xFFFFu, entry(a, pb));
                if (old == (a & 0xFFFFu))
                    return;
                pa = target(a, old);
            } else {
                a = pa;
                pa = next(a);
            }
        }
    }
};

template <int W, int TXc, int TYc, bool kMeasure>
__device__ __forceinline__ void sweep_whole(const Whole &w, uint8_t *spins, uint32_t *rng_state, uint8_t *rng_sel,
                                            uint32_t *rng_iter, const uint32_t thr, const MeasureArgs &meas,
                                            unsigned int *fault, unsigned char *smem)
{
    namespace cg = cooperative_groups;
    const cg::cluster_group cluster = cg::this_cluster();
    const Geo &g = w.g;
    const WholeSmem S = whole_smem(w, W);
    const uint32_t TY = TYc ? TYc : g.TY, P = w.pitch, rank = w.ctas > 1 ? cluster.block_rank() : 0;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    uint32_t *parent = reinterpret_cast<uint32_t *>(smem);
    uint2 *raw = reinterpret_cast<uint2 *>(smem + S.raw);
    uint32_t *spin = reinterpret_cast<uint32_t *>(smem + S.spin);
    uint32_t *counts = reinterpret_cast<uint32_t *>(smem + S.counts);
    int *sums = reinterpret_cast<int *>(smem + S.sums);
    uint2 *pairs = reinterpret_cast<uint2 *>(smem + S.pairs);
    const uint32_t y0 = min(rank * w.tr * TY, g.L1), rows = min(w.tr * TY, g.L1 - y0);  // the CTA's rows (0: none)
    const uint32_t used = (g.n1 + w.tr - 1) / w.tr;                                     // CTAs that have rows
    const uint32_t npieces = w.strips * ((rows + TY - 1) / TY);

    if (threadIdx.x < 5) {
        pairs[threadIdx.x] = make_uint2(lcg_param_a(threadIdx.x), lcg_param_c(threadIdx.x));
        if (threadIdx.x < 4)
            sums[threadIdx.x] = 0;
    }
    __syncthreads();
    after_previous();

    // ---- draws and bonds of every piece
    for (uint32_t pc = warp; pc < npieces; pc += nwarps) {
        const uint32_t band = pc / w.strips, strip = pc - band * w.strips;
        const uint32_t r0 = band * TY, n = min(TY, rows - r0), xs = strip * 32, ncols = min(32u, g.L0 - xs);
        const uint32_t trow = rank * w.tr + band;
        uint32_t *d = reinterpret_cast<uint32_t *>(smem + S.work) + pc * S.wcap;
        const StripTile first = strip_stream<W, TXc, TYc>(g, 0, 0, strip, trow, 1, 0, rng_state, rng_sel, rng_iter);
        uint32_t s = 0, right = 0;
        if (lane < n) {
            const uint8_t *row = spins + (size_t)(y0 + r0 + lane) * g.L0;
            s = strip_row_bits(row + xs, ncols, (g.L0 & 15u) == 0 ? 16 : (g.L0 & 3u) == 0 ? 4 : 2);
            right = row[xs + ncols < g.L0 ? xs + ncols : 0u];
        }
        const uint32_t yh = y0 + r0 + n, hy = yh < g.L1 ? yh : 0u;
        const uint32_t hb = lane < ncols ? spins[(size_t)hy * g.L0 + xs + lane] : 0u;
        const uint32_t below = __ballot_sync(0xffffffffu, hb != 0);
        strip_draws<W, TXc, TYc>(g, 0, 0, strip, trow, 1, first, d, S.slots, pairs, rng_state, rng_sel, rng_iter, thr);
        __syncwarp();
        uint32_t down = __shfl_down_sync(0xffffffffu, s, 1);
        if (lane + 1 == n)
            down = below;
        const uint32_t colm = 0xFFFFFFFFu >> (32 - ncols);
        const uint32_t dx = s ^ (s >> 1 | right << (ncols - 1)), dy = s ^ down;
        if (lane < n) {
            uint32_t AX, AY;
            strip_accept<W, TXc, TYc>(g, d, S.slots, lane, n, ncols, AX, AY);
            raw[strip * S.rows + r0 + lane] = make_uint2(~dx & AX & colm, ~dy & AY & colm);
            spin[strip * S.rows + r0 + lane] = s;
        }
        if constexpr (kMeasure) {
            int e = 0, m = 0;
            if (lane < n) {
                e = 2 * (int)ncols - 2 * (__popc(dx & colm) + __popc(dy & colm));
                m = 2 * __popc(s) - (int)ncols;
            }
            e = __reduce_add_sync(0xffffffffu, e);
            m = __reduce_add_sync(0xffffffffu, m);
            if (lane == 0) {
                atomicAdd(sums, e);
                atomicAdd(sums + 1, m);
            }
        }
        __syncwarp();

        // ---- scan (as assign_strips) and the piece's unions
        uint4 *scan = reinterpret_cast<uint4 *>(smem + S.scan) + strip * S.rows + r0;
        if (lane < n) {
            const uint32_t X = raw[strip * S.rows + r0 + lane].x;
            uint32_t Yu = 0, U = 0;
            if (lane) {
                const uint2 up = raw[strip * S.rows + r0 + lane - 1];
                Yu = up.y;
                U = Yu & ~((Yu & X & up.x) << 1);
            }
            scan[lane] = make_uint4(~X, Yu | ~X | 0x80000000u, Yu, U);
        }
        __syncwarp();
        const uint32_t under = (1u << lane) - 1u, bit = 1u << lane;
        uint32_t above = 0, base = r0 * P + xs;
        for (uint32_t r = 0; r < n; ++r, base += P) {
            const uint4 v = scan[r];
            int last_gap;  // -1: none
            asm("bfind.u32 %0, %1;" : "=r"(last_gap) : "r"(v.x & under));
            const uint32_t rs = last_gap + 1;
            const uint32_t pos = __clz(__brev(v.y & (0xFFFFFFFFu << rs)));
            const uint32_t rep = __shfl_sync(0xffffffffu, above, pos);
            const uint32_t lab = (v.z & (1u << pos)) ? rep : base + rs;
            const uint32_t m = __ballot_sync(0xffffffffu, (v.w & bit) && above != lab);
            if (lane == 0)
                d[r] = m;
            parent[base + lane] = lab;
            above = lab;
        }
        __syncwarp();
    }
    __syncthreads();

    // ---- the unions (as assign_strips): a piece's marked sites, its first row's bonds to the row above it
    // in the CTA (periodic where one CTA holds the lattice), and the bonds from its last column into the
    // next strip (periodic)
    for (uint32_t pc = warp; pc < npieces; pc += nwarps) {
        const uint32_t band = pc / w.strips, strip = pc - band * w.strips;
        const uint32_t r0 = band * TY, n = min(TY, rows - r0), xs = strip * 32, last = min(32u, g.L0 - xs) - 1;
        const bool end_strip = strip + 1 == w.strips;
        uint32_t *d = reinterpret_cast<uint32_t *>(smem + S.work) + pc * S.wcap;
        uint32_t mine = lane < n ? d[lane] : 0u, across = 0;
        if (lane == 0 && (band != 0 || used == 1)) {
            const uint2 up = raw[strip * S.rows + (r0 ? r0 : rows) - 1];
            mine = up.y & ~((up.y & up.x & raw[strip * S.rows + r0].x) << 1);
        }
        if (lane < n) {
            const uint32_t r = r0 + lane, ns = end_strip ? 0 : strip + 1;
            across = (raw[strip * S.rows + r].x >> last) & 1u;
            if (r) {  // not where the rows above join the same runs
                const uint2 a = raw[strip * S.rows + r - 1];
                across &= ~(((a.x & a.y) >> last) & raw[ns * S.rows + r - 1].y);
            }
        }
        __syncwarp();
        uint32_t end = __popc(mine) + across;
#pragma unroll
        for (uint32_t o = 1; o < 32; o *= 2) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, end, o);
            if (lane >= o)
                end += v;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, end, 31), l0 = (r0 + lane) * P + xs;
        for (uint32_t b0 = 0; b0 < total; b0 += kWholeList) {
            __syncwarp();
            uint32_t k = end - __popc(mine) - across - b0;
            for (uint32_t left = mine; left; left &= left - 1, ++k)
                if (k < kWholeList)  // unsigned: also false before the window
                    d[k] = l0 + __ffs(left) - 1;
            if (across && k < kWholeList)
                d[k] = kLocalFlag | (l0 + last);
            __syncwarp();
            const uint32_t listed = min(total - b0, kWholeList);
            for (uint32_t i = lane; i < listed; i += 32) {
                const uint32_t v = d[i], l = v & kLocalMask;
                const uint32_t to = (v & kLocalFlag) ? (end_strip ? l + 1 - g.L0 : l + 1) : (l >= P ? l : l + rows * P) - P;
                d[i] = uf_union_link(parent, parent[to], parent[l]);
            }
        }
        if (lane == 0) {
            counts[pc] = min(total, kWholeList);
            if (total > kWholeList)
                sums[2] = 1;  // the list no longer holds every linked label
        }
    }
    __syncthreads();
    const bool deep = sums[2] != 0;
    for (uint32_t pc = warp; pc < npieces; pc += nwarps) {
        const uint32_t *d = reinterpret_cast<const uint32_t *>(smem + S.work) + pc * S.wcap;
        for (uint32_t i = lane; i < counts[pc]; i += 32)
            if (d[i] != kNoLink)
                uf_flatten(parent, d[i]);
    }
    __syncthreads();

    if (used > 1) {
        uint32_t *edge = reinterpret_cast<uint32_t *>(smem + S.edge);  // [0] first row, [pitch] last row
        for (uint32_t i = threadIdx.x; rows && i < 2 * P; i += blockDim.x)
            edge[i] = uf_find(parent, parent[i < P ? i : (rows - 2) * P + i]);
        cluster.sync();  // every CTA's labels stand
        // ---- the last row's y-bonds into the next CTA's first row, one lane per pair of roots
        const ClusterNodes nodes{parent, rank};
        const uint32_t after = rank + 1 < used ? rank + 1 : 0;
        const volatile uint32_t *top = cluster.map_shared_rank(edge, after);
        for (uint32_t strip = warp; rows && strip < w.strips; strip += nwarps) {
            const uint32_t x = strip * 32 + lane;
            const bool go = (raw[strip * S.rows + rows - 1].y >> lane) & 1u;
            const uint32_t ra = edge[P + x], rb = go ? top[x] : 0u, key = go ? ra << 16 | rb : 0xFFFF0000u | lane;
            const uint32_t same = __match_any_sync(0xffffffffu, key);
            if (go && lane == __ffs(same) - 1)
                nodes.unite(rank << 16 | ra, after << 16 | rb, fault);
        }
        cluster.sync();  // no union is left
        // ---- every root that was linked is the root of a site in its CTA's first or last row: it is pointed at
        // the cluster's root.  Every step is stored, so that the CTAs' walks shorten one another's.
        for (uint32_t i = threadIdx.x; rows && i < 2 * P; i += blockDim.x) {
            const uint32_t r = edge[i];
            const uint32_t same = __match_any_sync(0xffffffffu, r);  // whole warps: 2 P and the step are multiples of 32
            if (lane == __ffs(same) - 1 && ((volatile uint32_t *)parent)[r] != r) {
                uint32_t t = nodes.next(rank << 16 | r);
                for (uint32_t n = 0; n < kChainCap; ++n) {
                    ((volatile uint32_t *)parent)[r] = t + 0x10000u;
                    const uint32_t u = nodes.next(t);
                    if (u == t)
                        break;
                    t = u;
                }
            }
        }
        cluster.barrier_arrive();  // this CTA reads no other's labels any more
    }
    __syncthreads();

    // ---- flip: a site's label, its root in the CTA, the cluster's root are at most three lookups away; the
    // root's offset is odd iff its site index is (extents and pitch are even)
    auto odd = [&](uint32_t v) {  // v: a site's entry
        v = v < 0x10000u ? parent[v] : v;
        v = v < 0x10000u ? parent[v] : v;
        while (deep && v < 0x10000u && parent[v] != v)
            v = parent[v];
        return v & 1u;
    };
    if ((g.L0 & 3u) == 0) {
        const uint32_t nq = (g.L0 + 127) / 128;  // 128 columns per warp and step
        for (uint32_t i = warp; i < rows * nq; i += nwarps) {
            const uint32_t r = i / nq, x = (i - r * nq) * 128 + lane * 4;
            if (x < g.L0) {
                const uint4 pp = *reinterpret_cast<const uint4 *>(parent + r * P + x);
                const uint32_t f = odd(pp.x) | odd(pp.y) << 8 | odd(pp.z) << 16 | odd(pp.w) << 24;
                const uint32_t b = (spin[(x >> 5) * S.rows + r] >> (x & 31)) & 15u;
                reinterpret_cast<uint32_t *>(spins + (size_t)(y0 + r) * g.L0)[x >> 2] =
                    ((b * 0x00204081u) & 0x01010101u) ^ f;
            }
        }
    } else {
        for (uint32_t i = warp; i < rows * w.strips; i += nwarps) {
            const uint32_t r = i / w.strips, strip = i - r * w.strips, x = strip * 32 + lane;
            if (x < g.L0)
                spins[(size_t)(y0 + r) * g.L0 + x] =
                    (uint8_t)(((spin[strip * S.rows + r] >> lane) & 1u) ^ odd(parent[r * P + x]));
        }
    }
    if constexpr (kMeasure) {
        if (threadIdx.x == 0)
            obs_add_part(meas.obs, meas.series, meas.cap, (size_t)g.L0 * g.L1, w.ctas, sums[0], sums[1], 1);
    }
    if (used > 1)
        cluster.barrier_wait();  // the others are done with this CTA's labels
}

}  // namespace swb
