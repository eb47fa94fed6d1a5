// The assign phase of a 2D sweep: lcg32 draws, bonds and connected components of a block (up to
// 128 x 32 sites), from spins and streams in global memory to the encoded labels.  Shared by the
// single-lattice and the batched kernels.
//
// A warp owns a piece of the block, 32 columns (a strip) of a band of tile rows, from the draws to
// the labelling and exchanges nothing with the others until the pieces are joined:
//
//   spins    lane r packs row r of the piece (32 bytes) into one word;
//   draws    one W-lane segment per tile, 32 / W tiles per pass; every update's warp ballot of the
//            accept bits goes to the piece's shared words;
//   bonds    lane r forms row r's x- and y-bond words from the spin words and the ballots;
//   scan     lane k holds column k: row after row, every x-run takes the label above its leftmost
//            y-bonded site, or its own first site as a new label, and stores it as the site's parent;
//            y-bonds that meet another label are marked, listed and united together, one per lane;
//   join     bonds across the pieces; labels that a union hung below another are pointed at their
//            root; every site's label is two lookups away.
//
// With many blocks a block is one band (4 warps: no seams between bands, and instruction issue is what
// bounds it: 2.5 warp instructions per site, of which scan 0.8, draws 0.7, unions 0.5, labels 0.3, the
// rest 0.2); with few, a band per tile row (up to 16 warps), which shortens every warp's serial walk.
// 16384^2 with 16 x 8 tiles: 903 us a launch (1305 with staged spins, bond words through shared memory and
// a find per site).
#pragma once

#include "sw_core.cuh"

namespace swb {

constexpr uint32_t kStripThreads = 128;  // one band: a warp per strip, blocks are at most 128 columns wide
constexpr uint32_t kBandsMax = 4;        // bands of a block that is short of company
// A piece's list of unions, in the draws' words (dead by then).  A 32 x 32 piece has 20 to 110 at T in
// [1.5, 3.5]; more take further rounds.
constexpr uint32_t kStripList = 128;

// Bands of a block by a CTA of `threads`: whole tile rows, tpb of them each.
__host__ __device__ inline uint32_t band_tile_rows(const Geo &g, uint32_t bands) { return (g.TBY + bands - 1) / bands; }

struct StripSmem {
    uint32_t parent, words, last, draws, sums, pairs, total;  // byte offsets
    uint32_t slots, dcap;                              // updates per pass; words per piece
};

__host__ __device__ inline StripSmem strip_smem(const Geo &g, uint32_t W, uint32_t bands)
{
    StripSmem s{};
    const uint32_t ns = (g.BX + 31) / 32, tps = 32 / g.TX;
    s.slots = draw_slots(g, W);
    const uint32_t nd = (band_tile_rows(g, bands) * tps * W + 31) / 32 * s.slots;
    s.dcap = nd > kStripList ? nd : kStripList;
    s.parent = 0;                                      // [BY][kBlockPitch] uint32
    s.words = g.BY * kBlockPitch * 4;                  // [strip][BY] row words (below)
    s.last = s.words + ns * g.BY * 16;                 // [band][strip] {y, x} bonds of the piece's last row
    s.draws = s.last + ns * bands * 8;                 // [band][strip][dcap]
    s.sums = s.draws + ns * bands * s.dcap * 4;        // energy and magnetisation sums, deep flag, edge words 0, 5, 6
    s.pairs = (s.sums + 32 + 7) & ~7u;                 // the five (a, c) pairs of lcg32, 8 bytes each
    s.total = s.pairs + 40;
    return s;
}

// The largest strip_smem of any tile shape with lcg width W.
inline uint32_t strip_smem_max(uint32_t W, uint32_t bands)
{
    uint32_t m = 0;
    for (uint32_t tx = 8; tx <= 32; tx *= 2)
        for (uint32_t ty = 2; ty <= 32; ++ty) {
            const uint32_t t = strip_smem(make_geo(128, 32, tx, ty), W, bands).total;
            m = t > m ? t : m;
        }
    return m;
}

// Bits of the `n` (even, up to 32) spins at p: 16-byte loads where p allows them, else 4- or 2-byte
// loads (extents and block offsets are even, so 2-byte alignment always holds).
__device__ __forceinline__ uint32_t strip_row_bits(const uint8_t *p, const uint32_t n, const uint32_t align)
{
    if (align >= 16 && n == 32) {
        const uint4 a = reinterpret_cast<const uint4 *>(p)[0], b = reinterpret_cast<const uint4 *>(p)[1];
        return spin_nibble(a.x) | spin_nibble(a.y) << 4 | spin_nibble(a.z) << 8 | spin_nibble(a.w) << 12 |
               spin_nibble(b.x) << 16 | spin_nibble(b.y) << 20 | spin_nibble(b.z) << 24 | spin_nibble(b.w) << 28;
    }
    uint32_t s = 0;
    if (align >= 4) {  // n is a multiple of 4
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k)
            if (4 * k < n)
                s |= spin_nibble(reinterpret_cast<const uint32_t *>(p)[k]) << (4 * k);
    } else {
#pragma unroll
        for (uint32_t k = 0; k < 16; ++k)
            if (2 * k < n) {
                const uint32_t v = reinterpret_cast<const uint16_t *>(p)[k];
                s |= ((v | v >> 7) & 3u) << (2 * k);
            }
    }
    return s;
}

// The draws of one sweep for a piece: tile rows [trow0, trow0 + trows) of the block, one strip.  Tile q of
// the piece (tile rows outer, the strip's 32 / TX tile columns inner) is segment q % (32 / W) of pass
// q / (32 / W); update u of pass p leaves its ballot in d[p * slots + u].  Row request r (tile_x numbers;
// element k is lane k % W after update k / W + 1 of the request) starts at update r * Ur, the merge
// request (tile_x + tile_y numbers: bottom edge, then right edge) at update (2 tile_y - 1) * Ur; a tile
// shorter than tile_y idles through the rows it lacks.  Lanes past a request's end leave bits that no
// reader takes.
struct StripTile {  // a lane's stream in one pass
    uint32_t tile, jjmax, st, sel, it;
    bool on;
};

template <int W, int TXc, int TYc>
__device__ __forceinline__ StripTile strip_stream(const Geo &g, const uint32_t bxi, const uint32_t byi,
                                                  const uint32_t strip, const uint32_t trow0, const uint32_t trows,
                                                  const uint32_t p, const uint32_t *rng_state, const uint8_t *rng_sel,
                                                  const uint32_t *rng_iter)
{
    constexpr uint32_t kTps = 32 / TXc, kPer = 32 / W;
    const uint32_t TY = TYc ? TYc : g.TY, lane32 = threadIdx.x & 31;
    const uint32_t q = p * kPer + lane32 / W, trow = q / kTps, tcol = strip * kTps + q % kTps;
    const uint32_t tgx = bxi * g.TBX + tcol, tgy = byi * g.TBY + trow0 + trow;
    StripTile t;
    t.on = trow < trows && tcol < g.TBX && tgx < g.n0 && tgy < g.n1;
    t.tile = tgy * g.n0 + tgx;
    t.jjmax = t.on ? min(TY, g.L1 - tgy * TY) : 0;
    t.st = t.sel = t.it = 0;
    if (t.on) {
        t.st = rng_state[(size_t)t.tile * W + lane32 % W];
        t.sel = rng_sel[(size_t)t.tile * W + lane32 % W];
        t.it = rng_iter[t.tile];
    }
    return t;
}

// `first` is pass 0's strip_stream; every pass loads the next one's while it draws.
template <int W, int TXc, int TYc>
__device__ __forceinline__ void strip_draws(const Geo &g, const uint32_t bxi, const uint32_t byi, const uint32_t strip,
                                            const uint32_t trow0, const uint32_t trows, const StripTile &first_tile,
                                            uint32_t *d, const uint32_t slots, const uint2 *pairs,
                                            uint32_t *__restrict__ rng_state, uint8_t *__restrict__ rng_sel,
                                            uint32_t *__restrict__ rng_iter, const uint32_t thr)
{
    constexpr uint32_t kTps = 32 / TXc, kPer = 32 / W;
    const uint32_t TY = TYc ? TYc : g.TY;
    const uint32_t lane32 = threadIdx.x & 31, lane = lane32 % W;
    const uint32_t passes = (trows * kTps + kPer - 1) / kPer;
    StripTile next_tile = first_tile;
    for (uint32_t p = 0; p < passes; ++p, d += slots) {
        const StripTile t = next_tile;
        if (p + 1 < passes)
            next_tile = strip_stream<W, TXc, TYc>(g, bxi, byi, strip, trow0, trows, p + 1, rng_state, rng_sel, rng_iter);
        const uint32_t tile = t.tile, jjmax = t.jjmax;
        const bool on = t.on;
        const uint32_t onm = __ballot_sync(0xffffffffu, on);
        if (onm == 0)
            continue;
        // swb_sweep_static's indices are its caller's: one past the last pair acts as the last, as in lcg_param_a,
        // and reads nothing behind the table of pairs.  (Not where they are loaded, which would wait for the
        // load a pass early: 16384^2 sweep 1.32 -> 1.36 ms.)
        uint32_t st = t.st, sel = min(t.sel, 4u), it = t.it;
        uint2 ac = pairs[sel];
        // The parameter rotation of LCG32_State::Update (random/src/lcg32.cpp:51-84): before
        // update itn when itn is a multiple of 15, the (a, c) pairs rotate by
        // state[itn & (W-1)] + (itn odd ? 0 : 1).
        auto rotate = [&](const uint32_t itn, const bool rot) {
            const uint32_t src = __shfl_sync(0xffffffffu, st, itn & (W - 1), W);
            const uint32_t from = (lane + src + ((itn & 1u) ? 0u : 1u)) & (W - 1);
            const uint32_t s2 = __shfl_sync(0xffffffffu, sel, from, W);
            if (rot) {
                sel = s2;
                ac = pairs[sel];
            }
        };
        auto draw = [&](const uint32_t k) {
            st = ac.x * st + ac.y;
            const uint32_t word = __ballot_sync(0xffffffffu, lcg_accept(st, thr));
            if (lane32 == 0)
                d[k] = word;
        };
        // Full-height tiles whose iteration counts agree (they do unless a program imported streams
        // or a lattice's last tile row is cut short): nothing is predicated and the rotations come
        // before the same updates for the whole warp.  Segments off the lattice run along and store
        // nothing.
        const uint32_t itu = __shfl_sync(0xffffffffu, it, __ffs(onm) - 1);
        if (__all_sync(0xffffffffu, !on || (jjmax == TY && it == itu))) {
            const uint32_t first = kShuffleDistance - 1 - itu % kShuffleDistance;  // the first update with a rotation
            if constexpr (TYc != 0) {
                // compile-time count: one straight-line sequence per rotation phase
                constexpr uint32_t kN = (2 * TYc - 1) * ((TXc + W - 1) / W) + (TXc + TYc + W - 1) / W;
                auto run = [&](auto phase) {
                    draw_sequence<decltype(phase)::value>(std::make_integer_sequence<uint32_t, kN>{}, rotate, draw, itu);
                };
                switch (first) {
                case 0: run(U32<0>{}); break;
                case 1: run(U32<1>{}); break;
                case 2: run(U32<2>{}); break;
                case 3: run(U32<3>{}); break;
                case 4: run(U32<4>{}); break;
                case 5: run(U32<5>{}); break;
                case 6: run(U32<6>{}); break;
                case 7: run(U32<7>{}); break;
                case 8: run(U32<8>{}); break;
                case 9: run(U32<9>{}); break;
                case 10: run(U32<10>{}); break;
                case 11: run(U32<11>{}); break;
                case 12: run(U32<12>{}); break;
                case 13: run(U32<13>{}); break;
                default: run(U32<14>{}); break;
                }
            } else {
                for (uint32_t k = 0, next = first; k < slots; ++k) {
                    if (k == next) {
                        rotate(itu + k + 1, true);
                        next += kShuffleDistance;
                    }
                    draw(k);
                }
            }
            it += slots;
        } else {
            constexpr uint32_t Ur = (TXc + W - 1) / W;
            const uint32_t Um = (TXc + TY + W - 1) / W;
            const uint32_t nrow = on ? 2 * jjmax - 1 : 0;
            uint32_t to_rot = kShuffleDistance - it % kShuffleDistance;  // updates until the next rotation
            auto advance = [&](const uint32_t u, const bool upd) {
                const bool rot = upd && to_rot == 1;
                if (__any_sync(0xffffffffu, rot))
                    rotate(it + 1, rot);
                if (upd) {
                    it += 1;
                    st = ac.x * st + ac.y;
                    to_rot = rot ? kShuffleDistance : to_rot - 1;
                }
                const uint32_t word = __ballot_sync(0xffffffffu, upd && lcg_accept(st, thr));
                if (lane32 == 0)
                    d[u] = word;
            };
            uint32_t u = 0;
            for (uint32_t req = 0; req < 2 * TY - 1; ++req)
                for (uint32_t sub = 0; sub < Ur; ++sub, ++u)
                    advance(u, req < nrow);
            for (uint32_t sub = 0; sub < Um; ++sub, ++u)
                advance(u, on);
        }
        if (on) {
            rng_state[(size_t)tile * W + lane] = st;
            rng_sel[(size_t)tile * W + lane] = (uint8_t)sel;
            if (lane == 0)
                rng_iter[tile] = it;
        }
    }
}

// Accept bits (x bonds, y bonds) of row r of a piece of `rows` rows, one bit per column, from the ballots.
template <int W, int TXc, int TYc>
__device__ __forceinline__ void strip_accept(const Geo &g, const uint32_t *d, const uint32_t slots, const uint32_t r,
                                             const uint32_t rows, const uint32_t ncols, uint32_t &AX, uint32_t &AY)
{
    constexpr uint32_t kTps = 32 / TXc, Ur = (TXc + W - 1) / W;
    const uint32_t TY = TYc ? TYc : g.TY, um = (2 * TY - 1) * Ur;
    const uint32_t trow = r / TY, jj = r - trow * TY, jjmax = min(TY, rows - trow * TY);
    AX = AY = 0;
    if constexpr (TXc == W) {
        if (ncols == 32) {  // the ballot of a row's update is the row's accept word
            constexpr uint32_t kOnes = TXc == 8 ? 0x01010101u : TXc == 16 ? 0x00010001u : 1u;
            const uint32_t *t = d + trow * slots;
            const uint32_t m = (t[um + 1 + jj / W] >> (jj % W)) & kOnes;  // right edges: element tile_x + jj
            AX = (t[jj] & ~(kOnes << (TXc - 1))) | m << (TXc - 1);
            AY = t[jj + 1 < jjmax ? jjmax + jj : um];
            return;
        }
    }
    const DrawWords<W> dw{d, slots};
#pragma unroll
    for (uint32_t k = 0; k < kTps; ++k) {
        if (k * TXc < ncols) {
            const uint32_t q = trow * kTps + k, iimax = min((uint32_t)TXc, ncols - k * TXc);
            const uint32_t tmask = 0xFFFFFFFFu >> (32 - iimax);
            const uint32_t xb = (dw.req(q, jj * Ur, Ur) & (tmask >> 1)) | dw.bit(q, um, TXc + jj) << (iimax - 1);
            const uint32_t yb = dw.req(q, jj + 1 < jjmax ? (jjmax + jj) * Ur : um, Ur) & tmask;
            AX |= xb << (k * TXc);
            AY |= yb << (k * TXc);
        }
    }
}

// Block (bxi, byi) of a lattice by a CTA of 32 threads per strip and band; smem holds
// strip_smem(g, W, bands).total bytes.  kMeasure: also add the block's energy and magnetisation sums
// (of the spins the sweep starts from) to meas.obs.  kMayDump: `dump` may ask for the bonds and the
// block's labels.  kEarly: the kernel was launched by launch_next; the draws come before the wait
// for the previous kernel, which must not write the streams (the previous sweep's assign, which does, is two
// or more kernels back).
template <int W, int TXc, int TYc, bool kMeasure, bool kMayDump, bool kEarly>
__device__ __forceinline__ void assign_strips(const Geo &g, const uint32_t bxi, const uint32_t byi,
                                              const uint32_t bands, const uint8_t *spins,
                                              uint32_t *labels, uint32_t *__restrict__ rng_state,
                                              uint8_t *__restrict__ rng_sel, uint32_t *__restrict__ rng_iter,
                                              const uint32_t thr, uint32_t *edge, const AssignDump &dump,
                                              const MeasureArgs &meas, unsigned char *smem)
{
    const StripSmem L = strip_smem(g, W, bands);
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nstrips = (g.BX + 31) / 32;
    const uint32_t band = bands == 1 ? 0 : warp / nstrips, strip = warp - band * nstrips;
    const uint32_t x0 = bxi * g.BX, y0 = byi * g.BY, xs = strip * 32;
    const uint32_t bxv = min(g.BX, g.L0 - x0), byv = min(g.BY, g.L1 - y0);
    // the piece: ncols columns from xs, rows [r0, r0 + rows) of the block (ncols 0: none)
    const uint32_t tpb = band_tile_rows(g, bands), TY = TYc ? TYc : g.TY;
    const uint32_t r0 = band * tpb * TY, rows = min(tpb * TY, byv - min(r0, byv));
    const uint32_t ncols = strip < nstrips && band < bands && rows != 0 && xs < bxv ? min(32u, bxv - xs) : 0u;
    uint32_t *parent = reinterpret_cast<uint32_t *>(smem + L.parent);
    uint4 *words = reinterpret_cast<uint4 *>(smem + L.words) + strip * g.BY + r0;  // lane r: row r0 + r
    uint2 *last = reinterpret_cast<uint2 *>(smem + L.last) + warp;
    uint32_t *d = reinterpret_cast<uint32_t *>(smem + L.draws) + warp * L.dcap;
    uint32_t *eblk = edge + ((size_t)byi * g.nbx + bxi) * kEdgeWords;
    int *sums = reinterpret_cast<int *>(smem + L.sums);
    uint2 *pairs = reinterpret_cast<uint2 *>(smem + L.pairs);
    if (threadIdx.x < 5) {
        pairs[threadIdx.x] = make_uint2(lcg_param_a(threadIdx.x), lcg_param_c(threadIdx.x));
    }
    if (threadIdx.x < 6)
        sums[threadIdx.x] = 0;
    const uint32_t trow0 = band * tpb, trows = ncols ? min(tpb, g.TBY - trow0) : 0;
    const StripTile first_tile =
        strip_stream<W, TXc, TYc>(g, bxi, byi, strip, trow0, trows, 0, rng_state, rng_sel, rng_iter);
    __syncthreads();

    if (ncols != 0) {
        strip_draws<W, TXc, TYc>(g, bxi, byi, strip, trow0, trows, first_tile, d, L.slots, pairs, rng_state, rng_sel,
                                 rng_iter, thr);
        if constexpr (kEarly)
            after_previous();

        // spins: lane r's row word S, the bit right of its last column, the row below the piece
        uint32_t S = 0, right = 0;
        {
            const uint32_t both = g.L0 | x0, align = (both & 15u) == 0 ? 16 : (both & 3u) == 0 ? 4 : 2;
            const uint32_t xe = x0 + xs + ncols;
            if (lane < rows) {
                const uint8_t *row = spins + (size_t)(y0 + r0 + lane) * g.L0;
                S = strip_row_bits(row + x0 + xs, ncols, align);
                right = row[xe < g.L0 ? xe : 0u];
            }
        }
        const uint32_t yh = y0 + r0 + rows, hy = yh < g.L1 ? yh : 0u;  // row below the piece (periodic)
        const uint32_t hb = lane < ncols ? spins[(size_t)hy * g.L0 + x0 + xs + lane] : 0u;
        const uint32_t below_row = __ballot_sync(0xffffffffu, hb != 0);

        __syncwarp();

        // bonds: equal spins and an accepted draw
        uint32_t D = __shfl_down_sync(0xffffffffu, S, 1);
        if (lane + 1 == rows)
            D = below_row;
        const uint32_t colm = 0xFFFFFFFFu >> (32 - ncols);
        const uint32_t dx = S ^ (S >> 1 | right << (ncols - 1)), dy = S ^ D;
        uint32_t X = 0, Y = 0;
        if (lane < rows) {
            uint32_t AX, AY;
            strip_accept<W, TXc, TYc>(g, d, L.slots, lane, rows, ncols, AX, AY);
            X = ~dx & AX & colm;
            Y = ~dy & AY & colm;
            if (lane + 1 == rows) {
                *last = make_uint2(Y, X);
                if (r0 + rows == byv) {
                    eblk[1 + strip] = Y;  // bonds out of the block's last row
                    eblk[kEdgeXLast + strip] = X;
                }
            }
            if (r0 + lane == 0)
                eblk[kEdgeXFirst + strip] = X;
        }
        // Row words: the gaps ~X; the first y-bond up or run end from a run's start is the run's first
        // set bit of the second (bit 31 always ends a strip run); the bonds Yu to the row above; and of
        // those the ones that may unite: a bond whose left neighbour is bonded up too, with both
        // rows bonded across, meets the same two runs as that neighbour's.
        {
            uint32_t Yu = __shfl_up_sync(0xffffffffu, Y, 1);
            const uint32_t Xu = __shfl_up_sync(0xffffffffu, X, 1);
            if (lane == 0)
                Yu = 0;
            if (lane < rows)
                words[lane] = make_uint4(~X, Yu | ~X | 0x80000000u, Yu, Yu & ~((Yu & X & Xu) << 1));
        }
        if (xs + 32 >= bxv) {  // bonds out of the block's last column, and along it
            const uint32_t e = __ballot_sync(0xffffffffu, (X >> (ncols - 1)) & 1u);
            const uint32_t yl = __ballot_sync(0xffffffffu, (Y >> (ncols - 1)) & 1u);
            if (lane == 0) {
                atomicOr(reinterpret_cast<unsigned int *>(sums) + 3, e << r0);
                atomicOr(reinterpret_cast<unsigned int *>(sums) + 4, yl << r0);
            }
        }
        if (strip == 0) {
            const uint32_t yf = __ballot_sync(0xffffffffu, Y & 1u);
            if (lane == 0)
                atomicOr(reinterpret_cast<unsigned int *>(sums) + 5, yf << r0);
        }
        if constexpr (kMeasure) {  // s (s_right + s_down) and s: +1 per equal pair, -1 per unequal one
            int e = 0, m = 0;
            if (lane < rows) {
                e = 2 * (int)ncols - 2 * (__popc(dx & colm) + __popc(dy & colm));
                m = 2 * __popc(S) - (int)ncols;
            }
            e = __reduce_add_sync(0xffffffffu, e);
            m = __reduce_add_sync(0xffffffffu, m);
            if (lane == 0) {
                atomicAdd(sums, e);
                atomicAdd(sums + 1, m);
            }
        }
        __syncwarp();

        // Scan.  A run (x-bonded sites of the strip row; its first lane from the gap mask below the
        // lane) takes the label above its leftmost y-bonded site, or with none its own first site as a
        // new label.  A y-bond of the run that meets a different label unites the two: such sites are
        // only marked here (one ballot per row).  Deferring the unions changes no label, and the
        // union-find's roots (each set's minimum) do not depend on the order of the unions.
        const uint32_t under = (1u << lane) - 1u, bit = 1u << lane;
        uint32_t above = 0, base = r0 * kBlockPitch + xs;
#pragma unroll 4
        for (uint32_t r = 0; r < rows; ++r, base += kBlockPitch) {
            const uint4 w = words[r];
            int last_gap;  // -1: none
            asm("bfind.u32 %0, %1;" : "=r"(last_gap) : "r"(w.x & under));
            const uint32_t rs = last_gap + 1;
            const uint32_t pos = __clz(__brev(w.y & (0xFFFFFFFFu << rs)));
            const uint32_t rep = __shfl_sync(0xffffffffu, above, pos);
            const uint32_t lab = (w.z & (1u << pos)) ? rep : base + rs;
            const uint32_t m = __ballot_sync(0xffffffffu, (w.w & bit) && above != lab);
            if (lane == 0)
                d[r] = m;
            parent[base + lane] = lab;
            above = lab;
        }
        __syncwarp();
    }
    if (kEarly && ncols == 0)
        after_previous();
    __syncthreads();

    // The unions, within the pieces and across them: lane r lists row r's marked sites (a band's first row:
    // those bonded to the band above) and the bond from its last column into the next strip (unless the
    // rows above join the same runs); then the list is worked off one entry per lane -- inside the scan
    // they would run, divergent, on almost every row.  Each entry becomes the label its union hung below
    // another (every label at most once), or none.
    uint32_t listed = 0;
    if (ncols != 0) {
        uint32_t mine = lane < rows ? d[lane] : 0u, across = 0;
        if (lane == 0 && band != 0) {
            const uint2 up = last[-(int)nstrips];  // {y, x} bonds of the row above the piece
            mine = up.x & ~((up.x & up.y & ~words[0].x) << 1);
        }
        if (ncols == 32 && xs + 32 < bxv && lane < rows) {
            const uint4 a = words[lane], b = words[g.BY + lane];
            const bool same = lane != 0 && (~words[lane - (lane != 0)].x & a.z) >> 31 && (b.z & 1u);
            across = !(a.x >> 31) && !same;
        }
        __syncwarp();
        uint32_t end = __popc(mine) + across;  // inclusive prefix sum over the rows
#pragma unroll
        for (uint32_t o = 1; o < 32; o *= 2) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, end, o);
            if (lane >= o)
                end += v;
        }
        listed = __shfl_sync(0xffffffffu, end, 31);
        const uint32_t l0 = (r0 + lane) * kBlockPitch + xs;
        for (uint32_t b0 = 0; b0 < listed; b0 += kStripList) {
            __syncwarp();
            uint32_t k = end - __popc(mine) - across - b0;
            for (uint32_t left = mine; left; left &= left - 1, ++k)
                if (k < kStripList)  // unsigned: also false before the window
                    d[k] = l0 + __ffs(left) - 1;
            if (across && k < kStripList)
                d[k] = kLocalFlag | (l0 + 31);
            __syncwarp();
            const uint32_t n = min(listed - b0, kStripList);
            for (uint32_t i = lane; i < n; i += 32) {
                const uint32_t v = d[i], l = v & kLocalMask;
                d[i] = uf_union_link(parent, parent[(v & kLocalFlag) ? l + 1 : l - kBlockPitch], parent[l]);
            }
        }
        if (listed > kStripList && lane == 0)
            sums[2] = 1;  // the list no longer holds every linked label
    }
    if (threadIdx.x < 3)
        eblk[threadIdx.x == 0 ? 0 : kEdgeYLast - 1 + threadIdx.x] = (uint32_t)sums[3 + threadIdx.x];
    __syncthreads();

    // Point every linked label straight at its root (they are the only labels that are not roots), so
    // that a site's root is two lookups away; concurrent writers only shorten each other's paths.  A
    // block in bands skips this pass and its barrier: its few sites per thread walk to their roots.
    bool deep = bands != 1;
    if (!deep) {
        for (uint32_t i = lane; i < min(listed, kStripList); i += 32) {
            const uint32_t b = d[i];
            if (b != kNoLink)
                uf_flatten(parent, b);
        }
        __syncthreads();
        deep = sums[2] != 0;
    }

    // Labels: a block root stores its global site index (the merge links these), every other site
    // kLocalFlag | the block-local index of its root.  (The test is on BX: one on nstrips changes the registers of
    // whole instances, 960 x 2336 with 16 x 4 tiles 32 -> 40 us a sweep.)
    if ((g.L0 & 3u) == 0 && g.BX > 32) {
        // four sites per lane and row: one 16-byte load of parents, four lookups, one 16-byte store
        // (rows and x0 are 16-byte aligned)
        const uint32_t x4 = lane * 4, rstep = blockDim.x >> 5;
        if (x4 < bxv) {
            uint32_t l = warp * kBlockPitch + x4, gb = (y0 + warp) * g.L0 + x0 + x4;
#pragma unroll 2
            for (uint32_t yl = warp; yl < byv; yl += rstep, l += rstep * kBlockPitch, gb += rstep * g.L0) {
                const uint4 pp = *reinterpret_cast<const uint4 *>(parent + l);
                uint32_t r[4] = {parent[pp.x], parent[pp.y], parent[pp.z], parent[pp.w]};
                while (deep) {  // the four walks advance together
                    uint32_t z[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        z[k] = parent[r[k]];
                    if (z[0] == r[0] && z[1] == r[1] && z[2] == r[2] && z[3] == r[3])
                        break;
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        r[k] = z[k];
                }
                uint4 o;
                o.x = r[0] == l ? gb : (kLocalFlag | r[0]);
                o.y = r[1] == l + 1 ? gb + 1 : (kLocalFlag | r[1]);
                o.z = r[2] == l + 2 ? gb + 2 : (kLocalFlag | r[2]);
                o.w = r[3] == l + 3 ? gb + 3 : (kLocalFlag | r[3]);
                *reinterpret_cast<uint4 *>(labels + gb) = o;
            }
        }
    } else if (ncols != 0) {
        // Rows of L0 = 2 mod 4 are 8-byte aligned (x0 is a multiple of 8), and a block of one strip would leave most
        // lanes idle above: the warp takes two sites a lane and two rows of its piece at a time.  514^2 with 8 x 8
        // tiles 43.5 us a sweep with a site a lane and a find for each, now 33; 32 x 262144 at T_c 110 with the loop
        // above, now 104.
        const uint32_t x2 = (lane & 15) * 2;
#pragma unroll 2
        for (uint32_t yl = r0 + (lane >> 4); x2 < ncols && yl < r0 + rows; yl += 2) {
            const uint32_t l = yl * kBlockPitch + xs + x2, gb = (y0 + yl) * g.L0 + x0 + xs + x2;
            const uint2 pp = *reinterpret_cast<const uint2 *>(parent + l);
            uint32_t ra = parent[pp.x], rb = parent[pp.y];
            while (deep) {
                const uint32_t za = parent[ra], zb = parent[rb];
                if (za == ra && zb == rb)
                    break;
                ra = za;
                rb = zb;
            }
            *reinterpret_cast<uint2 *>(labels + gb) =
                make_uint2(ra == l ? gb : (kLocalFlag | ra), rb == l + 1 ? gb + 1 : (kLocalFlag | rb));
        }
    }
    if constexpr (kMeasure) {
        if (threadIdx.x == 0)  // the block's sums (complete since the first barrier)
            obs_add_part(meas.obs, meas.series, meas.cap, (size_t)g.L0 * g.L1, g.nbx * g.nby, sums[0], sums[1], 1);
    }
    if (kMayDump && (dump.bonds || dump.block_labels)) {  // recording only
        __syncthreads();
        for (uint32_t r = 0; lane < ncols && r < rows; ++r) {
            const size_t site = (size_t)(y0 + r0 + r) * g.L0 + x0 + xs + lane;
            const uint32_t Y = r + 1 < rows ? words[r + 1].z : last->x;
            if (dump.bonds)
                dump.bonds[site] = (uint8_t)(((~words[r].x >> lane) & 1u) | ((Y >> lane) & 1u) << 1);
            if (dump.block_labels)
                dump.block_labels[site] = label_global(g, bxi, byi, labels[site]);
        }
    }
}

// assign_strips with the tile width, and the common tile heights, as constants; kManyShapes false
// keeps only 16 x 8 and 16 x 4 of lcg width 16 (the tiles the B200 table picks).
template <int W, bool kMeasure, bool kMayDump, bool kEarly, bool kManyShapes = true>
__device__ __forceinline__ void assign_strips_any(const Geo &g, const uint32_t bxi, const uint32_t byi,
                                                  const uint32_t bands, const uint8_t *spins, uint32_t *labels,
                                                  uint32_t *__restrict__ rng_state, uint8_t *__restrict__ rng_sel,
                                                  uint32_t *__restrict__ rng_iter, const uint32_t thr,
                                                  uint32_t *edge, const AssignDump &dump,
                                                  const MeasureArgs &meas, unsigned char *smem)
{
#define SWB_STRIPS(tx, ty)                                                                                            \
    {                                                                                                                 \
        assign_strips<W, tx, ty, kMeasure, kMayDump, kEarly>(g, bxi, byi, bands, spins, labels, rng_state, rng_sel,   \
                                                             rng_iter, thr, edge, dump, meas, smem);                  \
        return;                                                                                                       \
    }
    if constexpr (W == 16) {
        if (g.TX == 16 && g.TY == 8) SWB_STRIPS(16, 8)
        if (g.TX == 16 && g.TY == 4) SWB_STRIPS(16, 4)
    }
    if constexpr (W != 16 || kManyShapes) {
        if (g.TX == 8) SWB_STRIPS(8, 0)
        if (g.TX == 16) SWB_STRIPS(16, 0)
        SWB_STRIPS(32, 0)
    }
#undef SWB_STRIPS
}

}  // namespace swb
