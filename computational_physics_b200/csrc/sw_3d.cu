// Swendsen-Wang sweep for the 3D Ising model (J = 1, periodic L0 x L1 x L2) on one B200.  The
// reference names the 3D case only (ising/include/swendsen_wang_selflabeling.hpp:20-22); this
// engine extends the 2D conventions: spins uint8 0/1 with site index (z L1 + y) L0 + x, one lcg32
// stream per tile of tx x ty x tz sites seeded seed_base + tile id, the draw order of
// oracle/sw_oracle.c's orc3_sw_sweep (per row: +x requests, then +y, then +z, then one face
// request for the tile's +y, +x and +z faces), the integer accept threshold, labels = minimum
// site index of each cluster, a cluster flips iff its label is odd.
//
// One sweep = four kernels, the 2D split:
//   k3_assign   one CTA per block of tiles: draws, bonds and labels (labels in the 2D encoding: block
//               roots their global index, others kLocalFlag | block-local root) and the block's three
//               outgoing face bitmaps.
//   k3_merge    unions across the +x, +y, +z faces on the global label array, each recording the root
//               it linked.
//   k3_resolve  every linked root's chain walked to the cluster root.
//   k3_flip     every site reads its root's resolved label and flips iff it is odd.
//
// k3_assign is the 2D strip form (sw_strip.cuh) with a third direction.  A block is 32 columns by up to
// 16 rows by up to 16 layers; a warp owns a piece of it, 32 columns of one tile layer's rows (R = 32
// rows of sites for the default tile), and
//   packs row r of the piece, and the rows after it in y and z, into words (lane r);
//   runs its tiles' draws, leaving every update's ballot in shared memory;
//   forms row r's x-, y- and z-bond words (lane r), which the block shares;
//   scans its rows in order (lane k is column k): a run takes the label of its leftmost site that is
//   bonded back in y or z, or its own first site; other bonds back that meet another label are marked,
//   listed and united together, one per lane;
// then the bonds between pieces are united the same way, linked labels are pointed at their roots and
// every site's label is two lookups away.  A site-by-site form (one union-find node and up to three
// unions per site) took 12 (default tile on whole blocks) to 31 (any other) warp instructions per
// site; this one 4.1.  256^3 sweep 397 -> 175 us (assign 278 -> 112, merge 71 -> 32, resolve 37 -> 17), 90 x 76 x
// 54 169 -> 53 us.

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "../../include/swb200.h"
#include "sw_3d.cuh"
#include "sw_core.cuh"
#include "sw_strip.cuh"

namespace swb {

// Global site index of a label read at a site of block (bxi, byi, bzi).
__device__ __forceinline__ uint32_t label_global3(const Geo3 &g, uint32_t bxi, uint32_t byi, uint32_t bzi, uint32_t v)
{
    if (!(v & kLocalFlag))
        return v;
    const uint32_t r = v & kLocalMask, zl = r / k3Layer, yl = r / k3Pitch % k3Rows, xl = r % k3Pitch;
    return ((bzi * g.BZ + zl) * g.L1 + byi * g.BY + yl) * g.L0 + bxi * g.BX + xl;
}

// The draws of one sweep for a piece (tile rows [ty0, ty0 + nty) of tile layer tz, every tile column of
// the block), as strip_draws: tile q (tile rows outer, columns inner) is segment q % (32 / W) of pass
// q / (32 / W); update u of pass p leaves its ballot in d[p * total + u].  A tile that lacks a row idles
// through it.  This warp takes the passes first, first + step, ...
template <int W, int TX>
__device__ __forceinline__ void draws_piece3(const Geo3 &g, const uint32_t bxi, const uint32_t ty_first,
                                             const uint32_t nty, const uint32_t tz, uint32_t *d, const Draws3 &D,
                                             const uint32_t first, const uint32_t step, const uint2 *pairs,
                                             uint32_t *__restrict__ rng_state, uint8_t *__restrict__ rng_sel,
                                             uint32_t *__restrict__ rng_iter, const uint32_t thr)
{
    constexpr uint32_t kTps = 32 / TX, kPer = 32 / W;
    const uint32_t TY = g.TY, TZ = g.TZ, lane32 = threadIdx.x & 31, lane = lane32 % W;
    d += first * D.total;
    for (uint32_t p = first; p * kPer < nty * kTps; p += step, d += step * D.total) {
        const uint32_t q = p * kPer + lane32 / W, tcol = q % kTps;
        const uint32_t tgx = bxi * g.TBX + tcol, tgy = ty_first + q / kTps;
        const bool on = q < nty * kTps && tcol < g.TBX && tgx < g.n0 && tgy < g.n1;
        const uint32_t onm = __ballot_sync(0xffffffffu, on);
        if (onm == 0)
            continue;
        const uint32_t tile = (tz * g.n1 + tgy) * g.n0 + tgx;
        const uint32_t jjmax = on ? min(TY, g.L1 - tgy * TY) : 0, kkmax = on ? min(TZ, g.L2 - tz * TZ) : 0;
        uint32_t st = 0, sel = 0, it = 0;
        if (on) {
            st = rng_state[(size_t)tile * W + lane];
            sel = rng_sel[(size_t)tile * W + lane];
            it = rng_iter[tile];
        }
        uint2 ac = pairs[sel];
        // the parameter rotation of LCG32_State::Update (random/src/lcg32.cpp:51-84), as in strip_draws
        auto rotate = [&](const uint32_t itn, const bool rot) {
            const uint32_t src = __shfl_sync(0xffffffffu, st, itn & (W - 1), W);
            const uint32_t from = (lane + src + ((itn & 1u) ? 0u : 1u)) & (W - 1);
            const uint32_t s2 = __shfl_sync(0xffffffffu, sel, from, W);
            if (rot) {
                sel = s2;
                ac = pairs[sel];
            }
        };
        const uint32_t itu = __shfl_sync(0xffffffffu, it, __ffs(onm) - 1);
        if (__all_sync(0xffffffffu, !on || (jjmax == TY && kkmax == TZ && it == itu))) {
            // whole tiles in step: nothing predicated, groups of 15 updates between the rotations
            uint32_t k = 0, next = kShuffleDistance - 1 - itu % kShuffleDistance;
            auto draw = [&](const uint32_t u) {
                st = ac.x * st + ac.y;
                const uint32_t word = __ballot_sync(0xffffffffu, lcg_accept(st, thr));
                if (lane32 == 0)
                    d[u] = word;
            };
            for (; k < min(next, D.total); ++k)
                draw(k);
            while (k < D.total) {
                rotate(itu + k + 1, true);
                if (k + kShuffleDistance <= D.total) {
#pragma unroll
                    for (uint32_t u = 0; u < kShuffleDistance; ++u)
                        draw(k + u);
                    k += kShuffleDistance;
                } else {
                    for (; k < D.total; ++k)
                        draw(k);
                }
            }
            it += D.total;
        } else {
            uint32_t to_rot = kShuffleDistance - it % kShuffleDistance, u = 0;
            auto advance = [&](const bool upd) {
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
                ++u;
            };
            for (uint32_t dir = 0; dir < 3; ++dir) {
                const uint32_t nj = dir == 1 ? TY - 1 : TY, nk = dir == 2 ? TZ - 1 : TZ;
                for (uint32_t kk = 0; kk < nk; ++kk)
                    for (uint32_t jj = 0; jj < nj; ++jj) {
                        const bool row = dir == 0 ? (kk < kkmax && jj < jjmax)
                                       : dir == 1 ? (kk < kkmax && jj + 1 < jjmax) : (kk + 1 < kkmax && jj < jjmax);
                        for (uint32_t n = 0; n < D.ur; ++n)
                            advance(row);
                    }
            }
            while (u < D.total)
                advance(on);
        }
        if (on) {
            rng_state[(size_t)tile * W + lane] = st;
            rng_sel[(size_t)tile * W + lane] = (uint8_t)sel;
            if (lane == 0)
                rng_iter[tile] = it;
        }
    }
}

// Elements [e, e + n) (n <= 32) of tile q's request that starts at update u.
template <int W>
__device__ __forceinline__ uint32_t request_bits(const DrawWords<W> &dw, const uint32_t q, const uint32_t u,
                                                 const uint32_t e, const uint32_t n)
{
    uint32_t v = 0;
    for (uint32_t k = 0; k < n;) {
        const uint32_t o = (e + k) % W;
        v |= (dw.seg(q, u + (e + k) / W) >> o) << k;
        k += W - o;
    }
    return v & (0xFFFFFFFFu >> (32 - n));
}

// Unions of the marked bonds of a piece: lane r holds row r's marks of each group of 32 rows, my for the
// bonds to the row before, mz for those to the layer before.  They are listed window by window and
// worked off one per lane; the labels that a union hung below another are appended to links.
template <int kGroups>
__device__ __forceinline__ void unite_marked3(uint32_t *parent, uint16_t *list, uint16_t *links, uint32_t &nlinks,
                                              const uint32_t (&my)[kGroups], const uint32_t (&mz)[kGroups],
                                              const uint32_t (&lrow)[kGroups])
{
    const uint32_t lane = threadIdx.x & 31;
#pragma unroll
    for (int g = 0; g < kGroups; ++g) {
        const uint32_t mine = __popc(my[g]) + __popc(mz[g]);
        uint32_t end = mine;
#pragma unroll
        for (uint32_t o = 1; o < 32; o *= 2) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, end, o);
            if (lane >= o)
                end += v;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, end, 31);
        for (uint32_t b0 = 0; b0 < total; b0 += k3Window) {
            __syncwarp();
            uint32_t k = end - mine - b0;
            for (uint32_t left = my[g]; left; left &= left - 1, ++k)
                if (k < k3Window)  // unsigned: also false before the window
                    list[k] = (uint16_t)(lrow[g] + __ffs(left) - 1);
            for (uint32_t left = mz[g]; left; left &= left - 1, ++k)
                if (k < k3Window)
                    list[k] = (uint16_t)((lrow[g] + __ffs(left) - 1) | 0x8000u);
            __syncwarp();
            const uint32_t n = min(total - b0, k3Window);
            for (uint32_t i0 = 0; i0 < n; i0 += 32) {
                uint32_t link = kNoLink;
                if (i0 + lane < n) {
                    const uint32_t v = list[i0 + lane], l = v & 0x7FFFu;
                    link = uf_union_link(parent, parent[l - ((v & 0x8000u) ? k3Layer : k3Pitch)], parent[l]);
                }
                __syncwarp();
                const uint32_t m = __ballot_sync(0xffffffffu, link != kNoLink);
                const uint32_t at = nlinks + __popc(m & ((1u << lane) - 1u));
                if (link != kNoLink && at < k3Links)
                    links[at] = (uint16_t)link;
                nlinks += __popc(m);
            }
        }
    }
}

// kGroups: groups of 32 rows a piece has (2 for tiles of more than 32 rows).  kMeasure: also measure
// the spins the sweep starts from.
template <int W, int TX, int kGroups, bool kMeasure>
__global__ void __launch_bounds__(k3MaxThreads, kGroups == 1 ? 2 : 1)
k3_assign(const Geo3 g, const uint8_t *spins, uint32_t *labels, uint32_t *__restrict__ rng_state,
          uint8_t *__restrict__ rng_sel, uint32_t *__restrict__ rng_iter, const uint32_t thr, uint32_t *faces,
          uint8_t *dump_bonds, const MeasureArgs meas, const uint32_t share)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const Assign3Smem S = assign3_smem<W>(g);
    const Draws3 D = draws3<W>(TX, g.TY, g.TZ);
    constexpr uint32_t kTps = 32 / TX;
    uint32_t *parent = reinterpret_cast<uint32_t *>(smem);
    uint4 *raw = reinterpret_cast<uint4 *>(smem + S.raw);
    int *sums = reinterpret_cast<int *>(smem + S.sums);
    uint2 *pairs = reinterpret_cast<uint2 *>(smem + S.pairs);
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const uint32_t bxi = blockIdx.x, byi = blockIdx.y, bzi = blockIdx.z;
    const uint32_t x0 = bxi * g.BX, y0 = byi * g.BY, z0 = bzi * g.BZ;
    const uint32_t bxv = min(g.BX, g.L0 - x0), byv = min(g.BY, g.L1 - y0), bzv = min(g.BZ, g.L2 - z0);
    const size_t plane = (size_t)g.L0 * g.L1;
    // the piece: rows [yp, yp + nj) of layers [zp, zp + nk) of the block.  `share` warps take its draws
    // between them (draw_share3), the first of them all the rest.
    const uint32_t np = pieces3(g), turn = share == 1 ? 0 : warp / np, piece = warp - turn * np;
    const uint32_t tz = piece / g.pcy, typ = (piece - tz * g.pcy) * g.py;
    const uint32_t yp = typ * g.TY, zp = tz * g.TZ, PY = g.py * g.TY;
    const bool exists = yp < byv && zp < bzv, here = exists && turn == 0;
    const uint32_t nj = here ? min(PY, byv - yp) : 0, nk = here ? min(g.TZ, bzv - zp) : 0;
    uint32_t *work = reinterpret_cast<uint32_t *>(smem + S.work) + piece * S.wcap;
    uint16_t *links = reinterpret_cast<uint16_t *>(smem + S.links) + piece * k3Links;
    uint4 *scan = reinterpret_cast<uint4 *>(smem + S.scan) + piece * S.rows * 2;
    uint32_t *fblk = faces + (((size_t)bzi * g.nby + byi) * g.nbx + bxi) * k3FaceWords;

    if (threadIdx.x < 5) {
        pairs[threadIdx.x] = make_uint2(lcg_param_a(threadIdx.x), lcg_param_c(threadIdx.x));
        if (threadIdx.x < 4)
            sums[threadIdx.x] = 0;
    }
    __syncthreads();
    if (exists)
        draws_piece3<W, TX>(g, bxi, byi * g.TBY + typ, min(g.py, g.TBY - typ), bzi * g.TBZ + tz, work, D, turn,
                            share, pairs, rng_state, rng_sel, rng_iter, thr);
    if (share == 1)
        __syncwarp();
    else
        __syncthreads();
    after_previous();

    // ---- bonds, lane r of a group: row r = kk * PY + j of the piece
    const uint32_t colm = 0xFFFFFFFFu >> (32 - bxv);
    uint32_t rj[kGroups], rk[kGroups];  // the row's j and kk
    bool row_on[kGroups];
#pragma unroll
    for (int q = 0; q < kGroups; ++q) {
        const uint32_t r = q * 32 + lane;
        rk[q] = r / PY;
        rj[q] = r - rk[q] * PY;
        row_on[q] = rj[q] < nj && rk[q] < nk;
        if (row_on[q]) {
            const uint32_t yl = yp + rj[q], zl = zp + rk[q], y = y0 + yl, z = z0 + zl;
            const uint32_t yn = y + 1 < g.L1 ? y + 1 : 0, zn = z + 1 < g.L2 ? z + 1 : 0, xe = x0 + bxv;
            const uint32_t both = g.L0 | x0, align = (both & 15u) == 0 ? 16 : (both & 3u) == 0 ? 4 : 2;
            const uint8_t *row = spins + z * plane + (size_t)y * g.L0;
            const uint32_t s = strip_row_bits(row + x0, bxv, align), right = row[xe < g.L0 ? xe : 0u];
            const uint32_t sy = strip_row_bits(spins + z * plane + (size_t)yn * g.L0 + x0, bxv, align);
            const uint32_t sz = strip_row_bits(spins + zn * plane + (size_t)y * g.L0 + x0, bxv, align);
            const uint32_t dx = (s ^ (s >> 1 | right << (bxv - 1))) & colm, dy = s ^ sy, dz = s ^ sz;
            if constexpr (kMeasure) {
                atomicAdd(sums, 3 * (int)bxv - 2 * (__popc(dx) + __popc(dy) + __popc(dz)));
                atomicAdd(sums + 1, 2 * __popc(s) - (int)bxv);
            }
            // accepted draws: requests of the tile's rows, or elements of its face request (y face, x face,
            // z face) for the last row, column, layer of the tile
            const uint32_t t = rj[q] / g.TY, jj = rj[q] - t * g.TY, kk = rk[q];
            const uint32_t jjmax = min(g.TY, nj - t * g.TY), fy = TX * g.TZ, fz = fy + g.TY * g.TZ;
            const DrawWords<W> dw{work, D.total};
            uint32_t AX = 0, AY = 0, AZ = 0;
#pragma unroll
            for (uint32_t c = 0; c < kTps; ++c) {
                if (c * TX < bxv) {
                    const uint32_t tq = t * kTps + c, n = min((uint32_t)TX, bxv - c * TX);
                    const uint32_t tmask = 0xFFFFFFFFu >> (32 - n);
                    const uint32_t ax = dw.req(tq, (kk * g.TY + jj) * D.ur, D.ur) & (tmask >> 1);
                    const uint32_t last = dw.bit(tq, D.face, fy + kk * g.TY + jj);
                    const uint32_t ay = jj + 1 < jjmax ? dw.req(tq, D.y + (kk * (g.TY - 1) + jj) * D.ur, D.ur)
                                                       : request_bits<W>(dw, tq, D.face, kk * TX, TX);
                    const uint32_t az = kk + 1 < nk ? dw.req(tq, D.z + (kk * g.TY + jj) * D.ur, D.ur)
                                                    : request_bits<W>(dw, tq, D.face, fz + jj * TX, TX);
                    AX |= (ax | last << (n - 1)) << (c * TX);
                    AY |= (ay & tmask) << (c * TX);
                    AZ |= (az & tmask) << (c * TX);
                }
            }
            const uint32_t X = ~dx & AX & colm, Y = ~dy & AY & colm, Z = ~dz & AZ & colm;
            raw[zl * k3Rows + yl] = make_uint4(X, Y, Z, 0);
            if (yl + 1 == byv)
                fblk[k3FaceX + zl] = Y;
            if (zl + 1 == bzv)
                fblk[k3FaceX + k3FaceY + yl] = Z;
            if (dump_bonds)
                for (uint32_t x = 0; x < bxv; ++x)
                    dump_bonds[z * plane + (size_t)y * g.L0 + x0 + x] =
                        (uint8_t)(((X >> x) & 1u) | ((Y >> x) & 1u) << 1 | ((Z >> x) & 1u) << 2);
        }
    }
    __syncthreads();

    // +x face: a bit per row, 32 rows (two layers) per word
    for (uint32_t w = warp; 2 * w < bzv; w += nwarps) {
        const uint32_t r = w * 32 + lane;
        const bool on = r % k3Rows < byv && r / k3Rows < bzv;
        const uint32_t m = __ballot_sync(0xffffffffu, on && ((raw[r < g.BZ * k3Rows ? r : 0].x >> (bxv - 1)) & 1u));
        if (lane == 0)
            fblk[w] = m;
    }

    uint32_t nlinks = 0, my[kGroups], mz[kGroups], lrow[kGroups];
    if (here) {
        // Scan words of row r: the gaps ~X; the first bond back or run end from a run's start is the run's
        // first set bit of the second; the bonds back in y or z; those in y; and the ones in y and in z that
        // may unite (a bond whose left neighbour is bonded back too, with both rows bonded across, meets
        // the same two runs).  Bonds back into another piece wait for the join (my, mz).
#pragma unroll
        for (int q = 0; q < kGroups; ++q) {
            my[q] = mz[q] = 0;
            lrow[q] = ((zp + rk[q]) * k3Rows + yp + rj[q]) * k3Pitch;
            if (row_on[q]) {
                const uint32_t row = (zp + rk[q]) * k3Rows + yp + rj[q];
                const uint32_t X = raw[row].x;
                uint32_t Yu = 0, Uy = 0, Zu = 0, Uz = 0;
                if (yp + rj[q]) {
                    const uint4 w = raw[row - 1];
                    Yu = w.y;
                    Uy = Yu & ~((Yu & X & w.x) << 1);
                }
                if (zp + rk[q]) {
                    const uint4 w = raw[row - k3Rows];
                    Zu = w.z;
                    Uz = Zu & ~((Zu & X & w.x) << 1);
                }
                if (rj[q] == 0) {
                    my[q] = Uy;
                    Yu = Uy = 0;
                }
                if (rk[q] == 0) {
                    mz[q] = Uz;
                    Zu = Uz = 0;
                }
                const uint32_t r = q * 32 + lane;
                scan[2 * r] = make_uint4(~X, Yu | Zu | ~X | 0x80000000u, Yu | Zu, Yu);
                scan[2 * r + 1] = make_uint4(Uy, Uz, 0, 0);
            }
        }
        __syncwarp();

        const uint32_t under = (1u << lane) - 1u, bit = 1u << lane;
        for (uint32_t kk = 0; kk < nk; ++kk) {
            uint32_t above = 0, base = ((zp + kk) * k3Rows + yp) * k3Pitch, r = kk * PY;
            for (uint32_t j = 0; j < nj; ++j, ++r, base += k3Pitch) {
                const uint4 w = scan[2 * r];
                const uint2 u = *reinterpret_cast<const uint2 *>(scan + 2 * r + 1);
                const uint32_t before = kk ? parent[base + lane - k3Layer] : 0u;
                int last_gap;  // -1: none
                asm("bfind.u32 %0, %1;" : "=r"(last_gap) : "r"(w.x & under));
                const uint32_t rs = last_gap + 1;
                const uint32_t pos = __clz(__brev(w.y & (0xFFFFFFFFu << rs)));
                const uint32_t rep = __shfl_sync(0xffffffffu, (w.w & bit) ? above : before, pos);
                const uint32_t lab = (w.z & (1u << pos)) ? rep : base + rs;
                const uint32_t ny = __ballot_sync(0xffffffffu, (u.x & bit) && above != lab);
                const uint32_t nz = __ballot_sync(0xffffffffu, (u.y & bit) && before != lab);
                if (lane == 0)
                    *reinterpret_cast<uint2 *>(work + 2 * r) = make_uint2(ny, nz);
                parent[base + lane] = lab;
                above = lab;
            }
        }
        __syncwarp();
        uint32_t iy[kGroups], iz[kGroups];
#pragma unroll
        for (int q = 0; q < kGroups; ++q) {
            const uint2 v = row_on[q] ? *reinterpret_cast<const uint2 *>(work + 2 * (q * 32 + lane)) : make_uint2(0, 0);
            iy[q] = v.x;
            iz[q] = v.y;
        }
        __syncwarp();
        unite_marked3<kGroups>(parent, reinterpret_cast<uint16_t *>(work), links, nlinks, iy, iz, lrow);
    }
    __syncthreads();

    // ---- join the pieces
    if (here) {
        unite_marked3<kGroups>(parent, reinterpret_cast<uint16_t *>(work), links, nlinks, my, mz, lrow);
        if (nlinks > k3Links && lane == 0)
            sums[2] = 1;  // the list does not hold every linked label
    }
    __syncthreads();
    __syncwarp();
    for (uint32_t i = lane; i < min(nlinks, k3Links); i += 32)
        uf_flatten(parent, links[i]);
    __syncthreads();
    const bool deep = sums[2] != 0;

    // ---- labels: block roots their global index, others kLocalFlag | the block-local root
    if ((g.L0 & 3u) == 0) {  // four sites per lane, four rows per warp; rows and x0 are 16-byte aligned
        const uint32_t x4 = (lane & 7) * 4;
        for (uint32_t r = warp * 4 + (lane >> 3); r < bzv * k3Rows; r += nwarps * 4) {
            const uint32_t yl = r % k3Rows, zl = r / k3Rows;
            if (yl >= byv || x4 >= bxv)
                continue;
            const uint32_t l = r * k3Pitch + x4;
            const uint4 pp = *reinterpret_cast<const uint4 *>(parent + l);
            uint32_t v[4] = {parent[pp.x], parent[pp.y], parent[pp.z], parent[pp.w]};
            while (deep) {
                uint32_t n[4];
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    n[k] = parent[v[k]];
                if (n[0] == v[0] && n[1] == v[1] && n[2] == v[2] && n[3] == v[3])
                    break;
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    v[k] = n[k];
            }
            const uint32_t gb = ((z0 + zl) * g.L1 + y0 + yl) * g.L0 + x0 + x4;
            uint4 o;
            o.x = v[0] == l ? gb : (kLocalFlag | v[0]);
            o.y = v[1] == l + 1 ? gb + 1 : (kLocalFlag | v[1]);
            o.z = v[2] == l + 2 ? gb + 2 : (kLocalFlag | v[2]);
            o.w = v[3] == l + 3 ? gb + 3 : (kLocalFlag | v[3]);
            *reinterpret_cast<uint4 *>(labels + gb) = o;
        }
    } else {
        for (uint32_t r = warp; lane < bxv && r < bzv * k3Rows; r += nwarps) {
            const uint32_t yl = r % k3Rows, zl = r / k3Rows;
            if (yl >= byv)
                continue;
            const uint32_t l = r * k3Pitch + lane, v = uf_find(parent, l);
            const uint32_t gs = ((z0 + zl) * g.L1 + y0 + yl) * g.L0 + x0 + lane;
            labels[gs] = v == l ? gs : (kLocalFlag | v);
        }
    }
    if constexpr (kMeasure) {
        if (threadIdx.x == 0)
            obs_add_part(meas.obs, meas.series, meas.cap, plane * g.L2, g.nbx * g.nby * g.nbz, sums[0], sums[1], 1);
    }
}

// Unions across block (bxi, byi, bzi)'s +x, +y and +z faces (periodic).  The active face bonds (a quarter
// of the face sites near the critical temperature) are listed first, so that the label loads and walks
// run on full warps; slot i + 1 of the block's receives the root that the i-th listed bond's union
// linked, slot 0 their number.
__global__ void __launch_bounds__(k3MergeThreads) k3_merge(const Geo3 g, const uint32_t *faces, uint32_t *labels,
                                                           unsigned int *fault, uint32_t *linked)
{
    __shared__ uint16_t list[k3FaceSites];
    __shared__ uint32_t count;
    if (threadIdx.x == 0)
        count = 0;
    __syncthreads();
    after_previous();
    const uint32_t bxi = blockIdx.x, byi = blockIdx.y, bzi = blockIdx.z;
    const uint32_t x0 = bxi * g.BX, y0 = byi * g.BY, z0 = bzi * g.BZ;
    const uint32_t bxv = min(g.BX, g.L0 - x0), byv = min(g.BY, g.L1 - y0), bzv = min(g.BZ, g.L2 - z0);
    const size_t blk = ((size_t)bzi * g.nby + byi) * g.nbx + bxi;
    const uint32_t *f = faces + blk * k3FaceWords;
    uint32_t *slots = linked + blk * k3Slots;
    for (uint32_t w = threadIdx.x; w < k3FaceWords; w += blockDim.x) {
        const bool on = w < k3FaceX ? 2 * w < bzv : w < k3FaceX + k3FaceY ? w - k3FaceX < bzv
                                                                         : w - k3FaceX - k3FaceY < byv;
        uint32_t bits = on ? f[w] : 0u;
        uint32_t at = bits ? atomicAdd(&count, __popc(bits)) : 0u;
        for (; bits; bits &= bits - 1)
            list[at++] = (uint16_t)(w * 32 + __ffs(bits) - 1);
    }
    __syncthreads();
    const uint32_t n = count;
    if (threadIdx.x == 0)
        slots[0] = n;
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
        const uint32_t t = list[i], w = t / 32, b = t % 32;
        uint32_t xl, yl, zl, nx, ny, nz, nbx = bxi, nby = byi, nbz = bzi;
        if (w < k3FaceX) {
            zl = t / k3Rows; yl = t % k3Rows; xl = bxv - 1;
            nx = x0 + bxv < g.L0 ? x0 + bxv : 0; ny = y0 + yl; nz = z0 + zl;
            nbx = bxi + 1 == g.nbx ? 0 : bxi + 1;
        } else if (w < k3FaceX + k3FaceY) {
            zl = w - k3FaceX; yl = byv - 1; xl = b;
            nx = x0 + xl; ny = y0 + byv < g.L1 ? y0 + byv : 0; nz = z0 + zl;
            nby = byi + 1 == g.nby ? 0 : byi + 1;
        } else {
            yl = w - k3FaceX - k3FaceY; zl = bzv - 1; xl = b;
            nx = x0 + xl; ny = y0 + yl; nz = z0 + bzv < g.L2 ? z0 + bzv : 0;
            nbz = bzi + 1 == g.nbz ? 0 : bzi + 1;
        }
        const volatile uint32_t *vl = labels;
        const size_t s = ((size_t)(z0 + zl) * g.L1 + y0 + yl) * g.L0 + x0 + xl;
        const size_t nb = ((size_t)nz * g.L1 + ny) * g.L0 + nx;
        const uint32_t a = label_global3(g, bxi, byi, bzi, vl[s]), c = label_global3(g, nbx, nby, nbz, vl[nb]);
        slots[1 + i] = a != c ? guf_union_pair(labels, a, c, g.L0 * g.L1 * g.L2, fault) : kNoLink;
    }
}

__global__ void __launch_bounds__(k3MergeThreads) k3_resolve(const Geo3 g, const uint32_t *linked, uint32_t *labels,
                                                             unsigned int *fault)
{
    after_previous();
    const uint32_t *slots = linked + (((size_t)blockIdx.z * g.nby + blockIdx.y) * g.nbx + blockIdx.x) * k3Slots;
    const uint32_t n = min(slots[0], k3FaceSites);
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
        const uint32_t b = slots[1 + i];
        if (b != kNoLink)
            labels[b] = guf_find(labels, b, g.L0 * g.L1 * g.L2, fault);
    }
}

// Every block root's label is its cluster's root after k3_resolve; every site reads its root's
// and flips iff it is odd.  With write_labels the resolved labels are stored (a dumped sweep).
// Where rows allow 16-byte accesses each thread holds four quads of four sites (one 16-byte label load
// and one 4-byte spin load each) from the first pass to the second.
__global__ void __launch_bounds__(k3FlipThreads, 3) k3_flip(const Geo3 g, uint8_t *spins, uint32_t *labels,
                                                            const int write_labels)
{
    extern __shared__ __align__(16) unsigned char smem[];
    uint32_t *res = reinterpret_cast<uint32_t *>(smem);
    after_previous();
    const uint32_t x0 = blockIdx.x * g.BX, y0 = blockIdx.y * g.BY, z0 = blockIdx.z * g.BZ;
    const uint32_t bxv = min(g.BX, g.L0 - x0), byv = min(g.BY, g.L1 - y0), bzv = min(g.BZ, g.L2 - z0);
    if ((g.L0 & 3u) == 0) {
        constexpr int kQuads = k3Layers * k3Layer / 4 / k3FlipThreads;
        const uint32_t x4 = (threadIdx.x & 7) * 4;
        uint4 lab[kQuads];
        uint32_t spn[kQuads], site[kQuads];
#pragma unroll
        for (int k = 0; k < kQuads; ++k) {
            const uint32_t r = (threadIdx.x + k * k3FlipThreads) >> 3, yl = r % k3Rows, zl = r / k3Rows;
            site[k] = kNoLink;
            if (zl < bzv && yl < byv && x4 < bxv) {
                site[k] = ((z0 + zl) * g.L1 + y0 + yl) * g.L0 + x0 + x4;
                lab[k] = *reinterpret_cast<const uint4 *>(labels + site[k]);
                spn[k] = *reinterpret_cast<const uint32_t *>(spins + site[k]);
            }
        }
#pragma unroll
        for (int k = 0; k < kQuads; ++k) {
            const uint32_t l = (threadIdx.x + k * k3FlipThreads) * 4;
            const uint32_t v[4] = {lab[k].x, lab[k].y, lab[k].z, lab[k].w};
            if (site[k] != kNoLink) {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (!(v[j] & kLocalFlag))
                        res[l + j] = v[j];
            }
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kQuads; ++k) {
            const uint32_t l = (threadIdx.x + k * k3FlipThreads) * 4;
            const uint32_t v[4] = {lab[k].x, lab[k].y, lab[k].z, lab[k].w};
            if (site[k] != kNoLink) {
                uint32_t rr[4], flip = 0;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    rr[j] = res[(v[j] & kLocalFlag) ? (v[j] & kLocalMask) : l + j];
                    flip |= (rr[j] & 1u) << (8 * j);
                }
                *reinterpret_cast<uint32_t *>(spins + site[k]) = spn[k] ^ flip;
                if (write_labels)
                    *reinterpret_cast<uint4 *>(labels + site[k]) = make_uint4(rr[0], rr[1], rr[2], rr[3]);
            }
        }
        return;
    }
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    for (uint32_t r = warp; lane < bxv && r < bzv * k3Rows; r += nwarps) {
        if (r % k3Rows < byv) {
            const uint32_t v = labels[((z0 + r / k3Rows) * g.L1 + y0 + r % k3Rows) * g.L0 + x0 + lane];
            if (!(v & kLocalFlag))
                res[r * k3Pitch + lane] = v;
        }
    }
    __syncthreads();
    for (uint32_t r = warp; lane < bxv && r < bzv * k3Rows; r += nwarps) {
        if (r % k3Rows < byv) {
            const uint32_t s = ((z0 + r / k3Rows) * g.L1 + y0 + r % k3Rows) * g.L0 + x0 + lane;
            const uint32_t v = labels[s], c = res[(v & kLocalFlag) ? (v & kLocalMask) : r * k3Pitch + lane];
            spins[s] ^= (uint8_t)(c & 1u);
            if (write_labels)
                labels[s] = c;
        }
    }
}

// Row words: a warp takes 32 rows, lane r packs 32 columns of row r and of the rows after it in y and z.
__global__ void __launch_bounds__(256) k3_measure(const Geo3 g, const uint8_t *spins, Obs *obs, long long *series,
                                                  const unsigned long long cap, const int accumulate)
{
    after_previous();
    const uint32_t rows = g.L1 * g.L2, segs = (g.L0 + 31) / 32, align = (g.L0 & 15u) == 0 ? 16 : (g.L0 & 3u) == 0 ? 4 : 2;
    const size_t plane = (size_t)g.L0 * g.L1, items = (size_t)rows * segs;
    long long e = 0, m = 0;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < items; i += (size_t)gridDim.x * blockDim.x) {
        const uint32_t row = (uint32_t)(i % rows), x = (uint32_t)(i / rows) * 32, z = row / g.L1, y = row - z * g.L1;
        const uint32_t n = min(32u, g.L0 - x), mask = 0xFFFFFFFFu >> (32 - n);
        const uint8_t *p = spins + z * plane + (size_t)y * g.L0;
        const uint32_t s = strip_row_bits(p + x, n, align);
        const uint32_t sx = s >> 1 | (uint32_t)p[x + n < g.L0 ? x + n : 0] << (n - 1);
        const uint32_t sy = strip_row_bits(spins + z * plane + (size_t)(y + 1 < g.L1 ? y + 1 : 0) * g.L0 + x, n, align);
        const uint32_t sz = strip_row_bits(spins + (z + 1 < g.L2 ? z + 1 : 0) * plane + (size_t)y * g.L0 + x, n, align);
        e += 3 * (int)n - 2 * (__popc((s ^ sx) & mask) + __popc(s ^ sy) + __popc(s ^ sz));
        m += 2 * __popc(s) - (int)n;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        e += __shfl_xor_sync(0xffffffffu, e, o);
        m += __shfl_xor_sync(0xffffffffu, m, o);
    }
    __shared__ long long se[8], sm[8];
    if ((threadIdx.x & 31) == 0) {
        se[threadIdx.x >> 5] = e;
        sm[threadIdx.x >> 5] = m;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        long long be = 0, bm = 0;
        for (uint32_t k = 0; k < blockDim.x / 32; ++k) {
            be += se[k];
            bm += sm[k];
        }
        obs_add_part(obs, series, cap, (size_t)rows * g.L0, gridDim.x, be, bm, accumulate);
    }
}

template <int W>
__global__ void k3_rng_init(const uint32_t n_tiles, const uint32_t seed_base, uint32_t *state, uint8_t *sel,
                           uint32_t *iter)
{
    rng_init_tile<W>(n_tiles, seed_base, state, sel, iter);
}

__global__ void k3_hot_start(const size_t n, const uint32_t seed, uint8_t *spins)
{
    hot_start_chunk(n, seed, spins);
}

__global__ void k3_check_spins(const size_t n, const uint8_t *p, unsigned int *bad)
{
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        if (p[i] > 1)
            atomicOr(bad, 1u);
}

}  // namespace swb

using namespace swb;

struct swb_lattice3 {
    int device = 0;
    cudaStream_t stream = nullptr;
    Geo3 g{};
    uint32_t W = 16, n_tiles = 0, n_blocks = 0, smem_assign = 0;
    size_t n = 0;
    uint8_t *spins = nullptr;
    uint32_t *labels = nullptr, *rng_state = nullptr, *rng_iter = nullptr, *faces = nullptr, *linked = nullptr;
    uint8_t *rng_sel = nullptr;
    Obs *obs = nullptr;
    long long *series = nullptr;
    unsigned long long series_cap = 1ull << 16;
    unsigned int *fault = nullptr, *flag = nullptr;
    int measure_grid = 1;
    bool measure_pending = false;  // a sample of the current spins is still to be taken
};

namespace {

int set_device3(const swb_lattice3 *h)
{
    SWB_CUDA(cudaSetDevice(h->device));
    return SWB_OK;
}

int check_fault3(swb_lattice3 *h)
{
    unsigned int f = 0;
    SWB_CUDA(cudaMemcpyAsync(&f, h->fault, sizeof(f), cudaMemcpyDeviceToHost, h->stream));
    SWB_CUDA(cudaStreamSynchronize(h->stream));
    if (f)
        return fail(SWB_ERR_STATE, "label union-find fault (word %u: 1 chain over %u steps, 2 union retries, 4 label outside the lattice)", f, kChainCap);
    return SWB_OK;
}

bool early_launch3(const swb_lattice3 *h) { return h->n_blocks < kEarlyBlocks; }

// Warps that take a piece's draws between them: where blocks are for at most one SM each, the warps that a CTA
// may have beyond its pieces help (90 x 76 x 54 with the default tile 57.6 -> 53.4 us a sweep, 8 x 8 x 8 with W 32 on 64^3
// 60 -> 52).  Beyond that the blocks share the SMs: with 256 blocks of 128^3 8 x 8 x 8 tiles 69 -> 91 us, 16 x 4 x 4 on
// 256^3 182 -> 224.
template <int W>
uint32_t draw_share3(const Geo3 &g)
{
    if (g.nbx * g.nby * g.nbz > k3ShareBlocks)
        return 1;
    return std::max(1u, std::min(passes3(g, W), k3MaxThreads / 32 / pieces3(g)));
}

template <int W, int TX>
int launch_assign3(swb_lattice3 *h, uint32_t thr, uint8_t *dump_bonds, const MeasureArgs &meas)
{
    const Geo3 &g = h->g;
    const bool two = g.py * g.TY * g.TZ > 32;
    const uint32_t share = draw_share3<W>(g);
    auto k = two ? (meas.obs ? k3_assign<W, TX, 2, true> : k3_assign<W, TX, 2, false>)
                 : (meas.obs ? k3_assign<W, TX, 1, true> : k3_assign<W, TX, 1, false>);
    return launch_next(early_launch3(h), k, dim3(g.nbx, g.nby, g.nbz), pieces3(g) * share * 32, h->smem_assign, h->stream, g,
                       h->spins, h->labels, h->rng_state, h->rng_sel, h->rng_iter, thr, h->faces, dump_bonds, meas, share);
}

template <int W>
int launch_assign3(swb_lattice3 *h, uint32_t thr, uint8_t *dump_bonds, const MeasureArgs &meas)
{
    switch (h->g.TX) {
    case 8: return launch_assign3<W, 8>(h, thr, dump_bonds, meas);
    case 16: return launch_assign3<W, 16>(h, thr, dump_bonds, meas);
    default: return launch_assign3<W, 32>(h, thr, dump_bonds, meas);
    }
}

// More than 48 KiB of shared memory per CTA is asked for once per kernel.
template <int W, int TX>
cudaError_t allow_smem3(uint32_t bytes)
{
    for (auto k : {k3_assign<W, TX, 1, false>, k3_assign<W, TX, 1, true>, k3_assign<W, TX, 2, false>,
                   k3_assign<W, TX, 2, true>})
        if (cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes))
            return e;
    return cudaSuccess;
}

template <int W>
cudaError_t allow_smem3(uint32_t TX, uint32_t bytes)
{
    return TX == 8 ? allow_smem3<W, 8>(bytes) : TX == 16 ? allow_smem3<W, 16>(bytes) : allow_smem3<W, 32>(bytes);
}

// measure: the assign also measures the spins the sweep starts from.
int launch_sweep3(swb_lattice3 *h, float temperature, uint8_t *dump_bonds, bool write_labels, bool measure = false)
{
    const Geo3 &g = h->g;
    const dim3 grid(g.nbx, g.nby, g.nbz);
    const uint32_t thr = accept_threshold(swb_p_add(temperature));
    const MeasureArgs meas = measure ? MeasureArgs{h->obs, h->series, h->series_cap} : MeasureArgs{};
    const bool early = early_launch3(h);
    if (int rc = h->W == 8    ? launch_assign3<8>(h, thr, dump_bonds, meas)
                 : h->W == 16 ? launch_assign3<16>(h, thr, dump_bonds, meas)
                              : launch_assign3<32>(h, thr, dump_bonds, meas))
        return rc;
    if (int rc = launch_next(early, k3_merge, grid, k3MergeThreads, 0, h->stream, g, h->faces, h->labels, h->fault,
                             h->linked))
        return rc;
    if (int rc = launch_next(early, k3_resolve, grid, k3MergeThreads, 0, h->stream, g, h->linked, h->labels, h->fault))
        return rc;
    return launch_next(early, k3_flip, grid, k3FlipThreads, k3Layers * k3Layer * 4, h->stream, g, h->spins, h->labels,
                       write_labels ? 1 : 0);
}

int launch_measure3(swb_lattice3 *h, int accumulate)
{
    return launch_next(early_launch3(h), k3_measure, h->measure_grid, 256, 0, h->stream, h->g, h->spins, h->obs,
                       h->series, h->series_cap, accumulate);
}

// A sample that swb3_sweep left for the next sweep's assign phase is taken now: before anything reads
// the observables, changes the spins or sweeps without measuring.
int flush_measure3(swb_lattice3 *h)
{
    if (!h->measure_pending)
        return SWB_OK;
    h->measure_pending = false;
    return launch_measure3(h, 1);
}

bool valid_temperature(float T) { return T > 0.0f && std::isfinite(T); }

}  // namespace

extern "C" {

int swb3_create(swb_lattice3 **out, uint32_t L0, uint32_t L1, uint32_t L2, uint32_t tile_x, uint32_t tile_y,
                uint32_t tile_z, uint32_t lcg_width, uint32_t seed_base, int device)
{
    if (!out)
        return fail(SWB_ERR_ARGUMENT, "out is NULL");
    *out = nullptr;
    if (L0 == 0 || L1 == 0 || L2 == 0 || L0 % 2 || L1 % 2 || (L2 % 2 && L2 != 1))
        return fail(SWB_ERR_ARGUMENT, "SwendsenWang_3D requires even extents (L2 = 1 allowed), got %u x %u x %u", L0, L1,
                    L2);
    if ((uint64_t)L0 * L1 * L2 > 0x7FFFFFFFull)
        return fail(SWB_ERR_ARGUMENT, "lattice of %u x %u x %u sites exceeds 2^31 - 1 labels", L0, L1, L2);
    if (!(tile_x == 8 || tile_x == 16 || tile_x == 32) || tile_y < 1 || tile_y > 8 || tile_z < 1 || tile_z > 8)
        return fail(SWB_ERR_ARGUMENT, "unsupported tile %u x %u x %u (tile_x in {8,16,32}, 1 <= tile_y, tile_z <= 8)",
                    tile_x, tile_y, tile_z);
    if (!(lcg_width == 8 || lcg_width == 16 || lcg_width == 32))
        return fail(SWB_ERR_ARGUMENT, "unsupported lcg32 width %u (8, 16 or 32)", lcg_width);
    Geo3 g = make_geo3(L0, L1, L2, tile_x, tile_y, tile_z);
    spread3(g, lcg_width);
    if (g.nby > 65535 || g.nbz > 65535)
        return fail(SWB_ERR_ARGUMENT, "lattice of %u x %u x %u sites needs too many block rows or layers", L0, L1, L2);
    swb_lattice3 *h = new swb_lattice3();
    h->device = device;
    h->W = lcg_width;
    h->g = g;
    h->n = (size_t)L0 * L1 * L2;
    h->n_tiles = g.n0 * g.n1 * g.n2;
    h->n_blocks = g.nbx * g.nby * g.nbz;
    h->smem_assign = lcg_width == 8    ? assign3_smem<8>(g).total
                     : lcg_width == 16 ? assign3_smem<16>(g).total
                                       : assign3_smem<32>(g).total;
    auto cleanup = [&](int rc) {
        swb3_destroy(h);
        return rc;
    };
#define SWB_TRY(call)                                                                              \
    do {                                                                                           \
        cudaError_t err__ = (call);                                                                \
        if (err__ != cudaSuccess)                                                                  \
            return cleanup(fail(SWB_ERR_CUDA, "%s failed: %s", #call, cudaGetErrorString(err__))); \
    } while (0)
    SWB_TRY(cudaSetDevice(device));
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    h->measure_grid = (int)std::max<size_t>(1, std::min<size_t>((h->n / 32 + 255) / 256, (size_t)sms * 8));
    SWB_TRY(cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking));
    SWB_TRY(cudaMalloc(&h->spins, h->n + 16));
    SWB_TRY(cudaMalloc(&h->labels, h->n * 4 + 16));
    SWB_TRY(cudaMalloc(&h->rng_state, (size_t)h->n_tiles * h->W * 4));
    SWB_TRY(cudaMalloc(&h->rng_sel, (size_t)h->n_tiles * h->W));
    SWB_TRY(cudaMalloc(&h->rng_iter, (size_t)h->n_tiles * 4));
    SWB_TRY(cudaMalloc(&h->faces, (size_t)h->n_blocks * k3FaceWords * 4));
    SWB_TRY(cudaMalloc(&h->linked, (size_t)h->n_blocks * k3Slots * 4));
    SWB_TRY(cudaMalloc(&h->obs, sizeof(Obs)));
    SWB_TRY(cudaMalloc(&h->series, h->series_cap * 16));
    SWB_TRY(cudaMalloc(&h->fault, 4));
    SWB_TRY(cudaMalloc(&h->flag, 4));
    SWB_TRY(cudaMemsetAsync(h->fault, 0, 4, h->stream));
    SWB_TRY(cudaMemsetAsync(h->spins, 0, h->n + 16, h->stream));
    SWB_TRY(cudaMemsetAsync(h->obs, 0, sizeof(Obs), h->stream));
    if (h->smem_assign > k3SmemMax)
        return cleanup(fail(SWB_ERR_ARGUMENT, "block of %u x %u x %u sites needs %u bytes of shared memory", g.BX, g.BY,
                            g.BZ, h->smem_assign));
    SWB_TRY(h->W == 8    ? allow_smem3<8>(tile_x, k3SmemMax)
            : h->W == 16 ? allow_smem3<16>(tile_x, k3SmemMax)
                         : allow_smem3<32>(tile_x, k3SmemMax));
    const unsigned grid = (h->n_tiles + 127) / 128;
    switch (h->W) {
    case 8: k3_rng_init<8><<<grid, 128, 0, h->stream>>>(h->n_tiles, seed_base, h->rng_state, h->rng_sel, h->rng_iter); break;
    case 16: k3_rng_init<16><<<grid, 128, 0, h->stream>>>(h->n_tiles, seed_base, h->rng_state, h->rng_sel, h->rng_iter); break;
    default: k3_rng_init<32><<<grid, 128, 0, h->stream>>>(h->n_tiles, seed_base, h->rng_state, h->rng_sel, h->rng_iter); break;
    }
    g_launches.fetch_add(1);
    SWB_TRY(cudaGetLastError());
    SWB_TRY(cudaStreamSynchronize(h->stream));
#undef SWB_TRY
    *out = h;
    return SWB_OK;
}

int swb3_destroy(swb_lattice3 *h)
{
    if (!h)
        return SWB_OK;
    cudaSetDevice(h->device);
    if (h->stream)
        cudaStreamSynchronize(h->stream);
    cudaFree(h->spins);
    cudaFree(h->labels);
    cudaFree(h->rng_state);
    cudaFree(h->rng_sel);
    cudaFree(h->rng_iter);
    cudaFree(h->faces);
    cudaFree(h->linked);
    cudaFree(h->obs);
    cudaFree(h->series);
    cudaFree(h->fault);
    cudaFree(h->flag);
    if (h->stream)
        cudaStreamDestroy(h->stream);
    delete h;
    return SWB_OK;
}

int swb3_geometry(swb_lattice3 *h, uint32_t *geometry)
{
    if (!h || !geometry)
        return fail(SWB_ERR_ARGUMENT, "NULL argument");
    const Geo3 &g = h->g;
    const uint32_t v[12] = {g.L0, g.L1, g.L2, g.TX, g.TY, g.TZ, g.BX, g.BY, g.BZ, g.nbx, g.nby, g.nbz};
    std::memcpy(geometry, v, sizeof(v));
    return SWB_OK;
}

int swb3_set_spins(swb_lattice3 *h, const uint8_t *host_spins)
{
    if (!h || !host_spins)
        return fail(SWB_ERR_ARGUMENT, "NULL argument");
    if (int rc = set_device3(h))
        return rc;
    if (int rc = flush_measure3(h))
        return rc;
    SWB_CUDA(cudaMemcpyAsync(h->spins, host_spins, h->n, cudaMemcpyHostToDevice, h->stream));
    SWB_CUDA(cudaMemsetAsync(h->flag, 0, 4, h->stream));
    k3_check_spins<<<h->measure_grid, 256, 0, h->stream>>>(h->n, h->spins, h->flag);
    SWB_LAUNCHED();
    unsigned int bad = 0;
    SWB_CUDA(cudaMemcpyAsync(&bad, h->flag, 4, cudaMemcpyDeviceToHost, h->stream));
    SWB_CUDA(cudaStreamSynchronize(h->stream));
    if (bad)
        return fail(SWB_ERR_ARGUMENT, "spins must be 0 or 1");
    return SWB_OK;
}

int swb3_get_spins(swb_lattice3 *h, uint8_t *host_spins)
{
    if (!h || !host_spins)
        return fail(SWB_ERR_ARGUMENT, "NULL argument");
    if (int rc = set_device3(h))
        return rc;
    SWB_CUDA(cudaMemcpyAsync(host_spins, h->spins, h->n, cudaMemcpyDeviceToHost, h->stream));
    SWB_CUDA(cudaStreamSynchronize(h->stream));
    return check_fault3(h);
}

int swb3_hot_start(swb_lattice3 *h, uint32_t seed)
{
    if (!h)
        return fail(SWB_ERR_ARGUMENT, "NULL handle");
    if (int rc = set_device3(h))
        return rc;
    if (int rc = flush_measure3(h))
        return rc;
    const size_t chunks = (h->n + 63) / 64;
    k3_hot_start<<<(unsigned)((chunks + 255) / 256), 256, 0, h->stream>>>(h->n, seed, h->spins);
    SWB_LAUNCHED();
    return SWB_OK;
}

int swb3_sweep(swb_lattice3 *h, float temperature, uint32_t n_sweeps, uint32_t measure_every)
{
    if (!h)
        return fail(SWB_ERR_ARGUMENT, "NULL handle");
    if (!valid_temperature(temperature))
        return fail(SWB_ERR_ARGUMENT, "temperature must be positive and finite");
    if (int rc = set_device3(h))
        return rc;
    for (uint32_t s = 1; s <= n_sweeps; ++s) {
        // a pending sample of the spins this sweep starts from is taken by its assign phase
        const bool fused = h->measure_pending;
        h->measure_pending = false;
        if (int rc = launch_sweep3(h, temperature, nullptr, false, fused))
            return rc;
        if (measure_every && s % measure_every == 0)
            h->measure_pending = true;
    }
    return SWB_OK;
}

int swb3_sweep_dumped(swb_lattice3 *h, float temperature, uint8_t *bonds, uint32_t *labels_final)
{
    if (!h)
        return fail(SWB_ERR_ARGUMENT, "NULL handle");
    if (!valid_temperature(temperature))
        return fail(SWB_ERR_ARGUMENT, "temperature must be positive and finite");
    if (int rc = set_device3(h))
        return rc;
    if (int rc = flush_measure3(h))
        return rc;
    uint8_t *d_bonds = nullptr;
    if (bonds)
        SWB_CUDA(cudaMallocAsync(&d_bonds, h->n, h->stream));
    int rc = launch_sweep3(h, temperature, d_bonds, true);
    if (rc == SWB_OK) {
        if (bonds)
            SWB_CUDA(cudaMemcpyAsync(bonds, d_bonds, h->n, cudaMemcpyDeviceToHost, h->stream));
        if (labels_final)
            SWB_CUDA(cudaMemcpyAsync(labels_final, h->labels, h->n * 4, cudaMemcpyDeviceToHost, h->stream));
    }
    if (d_bonds)
        cudaFreeAsync(d_bonds, h->stream);
    SWB_CUDA(cudaStreamSynchronize(h->stream));
    return rc ? rc : check_fault3(h);
}

int swb3_sweep_timed(swb_lattice3 *h, float temperature, uint32_t n_sweeps, float *ms)
{
    if (!h || !ms)
        return fail(SWB_ERR_ARGUMENT, "NULL argument");
    if (!valid_temperature(temperature))
        return fail(SWB_ERR_ARGUMENT, "temperature must be positive and finite");
    if (int rc = set_device3(h))
        return rc;
    if (int rc = flush_measure3(h))
        return rc;
    cudaEvent_t a, b;
    SWB_CUDA(cudaEventCreate(&a));
    SWB_CUDA(cudaEventCreate(&b));
    SWB_CUDA(cudaEventRecord(a, h->stream));
    int rc = SWB_OK;
    for (uint32_t s = 0; s < n_sweeps && rc == SWB_OK; ++s)
        rc = launch_sweep3(h, temperature, nullptr, false);
    SWB_CUDA(cudaEventRecord(b, h->stream));
    SWB_CUDA(cudaEventSynchronize(b));
    SWB_CUDA(cudaEventElapsedTime(ms, a, b));
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    return rc ? rc : check_fault3(h);
}

int swb3_energy_magnetization(swb_lattice3 *h, double *out, int64_t *e_sum, int64_t *m_sum)
{
    if (!h)
        return fail(SWB_ERR_ARGUMENT, "NULL handle");
    if (int rc = set_device3(h))
        return rc;
    if (int rc = flush_measure3(h))
        return rc;
    if (int rc = launch_measure3(h, 0))
        return rc;
    Obs o;
    SWB_CUDA(cudaMemcpyAsync(&o, h->obs, sizeof(Obs), cudaMemcpyDeviceToHost, h->stream));
    SWB_CUDA(cudaStreamSynchronize(h->stream));
    if (out) {
        out[0] = -(double)o.last_e / (double)h->n;
        out[1] = (double)o.last_m / (double)h->n;
    }
    if (e_sum) *e_sum = o.last_e;
    if (m_sum) *m_sum = o.last_m;
    return SWB_OK;
}

int swb3_samples(swb_lattice3 *h, int64_t *em, uint64_t capacity, uint64_t *count, double *acc)
{
    if (!h || !count)
        return fail(SWB_ERR_ARGUMENT, "NULL argument");
    if (int rc = set_device3(h))
        return rc;
    if (int rc = flush_measure3(h))
        return rc;
    Obs o;
    SWB_CUDA(cudaMemcpyAsync(&o, h->obs, sizeof(Obs), cudaMemcpyDeviceToHost, h->stream));
    SWB_CUDA(cudaStreamSynchronize(h->stream));
    *count = o.n_samples;
    if (acc)
        std::memcpy(acc, o.acc, sizeof(o.acc));
    if (o.n_samples > h->series_cap)
        return fail(SWB_ERR_CAPACITY, "%llu samples recorded, series keeps %llu", o.n_samples, h->series_cap);
    const uint64_t k = std::min<uint64_t>(o.n_samples, capacity);
    if (k && em) {
        SWB_CUDA(cudaMemcpyAsync(em, h->series, k * 16, cudaMemcpyDeviceToHost, h->stream));
        SWB_CUDA(cudaStreamSynchronize(h->stream));
    }
    return SWB_OK;
}

int swb3_get_rng(swb_lattice3 *h, uint32_t *state, uint32_t *a, uint32_t *c, uint32_t *iteration)
{
    if (!h || !state || !a || !c || !iteration)
        return fail(SWB_ERR_ARGUMENT, "NULL argument");
    if (int rc = set_device3(h))
        return rc;
    const size_t nw = (size_t)h->n_tiles * h->W;
    std::vector<uint8_t> sel(nw);
    SWB_CUDA(cudaMemcpyAsync(state, h->rng_state, nw * 4, cudaMemcpyDeviceToHost, h->stream));
    SWB_CUDA(cudaMemcpyAsync(sel.data(), h->rng_sel, nw, cudaMemcpyDeviceToHost, h->stream));
    SWB_CUDA(cudaMemcpyAsync(iteration, h->rng_iter, (size_t)h->n_tiles * 4, cudaMemcpyDeviceToHost, h->stream));
    SWB_CUDA(cudaStreamSynchronize(h->stream));
    for (size_t i = 0; i < nw; ++i) {
        a[i] = lcg_param_a(sel[i]);
        c[i] = lcg_param_c(sel[i]);
    }
    return SWB_OK;
}

int swb3_rng_shape(swb_lattice3 *h, uint32_t *n_tiles, uint32_t *lcg_width)
{
    if (!h)
        return fail(SWB_ERR_ARGUMENT, "NULL handle");
    if (n_tiles) *n_tiles = h->n_tiles;
    if (lcg_width) *lcg_width = h->W;
    return SWB_OK;
}

}  // extern "C"
