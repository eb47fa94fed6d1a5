// Shared device code of the Swendsen-Wang engine: lattice geometry, the per-block assign
// phase (lcg32 draws, bonds, shared-memory union-find) and the per-block edge merge.  Used by
// the single-lattice kernels (sw_plain.cu) and the batched kernels (sw_batch.cu).
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <string>
#include <utility>

#include "../../include/swb200.h"
#include "sw_device.cuh"

namespace swb {

// ------------------------------------------------------------------------------------------
// errors and launch accounting (defined in sw_plain.cu)

extern thread_local std::string g_last_error;
extern std::atomic<uint64_t> g_launches;
int fail(int code, const char *fmt, ...);

// swb_sweep_static's scratch: one file-scope device array (sw_static_scratch.cu) holding the
// label array, the block edge words and the fault word of a lattice of at most 2048 x 2048 sites.
constexpr uint64_t kStaticMaxSites = 1ull << 22;               // 2048 x 2048 sites
constexpr size_t kStaticScratchBytes = (24ull << 20) + 1024;   // labels 16 MiB + edge words + fault
// Device address of that array on `device`, which must be current (looked up once per device).
int static_scratch_base(int device, unsigned char **base);

#define SWB_CUDA(call)                                                                          \
    do {                                                                                        \
        cudaError_t err__ = (call);                                                             \
        if (err__ != cudaSuccess)                                                               \
            return ::swb::fail(SWB_ERR_CUDA, "%s failed: %s", #call, cudaGetErrorString(err__)); \
    } while (0)

#define SWB_LAUNCHED()                                                                           \
    do {                                                                                         \
        ::swb::g_launches.fetch_add(1, std::memory_order_relaxed);                               \
        cudaError_t err__ = cudaGetLastError();                                                  \
        if (err__ != cudaSuccess)                                                                \
            return ::swb::fail(SWB_ERR_CUDA, "kernel launch failed: %s", cudaGetErrorString(err__)); \
    } while (0)

// ------------------------------------------------------------------------------------------
// Kernels of one sweep, launched back to back.  A kernel launched by launch_next may start while the
// one before it still runs: it calls after_previous() before it touches anything the previous
// kernels write (that returns once they have completed), which also lets the kernel after it
// start, so any kernel runs at most beside its predecessor.  What it reads then must not go through
// the read-only path (no __ldg, no const __restrict__): that assumes data no one writes while the
// kernel lives.  Hides the launch and the drain of a phase: 256^2 sweep
// 25.7 -> 19.5 us, 1024^2 34.9 -> 27.2 us.

__device__ __forceinline__ void after_previous()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// early false: an ordinary launch of such a kernel.
template <class... P, class... A>
int launch_next(bool early, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args)
{
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = early ? 1 : 0;
    g_launches.fetch_add(1, std::memory_order_relaxed);
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return fail(SWB_ERR_CUDA, "kernel launch failed: %s", cudaGetErrorString(e));
    }
    return SWB_OK;
}

// ------------------------------------------------------------------------------------------
// geometry

// Lattices of at least this many (full-width) blocks launch their kernels the ordinary way: they fill the GPU for
// longer than a launch takes, and CTAs that wait early hold slots that the running kernel's last
// waves and other streams' kernels could use (16384^2 sweep 1.44 -> 1.54 ms early; 2048^2 46.3 ->
// 40.3 us).
constexpr uint32_t kEarlyBlocks = 2048;

struct Geo {
    uint32_t L0, L1;    // extent
    uint32_t TX, TY;    // tile
    uint32_t TBX, TBY;  // tiles per block
    uint32_t BX, BY;    // block in sites
    uint32_t n0, n1;    // tiles per direction
    uint32_t nbx, nby;  // blocks per direction
};

// Tiles per block: blocks of up to 128 x 32 sites.  tbx / tby (tiles per block) of 0 pick the largest
// such block; explicit values are clamped to it.
inline Geo make_geo(uint32_t L0, uint32_t L1, uint32_t TX, uint32_t TY, uint32_t tbx = 0, uint32_t tby = 0)
{
    Geo g{};
    g.L0 = L0; g.L1 = L1; g.TX = TX; g.TY = TY;
    g.n0 = (L0 + TX - 1) / TX;
    g.n1 = (L1 + TY - 1) / TY;
    g.TBX = 128 / TX;
    g.TBY = TY >= 32 ? 1 : 32 / TY;
    if (tbx && tbx < g.TBX)
        g.TBX = tbx;
    if (tby && tby < g.TBY)
        g.TBY = tby;
    // Do not make blocks larger than the lattice needs.
    while (g.TBX > 1 && (g.TBX / 2) * TX >= L0)
        g.TBX /= 2;
    while (g.TBY > 1 && (g.TBY / 2) * TY >= L1)
        g.TBY /= 2;
    g.BX = g.TBX * TX;
    g.BY = g.TBY * TY;
    g.nbx = (L0 + g.BX - 1) / g.BX;
    g.nby = (L1 + g.BY - 1) / g.BY;
    return g;
}

// Updates Ks... of a sweep as straight-line code, the rotation before every update k with
// k % 15 == kFirst (the rotating updates of a warp whose tiles share their iteration count).
template <uint32_t kFirst, uint32_t... Ks, class Rotate, class Draw>
__device__ __forceinline__ void draw_sequence(std::integer_sequence<uint32_t, Ks...>, Rotate &rotate, Draw &draw,
                                              const uint32_t it)
{
    ((Ks % kShuffleDistance == kFirst ? rotate(it + Ks + 1, true) : (void)0, draw(Ks)), ...);
}

template <uint32_t V>
struct U32 {  // a compile-time uint32_t passed as a value
    static constexpr uint32_t value = V;
};

constexpr uint32_t kMaxGridY = 65535;  // block rows of a lattice: the kernels' grid y
// Edge words of a block: what its merge needs.  [0] bonds out of the last column (a bit per row), [1..4] out
// of the last row (a bit per column); then, to leave out bonds that join the same two runs as the bond
// before them: [5] y-bonds in the last column, [6] in the first column (a bit per row), [7..10] x-bonds in
// the last row, [11..14] in the first row.  A recorded sweep leaves [5..14] zero: nothing is left out.
constexpr uint32_t kEdgeWords = 16;
constexpr uint32_t kEdgeYLast = 5, kEdgeYFirst = 6, kEdgeXLast = 7, kEdgeXFirst = 11;
constexpr uint32_t kEdgeParts = 5;       // words [0..4]
constexpr uint32_t kMergeList = kEdgeParts * 32;  // edge bonds of a block, at most
constexpr uint32_t kMergeThreads = 160;  // merge, resolve: one warp or several per block

// Label encoding between the assign and flip phases of a sweep.  A block root holds its global
// site index (< 2^31); these are the only entries the merge reads and links.  Every other site
// holds kLocalFlag | the block-local index (yl * kBlockPitch + xl, whatever the block's width) of its
// root, which needs no division to resolve and marks the site as a non-root.  Resolved labels
// (global) are written only by a recorded sweep.
constexpr uint32_t kLocalFlag = 0x80000000u;
constexpr uint32_t kLocalMask = 0x0000FFFFu;
constexpr uint32_t kBlockPitch = 128;  // blocks are at most 128 x 32 sites

// Global site index of a label read at a site of block (bxi, byi).
__device__ __forceinline__ uint32_t label_global(const Geo &g, uint32_t bxi, uint32_t byi, uint32_t v)
{
    if (!(v & kLocalFlag))
        return v;
    const uint32_t r = v & kLocalMask;
    return (byi * g.BY + r / kBlockPitch) * g.L0 + bxi * g.BX + r % kBlockPitch;
}

// Observables.  Per-sweep integer sums land in obs->e / obs->m; the last CTA turns them into
// E/N, M/N, accumulates E, E^2, |M| in FP64 and appends (e, m) to the sample series.
struct Obs {
    unsigned long long e, m;       // running int64 sums (two's complement) of this measurement
    unsigned int done;             // CTAs finished
    unsigned int pad;
    long long last_e, last_m;      // sums of the last measurement
    double acc[4];                 // sum E/N, sum (E/N)^2, sum |M/N|, samples
    unsigned long long n_samples;  // samples recorded (may exceed capacity)
};

// LCG32_State<W>::Init (random/src/lcg32.cpp:27-49) of tile t = this thread, seeded seed_base + t:
// drand48 draws pick each lane's (a, c) pair and the first lane's start, the others follow from
// it.  The two double multiplications are rounded as the host's (__dmul_rn).
template <int W>
__device__ __forceinline__ void rng_init_tile(const uint32_t n_tiles, const uint32_t seed_base, uint32_t *state,
                                              uint8_t *sel, uint32_t *iter)
{
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n_tiles)
        return;
    uint64_t x = drand48_seed(seed_base + t);
    uint32_t s[W];
#pragma unroll
    for (int i = 0; i < W; ++i) {
        x = drand48_step(x);
        s[i] = ((uint32_t)__dmul_rn(1000.0, drand48_value(x))) % 5u;
        sel[(size_t)t * W + i] = (uint8_t)s[i];
    }
    x = drand48_step(x);
    uint32_t v = lcg_param_a(s[0]) * ((uint32_t)__dmul_rn(4026531839.0, drand48_value(x)) + 1u) + lcg_param_c(s[0]);
    state[(size_t)t * W] = v;
#pragma unroll
    for (int i = 1; i < W; ++i) {
        v = lcg_param_a(s[i]) * v + lcg_param_c(s[i]);
        state[(size_t)t * W + i] = v;
    }
    iter[t] = 0;
}

// Hot start of Lattice<2> (ising/src/lattice.cpp:15-27), one 64-site chunk per thread: site i
// takes drand48 draw i + 1 after srand48(seed); drand48() < 0.5 iff bit 47 of the 48-bit state is
// clear.  The chunk's first state comes by jump-ahead; whole chunks store 8 sites at a time.
__device__ __forceinline__ void hot_start_chunk(const size_t n, const uint32_t seed, uint8_t *spins)
{
    constexpr uint32_t kChunk = 64;
    const size_t first = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * kChunk;
    if (first >= n)
        return;
    uint64_t A, C;
    drand48_jump(first, A, C);
    uint64_t x = (A * drand48_seed(seed) + C) & kDrandMask;
    const size_t last = first + kChunk < n ? first + kChunk : n;
    if (last - first == kChunk && (reinterpret_cast<uintptr_t>(spins) & 7u) == 0) {
#pragma unroll
        for (uint32_t q = 0; q < kChunk / 8; ++q) {
            uint64_t v = 0;
#pragma unroll
            for (uint32_t k = 0; k < 8; ++k) {
                x = drand48_step(x);
                v |= (x >> 47) << (8 * k);
            }
            reinterpret_cast<uint64_t *>(spins + first)[q] = v;
        }
        return;
    }
    for (size_t i = first; i < last; ++i) {
        x = drand48_step(x);
        spins[i] = (uint8_t)(x >> 47);
    }
}

// One part of a measurement: adds this part's integer sums (e = sum s (s_right + s_down),
// m = sum s over its sites) and, if it is the last of n_parts, turns the totals into E/N and
// M/N, accumulates E, E^2, |M| in FP64 (with accumulate), appends (e, m) to the series and
// clears the sums for the next measurement.  Called by one thread per part.
__device__ __forceinline__ void obs_add_part(Obs *obs, long long *series, const unsigned long long cap, const size_t n,
                                             const unsigned int n_parts, const long long e, const long long m,
                                             const int accumulate)
{
    atomicAdd(&obs->e, (unsigned long long)e);
    atomicAdd(&obs->m, (unsigned long long)m);
    __threadfence();
    const unsigned int ticket = atomicAdd(&obs->done, 1u);
    if (ticket == n_parts - 1) {
        __threadfence();
        const long long te = (long long)atomicAdd(&obs->e, 0ull);
        const long long tm = (long long)atomicAdd(&obs->m, 0ull);
        obs->last_e = te;
        obs->last_m = tm;
        if (accumulate) {
            const double E = -(double)te / (double)n, M = (double)tm / (double)n;
            obs->acc[0] += E;
            obs->acc[1] += E * E;
            obs->acc[2] += fabs(M);
            obs->acc[3] += 1.0;
            const unsigned long long k = obs->n_samples;
            if (k < cap) {
                series[2 * k] = te;
                series[2 * k + 1] = tm;
            }
            obs->n_samples = k + 1;
        }
        obs->e = 0;
        obs->m = 0;
        obs->done = 0;
    }
}

// A measurement of the spins a sweep starts from, made by its assign phase (obs null: none).
// The blocks of the sweep are its parts.
struct MeasureArgs {
    Obs *obs;
    long long *series;
    unsigned long long cap;
};

// Optional dumps of the assign phase to device buffers (one entry per site, row-major).  All
// null in a plain sweep; set by the recording entry points.  bonds: bit 0 +x, bit 1 +y (every
// bond of the sweep, block edges and the periodic wrap included); block_labels: the minimum
// global site index of the site's component over the bonds inside its block (the labels the
// assign phase hands to the merge); tile_labels: the same inside the site's tile (the
// reference's AssignLabels stage), which only the tile-by-tile form below computes.
struct AssignDump {
    uint8_t *bonds;
    uint32_t *block_labels;
    uint32_t *tile_labels;
};

struct AssignSmem {
    uint32_t parent, draws, slots, edge, bond, sp, total, pitch;
};

// Updates of every lcg32 lane in one sweep: 2 tile_y - 1 row requests of tile_x numbers and
// the merge request of tile_x + tile_y numbers, W numbers per update.
__host__ __device__ inline uint32_t draw_slots(const Geo &g, uint32_t W)
{
    return (2 * g.TY - 1) * ((g.TX + W - 1) / W) + (g.TX + g.TY + W - 1) / W;
}

__host__ __device__ inline AssignSmem assign_smem(const Geo &g, uint32_t W)
{
    AssignSmem s{};
    const uint32_t ns = g.BX * g.BY, ntb = g.TBX * g.TBY;
    s.pitch = g.BX + 1;
    s.slots = draw_slots(g, W);
    s.parent = 0;
    s.draws = s.parent + ns * 4;                                  // [warp][slot] ballot words
    s.edge = s.draws + ((ntb * W + 31) / 32) * s.slots * 4;
    s.bond = s.edge + kEdgeWords * 4;
    s.sp = (s.bond + ns + 15) & ~15u;
    s.total = s.sp + (g.BY + 1) * s.pitch;
    return s;
}

// Accepted draws of a block's tiles, read back from the warps' ballot words: bit k of a request
// word is element k of the request.  Tile tb's lanes are bits (tb * W) % 32 .. + W of warp
// (tb * W) / 32's words; a request starting at update u spans updates u .. u + ceil(n / W).
template <int W>
struct DrawWords {
    const uint32_t *d;
    uint32_t slots;
    __device__ __forceinline__ uint32_t seg(uint32_t tb, uint32_t u) const
    {
        const uint32_t v = d[((tb * W) >> 5) * slots + u] >> ((tb * W) & 31);
        return W == 32 ? v : v & ((1u << (W & 31)) - 1u);
    }
    // elements [0, ur * W) of the request at update u (ur * W <= 32)
    __device__ __forceinline__ uint32_t req(uint32_t tb, uint32_t u, uint32_t ur) const
    {
        uint32_t v = seg(tb, u);
        for (uint32_t s = 1; s < ur; ++s)
            v |= seg(tb, u + s) << (s * W);
        return v;
    }
    // element k of the request at update u
    __device__ __forceinline__ uint32_t bit(uint32_t tb, uint32_t u, uint32_t k) const
    {
        return (seg(tb, u + k / W) >> (k % W)) & 1u;
    }
};

// ------------------------------------------------------------------------------------------
// kernels

// Bit k of the result = bit 0 of byte k of v: multiplying the masked bytes by
// 2^28 + 2^21 + 2^14 + 2^7 lands byte k's bit at bit 28 + k, every cross term below bit 28.
__device__ __forceinline__ uint32_t spin_nibble(uint32_t v)
{
    return ((v & 0x01010101u) * 0x10204080u) >> 28;
}

// Energy / magnetisation sums of the `cnt` sites x0 .. x0 + cnt - 1 of row y of an L0 x L1
// periodic lattice: e = sum s (s_right + s_down), m = sum s, s = 2 b - 1.  Rows 16-byte aligned
// (L0 % 16 == 0) and 16-site aligned pieces go 16 sites at a time through bit masks (two 16-byte
// loads, the byte after them, popcounts); anything else site by site.  No per-site division.
__device__ __forceinline__ void row_em(const uint8_t *spins, const uint32_t L0, const uint32_t L1,
                                       const uint32_t y, uint32_t x0, uint32_t cnt, int &e, int &m)
{
    const uint8_t *row = spins + (size_t)y * L0, *down = spins + (size_t)(y + 1 == L1 ? 0 : y + 1) * L0;
    if ((L0 & 15u) == 0) {
        for (; cnt >= 16 && (x0 & 15u) == 0; x0 += 16, cnt -= 16) {
            const uint4 a = *reinterpret_cast<const uint4 *>(row + x0), d = *reinterpret_cast<const uint4 *>(down + x0);
            const uint32_t S = spin_nibble(a.x) | spin_nibble(a.y) << 4 | spin_nibble(a.z) << 8 | spin_nibble(a.w) << 12;
            const uint32_t D = spin_nibble(d.x) | spin_nibble(d.y) << 4 | spin_nibble(d.z) << 8 | spin_nibble(d.w) << 12;
            const uint32_t R = (S >> 1) | ((uint32_t)row[x0 + 16 == L0 ? 0 : x0 + 16] << 15);
            e += 32 - 2 * (__popc(S ^ R) + __popc(S ^ D));
            m += 2 * __popc(S) - 16;
        }
    }
    for (; cnt; ++x0, --cnt) {
        const int v = 2 * row[x0] - 1;
        e += v * ((2 * row[x0 + 1 == L0 ? 0 : x0 + 1] - 1) + (2 * down[x0] - 1));
        m += v;
    }
}

// Block (bxi, byi) of a recorded sweep, labelled tile by tile as the reference does (its AssignLabels,
// then the in-block part of its MergeLabels), so that the tile stage can be dumped: lcg32 draws,
// bonds and a union-find with one node per site in shared memory.  Runs on all threads of the
// CTA (whole warps); smem holds assign_smem(g, W).total bytes.  Plain sweeps take assign_strips
// (sw_strip.cuh).
template <int W>
__device__ __forceinline__ void assign_block_tiles(const Geo &g, const uint32_t bxi, const uint32_t byi,
                                                   const uint8_t *__restrict__ spins, uint32_t *__restrict__ labels,
                                                   uint32_t *__restrict__ rng_state, uint8_t *__restrict__ rng_sel,
                                                   uint32_t *__restrict__ rng_iter, const uint32_t thr,
                                                   uint32_t *__restrict__ edge, const AssignDump dump,
                                                   unsigned char *smem)
{
    const AssignSmem L = assign_smem(g, W);
    const uint32_t TX = g.TX, TY = g.TY;
    uint32_t *parent = reinterpret_cast<uint32_t *>(smem + L.parent);
    uint32_t *edge_s = reinterpret_cast<uint32_t *>(smem + L.edge);
    uint8_t *bond = smem + L.bond;
    uint8_t *sp = smem + L.sp;

    const uint32_t tid = threadIdx.x, nthr = blockDim.x;
    const uint32_t BX = g.BX, BY = g.BY, NS = BX * BY, ntb = g.TBX * g.TBY;
    const uint32_t x0 = bxi * BX, y0 = byi * BY;
    const uint32_t bxv = min(BX, g.L0 - x0), byv = min(BY, g.L1 - y0);
    const uint32_t pitch = L.pitch;

    if (tid < kEdgeWords)
        edge_s[tid] = 0;

    // ---- 1. spins of the block and its halo (column x0+bxv and row y0+byv, periodic)
    for (uint32_t i = tid; i < (bxv + 1) * (byv + 1); i += nthr) {
        const uint32_t yl = i / (bxv + 1), xl = i - yl * (bxv + 1);
        const uint32_t gx = x0 + xl < g.L0 ? x0 + xl : 0u, gy = y0 + yl < g.L1 ? y0 + yl : 0u;
        sp[yl * pitch + xl] = spins[(size_t)gy * g.L0 + gx];
    }

    // ---- 2. lcg32 draws of this sweep, one W-lane segment per tile; every update's ballot of the
    // accept bits goes to shared memory (DrawWords reads a tile's requests back); a tile shorter
    // than tile_y idles through the rows it lacks.
    for (uint32_t t0 = 0; t0 < ntb * W; t0 += nthr) {
        const uint32_t vt = t0 + tid, tb = vt / W, lane = tid % W, lane32 = tid & 31;
        const uint32_t tbr = tb / g.TBX;
        const uint32_t tgx = bxi * g.TBX + (tb - tbr * g.TBX), tgy = byi * g.TBY + tbr;
        const bool on = tb < ntb && tgx < g.n0 && tgy < g.n1;
        const uint32_t tile = tgy * g.n0 + tgx;
        const uint32_t jjmax = on ? min(TY, g.L1 - tgy * TY) : 0;
        uint32_t *draws = reinterpret_cast<uint32_t *>(smem + L.draws) + (vt >> 5) * L.slots;
        const bool wr = lane32 == 0 && vt < ntb * W;  // one writer per warp that holds tiles
        uint32_t st = 0, sel = 0, it = 0;
        if (on) {
            st = rng_state[(size_t)tile * W + lane];
            sel = rng_sel[(size_t)tile * W + lane];
            it = rng_iter[tile];
        }
        uint32_t a = lcg_param_a(sel), c = lcg_param_c(sel);
        const uint32_t Ur = (TX + W - 1) / W, Um = (TX + TY + W - 1) / W;
        const uint32_t nrow = on ? 2 * jjmax - 1 : 0;
        uint32_t to_rot = kShuffleDistance - it % kShuffleDistance;  // updates until the next rotation
        // The parameter rotation of LCG32_State::Update (random/src/lcg32.cpp:51-84): before
        // update itn when itn is a multiple of 15, the (a, c) pairs rotate by
        // state[itn & (W-1)] + (itn odd ? 0 : 1).
        auto advance = [&](const bool upd) {
            const bool rot = upd && to_rot == 1;
            if (__any_sync(0xffffffffu, rot)) {
                const uint32_t itn = it + 1;
                const uint32_t src = __shfl_sync(0xffffffffu, st, itn & (W - 1), W);
                const uint32_t from = (lane + src + ((itn & 1u) ? 0u : 1u)) & (W - 1);
                const uint32_t a2 = __shfl_sync(0xffffffffu, a, from, W);
                const uint32_t c2 = __shfl_sync(0xffffffffu, c, from, W);
                const uint32_t s2 = __shfl_sync(0xffffffffu, sel, from, W);
                if (rot) {
                    a = a2;
                    c = c2;
                    sel = s2;
                }
            }
            if (upd) {
                it += 1;
                st = a * st + c;
                to_rot = rot ? kShuffleDistance : to_rot - 1;
            }
        };
        uint32_t u = 0;
        for (uint32_t req = 0; req < 2 * TY - 1; ++req) {
            const bool upd = req < nrow;
            for (uint32_t sub = 0; sub < Ur; ++sub, ++u) {
                advance(upd);
                const uint32_t word = __ballot_sync(0xffffffffu, upd && sub * W + lane < TX && lcg_accept(st, thr));
                if (wr)
                    draws[u] = word;
            }
        }
        for (uint32_t sub = 0; sub < Um; ++sub, ++u) {
            advance(on);
            const uint32_t word = __ballot_sync(0xffffffffu, on && sub * W + lane < TX + TY && lcg_accept(st, thr));
            if (wr)
                draws[u] = word;
        }
        if (on) {
            rng_state[(size_t)tile * W + lane] = st;
            rng_sel[(size_t)tile * W + lane] = (uint8_t)sel;
            if (lane == 0)
                rng_iter[tile] = it;
        }
    }
    __syncthreads();

    // ---- 3. bonds (bit 0 +x, bit 1 +y): equal spins and an accepted draw.  The last
    // column / row of a tile bonds through the merge draw: [0, TX) bottom, [TX, TX+TY) right.
    const uint32_t Ur = (TX + W - 1) / W, um = (2 * TY - 1) * Ur;
    const DrawWords<W> dw{reinterpret_cast<const uint32_t *>(smem + L.draws), L.slots};
    for (uint32_t l = tid; l < NS; l += nthr) {
        const uint32_t xl = l % BX, yl = l / BX;
        uint8_t b = 0;
        if (xl < bxv && yl < byv) {
            const uint32_t tbx = xl / TX, tby = yl / TY, tb = tby * g.TBX + tbx;
            const uint32_t ii = xl - tbx * TX, jj = yl - tby * TY;
            const uint32_t iimax = min(TX, bxv - tbx * TX), jjmax = min(TY, byv - tby * TY);
            const uint8_t s = sp[yl * pitch + xl];
            const uint32_t xa = (ii + 1 < iimax) ? dw.bit(tb, jj * Ur, ii) : dw.bit(tb, um, TX + jj);
            const uint32_t ya = (jj + 1 < jjmax) ? dw.bit(tb, (jjmax + jj) * Ur, ii) : dw.bit(tb, um, ii);
            b = (uint8_t)(((xa & 1u) && s == sp[yl * pitch + xl + 1]) | (((ya & 1u) && s == sp[(yl + 1) * pitch + xl]) << 1));
        }
        bond[l] = b;
        parent[l] = l;
    }
    __syncthreads();

    // ---- 4. tile-local components (the reference's AssignLabels result)
    for (uint32_t l = tid; l < NS; l += nthr) {
        const uint8_t b = bond[l];
        if (!b)
            continue;
        const uint32_t xl = l % BX, yl = l / BX;
        const uint32_t tbx = xl / TX, tby = yl / TY;
        const uint32_t ii = xl - tbx * TX, jj = yl - tby * TY;
        const uint32_t iimax = min(TX, bxv - tbx * TX), jjmax = min(TY, byv - tby * TY);
        if ((b & 1) && ii + 1 < iimax)
            uf_union(parent, l, l + 1);
        if ((b & 2) && jj + 1 < jjmax)
            uf_union(parent, l, l + BX);
    }
    __syncthreads();
    if (dump.bonds || dump.tile_labels) {
        for (uint32_t l = tid; l < NS; l += nthr) {
            const uint32_t xl = l % BX, yl = l / BX;
            if (xl < bxv && yl < byv) {
                const size_t site = (size_t)(y0 + yl) * g.L0 + x0 + xl;
                if (dump.tile_labels) {
                    const uint32_t r = uf_find(parent, l);
                    dump.tile_labels[site] = (y0 + r / BX) * g.L0 + x0 + r % BX;
                }
                if (dump.bonds)
                    dump.bonds[site] = bond[l];
            }
        }
        __syncthreads();
    }

    // ---- 5. bonds between tiles of this block; bonds leaving the block go to k_merge
    for (uint32_t l = tid; l < NS; l += nthr) {
        const uint8_t b = bond[l];
        if (!b)
            continue;
        const uint32_t xl = l % BX, yl = l / BX;
        const uint32_t tbx = xl / TX, tby = yl / TY;
        const uint32_t ii = xl - tbx * TX, jj = yl - tby * TY;
        const uint32_t iimax = min(TX, bxv - tbx * TX), jjmax = min(TY, byv - tby * TY);
        if ((b & 1) && ii + 1 == iimax) {
            if (xl + 1 < bxv)
                uf_union(parent, l, l + 1);
            else
                atomicOr(edge_s, 1u << yl);
        }
        if ((b & 2) && jj + 1 == jjmax) {
            if (yl + 1 < byv)
                uf_union(parent, l, l + BX);
            else
                atomicOr(edge_s + 1 + (xl >> 5), 1u << (xl & 31));
        }
    }
    __syncthreads();

    // ---- 6. labels: a block root stores its global site index, every other site
    // kLocalFlag | the block-local index of its root
    for (uint32_t l = tid; l < NS; l += nthr) {
        const uint32_t xl = l % BX, yl = l / BX;
        if (xl < bxv && yl < byv) {
            const uint32_t r = uf_find(parent, l);
            labels[(size_t)(y0 + yl) * g.L0 + x0 + xl] =
                r == l ? (y0 + yl) * g.L0 + x0 + xl : (kLocalFlag | (r / BX * kBlockPitch + r % BX));
        }
    }
    if (tid < kEdgeWords)
        edge[((size_t)byi * g.nbx + bxi) * kEdgeWords + tid] = edge_s[tid];
}

constexpr uint32_t kMidWarps = 3;

// Warps per block in merge and resolve: one per edge word while the blocks leave the GPU's warps free, fewer
// with lists beyond.  Measured with 1 / 2 / 3 / 4 listing warps: 16384^2 sweep 1354 / 1360 / 1377 / 1386 us (a
// thread per edge site: 1418); 4096^2 at T = 2.0 132.7 / 132.8 / 127.3 / 126.2, at T = 3.0 97.3 / 94.0 / 97.4 /
// 98.3; 512-lattice mix round 269.6 / 269.7 / 267.5 / 270.3; 16 lattices 35.7 / 32.9 / 30.6 / 30.2 (by edge
// site 29.0).
inline uint32_t merge_warps(uint32_t blocks) { return blocks < 4096 ? kEdgeParts : blocks < 16384 ? kMidWarps : 1; }
inline uint32_t merge_grid(uint32_t blocks)
{
    constexpr uint32_t kWarps = kMergeThreads / 32;
    const uint32_t n = (blocks * merge_warps(blocks) + kWarps - 1) / kWarps;
    return n ? n : 1;
}

// Merge slots of a block: the root that each edge bond's union linked (kNoLink for none) -- by edge site, or
// with lists by their order and their number after the last; a multiple of 32 bytes.
constexpr uint32_t kMergeSlots = kMergeList + 8;

// Unions across the right and bottom edge (periodic) of block (bxi, byi), by warp `sub` of the kWarps
// that share the block.  With many blocks each warp lists the edge bonds that may join two clusters (at
// the critical temperature about a third of the edge sites: a thread per edge site left two lanes of
// three idle through the label loads and walks), then takes its share, one per lane; with kEdgeParts
// warps each takes one edge word as it is, the shorter way.  With `linked`, every block
// root the merge turns into a non-root appears in exactly one of its slots.  With active false (a
// lattice whose sweep budget is spent) nothing is written; the edge words are read all the same, so
// their load need not wait for the budget's.
template <uint32_t kWarps>
__device__ __forceinline__ void merge_block(const Geo &g, const uint32_t bxi, const uint32_t byi, const uint32_t sub,
                                            const uint32_t *edge, uint32_t *labels, unsigned int *fault,
                                            uint32_t *linked, uint8_t *list, const bool active = true)
{
    const uint32_t lane = threadIdx.x & 31, under = (1u << lane) - 1u;
    const uint32_t x0 = bxi * g.BX, y0 = byi * g.BY;
    const uint32_t bxv = min(g.BX, g.L0 - x0), byv = min(g.BY, g.L1 - y0);
    const uint32_t right = bxi + 1 == g.nbx ? 0 : bxi + 1, below = byi + 1 == g.nby ? 0 : byi + 1;
    const size_t blk = (size_t)byi * g.nbx + bxi;
    const uint32_t *e = edge + blk * kEdgeWords, *er = edge + ((size_t)byi * g.nbx + right) * kEdgeWords;
    const uint32_t *eb = edge + ((size_t)below * g.nbx + bxi) * kEdgeWords;
    uint32_t *slots = linked ? linked + blk * kMergeSlots : nullptr;
    // the bonds of edge word w, and of those the ones whose next neighbour would join the same runs
    auto part = [&](const uint32_t w, uint32_t &T) -> uint32_t {
        if (w == 0) {
            const uint32_t A = e[0];
            T = A & e[kEdgeYLast] & er[kEdgeYFirst];
            return A;
        }
        if ((w - 1) * 32 < bxv) {
            const uint32_t A = e[w];
            T = A & e[kEdgeXLast - 1 + w] & eb[kEdgeXFirst - 1 + w];
            return A;
        }
        T = 0;
        return 0;
    };
    auto unite = [&](const uint32_t i, const uint32_t t) {  // the i-th listed bond, edge site t
        uint32_t s, nb, nbx = bxi, nby = byi;               // the site, its neighbour, the neighbour's block
        if (t < 32) {
            s = (y0 + t) * g.L0 + x0 + bxv - 1;
            nb = (y0 + t) * g.L0 + (x0 + bxv < g.L0 ? x0 + bxv : 0u);
            nbx = right;
        } else {
            s = (y0 + byv - 1) * g.L0 + x0 + t - 32;
            nb = (y0 + byv < g.L1 ? y0 + byv : 0u) * g.L0 + x0 + t - 32;
            nby = below;
        }
        const volatile uint32_t *vl = labels;
        const uint32_t a = label_global(g, bxi, byi, vl[s]), b = label_global(g, nbx, nby, vl[nb]);
        const uint32_t link = a != b ? guf_union_pair(labels, a, b, g.L0 * g.L1, fault) : kNoLink;
        if (slots)
            slots[i] = link;
    };
    if constexpr (kWarps == kEdgeParts) {
        uint32_t T;
        const uint32_t A = part(sub, T), U = A & ~(T << 1);
        if (!active)
            return;
        if ((U >> lane) & 1u)
            unite(sub * 32 + lane, sub * 32 + lane);
        else if (slots)
            slots[sub * 32 + lane] = kNoLink;
        return;
    }
    uint32_t T = 0, n = 0;
    const uint32_t A = lane < kEdgeParts ? part(lane, T) : 0u;
    const uint32_t carry = __shfl_up_sync(0xffffffffu, T, 1) >> 31;
    const uint32_t U = A & ~(T << 1 | (lane < 2 ? 0u : carry));
#pragma unroll
    for (uint32_t w = 0; w < kEdgeParts; ++w) {
        const uint32_t word = __shfl_sync(0xffffffffu, U, w);
        if ((word >> lane) & 1u)
            list[n + __popc(word & under)] = (uint8_t)(w * 32 + lane);
        n += __popc(word);
    }
    __syncwarp();
    if (!active)
        return;
    if (slots && lane == 0 && sub == 0)
        slots[kMergeList] = n;
    for (uint32_t i = sub * 32 + lane; i < n; i += kWarps * 32)
        unite(i, list[i]);
}

// ResolveLabels for the roots the merge linked (block (bxi, byi)'s slots, after every merge of the sweep):
// the root's chain is walked to the cluster's root, which is stored in its label.  Afterwards every
// block root's label is its cluster's root, so the flip needs no chase; the chases of all blocks are
// in flight together here instead of behind each flip CTA's barrier.
template <uint32_t kWarps>
__device__ __forceinline__ void resolve_block(const Geo &g, const uint32_t bxi, const uint32_t byi, const uint32_t sub,
                                              const uint32_t *linked, uint32_t *labels, unsigned int *fault,
                                              const bool active = true)
{
    const uint32_t *slots = linked + ((size_t)byi * g.nbx + bxi) * kMergeSlots;
    uint32_t i = sub * 32 + (threadIdx.x & 31);
    uint32_t b = slots[i];
    const uint32_t n = !active ? 0u : kWarps == kEdgeParts ? kMergeList : min(slots[kMergeList], kMergeList);
    while (i < n) {
        if (b != kNoLink)
            labels[b] = guf_find(labels, b, g.L0 * g.L1, fault);  // the tree's minimum: other finds' atomicMin never undo it
        i += kWarps * 32;
        if (i < n)
            b = slots[i];
    }
}

// Shared memory of flip_block: the resolved label of every block root.
__host__ __device__ inline uint32_t flip_smem_bytes(const Geo &g)
{
    return g.BY * kBlockPitch * 4;
}

// ResolveLabels + FlipClusters for block (bxi, byi) after the merge.  Block roots (labels
// without kLocalFlag) follow their chain once (guf_find, which also compresses it for the other
// blocks) into shared memory, or with kResolved (resolve_block ran) take their label as it is;
// every site then reads its root's result there and flips iff the cluster's label is odd.
// kWriteLabels stores the resolved global labels (the reference's ResolveLabels output).
// With active false (a lattice whose sweep budget is spent) the block is read but nothing is
// written, so the loads need not wait for the budget's.
template <bool kWriteLabels, int kQuads = 2, bool kResolved = false>
__device__ __forceinline__ void flip_block(const Geo &g, const uint32_t bxi, const uint32_t byi, uint8_t *spins,
                                           uint32_t *labels, unsigned int *fault, unsigned char *smem,
                                           const bool active = true)
{
    const uint32_t L0 = g.L0;
    uint32_t *res = reinterpret_cast<uint32_t *>(smem);
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
    const uint32_t x0 = bxi * g.BX, y0 = byi * g.BY;
    const uint32_t bxv = min(g.BX, L0 - x0), byv = min(g.BY, g.L1 - y0);
    const uint32_t base = y0 * L0 + x0;
    const uint32_t nq = (bxv >> 2) * byv, qrow = bxv >> 2;
    // quads per row: a power of two (32 in a full 128-wide block) takes the shift path below
    const bool qpow2 = qrow && (qrow & (qrow - 1)) == 0;
    if ((L0 & 3u) == 0 && qpow2 && (blockDim.x & (qrow - 1)) == 0 && nq <= kQuads * blockDim.x) {
        // Every thread holds at most kQuads quads (4 labels + 4 spins each) in registers: one
        // round trip for the loads, the merged roots' chains, then the flips.  Quad k of a
        // thread is column xq of row yl0 + k * rstep (whole rows per step).
        const uint32_t lq = __ffs(qrow) - 1;
        const uint32_t rstep = blockDim.x >> lq, yl0 = tid >> lq, xq4 = 4 * (tid & (qrow - 1));
        uint4 lab[kQuads];
        uint32_t spn[kQuads];
#pragma unroll
        for (int k = 0; k < kQuads; ++k) {
            const uint32_t yl = yl0 + k * rstep;
            if (yl < byv) {
                const uint32_t s = base + yl * L0 + xq4;
                lab[k] = *reinterpret_cast<const uint4 *>(labels + s);
                spn[k] = reinterpret_cast<const uint32_t *>(spins)[s >> 2];
            }
        }
#pragma unroll
        for (int k = 0; k < kQuads; ++k) {
            const uint32_t yl = yl0 + k * rstep;
            if (yl < byv) {
                const uint32_t s = base + yl * L0 + xq4, l = yl * kBlockPitch + xq4;
                const uint32_t v[4] = {lab[k].x, lab[k].y, lab[k].z, lab[k].w};
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (!(v[j] & kLocalFlag))  // a block root: v is its parent (itself unless merged)
                        res[l + j] = kResolved || !active || v[j] == s + j ? v[j]
                                                                            : guf_find(labels, v[j], L0 * g.L1, fault);
            }
        }
        __syncthreads();
        if (!active)
            return;
#pragma unroll
        for (int k = 0; k < kQuads; ++k) {
            const uint32_t yl = yl0 + k * rstep;
            if (yl < byv) {
                const uint32_t s = base + yl * L0 + xq4, l = yl * kBlockPitch + xq4;
                const uint32_t v[4] = {lab[k].x, lab[k].y, lab[k].z, lab[k].w};
                uint32_t r[4], flip = 0;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    r[j] = res[(v[j] & kLocalFlag) ? (v[j] & kLocalMask) : l + j];
                    flip |= (r[j] & 1u) << (8 * j);
                }
                reinterpret_cast<uint32_t *>(spins)[s >> 2] = spn[k] ^ flip;
                if (kWriteLabels)
                    *reinterpret_cast<uint4 *>(labels + s) = make_uint4(r[0], r[1], r[2], r[3]);
            }
        }
        return;
    }
    for (uint32_t yl = warp; yl < byv; yl += nwarps)
        for (uint32_t xl = lane; xl < bxv; xl += 32) {
            const uint32_t site = base + yl * L0 + xl;
            const uint32_t v = labels[site];
            if (!(v & kLocalFlag))
                res[yl * kBlockPitch + xl] = kResolved || !active || v == site ? v : guf_find(labels, v, L0 * g.L1, fault);
        }
    __syncthreads();
    if (!active)
        return;
    if ((L0 & 3u) == 0) {
        for (uint32_t yl = warp; yl < byv; yl += nwarps) {
            const uint32_t row = base + yl * L0;
            for (uint32_t q = lane; 4 * q < bxv; q += 32) {
                const uint32_t s = row + 4 * q;
                const uint4 lab = *reinterpret_cast<const uint4 *>(labels + s);
                const uint32_t v[4] = {lab.x, lab.y, lab.z, lab.w};
                uint32_t r[4], flip = 0;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    r[k] = res[(v[k] & kLocalFlag) ? (v[k] & kLocalMask) : yl * kBlockPitch + 4 * q + k];
                    flip |= (r[k] & 1u) << (8 * k);
                }
                reinterpret_cast<uint32_t *>(spins)[s >> 2] ^= flip;
                if (kWriteLabels)
                    *reinterpret_cast<uint4 *>(labels + s) = make_uint4(r[0], r[1], r[2], r[3]);
            }
        }
    } else {
        for (uint32_t yl = warp; yl < byv; yl += nwarps)
            for (uint32_t xl = lane; xl < bxv; xl += 32) {
                const uint32_t s = base + yl * L0 + xl;
                const uint32_t v = labels[s];
                const uint32_t r = res[(v & kLocalFlag) ? (v & kLocalMask) : yl * kBlockPitch + xl];
                spins[s] ^= (uint8_t)(r & 1u);
                if (kWriteLabels)
                    labels[s] = r;
            }
    }
}


}  // namespace swb
