// Throughput kernel of the lcg32 generator on its own: the equivalent of the reference's
// TestRNG --target program (random/src/test_rng.cpp, random/src/test_rng_amd_gpu.cpp:44-133,
// random/src/test_rng_cpu.cpp).  Many independent streams, stream i seeded seed_base + i as
// LCG32_State::Init does (random/src/lcg32.cpp:27-49); each update of a stream's W lanes
// yields W numbers 2^-32 * (float)u in the order of LCG32<CPU>::NextReal (element k is lane
// k % W after update k / W + 1, random/src/lcg32.cpp:103-129), with the parameter rotation
// before every 15th update (random/src/lcg32.cpp:51-84).
//
// One stream lives in the registers of a W-lane warp segment.  What a program can observe is
// kept: the last 64 numbers of one chosen stream (the reference's 64-number buffer) and an XOR
// of the bits of every number generated, so that no number is dead code.
#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>
#include <mutex>
#include <vector>

#include "../../include/swb200.h"
#include "sw_core.cuh"

namespace swb {
namespace {

constexpr uint32_t kRngThreads = 256;
constexpr uint32_t kReport = 64;  // numbers kept of the reported stream

// drand48 jumps of 1 .. 33 steps: the lanes of a stream take their draws side by side.
struct DrandJumps {
    uint64_t A[34], C[34];
};
constexpr DrandJumps drand_jumps()
{
    DrandJumps j{};
    j.A[0] = 1;
    j.C[0] = 0;
    for (int k = 1; k < 34; ++k) {
        j.A[k] = (kDrandA * j.A[k - 1]) & kDrandMask;
        j.C[k] = (kDrandA * j.C[k - 1] + kDrandC) & kDrandMask;
    }
    return j;
}
__constant__ DrandJumps kJumps = drand_jumps();

// 2^-32 * (float)u without a conversion instruction: the halves of u go into the low mantissa bits
// of 2^23 (exact), the upper half's sum is exact, and the second fma rounds once, to nearest --
// the rounding of the conversion, which the scaling by a power of two leaves as it is.
__device__ __forceinline__ float unit_float_fma(const uint32_t u)
{
    const float hi = __uint_as_float(__byte_perm(u, 0x4B000000u, 0x7432));  // 2^23 + (u >> 16)
    const float lo = __uint_as_float(__byte_perm(u, 0x4B000000u, 0x7410));  // 2^23 + (u & 0xFFFF)
    const float t = fmaf(hi, 0x1p-16f, -0x1.0001p7f);                       // (u >> 16) 2^-16 - 2^-9, exact
    return fmaf(lo, 0x1p-32f, t);
}

// What bounds it: issue slots and the conversion.  An I2F runs at 16 per SM and clock, a quarter
// of the integer pipe's rate, so every second number is converted by fused multiply-adds instead
// (unit_float_fma): the two halves of the numbers use different pipes.  All streams share their
// iteration count, so the rotations sit at fixed places: groups of 15 updates, the last with the
// rotation, and no per-update test.  2.0e9 numbers (75776 streams x 1652 updates x 16 lanes):
// 711 us a launch with a test and a conversion per number, 377 us now (5.3 T numbers/s).
template <int W>
__global__ void __launch_bounds__(kRngThreads, 8) k_lcg32_bench(const uint32_t n_streams, const uint32_t seed_base,
                                                                const uint64_t updates, const uint32_t report_id,
                                                                float *__restrict__ report, unsigned int *checksum)
{
    constexpr uint32_t kLast = kReport / W;  // updates that fill the report buffer
    const uint32_t gid = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t stream = gid / W, lane = gid % W;
    const bool on = stream < n_streams;
    // LCG32_State::Init of this stream: drand48 draw i + 1 picks lane i's parameter pair, draw W + 1
    // seeds the first lane, every later lane follows by one step of its own pair.  Each lane jumps
    // to its draw; the lanes' steps are affine maps, composed by a scan.
    uint32_t st, a, c;
    {
        const uint64_t x0 = drand48_seed(seed_base + stream);
        const uint64_t xi = (kJumps.A[lane + 1] * x0 + kJumps.C[lane + 1]) & kDrandMask;
        const uint64_t xs = (kJumps.A[W + 1] * x0 + kJumps.C[W + 1]) & kDrandMask;
        const uint32_t sel = ((uint32_t)__dmul_rn(1000.0, drand48_value(xi))) % 5u;
        const uint32_t v = (uint32_t)__dmul_rn(4026531839.0, drand48_value(xs)) + 1u;
        a = lcg_param_a(sel);
        c = lcg_param_c(sel);
        uint32_t A = a, C = c;  // the map of lanes (lane - 2^k, lane]
#pragma unroll
        for (uint32_t o = 1; o < W; o *= 2) {
            const uint32_t pa = __shfl_up_sync(0xffffffffu, A, o, W), pc = __shfl_up_sync(0xffffffffu, C, o, W);
            if (lane >= o) {
                C = A * pc + C;
                A *= pa;
            }
        }
        st = A * v + C;
    }
    // the parameter rotation before update itn, a multiple of 15 (random/src/lcg32.cpp:51-84)
    auto rotate = [&](const uint32_t itn) {
        const uint32_t src = __shfl_sync(0xffffffffu, st, itn & (W - 1), W);
        const uint32_t from = (lane + src + ((itn & 1u) ? 0u : 1u)) & (W - 1);
        a = __shfl_sync(0xffffffffu, a, from, W);
        c = __shfl_sync(0xffffffffu, c, from, W);
    };
    uint32_t x = 0;
    uint64_t it = 0;
    for (const uint64_t groups_end = (updates - kLast) / kShuffleDistance * kShuffleDistance; it < groups_end;
         it += kShuffleDistance) {
#pragma unroll
        for (uint32_t k = 0; k < kShuffleDistance; ++k) {
            if (k == kShuffleDistance - 1)
                rotate((uint32_t)it + kShuffleDistance);
            st = a * st + c;
            x ^= __float_as_uint((k & 1) ? __uint2float_rn(st) * kTwoPowMinus32 : unit_float_fma(st));
        }
    }
    auto update = [&]() {
        ++it;
        if (it % kShuffleDistance == 0)
            rotate((uint32_t)it);
        st = a * st + c;
        const float f = unit_float_fma(st);
        x ^= __float_as_uint(f);
        return f;
    };
    while (it + kLast < updates)
        update();
    float last[kLast];
#pragma unroll
    for (uint32_t k = 0; k < kLast; ++k)
        last[k] = update();
    if (on && stream == report_id) {
#pragma unroll
        for (uint32_t k = 0; k < kLast; ++k)
            report[k * W + lane] = last[k];
    }
    x = __reduce_xor_sync(0xffffffffu, on ? x : 0u);
    if ((threadIdx.x & 31) == 0 && x)
        atomicXor(checksum, x);
}

template <int W>
int launch_bench(uint32_t n_streams, uint32_t seed_base, uint64_t updates, uint32_t report_id, float *d_report,
                 unsigned int *d_sum, cudaStream_t st)
{
    const uint64_t threads = (uint64_t)n_streams * W;
    const uint32_t grid = (uint32_t)((threads + kRngThreads - 1) / kRngThreads);
    k_lcg32_bench<W><<<grid, kRngThreads, 0, st>>>(n_streams, seed_base, updates, report_id, d_report, d_sum);
    SWB_LAUNCHED();
    return SWB_OK;
}

// What a call needs besides its kernel: a stream, two events and 65 words of device memory.
// Making and releasing them took 0.9 ms a call (cudaMalloc and cudaFree 0.68, the stream 0.10),
// twice the kernel of 2.0e9 numbers (a call: 1.31 ms, now 0.41), so up to kKeptWork are kept.  A call takes one off the list
// for itself (threads and devices never share one) and puts it back when its stream is idle; one
// that saw an error, or finds the list full, is released.
struct RngWork {
    int device = 0;
    cudaStream_t st = nullptr;
    cudaEvent_t ev[2] = {nullptr, nullptr};
    uint32_t *mem = nullptr;  // [0, kReport): the report (floats); [kReport]: the checksum

    int create(int dev)
    {
        device = dev;
        SWB_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
        for (auto &e : ev)
            SWB_CUDA(cudaEventCreate(&e));
        SWB_CUDA(cudaMalloc(&mem, (kReport + 1) * sizeof(uint32_t)));
        return SWB_OK;
    }
    void release()
    {
        if (st)
            cudaStreamSynchronize(st);
        for (auto &e : ev)
            if (e)
                cudaEventDestroy(e);
        cudaFree(mem);
        if (st)
            cudaStreamDestroy(st);
        *this = RngWork{};
    }
};
constexpr size_t kKeptWork = 4;
std::mutex g_work_mutex;
std::vector<RngWork> g_work;

}  // namespace
}  // namespace swb

using namespace swb;

extern "C" {

int swb_lcg32_benchmark(uint32_t n_streams, uint32_t lcg_width, uint32_t seed_base, uint64_t updates_per_stream,
                        uint32_t report_id, float *report, uint32_t *checksum, float *ms, int device)
{
    if (!report || !checksum || !ms)
        return fail(SWB_ERR_ARGUMENT, "NULL argument");
    if (!(lcg_width == 8 || lcg_width == 16 || lcg_width == 32))
        return fail(SWB_ERR_ARGUMENT, "unsupported lcg32 width %u (8, 16 or 32)", lcg_width);
    const uint64_t per = kReport / lcg_width;
    if (n_streams == 0 || report_id >= n_streams || updates_per_stream < per || updates_per_stream % per)
        return fail(SWB_ERR_ARGUMENT, "need n_streams > report_id and updates a positive multiple of %llu",
                    (unsigned long long)per);
    if ((uint64_t)n_streams * lcg_width > 0xFFFFFFFFull)
        return fail(SWB_ERR_ARGUMENT, "too many streams");
    SWB_CUDA(cudaSetDevice(device));
    RngWork w;
    {
        std::lock_guard<std::mutex> lock(g_work_mutex);
        for (size_t k = 0; k < g_work.size(); ++k)
            if (g_work[k].device == device) {
                w = g_work[k];
                g_work.erase(g_work.begin() + k);
                break;
            }
    }
    auto run = [&]() -> int {
        if (!w.mem)
            if (int rc = w.create(device))
                return rc;
        float *d_report = reinterpret_cast<float *>(w.mem);
        unsigned int *d_sum = w.mem + kReport;
        SWB_CUDA(cudaMemsetAsync(d_sum, 0, sizeof(unsigned int), w.st));
        SWB_CUDA(cudaEventRecord(w.ev[0], w.st));
        int rc = SWB_OK;
        switch (lcg_width) {
        case 8: rc = launch_bench<8>(n_streams, seed_base, updates_per_stream, report_id, d_report, d_sum, w.st); break;
        case 16: rc = launch_bench<16>(n_streams, seed_base, updates_per_stream, report_id, d_report, d_sum, w.st); break;
        default: rc = launch_bench<32>(n_streams, seed_base, updates_per_stream, report_id, d_report, d_sum, w.st); break;
        }
        if (rc)
            return rc;
        SWB_CUDA(cudaEventRecord(w.ev[1], w.st));
        uint32_t got[kReport + 1];
        SWB_CUDA(cudaMemcpyAsync(got, w.mem, sizeof(got), cudaMemcpyDeviceToHost, w.st));
        SWB_CUDA(cudaStreamSynchronize(w.st));
        SWB_CUDA(cudaEventElapsedTime(ms, w.ev[0], w.ev[1]));
        std::memcpy(report, got, kReport * sizeof(float));
        *checksum = got[kReport];
        return SWB_OK;
    };
    const int rc = run();
    if (rc == SWB_OK) {
        std::lock_guard<std::mutex> lock(g_work_mutex);
        if (g_work.size() < kKeptWork) {
            g_work.push_back(w);
            return SWB_OK;
        }
    }
    w.release();
    return rc;
}

}  // extern "C"
