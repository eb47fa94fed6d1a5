// Kernels and launch of the one-kernel sweep of a small lattice (sw_whole.cuh).
#include "sw_whole.cuh"

namespace swb {
namespace {

template <int W, int TXc, int TYc, bool kMeasure>
__global__ void __launch_bounds__(kWholeThreads, 1) k_whole(const Whole w, uint8_t *spins, uint32_t *rng_state,
                                                            uint8_t *rng_sel, uint32_t *rng_iter, const uint32_t thr,
                                                            const MeasureArgs meas, unsigned int *fault)
{
    extern __shared__ __align__(16) unsigned char smem[];
    sweep_whole<W, TXc, TYc, kMeasure>(w, spins, rng_state, rng_sel, rng_iter, thr, meas, fault, smem);
}

using WholeKernel = void (*)(Whole, uint8_t *, uint32_t *, uint8_t *, uint32_t *, uint32_t, MeasureArgs, unsigned int *);

template <int W, bool kMeasure>
WholeKernel kernel_for(uint32_t TX, uint32_t TY)
{
    if constexpr (W == 16) {
        if (TX == 16 && TY == 8) return k_whole<W, 16, 8, kMeasure>;
        if (TX == 16 && TY == 4) return k_whole<W, 16, 4, kMeasure>;
    }
    return TX == 8 ? k_whole<W, 8, 0, kMeasure> : TX == 16 ? k_whole<W, 16, 0, kMeasure> : k_whole<W, 32, 0, kMeasure>;
}

WholeKernel kernel_for(uint32_t W, uint32_t TX, uint32_t TY, bool measure)
{
    switch (W) {
    case 8: return measure ? kernel_for<8, true>(TX, TY) : kernel_for<8, false>(TX, TY);
    case 16: return measure ? kernel_for<16, true>(TX, TY) : kernel_for<16, false>(TX, TY);
    default: return measure ? kernel_for<32, true>(TX, TY) : kernel_for<32, false>(TX, TY);
    }
}

}  // namespace

namespace {

struct Config {
    cudaLaunchAttribute at[2] = {};
    cudaLaunchConfig_t cfg{};
    Config(const Whole &w, uint32_t W, cudaStream_t st)
    {
        at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[0].val.programmaticStreamSerializationAllowed = 1;
        at[1].id = cudaLaunchAttributeClusterDimension;
        at[1].val.clusterDim.x = w.ctas;
        at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
        const uint32_t pieces = w.strips * w.tr;
        cfg.gridDim = w.ctas;
        cfg.blockDim = 32 * (pieces < kWholeThreads / 32 ? pieces : kWholeThreads / 32);
        cfg.dynamicSmemBytes = whole_smem(w, W).total;
        cfg.stream = st;
        cfg.attrs = at;
        cfg.numAttrs = w.ctas > 1 ? 2 : 1;
    }
};

}  // namespace

cudaError_t allow_whole(const Whole &w, uint32_t W, bool *fits)
{
    *fits = false;
    if (whole_smem(w, W).total > kWholeSmemMax)
        return cudaSuccess;
    for (bool measure : {false, true}) {
        const WholeKernel k = kernel_for(W, w.g.TX, w.g.TY, measure);
        if (cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kWholeSmemMax))
            return e;
        if (cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1))
            return e;
        int clusters = 1;
        const Config c(w, W, nullptr);
        if (w.ctas > 1)
            if (cudaError_t e = cudaOccupancyMaxActiveClusters(&clusters, k, &c.cfg))
                return e;
        if (clusters < 1)  // no room for such a cluster on this device
            return cudaSuccess;
    }
    *fits = true;
    return cudaSuccess;
}

int launch_whole(const Whole &w, uint32_t W, uint8_t *spins, uint32_t *rng_state, uint8_t *rng_sel, uint32_t *rng_iter,
                 uint32_t thr, const MeasureArgs &meas, unsigned int *fault, cudaStream_t st)
{
    const Config c(w, W, st);
    g_launches.fetch_add(1, std::memory_order_relaxed);
    const cudaError_t e = cudaLaunchKernelEx(&c.cfg, kernel_for(W, w.g.TX, w.g.TY, meas.obs != nullptr), w, spins,
                                             rng_state, rng_sel, rng_iter, thr, meas, fault);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return fail(SWB_ERR_CUDA, "kernel launch failed: %s", cudaGetErrorString(e));
    }
    return SWB_OK;
}

}  // namespace swb
