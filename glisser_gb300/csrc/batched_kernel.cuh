// Ensemble (persistent work-queue) kernel template, included by the
// translation units that instantiate it (plain starters in batched.cu, the
// learned starter in batched_learned.cu; disjoint instantiations, internal
// linkage).
#pragma once
#include "tile.cuh"

namespace glisser {
namespace {

using namespace tile;

// Resident threads per SM the ensemble kernel's registers are sized for; a
// build-time tuning knob.  The kernel is bound by issue, and spills are
// instructions: 768 (80 registers, 6 CTAs of 128, 32 bytes of spill stores and loads)
// run the 256 giants systems' 512-step block in 34.8 ms, 1,024 (64 registers, 360
// bytes) in 37.2, 896 in 35.7 to 36.7, 640 in 36.2, 512 in 35.9.  Systems whose every drift is general
// (close-eccentric, bound by the FP64 pipe) run 1.5 % slower at 768 than at 1,024.
// The learned-starter kernel, which a block takes only when some drifts are wide,
// stays at 1,024: 2 % faster than at 768 where every drift runs the network.
#ifndef GLISSER_BATCHED_THREADS_PER_SM
#define GLISSER_BATCHED_THREADS_PER_SM 768
#endif
#ifndef GLISSER_BATCHED_THREADS_PER_SM_LEARNED
#define GLISSER_BATCHED_THREADS_PER_SM_LEARNED 1024
#endif

// Persistent kernel over (system, tile) work items.  The learned starter
// runs its network per lane, inline, only where the series starter is
// outside its domain.
template <int NP, int CTA, int PPT, bool LEARNED, bool KICK64>
__global__ void __launch_bounds__(CTA, (LEARNED ? GLISSER_BATCHED_THREADS_PER_SM_LEARNED
                                                : GLISSER_BATCHED_THREADS_PER_SM) / CTA)
    batched_kernel(const Common p, BatchSystems sys, const BatchItem* items, const uint32_t* n_items, uint32_t* queue)
{
    extern __shared__ __align__(128) double stage[];
    __shared__ CtaShared sh;
    init_barriers(sh);
    uint32_t phase[2] = { 0, 0 };
    const uint32_t total = *n_items;
    for (;;) {
        if (threadIdx.x == 0) sh.item = atomicAdd(queue, 1u);
        __syncthreads();
        const uint32_t it = sh.item;
        if (it >= total || sh.abort) break;
        const BatchItem w = items[it];
        load_planet_constants(p, sh, p.npl, sys.m + (size_t)w.system * p.npl, sys.rh + (size_t)w.system * p.npl,
                              sys.id + (size_t)w.system * p.npl);
        __syncthreads();
        bool ok = run_tile<NP, CTA, PPT, LEARNED, KICK64>(p, sys.log + (size_t)w.system * sys.log_stride, w.first,
                                                          w.count, stage, sh, phase);
        __syncthreads();   // sh.item / planet constants are rewritten by the next item
        if (!ok) break;
    }
}

template <int NP, int CTA, int PPT, bool LEARNED, bool KICK64>
cudaError_t launch_batched_t(const Common& p, const BatchSystems& sys, const BatchItem* items,
                             const uint32_t* n_items, uint32_t* queue, const BatchShape& shape, size_t smem,
                             cudaStream_t stream)
{
    uint32_t grid = shape.grid;
    auto kern = batched_kernel<NP, CTA, PPT, LEARNED, KICK64>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    if (grid == 0) {
        int dev = 0, sms = 0, per = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, CTA, smem);
        grid = (uint32_t)(sms * (per > 0 ? per : 1));
        // with fewer items than CTAs, which CTAs pop one is a matter of chance, and an
        // SM may hold several of them while others hold none: one CTA per item is
        // spread evenly (16 systems, 9,000 particles x 256 steps: 1.86 -> 0.64 ms)
        if (shape.items && shape.items < grid) grid = shape.items;
    }
    kern<<<grid, CTA, smem, stream>>>(p, sys, items, n_items, queue);
    return cudaGetLastError();
}

template <int NP, bool LEARNED, bool KICK64>
cudaError_t launch_batched_np(const Common& p, const BatchSystems& sys, const BatchItem* items,
                              const uint32_t* n_items, uint32_t* queue, const BatchShape& shape, size_t smem,
                              cudaStream_t stream)
{
    const int key = shape.cta * 10 + shape.ppt;
    switch (key) {
    case 641: return launch_batched_t<NP, 64, 1, LEARNED, KICK64>(p, sys, items, n_items, queue, shape, smem, stream);
    case 642: return launch_batched_t<NP, 64, 2, LEARNED, KICK64>(p, sys, items, n_items, queue, shape, smem, stream);
    case 1281: return launch_batched_t<NP, 128, 1, LEARNED, KICK64>(p, sys, items, n_items, queue, shape, smem, stream);
    case 1282: return launch_batched_t<NP, 128, 2, LEARNED, KICK64>(p, sys, items, n_items, queue, shape, smem, stream);
    case 2561: return launch_batched_t<NP, 256, 1, LEARNED, KICK64>(p, sys, items, n_items, queue, shape, smem, stream);
    case 2562: return launch_batched_t<NP, 256, 2, LEARNED, KICK64>(p, sys, items, n_items, queue, shape, smem, stream);
    default: return cudaErrorInvalidValue;
    }
}

// One kernel variant: four planets besides the Sun specialised, other counts
// on the generic planet loop.
template <bool LEARNED, bool KICK64>
cudaError_t launch_batched_variant(const Common& p, const BatchSystems& sys, const BatchItem* items,
                                   const uint32_t* n_items, uint32_t* queue, uint32_t npl, const BatchShape& shape,
                                   size_t smem, cudaStream_t stream)
{
    return npl == 5 ? launch_batched_np<4, LEARNED, KICK64>(p, sys, items, n_items, queue, shape, smem, stream)
                    : launch_batched_np<0, LEARNED, KICK64>(p, sys, items, n_items, queue, shape, smem, stream);
}

}  // namespace

// Launches of the variants compiled in other translation units (one variant
// per unit): plain starters with the FP64 kick (batched_kick64.cu), the
// learned starter with the float-float kick (batched_learned.cu) and with the
// FP64 kick (batched_learned_kick64.cu).
#define GLISSER_BATCHED_VARIANT_LAUNCH(name)                                                                     \
    cudaError_t name(const tile::Common& p, const BatchSystems& sys, const BatchItem* items,                     \
                     const uint32_t* n_items, uint32_t* queue, uint32_t npl, const BatchShape& shape, size_t smem, \
                     cudaStream_t stream)
GLISSER_BATCHED_VARIANT_LAUNCH(launch_batched_kick64);
GLISSER_BATCHED_VARIANT_LAUNCH(launch_batched_learned);
GLISSER_BATCHED_VARIANT_LAUNCH(launch_batched_learned_kick64);

}  // namespace glisser
