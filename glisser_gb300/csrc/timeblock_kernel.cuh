// Single-system time-block kernel template, included by the translation
// units that instantiate it (plain starters in timeblock.cu, the learned
// starter in timeblock_learned.cu; disjoint instantiations, internal linkage).
#pragma once
#include "tile.cuh"

namespace glisser {
namespace {

using namespace tile;

// CTAs per SM the register allocation is sized for: 16 CTAs of 64 threads (64
// registers, a few dozen bytes of spills; 32-step planet-log chunks, so that
// shared memory admits 16 with four planets).  12 CTAs measured 3 % slower on
// the giants and 5 % on planet crossers, 8 CTAs 4 and 9 %; only a run that leaves
// the SMs nearly empty (2,000 particles) gains, 4 to 6 %.
#ifndef GLISSER_TB_MIN_BLOCKS
#define GLISSER_TB_MIN_BLOCKS 16
#endif

// The learned-starter kernel runs the network per lane, inline, only where
// the series starter is outside its domain.  Sized for 14 CTAs of 64 (72
// registers; a second instance, below, for 16): the network's registers cost less
// there than its spills at 16 (64 registers): 14.46 against 14.66 ms for 64 steps of
// 1e6 close-eccentric particles; 5.31 against 5.15 ms on 1e6 scattered-disk
// particles, where 0.1 % of drifts take the network.  The network's shape (mlp_forward: four rows of the hidden
// layer per pass, two activation reads in flight) was chosen for a register
// budget.
#ifndef GLISSER_TB_MIN_BLOCKS_LEARNED
#define GLISSER_TB_MIN_BLOCKS_LEARNED 14
#endif
constexpr int TB_NET_ROWS = 4;
constexpr int TB_NET_QU = 2;

// Particles per thread of the plain-starter kernel (a build-time tuning
// knob; the learned kernel keeps one).  Two (118 registers, 8 CTAs per SM)
// measured 14 % slower on the plain-giants workload and 36 % on the
// scattered disk, where the warp-uniform Stumpff tiers diverge more often.
#ifndef GLISSER_TB_PPT
#define GLISSER_TB_PPT 1
#endif

template <int NP, bool LEARNED, bool KICK64, int CTAS_PER_SM>
__global__ void __launch_bounds__(BLOCK_THREADS, CTAS_PER_SM)
    timeblock_kernel(const Common p, const double* log, const double* m, const double* rh, const uint32_t* pid,
                     uint32_t n)
{
    extern __shared__ __align__(128) double stage[];
    __shared__ CtaShared sh;
    load_planet_constants(p, sh, p.npl, m, rh, pid);
    init_barriers(sh);
    __syncthreads();
    uint32_t phase[2] = { 0, 0 };
    constexpr int PPT = LEARNED ? 1 : GLISSER_TB_PPT;
    const uint32_t first = blockIdx.x * (uint32_t)(BLOCK_THREADS * PPT);
    run_tile<NP, BLOCK_THREADS, PPT, LEARNED, KICK64, TB_NET_ROWS, TB_NET_QU>(
        p, log, first, min((uint32_t)(BLOCK_THREADS * PPT), n - first), stage, sh, phase);
}

// The learned kernel's second instance, sized for the plain kernel's CTAs per SM,
// runs a grid that it takes in fewer waves: a wave of a few CTAs lasts as long as
// their serial chain.  100,000 close-eccentric particles x 128 steps (one wave of
// either) 3.40 ms with 14 CTAs and 4.44 with 16, 135,000 4.12 and 4.49, 140,000 (two
// waves of 14) 5.34 and 4.58, 150,000 5.70 and 4.83.  With many waves it matters little
// which runs, and 16, which the rule then takes, is not always the faster: 1e6
// particles x 64 steps 14.66 ms against 14.46 with 14 where every drift takes the
// network, 5.15 against 5.31 on the scattered disk.
inline bool learned_saves_a_wave(uint32_t grid, uint32_t sms)
{
    const uint32_t lean = sms * GLISSER_TB_MIN_BLOCKS_LEARNED, full = sms * GLISSER_TB_MIN_BLOCKS;
    return (grid + full - 1) / full < (grid + lean - 1) / lean;
}

template <int NP, bool LEARNED, bool KICK64, int CTAS_PER_SM>
cudaError_t launch_sized(const Common& p, const glisser_planet_block* pl, uint32_t n, uint32_t grid, size_t smem,
                         cudaStream_t stream)
{
    auto kern = timeblock_kernel<NP, LEARNED, KICK64, CTAS_PER_SM>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    kern<<<grid, BLOCK_THREADS, smem, stream>>>(p, pl->log, pl->m, pl->rh, pl->id, n);
    return cudaGetLastError();
}

template <int NP, bool LEARNED, bool KICK64>
cudaError_t launch_np(const Common& p, const glisser_planet_block* pl, uint32_t n, size_t smem, cudaStream_t stream)
{
    const uint32_t per_cta = (uint32_t)BLOCK_THREADS * (LEARNED ? 1u : (uint32_t)GLISSER_TB_PPT);
    const uint32_t grid = (n + per_cta - 1) / per_cta;
    if constexpr (LEARNED) {
        int dev = 0, sms = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return e;
        if (learned_saves_a_wave(grid, (uint32_t)sms))
            return launch_sized<NP, LEARNED, KICK64, GLISSER_TB_MIN_BLOCKS>(p, pl, n, grid, smem, stream);
        return launch_sized<NP, LEARNED, KICK64, GLISSER_TB_MIN_BLOCKS_LEARNED>(p, pl, n, grid, smem, stream);
    } else {
        return launch_sized<NP, LEARNED, KICK64, GLISSER_TB_MIN_BLOCKS>(p, pl, n, grid, smem, stream);
    }
}

// Dispatch over the planet count for one kernel variant.
template <bool LEARNED, bool KICK64>
cudaError_t launch_variant(const Common& p, const glisser_planet_block* pl, uint32_t n, size_t smem,
                           cudaStream_t stream)
{
    if constexpr (LEARNED) {
        // learned instantiations: one and four planets besides the Sun
        // specialised, other counts on the generic planet loop
        switch (pl->npl - 1) {
        case 1: return launch_np<1, true, KICK64>(p, pl, n, smem, stream);
        case 4: return launch_np<4, true, KICK64>(p, pl, n, smem, stream);
        default: return launch_np<0, true, KICK64>(p, pl, n, smem, stream);
        }
    } else {
        switch (pl->npl - 1) {
        case 1: return launch_np<1, false, KICK64>(p, pl, n, smem, stream);
        case 2: return launch_np<2, false, KICK64>(p, pl, n, smem, stream);
        case 3: return launch_np<3, false, KICK64>(p, pl, n, smem, stream);
        case 4: return launch_np<4, false, KICK64>(p, pl, n, smem, stream);
        case 5: return launch_np<5, false, KICK64>(p, pl, n, smem, stream);
        case 6: return launch_np<6, false, KICK64>(p, pl, n, smem, stream);
        case 7: return launch_np<7, false, KICK64>(p, pl, n, smem, stream);
        case 8: return launch_np<8, false, KICK64>(p, pl, n, smem, stream);
        default: return launch_np<0, false, KICK64>(p, pl, n, smem, stream);
        }
    }
}

}  // namespace

// Launches of the variants compiled in other translation units (each unit
// instantiates one variant, so that the units compile in parallel and keep
// their register allocations apart): plain starters with the FP64 kick
// (timeblock_kick64.cu), the learned starter with either kick
// (timeblock_learned.cu).
cudaError_t launch_timeblock_kick64(const tile::Common& p, const glisser_planet_block* pl, uint32_t n, size_t smem,
                                    cudaStream_t stream);
cudaError_t launch_timeblock_learned(const tile::Common& p, const glisser_planet_block* pl, uint32_t n, size_t smem,
                                     cudaStream_t stream);

}  // namespace glisser
