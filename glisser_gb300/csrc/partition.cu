// Stable three-way partition of the particle arrays: unflagged particles
// first, then particles in encounter ((flags & 0xFE) == 0, flags != 0), then
// the rest.  Replaces the unstable thrust::partition calls of the reference
// executor (src/executor.cu:663-665, 784-790, 865-869) with a deterministic
// order, so the host mirror and every output file are reproducible.
//
// Two launches over at most RANGES contiguous ranges of particles, one CTA each:
// the counts of each range's categories, then a scatter in which every CTA adds
// up the counts before its own (a few KB from L2) and walks its range in tiles of
// TILE, writing the 12 particle arrays to the output buffer.  HBM traffic is one
// read of the flags plus one read and one write of the 90-byte particle record.
//
// Bound: HBM.  A tile's record is read before its flags are ranked, and the next
// tile's before this one's is written, so that loads are in flight across the
// barriers.  A separate scan launch of one CTA between the two (per-tile
// counts, one particle per thread, the record read after the ranks) took 55 us
// for 1e6 particles and 197 us for 4e6; this takes 36.9 and 119 us, 0.72 and 0.89
// of the measured copy rate, and 8.4 against 14.5 us for 5,000.
#include <cuda.h>

#include <cstdio>
#include <mutex>

#include "timeblock.cuh"

namespace glisser {

namespace {

constexpr int TILE = 256;
// three CTAs of 256 threads (80 registers: two records) on each of GB300's 152 SMs; four at
// 64 registers measured 38 against 35 us for 1e6 particles
constexpr uint32_t RANGES = 152 * 3;

__device__ __forceinline__ int category(uint16_t f)
{
    if (f == 0) return 0;
    if ((f & 0xFE) == 0) return 1;
    return 2;
}

// Sums of two values over the CTA, returned to every thread.
__device__ __forceinline__ void cta_sum2(uint32_t& a, uint32_t& b, uint32_t (*buf)[TILE / 32])
{
    a = __reduce_add_sync(0xffffffffu, a);
    b = __reduce_add_sync(0xffffffffu, b);
    if ((threadIdx.x & 31) == 0) {
        buf[0][threadIdx.x >> 5] = a;
        buf[1][threadIdx.x >> 5] = b;
    }
    __syncthreads();
    a = b = 0;
#pragma unroll
    for (int w = 0; w < TILE / 32; w++) {
        a += buf[0][w];
        b += buf[1][w];
    }
    __syncthreads();
}

// Counts of categories 0 and 1 of range b = [b * per, (b + 1) * per) into
// counts[2 * b + {0, 1}].
__global__ void __launch_bounds__(TILE) count_kernel(const uint16_t* __restrict__ flags, uint32_t n, uint32_t per,
                                                     uint32_t* counts)
{
    __shared__ uint32_t buf[2][TILE / 32];
    const uint32_t lo = blockIdx.x * per, hi = n - lo < per ? n : lo + per;
    uint32_t c0 = 0, c1 = 0;
#pragma unroll 4
    for (uint32_t i = lo + threadIdx.x; i < hi; i += TILE) {
        const int cat = category(flags[i]);
        c0 += cat == 0;
        c1 += cat == 1;
    }
    cta_sum2(c0, c1, buf);
    if (threadIdx.x == 0) {
        counts[2 * blockIdx.x] = c0;
        counts[2 * blockIdx.x + 1] = c1;
    }
}

struct Record {
    double f[9];
    uint32_t dti, id;
    uint16_t flags;
};

__device__ __forceinline__ Record read_record(const glisser_particles& p, uint32_t i, bool valid)
{
    Record r = {};
    if (valid) {
        r.flags = p.flags[i];
        r.f[0] = p.rx[i]; r.f[1] = p.ry[i]; r.f[2] = p.rz[i];
        r.f[3] = p.vx[i]; r.f[4] = p.vy[i]; r.f[5] = p.vz[i];
        r.f[6] = p.ax[i]; r.f[7] = p.ay[i]; r.f[8] = p.az[i];
        r.dti = p.deathtime_index[i];
        r.id = p.id[i];
    }
    return r;
}

__global__ void __launch_bounds__(TILE, 3) scatter_kernel(glisser_particles in, glisser_particles out, uint32_t n,
                                                       uint32_t per, const uint32_t* __restrict__ counts,
                                                       uint32_t* n0p, uint32_t* n1p)
{
    __shared__ uint32_t buf[2][TILE / 32];
    __shared__ uint32_t warp_c[2][2][TILE / 32];
    const uint32_t lo = blockIdx.x * per, hi = n - lo < per ? n : lo + per;
    Record cur = read_record(in, lo + threadIdx.x, lo + threadIdx.x < hi);
    // category counts before this range, and in all
    uint32_t before0 = 0, before1 = 0, all0 = 0, all1 = 0;
    for (uint32_t b = threadIdx.x; b < gridDim.x; b += TILE) {
        const uint32_t c0 = counts[2 * b], c1 = counts[2 * b + 1];
        all0 += c0;
        all1 += c1;
        before0 += b < blockIdx.x ? c0 : 0u;
        before1 += b < blockIdx.x ? c1 : 0u;
    }
    cta_sum2(before0, before1, buf);
    cta_sum2(all0, all1, buf);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *n0p = all0;
        *n1p = all1;
    }
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5, lt = (1u << lane) - 1u;
    uint32_t parity = 0;
    for (uint32_t base = lo; base < hi; base += TILE, parity ^= 1u) {
        const uint32_t i = base + threadIdx.x;
        const Record next = read_record(in, i + TILE, i + TILE < hi);
        const int cat = i < hi ? category(cur.flags) : 3;
        const unsigned b0 = __ballot_sync(0xffffffffu, cat == 0), b1 = __ballot_sync(0xffffffffu, cat == 1);
        if (lane == 0) {
            warp_c[parity][0][warp] = __popc(b0);
            warp_c[parity][1][warp] = __popc(b1);
        }
        __syncthreads();     // the other parity's counts are rewritten only after the next one
        uint32_t r0 = before0 + __popc(b0 & lt), r1 = before1 + __popc(b1 & lt);
#pragma unroll
        for (unsigned w = 0; w < TILE / 32; w++) {
            const uint32_t c0 = warp_c[parity][0][w], c1 = warp_c[parity][1][w];
            r0 += w < warp ? c0 : 0u;
            r1 += w < warp ? c1 : 0u;
            before0 += c0;
            before1 += c1;
        }
        if (i < hi) {
            const uint32_t dst = cat == 0 ? r0 : cat == 1 ? all0 + r1 : all0 + all1 + (i - r0 - r1);
            out.rx[dst] = cur.f[0]; out.ry[dst] = cur.f[1]; out.rz[dst] = cur.f[2];
            out.vx[dst] = cur.f[3]; out.vy[dst] = cur.f[4]; out.vz[dst] = cur.f[5];
            out.ax[dst] = cur.f[6]; out.ay[dst] = cur.f[7]; out.az[dst] = cur.f[8];
            out.flags[dst] = cur.flags;
            out.deathtime_index[dst] = cur.dti;
            out.id[dst] = cur.id;
        }
        cur = next;
    }
}

__global__ void copy_range_kernel(glisser_particles src, glisser_particles dst, uint32_t begin, uint32_t end)
{
    uint32_t i = begin + blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= end) return;
    dst.rx[i] = src.rx[i]; dst.ry[i] = src.ry[i]; dst.rz[i] = src.rz[i];
    dst.vx[i] = src.vx[i]; dst.vy[i] = src.vy[i]; dst.vz[i] = src.vz[i];
    dst.ax[i] = src.ax[i]; dst.ay[i] = src.ay[i]; dst.az[i] = src.az[i];
    dst.flags[i] = src.flags[i];
    dst.deathtime_index[i] = src.deathtime_index[i];
    dst.id[i] = src.id[i];
}

}  // namespace

// Copies particles [begin, end) between two particle buffers.
int launch_copy_range(const glisser_particles* src, const glisser_particles* dst, size_t begin, size_t end,
                      cudaStream_t stream)
{
    if (end <= begin) return GLISSER_OK;
    uint32_t n = (uint32_t)(end - begin);
    copy_range_kernel<<<(n + 255) / 256, 256, 0, stream>>>(*src, *dst, (uint32_t)begin, (uint32_t)end);
    return cudaGetLastError() == cudaSuccess ? GLISSER_OK : GLISSER_E_CUDA;
}

size_t partition_scratch_bytes(size_t n)
{
    size_t tiles = (n + TILE - 1) / TILE;
    return 2 * tiles * sizeof(uint32_t) + 64;
}

namespace {

// Both launches; counts holds two words per range (at most RANGES ranges, and
// never more than one per TILE particles).
int launch_two(const glisser_particles* in, const glisser_particles* out, uint32_t n, uint32_t* counts, uint32_t* n0,
               uint32_t* n1, cudaStream_t stream)
{
    const uint32_t tiles = (uint32_t)(((uint64_t)n + TILE - 1) / TILE);
    const uint32_t per = (tiles + RANGES - 1) / RANGES * TILE;       // whole tiles per range
    const uint32_t ranges = (uint32_t)(((uint64_t)n + per - 1) / per);
    count_kernel<<<ranges, TILE, 0, stream>>>(in->flags, n, per, counts);
    scatter_kernel<<<ranges, TILE, 0, stream>>>(*in, *out, n, per, counts, n0, n1);
    return cudaGetLastError() == cudaSuccess ? GLISSER_OK : GLISSER_E_CUDA;
}

}  // namespace

int launch_partition(const glisser_particles* in, const glisser_particles* out, size_t n, void* scratch,
                     uint32_t* n0, uint32_t* n1, cudaStream_t stream)
{
    if (!in || !out || !scratch || !n0 || !n1) return GLISSER_E_INVALID;
    if (n > 0xFFFFFF00ull) return GLISSER_E_INVALID;
    if (n == 0) {
        cudaMemsetAsync(n0, 0, sizeof(uint32_t), stream);
        cudaMemsetAsync(n1, 0, sizeof(uint32_t), stream);
        return cudaGetLastError() == cudaSuccess ? GLISSER_OK : GLISSER_E_CUDA;
    }
    return launch_two(in, out, (uint32_t)n, reinterpret_cast<uint32_t*>(scratch), n0, n1, stream);
}


// ---------------------------------------------------------------------------
// Partition without allocation.
//
// For callers that must not allocate device memory at all: a host program
// that runs inside another framework's memory pool or under a fixed device
// budget, where a cudaMalloc would either be refused or would synchronise the
// whole device and stall work the caller has in flight.  Such a caller still
// owns the particle buffers and the two count words; the per-tile counts
// that glisser_partition keeps in caller-provided scratch live here in a
// file-scope device array instead.
//
// NOALLOC_MAX_PARTICLES bounds n: room for 2 counts per 256-particle tile (the
// ranges use fewer), 256 KiB in all, resident on every GPU that loads the library
// until the process exits.
// Every call shares that array and leaves the last call's counts in it.  No
// entry needs clearing before a call (count_kernel writes every range's counts
// before scatter_kernel reads them), but two calls whose work overlaps on the
// GPU, on one stream or several, race on the array and corrupt each other.
constexpr size_t NOALLOC_MAX_PARTICLES = 8u << 20;
constexpr size_t NOALLOC_TILES = NOALLOC_MAX_PARTICLES / TILE;

static __device__ __align__(256) uint32_t g_noalloc_counts[2 * NOALLOC_TILES];

namespace {

// Device address of g_noalloc_counts per device.  In host code the array's
// name is only a host-side stand-in; the address kernels need comes from
// cudaGetSymbolAddress, resolved with that device current.  The address
// belongs to the context the library's module was loaded into, so it is
// cached together with that context (the driver's cuCtxGetCurrent, reached
// through the runtime's entry-point query so that the library needs no link
// to the driver library) and looked up again when the current context
// differs: after a cudaDeviceReset, or under another context of the same
// device, a call resolves the array afresh instead of using a stale address.
constexpr int NOALLOC_MAX_DEVICES = 64;
std::mutex g_noalloc_mutex;
uint32_t* g_noalloc_ptr[NOALLOC_MAX_DEVICES] = {};
CUcontext g_noalloc_ctx[NOALLOC_MAX_DEVICES] = {};

using CtxGetCurrent = CUresult (*)(CUcontext*);

CtxGetCurrent ctx_get_current()
{
    static CtxGetCurrent fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            f = nullptr;
        return reinterpret_cast<CtxGetCurrent>(f);
    }();
    return fn;
}

CUcontext current_context()
{
    CUcontext c = nullptr;
    CtxGetCurrent fn = ctx_get_current();
    if (!fn || fn(&c) != CUDA_SUCCESS) return nullptr;
    return c;
}

int noalloc_scratch(uint32_t** out)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= NOALLOC_MAX_DEVICES) return GLISSER_E_CUDA;
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    const CUcontext ctx = current_context();
    if (!g_noalloc_ptr[dev] || !ctx || ctx != g_noalloc_ctx[dev]) {
        void* ptr = nullptr;
        if (cudaGetSymbolAddress(&ptr, g_noalloc_counts) != cudaSuccess || !ptr) return GLISSER_E_CUDA;
        g_noalloc_ptr[dev] = static_cast<uint32_t*>(ptr);
        g_noalloc_ctx[dev] = current_context();   // the context the lookup ran in
    }
    *out = g_noalloc_ptr[dev];
    return GLISSER_OK;
}

}  // namespace

size_t partition_noalloc_max_particles() { return NOALLOC_MAX_PARTICLES; }

int launch_partition_noalloc(const glisser_particles* in, const glisser_particles* out, size_t n, uint32_t* n0,
                             uint32_t* n1, cudaStream_t stream)
{
    if (!in || !out || !n0 || !n1) return GLISSER_E_INVALID;
    if (n > NOALLOC_MAX_PARTICLES) return GLISSER_E_INVALID;
    uint32_t* counts = nullptr;
    int rc = noalloc_scratch(&counts);
    if (rc != GLISSER_OK) return rc;
    if (n == 0) {
        cudaMemsetAsync(n0, 0, sizeof(uint32_t), stream);
        cudaMemsetAsync(n1, 0, sizeof(uint32_t), stream);
        return cudaGetLastError() == cudaSuccess ? GLISSER_OK : GLISSER_E_CUDA;
    }
    return launch_two(in, out, (uint32_t)n, counts, n0, n1, stream);
}

}  // namespace glisser
