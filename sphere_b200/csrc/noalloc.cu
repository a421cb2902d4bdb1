// noalloc.cu -- the cell list of device-resident positions without any
// device allocation (sph_cell_list_noalloc in include/sphk.h).
//
// Some callers cannot allocate device memory: a plugin whose host owns the
// whole device memory pool through its own allocator and forbids cudaMalloc,
// or a latency-critical loop that must not pay the implicit device-wide
// synchronisation of cudaMalloc/cudaFree.  This entry point computes the same
// cell list as the rest of libsphk (cell id of every particle, the stable
// (cell, particle index) order, cell start/end) using only the caller's
// input and output arrays and one fixed scratch array that lives in the
// library image: a file-scope __device__ array, which every GPU that loads
// the library holds until the process exits.
//
// The order is made by a stable least-significant-digit radix sort of the
// particles' bucket ids (the cell id, or one bucket after the last cell for
// a position outside the grid or not finite), the particle index as the
// value: every pass keeps equal digits in their order, so equal ids stay in
// particle-index order, and the work is linear in the number of particles
// whatever their spread over the cells.  Bucket ids have at most 20 bits:
// one pass where they fit one digit of 10 bits, otherwise two of half the
// bits.  The caller's two np-long outputs (sorted ids, permutation) are one
// of the sort's two buffer pairs, the scratch array the other; the passes end
// in the outputs.
//
// What bounds it: each pass waits for the scan of its digit counts, so the
// launches' latencies and, for many particles, the scatters' partial sectors.
// Seven launches where there were thirteen: 8-bit digits took three passes,
// and one block scanned all digit counts (104 of the 140 us of a pass at 1M
// particles).
//
// The host never passes the array's name to a kernel (in host code that
// name is a host-side stand-in, not a device address); it asks the runtime
// for the device address with cudaGetSymbolAddress once per device, with
// that device current, and passes that pointer.  All calls share the one
// scratch array, so calls that overlap on the GPU race; the array keeps the
// last call's contents, and every call overwrites what it reads before
// reading it.
#include "sphk_internal.cuh"
#include "../../include/sphk.h"

#include <algorithm>
#include <mutex>

namespace sphk {

// fixed capacity of the scratch array
constexpr uint32_t NA_MAX_NP = SPHK_NOALLOC_MAX_PARTICLES;
constexpr uint32_t NA_MAX_CELLS = SPHK_NOALLOC_MAX_CELLS;
// radix sort: digits of up to 10 bits; blocks of 512 threads, a tile of
// 1024 particles a block while that leaves an SM without one, 4096 beyond
// (every tile of the largest input is then resident at once; 8192, one block
// an SM, measured 22.5 us a scatter at 1M particles)
constexpr int NA_BLOCK = 512;
constexpr int NA_WARPS = NA_BLOCK / 32;
constexpr uint32_t NA_BINS = 1024;
constexpr uint32_t NA_SMALL_NP = 148 * 1024;
constexpr int NA_ITEMS_SMALL = 2, NA_ITEMS_LARGE = 8;
constexpr uint32_t NA_MAX_TILES = 256;
static_assert(NA_MAX_NP <= NA_MAX_TILES * NA_BLOCK * NA_ITEMS_LARGE &&
              NA_SMALL_NP <= NA_MAX_TILES * NA_BLOCK * NA_ITEMS_SMALL, "tiles of every input");
// layout in 32-bit words: the second key/value buffer pair, the digit counts
// of every tile (digit-major; scanned along the tiles in place), the digits'
// totals
constexpr size_t NA_OFF_KEYS = 0;
constexpr size_t NA_OFF_VALS = NA_OFF_KEYS + NA_MAX_NP;
constexpr size_t NA_OFF_HIST = NA_OFF_VALS + NA_MAX_NP;
constexpr size_t NA_OFF_TOTALS = NA_OFF_HIST + (size_t)NA_BINS * NA_MAX_TILES;
constexpr size_t NA_WORDS = NA_OFF_TOTALS + NA_BINS;

static __device__ __align__(256) uint32_t g_na_scratch[NA_WORDS];

struct NaGrid {
    uint32_t np, ncells, num[3];
    double origo[3], cellsize[3];
};

// The digit counts of the block's tile into hist[digit * ntiles + tile].
// key(i): the key of particle i.
template <int ITEMS, class Key>
__device__ __forceinline__ void na_tile_hist(uint32_t n, uint32_t shift, uint32_t bins,
                                             uint32_t *hist, uint32_t ntiles, Key key)
{
    __shared__ uint32_t cnt[NA_BINS];
    for (uint32_t k = threadIdx.x; k < bins; k += NA_BLOCK) cnt[k] = 0u;
    __syncthreads();
    const uint32_t base = blockIdx.x * (NA_BLOCK * ITEMS);
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        const uint32_t i = base + k * NA_BLOCK + threadIdx.x;
        if (i < n) atomicAdd(&cnt[(key(i) >> shift) & (bins - 1u)], 1u);
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < bins; k += NA_BLOCK) hist[k * ntiles + blockIdx.x] = cnt[k];
}

// The bucket of every particle (the cell list's rule: grid_cell), the sort's
// first keys, with the digit counts of the first pass; the blocks also clear
// the cells between them (empty: start 0xffffffff, end 0,
// src/device.cu:776-777), those past the tiles nothing else: without them
// 1,000 particles in 524,288 cells took 100 us, 31 with.
template <int ITEMS>
__global__ void __launch_bounds__(NA_BLOCK)
k_na_hash(NaGrid g, const double4 *__restrict__ x, uint32_t *keys, uint32_t bins, uint32_t *hist,
          uint32_t ntiles, uint32_t *cell_start, uint32_t *cell_end)
{
    for (uint32_t c = blockIdx.x * NA_BLOCK + threadIdx.x; c < g.ncells; c += gridDim.x * NA_BLOCK) {
        cell_start[c] = 0xffffffffu;
        cell_end[c] = 0u;
    }
    if (blockIdx.x >= ntiles) return;
    na_tile_hist<ITEMS>(g.np, 0u, bins, hist, ntiles, [&](uint32_t i) {
        const double4 p = x[i];
        uint32_t c;
        const uint32_t k = grid_cell(g, p.x, p.y, p.z, c) ? c : g.ncells;
        keys[i] = k;
        return k;
    });
}

template <int ITEMS>
__global__ void __launch_bounds__(NA_BLOCK)
k_na_hist(const uint32_t *__restrict__ keys, uint32_t n, uint32_t shift, uint32_t bins,
          uint32_t *hist, uint32_t ntiles)
{
    na_tile_hist<ITEMS>(n, shift, bins, hist, ntiles, [&](uint32_t i) { return keys[i]; });
}

// A warp per digit: the exclusive scan of its counts along the tiles, in
// place, and its total.  (The digits' own starts, a scan of at most 1024
// totals, are made by every scatter block for itself.)
__global__ void __launch_bounds__(256)
k_na_scan(uint32_t *hist, uint32_t ntiles, uint32_t bins, uint32_t *totals)
{
    const uint32_t dgt = blockIdx.x * 8u + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
    if (dgt >= bins) return;
    uint32_t *row = hist + (size_t)dgt * ntiles;
    uint32_t run = 0;
    for (uint32_t t0 = 0; t0 < ntiles; t0 += 32u) {
        const uint32_t t = t0 + lane;
        const uint32_t v = t < ntiles ? row[t] : 0u;
        uint32_t inc = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= (unsigned)o) inc += y;
        }
        if (t < ntiles) row[t] = run + inc - v;
        run += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (lane == 0) totals[dgt] = run;
}

// Stable scatter of one tile by the digit at `shift`.  Warp w takes the
// tile's w-th run of 32 ITEMS particles, 32 at a time in order; a particle's
// place is its digit's start, plus the particles with that digit in the
// tiles before (hist), in the earlier runs of the tile, in the earlier steps
// of its run, and in the lower lanes of its step.  vin nullptr: the values
// are the particle indices; label: keys from ncells on are written as
// 0xffffffff (the last pass: sph_get_cells' mark of the out-of-grid bucket).
template <int ITEMS>
__global__ void __launch_bounds__(NA_BLOCK)
k_na_scatter(const uint32_t *__restrict__ kin, const uint32_t *__restrict__ vin, uint32_t *kout,
             uint32_t *vout, uint32_t n, uint32_t shift, uint32_t bins,
             const uint32_t *__restrict__ hist, uint32_t ntiles,
             const uint32_t *__restrict__ totals, uint32_t ncells, int label)
{
    __shared__ uint16_t cnt[NA_WARPS][NA_BINS];   // counts in the tile: at most 4096
    __shared__ uint32_t start[NA_BINS];
    __shared__ uint32_t warp_tot[NA_WARPS];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, w = tid >> 5;
    for (uint32_t k = tid; k < NA_WARPS * NA_BINS / 2; k += NA_BLOCK)
        reinterpret_cast<uint32_t *>(&cnt[0][0])[k] = 0u;
    // the digits' starts: two totals a thread, scanned over the block
    {
        const uint32_t a = 2u * tid < bins ? totals[2u * tid] : 0u;
        const uint32_t b = 2u * tid + 1u < bins ? totals[2u * tid + 1u] : 0u;
        uint32_t inc = a + b;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= (unsigned)o) inc += y;
        }
        if (lane == 31) warp_tot[w] = inc;
        __syncthreads();
        uint32_t off = 0;
        for (uint32_t q = 0; q < w; ++q) off += warp_tot[q];
        const uint32_t at = off + inc - a - b;
        if (2u * tid < bins) start[2u * tid] = at + hist[(size_t)(2u * tid) * ntiles + blockIdx.x];
        if (2u * tid + 1u < bins)
            start[2u * tid + 1u] = at + a + hist[(size_t)(2u * tid + 1u) * ntiles + blockIdx.x];
    }
    const uint32_t run0 = blockIdx.x * (NA_BLOCK * ITEMS) + w * (32u * ITEMS);
    const uint32_t lt = (1u << lane) - 1u;
    uint32_t key[ITEMS];
    uint16_t rank[ITEMS];
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        const uint32_t i = run0 + k * 32u + lane;
        key[k] = i < n ? kin[i] : 0u;
    }
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        const bool ok = run0 + k * 32u + lane < n;
        const uint32_t dgt = ok ? ((key[k] >> shift) & (bins - 1u)) : NA_BINS;
        const uint32_t peers = __match_any_sync(0xffffffffu, dgt);
        const uint32_t before = ok ? cnt[w][dgt] : 0u;
        __syncwarp();
        if (ok && (peers & lt) == 0u) cnt[w][dgt] = (uint16_t)(before + __popc(peers));
        rank[k] = (uint16_t)(before + __popc(peers & lt));
        __syncwarp();
    }
    __syncthreads();
    for (uint32_t dgt = tid; dgt < bins; dgt += NA_BLOCK) {
        uint32_t at = 0;
#pragma unroll
        for (int r = 0; r < NA_WARPS; ++r) {
            const uint32_t c = cnt[r][dgt];
            cnt[r][dgt] = (uint16_t)at;
            at += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        const uint32_t i = run0 + k * 32u + lane;
        if (i >= n) continue;
        const uint32_t dgt = (key[k] >> shift) & (bins - 1u);
        const uint32_t dst = start[dgt] + cnt[w][dgt] + rank[k];
        kout[dst] = (label && key[k] >= ncells) ? 0xffffffffu : key[k];
        vout[dst] = vin ? vin[i] : i;
    }
}

// cell start/end from the sorted ids; the out-of-grid bucket has none
__global__ void k_na_bounds(const uint32_t *__restrict__ ids, uint32_t np, uint32_t ncells,
                            uint32_t *cell_start, uint32_t *cell_end)
{
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= np) return;
    const uint32_t c = ids[k];
    if (c >= ncells) return;
    if (k == 0 || ids[k - 1] != c) cell_start[c] = k;
    if (k + 1 == np || ids[k + 1] != c) cell_end[c] = k + 1;
}

// device address of the scratch array, looked up once per device
static std::mutex g_na_mutex;
static uint32_t *g_na_ptr[64] = {};

static int na_scratch_for_current_device(uint32_t **out)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return SPH_ERR_CUDA;
    std::lock_guard<std::mutex> lock(g_na_mutex);
    if (!g_na_ptr[dev]) {
        void *p = nullptr;
        if (cudaGetSymbolAddress(&p, g_na_scratch) != cudaSuccess || !p) return SPH_ERR_CUDA;
        g_na_ptr[dev] = static_cast<uint32_t *>(p);
    }
    *out = g_na_ptr[dev];
    return SPH_OK;
}

template <int ITEMS>
static void na_sort(const NaGrid &g, const double4 *x, uint32_t *cell_sorted, uint32_t *perm,
                    uint32_t *cell_start, uint32_t *cell_end, uint32_t *scratch, cudaStream_t st)
{
    const uint32_t np = g.np, ntiles = div_up(np, NA_BLOCK * ITEMS);
    // the buckets run to ncells (out of the grid)
    uint32_t bits = 1;
    while (g.ncells >> bits) ++bits;
    const int passes = bits > 10 ? 2 : 1;
    const uint32_t width = passes == 2 ? (bits + 1) / 2 : bits, bins = 1u << width;
    uint32_t *keys[2] = {scratch + NA_OFF_KEYS, cell_sorted};
    uint32_t *vals[2] = {scratch + NA_OFF_VALS, perm};
    uint32_t *hist = scratch + NA_OFF_HIST, *totals = scratch + NA_OFF_TOTALS;
    int cur = passes == 2 ? 1 : 0;   // the last pass writes the outputs
    const uint32_t clearing = std::min(sm_count(), div_up(g.ncells, NA_BLOCK));
    k_na_hash<ITEMS><<<std::max(ntiles, clearing), NA_BLOCK, 0, st>>>(g, x, keys[cur], bins, hist, ntiles, cell_start,
                                                  cell_end);
    for (int p = 0; p < passes; ++p) {
        const uint32_t shift = width * p;
        if (p > 0)
            k_na_hist<ITEMS><<<ntiles, NA_BLOCK, 0, st>>>(keys[cur], np, shift, bins, hist, ntiles);
        k_na_scan<<<div_up(bins, 8), 256, 0, st>>>(hist, ntiles, bins, totals);
        k_na_scatter<ITEMS><<<ntiles, NA_BLOCK, 0, st>>>(
            keys[cur], p > 0 ? vals[cur] : nullptr, keys[cur ^ 1], vals[cur ^ 1], np, shift, bins,
            hist, ntiles, totals, g.ncells, p == passes - 1);
        cur ^= 1;
    }
    k_na_bounds<<<div_up(np, 256), 256, 0, st>>>(cell_sorted, np, g.ncells, cell_start, cell_end);
}

static int na_run(const sph_config *cfg, const double *x_dev, uint32_t *cell_sorted,
                  uint32_t *perm, uint32_t *cell_start, uint32_t *cell_end, cudaStream_t st)
{
    uint32_t *scratch = nullptr;
    const int rc = na_scratch_for_current_device(&scratch);
    if (rc != SPH_OK) return rc;
    NaGrid g{};
    g.np = cfg->np;
    g.ncells = cfg->num[0] * cfg->num[1] * cfg->num[2];
    for (int k = 0; k < 3; ++k) {
        g.num[k] = cfg->num[k];
        g.origo[k] = cfg->origo[k];
        g.cellsize[k] = cfg->L[k] / (double)cfg->num[k];
    }
    const double4 *x = reinterpret_cast<const double4 *>(x_dev);
    if (g.np <= NA_SMALL_NP)
        na_sort<NA_ITEMS_SMALL>(g, x, cell_sorted, perm, cell_start, cell_end, scratch, st);
    else
        na_sort<NA_ITEMS_LARGE>(g, x, cell_sorted, perm, cell_start, cell_end, scratch, st);
    // a launch error of these kernels, without clearing one left by the
    // caller's own work (which is then reported too)
    return cudaPeekAtLastError() == cudaSuccess ? SPH_OK : SPH_ERR_CUDA;
}

}  // namespace sphk

using namespace sphk;

extern "C" int sph_cell_list_noalloc(const sph_config *cfg, const double *x_dev,
                                     uint32_t *cell_sorted, uint32_t *perm, uint32_t *cell_start,
                                     uint32_t *cell_end, void *stream)
{
    if (!cfg || !x_dev || !cell_sorted || !perm || !cell_start || !cell_end) return SPH_ERR_BAD_INPUT;
    const uint64_t ncells = (uint64_t)cfg->num[0] * cfg->num[1] * cfg->num[2];
    if (cfg->np == 0 || ncells == 0) return SPH_ERR_BAD_INPUT;
    if (cfg->np > NA_MAX_NP || ncells > NA_MAX_CELLS) return SPH_ERR_TOO_LARGE;
    // the caller's current device is put back before returning
    int caller_dev = 0;
    if (cudaGetDevice(&caller_dev) != cudaSuccess) return SPH_ERR_CUDA;
    if (cfg->device != caller_dev && cudaSetDevice(cfg->device) != cudaSuccess) return SPH_ERR_CUDA;
    const int rc = na_run(cfg, x_dev, cell_sorted, perm, cell_start, cell_end,
                          static_cast<cudaStream_t>(stream));
    if (cfg->device != caller_dev && cudaSetDevice(caller_dev) != cudaSuccess) return SPH_ERR_CUDA;
    return rc;
}
