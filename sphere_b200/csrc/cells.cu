// cells.cu -- the cell list of libsphk: hash, sort, cell start/end, relayout.
//
// The reference hashes every particle to a cell (calcParticleCellID,
// src/sorting.cuh:24-43), sorts (cellID, index) pairs with thrust's stable
// radix sort (src/device.cu:763-765) and marks cell ranges
// (reorderArrays, src/sorting.cuh:49-121).  The sorted order is "by cell, then
// by particle index".  Here the same order comes from a counting sort with
// the cell id as the radix, in one launch (rebuild.cuh).  The cell of every
// particle is computed by the step kernel from its new position; a step whose
// search sweeps has the list made again first, any other finds the launch's
// flag clear and leaves at once.
//
// Particles are stored in cell order (relayout), so neighbours are close in
// memory; k_relayout_* re-establish that order on demand.
#include <algorithm>

#include "rebuild.cuh"

namespace sphk {

constexpr int CELL_BLOCK = 256;

__global__ void k_cell_init(Dev d, int A)
{
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= d.np_all) return;
    const Params &P = prm_of(d, s);
    const double4 x = d.xr[A][s];
    uint32_t c;
    if (!grid_cell(P, x.x, x.y, x.z, c)) {
        atomicOr(d.status, ST_OUT_OF_GRID);
        c = d.ncells_all;
    } else {
        c += P.cell_base;
    }
    d.cell[s] = c;
}

// The cell list in one launch, a resident grid whose blocks wait for one
// another between the passes (a cooperative launch: they are on the device
// together).  As seven kernels behind a conditional graph node the node alone
// cost every step of a graph 6 to 7 us, taken or not.
constexpr int REBUILD_BLOCK = 512, REBUILD_BLOCKS_PER_SM = 2;
__global__ void __launch_bounds__(REBUILD_BLOCK, REBUILD_BLOCKS_PER_SM)
k_rebuild(const __grid_constant__ Dev d, int A)
{
    if (*(volatile const uint32_t *)&d.rebuild[REBUILD_NOW] == 0u || lists_given_up(d)) return;
    GridBar bar{&d.vs->bar_rebuild, 0};
    rebuild_grid<REBUILD_BLOCK>(d, A, bar);
}

void launch_cell_init(const Dev &d, uint32_t np, int a, cudaStream_t st)
{
    k_cell_init<<<div_up(np, CELL_BLOCK), CELL_BLOCK, 0, st>>>(d, a);
}

// A Verlet epoch from scratch after a state was put back: the cell list is
// rebuilt and every particle sweeps in the next step.
__global__ void k_epoch_reset(Dev d)
{
    Verlet V{};
    V.step = 1;
    V.all_rebuild = 1;
    *d.vs = V;
    d.rebuild[REBUILD_NOW] = 1u;
    d.rebuild[REBUILD_NEXT] = 0u;
}

void launch_epoch_reset(const Dev &d, cudaStream_t st)
{
    k_epoch_reset<<<1, 1, 0, st>>>(d);
}

cudaError_t launch_rebuild(const Dev &d, uint32_t np, uint32_t ncells, int a, cudaStream_t st)
{
    const uint32_t most = std::min(resident_blocks<k_rebuild, REBUILD_BLOCK>(), sm_count() * REBUILD_BLOCKS_PER_SM);
    const uint32_t grid = std::min(most, div_up(std::max<uint64_t>(np, (uint64_t)ncells + 1), REBUILD_BLOCK));
    return launch_together(k_rebuild, grid, REBUILD_BLOCK, st, d, a);
}

// ---- relayout: storage order := current cell order -----------------------
// inv[old storage index] = new storage index
__global__ void k_relayout_inv(Dev d, uint32_t *inv)
{
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= d.np_all) return;
    inv[d.cellorder[k]] = k;
}

template <typename T>
__global__ void k_gather(const T *__restrict__ src, T *__restrict__ dst, const uint32_t *order,
                         uint32_t n)
{
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) dst[k] = src[order[k]];
}

// contact rows: move the row and translate partner indices
// Tiled slot entries into the new storage order: entry e of the new tiles
// takes the old particle's entry, partners renamed through `inv` (empty
// slots keep whatever they held: an empty slot's entry is never read).  After a
// list that was given up `inv` may have gaps: a partner stays a particle.
__device__ __forceinline__ bool tile_entry(uint64_t e, uint32_t np, uint32_t &s, uint32_t &i)
{
    s = (uint32_t)((e / (32ull * NC)) * 32ull + (e & 31ull));
    i = (uint32_t)((e >> 5) % NC);
    return s < np;
}

__global__ void k_gather_rows(const uint32_t *src, uint32_t *dst, const uint32_t *order,
                              const uint32_t *inv, uint32_t np)
{
    const uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= tiled_size(np, NC)) return;
    uint32_t s, i;
    if (!tile_entry(e, np, s, i)) return;
    const uint32_t v = src[tile_at(order[s], i, NC)];
    dst[e] = (v < np) ? min(inv[v], np - 1u) : np;
}

__global__ void k_gather_dt(const P3 *src, P3 *dst, const uint32_t *order, uint32_t np)
{
    const uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= tiled_size(np, NC)) return;
    uint32_t s, i;
    if (!tile_entry(e, np, s, i)) return;
    dst[e] = src[tile_at(order[s], i, NC)];
}

__global__ void k_relayout_finish(Dev d, int A)
{
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= d.np_all) return;
    d.cellorder[k] = k;
    d.pos[k] = k;
    d.sidx[d.uid[k]] = k;
    if (k == 0) {
        // storage indices changed: every Verlet list is stale
        d.vs->all_rebuild = 1u;
        d.vs->moved = 0.0f;
    }
    const double4 x = d.xr[A][k];
    d.xs[A][k] = make_float4((float)x.x, (float)x.y, (float)x.z, (float)x.w);
}

template <typename T>
static void gather_back(T *arr, void *scratch, const uint32_t *order, uint32_t n, cudaStream_t st)
{
    T *tmp = static_cast<T *>(scratch);
    k_gather<T><<<div_up(n, CELL_BLOCK), CELL_BLOCK, 0, st>>>(arr, tmp, order, n);
    cudaMemcpyAsync(arr, tmp, sizeof(T) * (size_t)n, cudaMemcpyDeviceToDevice, st);
}

// Permute every per-particle array into the order of d.cellorder (which the
// rebuild kernels must have brought up to date).  `scratch` holds at least
// tiled_size(np, NC) * sizeof(P3) bytes plus np * sizeof(uint32_t) for the
// inverse.
void relayout(const Dev &d, uint32_t np, int a, void *scratch, cudaStream_t st)
{
    uint32_t *inv = reinterpret_cast<uint32_t *>(static_cast<char *>(scratch) +
                                                 tiled_size(np, NC) * sizeof(P3));
    const uint32_t *order = d.cellorder;
    k_relayout_inv<<<div_up(np, CELL_BLOCK), CELL_BLOCK, 0, st>>>(d, inv);
    gather_back(d.xr[a], scratch, order, np, st);
    gather_back(d.vel[a], scratch, order, np, st);
    gather_back(d.angvel[a], scratch, order, np, st);
    gather_back(d.vel0, scratch, order, np, st);
    gather_back(d.angvel0, scratch, order, np, st);
    gather_back(d.angpos, scratch, order, np, st);
    gather_back(d.xysum, scratch, order, np, st);
    gather_back(d.esv, scratch, order, np, st);
    gather_back(d.force, scratch, order, np, st);
    gather_back(d.torque, scratch, order, np, st);
    gather_back(d.acc, scratch, order, np, st);
    gather_back(d.angacc, scratch, order, np, st);
    gather_back(d.edp, scratch, order, np, st);
    gather_back(d.uid, scratch, order, np, st);
    gather_back(d.cell, scratch, order, np, st);
    gather_back(d.fixed, scratch, order, np, st);
    gather_back(d.cmask, scratch, order, np, st);
    gather_back(d.dmc, scratch, order, np, st);
    gather_back(d.wtouch, scratch, order, np, st);
    if (d.inst) gather_back(d.inst, scratch, order, np, st);
    const size_t ntile = tiled_size(np, NC);
    const unsigned int rows = div_up(ntile, CELL_BLOCK);
    {
        uint32_t *tmp = static_cast<uint32_t *>(scratch);
        k_gather_rows<<<rows, CELL_BLOCK, 0, st>>>(d.contacts, tmp, order, inv, np);
        cudaMemcpyAsync(d.contacts, tmp, sizeof(uint32_t) * ntile, cudaMemcpyDeviceToDevice, st);
    }
    {
        P3 *tmp = static_cast<P3 *>(scratch);
        k_gather_dt<<<rows, CELL_BLOCK, 0, st>>>(d.delta_t, tmp, order, np);
        cudaMemcpyAsync(d.delta_t, tmp, sizeof(P3) * ntile, cudaMemcpyDeviceToDevice, st);
    }
    k_relayout_finish<<<div_up(np, CELL_BLOCK), CELL_BLOCK, 0, st>>>(d, a);
}

}  // namespace sphk
