// rebuild.cuh -- the cell list as a device function of a whole grid, called by
// the kernel that only makes the list (cells.cu) and by the small scenes' step
// (k_small, step.cu):
//   count      histogram of cell ids                  (atomics in L2)
//   scan       exclusive scan of the histogram        (two passes)
//   scatter    each particle claims a position in its cell's range
//   rank       each particle's place is the number of its cell's members with
//              a smaller index: the list, its inverse and the float position
//              copy in list order; and the stamps of the cells whose particles'
//              lists a move upset
// The blocks wait for one another between the passes, so the kernel is
// launched cooperatively.  Arrays that a pass changes after another read them
// in the same launch are read past L1 (__ldcg).
#ifndef SPHK_REBUILD_CUH_
#define SPHK_REBUILD_CUH_

#include "barrier_count.h"
#include "sphk_internal.cuh"

namespace sphk {

// A barrier's counter and the end of this block's last round (thread 0's).
struct GridBar {
    unsigned long long *count;
    uint64_t end;
};

// Waits until every block of the grid is here; false when that did not happen
// within BULK_WAIT_NS (ST_TIMEOUT: the caller leaves, and no list is made before
// an upload has cleared the status, see lists_given_up).  bar: a counter that only this kernel's
// launches use, always with the same grid.
__device__ __forceinline__ bool grid_barrier(const Dev &d, GridBar &bar)
{
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        bar.end = barrier_round_end(bar.end, atomicAdd(bar.count, 1ull), gridDim.x);
        const uint64_t t0 = global_ns();
        ok = 1;
        while (!barrier_open(*(volatile const unsigned long long *)bar.count, bar.end)) {
            if (global_ns() - t0 > BULK_WAIT_NS) {
                atomicOr(d.status, ST_TIMEOUT);
                ok = 0;
                break;
            }
            __nanosleep(64);   // leaves the counter to those still arriving
        }
        __threadfence();
    }
    __syncthreads();
    return ok != 0;
}

// Whether a barrier has timed out since the upload.  The counters and cell_fill
// are then as the blocks that left found them: a list made from them would be
// written past its arrays.  The kernels that make lists leave at once until an
// upload has cleared all three.  (A half-made list is safe to read: every entry of
// every array is in range at any time.)
__device__ __forceinline__ bool lists_given_up(const Dev &d)
{
    return (*(volatile const uint32_t *)d.status & ST_TIMEOUT) != 0u;
}

// Every cell of the neighbourhood of the cells that a move left and entered
// (27 cells each, or with Params::wide 125) is stamped with this step's
// number; particles in stamped cells sweep their stencil again, or, around a
// particle that is back from outside a periodic boundary, look at their lists.
// Periodic axes wrap as in findDistMod.
//
// A thread a cell: one a move took 20 us for the one or two moves of a step, 125
// stores after one another.
__device__ __forceinline__ void stamp_moves(const Dev &d, uint32_t first, uint32_t stride)
{
    Verlet &V = *d.vs;
    const uint32_t n = min(__ldcg(&V.nmovers), MOVER_CAP), step = __ldcg(&V.step);
    for (uint32_t w = first; w < 2u * 125u * n; w += stride) {
        const uint32_t e = w / 125u;
        const uint2 mv = __ldcg(&d.movers[e >> 1]);
        const uint32_t cg = (e & 1u) ? mv.y : mv.x;
        if (cg >= d.ncells_all) continue;
        uint32_t *const stamps = mv.x == LOOK ? d.look : d.dirty;
        // the instance owning global cell cg (batched contexts)
        uint32_t inst = 0;
        if (d.inst) {
            uint32_t lo = 0, hi = d.ninst;
            while (hi - lo > 1) {
                const uint32_t mid = (lo + hi) >> 1;
                if (d.inst_cell_base[mid] <= cg) lo = mid; else hi = mid;
            }
            inst = lo;
        }
        const Params &P = d.prm[inst];
        const uint32_t c = cg - P.cell_base, o = w % 125u;
        const int32_t nx = (int32_t)P.num[0], ny = (int32_t)P.num[1], nz = (int32_t)P.num[2];
        const int32_t ox = (int32_t)(o % 5u) - 2, oy = (int32_t)(o / 5u % 5u) - 2, oz = (int32_t)(o / 25u) - 2;
        const int32_t R = P.wide ? 2 : 1;
        if (max(max(abs(ox), abs(oy)), abs(oz)) > R) continue;
        if (o == 62u) {   // the cell itself
            uint32_t *const when = mv.x == LOOK ? &V.look_step : &V.dirty_step;
            if (__ldcg(when) != step) *when = step;
        }
        int32_t x = (int32_t)(c % (uint32_t)nx) + ox, y = (int32_t)(c / (uint32_t)nx % (uint32_t)ny) + oy;
        const int32_t z = (int32_t)(c / (uint32_t)(nx * ny)) + oz;
        if (z < 0 || z >= nz) continue;
        if (y < 0 || y >= ny) {
            if (P.periodic != 1) continue;
            y = (y + ny) % ny;
        }
        if (x < 0 || x >= nx) {
            if (P.periodic != 1 && P.periodic != 2) continue;
            x = (x + nx) % nx;
        }
        stamps[P.cell_base + (uint32_t)x + (uint32_t)y * (uint32_t)nx + (uint32_t)(nx * ny) * (uint32_t)z] = step;
    }
}

// The exclusive scan over the block's threads of one value each, and their sum.
template <int BLOCK>
__device__ __forceinline__ uint32_t block_scan(uint32_t v, uint32_t &total)
{
    __shared__ uint32_t warp_tot[BLOCK / 32];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= (unsigned)o) inc += y;
    }
    if (lane == 31) warp_tot[warp] = inc;
    __syncthreads();
    uint32_t off = 0, sum = 0;
#pragma unroll
    for (int w = 0; w < BLOCK / 32; ++w) {
        const uint32_t t = warp_tot[w];
        if ((unsigned)w < warp) off += t;
        sum += t;
    }
    __syncthreads();
    total = sum;
    return off + inc - v;
}

// A cell with more members than this is put in order by one block, which looks
// for them among all particles in index order; below, every member counts the
// smaller indices of its cell for itself.  The first takes 2.4 us for each 512
// particles of the context, whatever the members, the second 0.5 us a member of
// the cell for a million particles, so they meet at about 10,000 members: a
// million particles in 16 cells 28.5 ms by counting, 4.6 by blocks, all in one
// cell 4.8.
constexpr uint32_t CROWD = 1u << 14;
// the crowded cells (at most 2^27 / CROWD), past the part of scan_tiles that the
// blocks' totals take
constexpr uint32_t CROWDED_AT = SCAN_TILES / 4, CROWDED_CAP = SCAN_TILES - CROWDED_AT;
static_assert(CROWDED_CAP >= (1u << 27) / CROWD, "every crowded cell has a place");

// The cell list of the positions in buffer A, by all blocks of the grid; false
// after a timeout.  BLOCK: the threads of a block.
//
// What bounds it: the barriers and L2 latency (17 us at 50,000 particles, 47 at a
// million).  One thread used to sort each cell's members by insertion, one load
// after another: 189 us a list where cells of four radii hold 12 grains each, and
// past the barrier's limit of 1 s at a few thousand.
template <int BLOCK>
__device__ __noinline__ bool rebuild_grid(const Dev &d, int A, GridBar &bar)
{
    const uint32_t first = blockIdx.x * BLOCK + threadIdx.x, stride = gridDim.x * BLOCK;
    const uint32_t np = d.np_all, n = d.ncells_all + 1u;   // buckets, the last for the outside
    Verlet &V = *d.vs;
    if (first == 0) {
        *d.alias_any = 0u;
        V.crowded = 0u;
    }
    for (uint32_t s = first; s < np; s += stride) atomicAdd(&d.cell_fill[d.cell[s]], 1u);
    if (!grid_barrier(d, bar)) return false;
    // the block's run of buckets: its sum, then after every block's the scan
    const uint32_t per = (n + gridDim.x - 1u) / gridDim.x;
    const uint32_t lo = min(n, blockIdx.x * per), hi = min(n, lo + per);
    uint32_t sum = 0, total = 0;
    for (uint32_t c = lo + threadIdx.x; c < hi; c += BLOCK) sum += __ldcg(&d.cell_fill[c]);
    block_scan<BLOCK>(sum, total);
    if (threadIdx.x == 0) d.scan_tiles[blockIdx.x] = total;
    if (!grid_barrier(d, bar)) return false;
    uint32_t run = 0;
    for (uint32_t b = threadIdx.x; b < blockIdx.x; b += BLOCK) run += __ldcg(&d.scan_tiles[b]);
    block_scan<BLOCK>(run, total);
    run = total;
    for (uint32_t c0 = lo; c0 < hi; c0 += BLOCK) {
        const uint32_t c = c0 + threadIdx.x;
        const uint32_t v = c < hi ? __ldcg(&d.cell_fill[c]) : 0u;
        const uint32_t at = run + block_scan<BLOCK>(v, total);
        if (c < hi) d.cell_start[c] = at;
        if (v > CROWD) {
            const uint32_t e = atomicAdd(&V.crowded, 1u);
            if (e < CROWDED_CAP) d.scan_tiles[CROWDED_AT + e] = c;
        }
        run += total;
    }
    if (first == 0) d.cell_start[n] = np;
    if (!grid_barrier(d, bar)) return false;
    // each particle takes a place of its cell's range; counters return to zero.
    // The members lie in the other buffer's float positions, which nothing
    // reads before this step's end writes them.
    uint32_t *const members = reinterpret_cast<uint32_t *>(d.xs[A ^ 1]);
    for (uint32_t s = first; s < np; s += stride) {
        const uint32_t c = d.cell[s];
        const uint32_t k = atomicSub(&d.cell_fill[c], 1u) - 1u;
        members[d.cell_start[c] + k] = s;
    }
    if (!grid_barrier(d, bar)) return false;
    // particle s at place k of the list
    auto place = [&](uint32_t s, uint32_t k) {
        const Params &P = prm_of(d, s);
        d.cellorder[k] = s;
        d.pos[s] = k;
        const double4 x = d.xr[A][s];
        d.xs[A][k] = make_float4((float)x.x, (float)x.y, (float)x.z, (float)x.w);
        // a particle whose floored coordinates leave the grid sits outside
        // its cell's box (saturated or aliased cell id): contact search must
        // then not prune cells by geometry
        if (cell_outside(P, x.x, x.y, x.z)) *d.alias_any = 1u;
    };
    for (uint32_t k = first; k < np; k += stride) {
        const uint32_t s = members[k], c = d.cell[s], key = d.uid[s];
        const uint32_t beg = d.cell_start[c], end = d.cell_start[c + 1];
        if (end - beg > CROWD) continue;
        uint32_t at = beg;
#pragma unroll 4
        for (uint32_t j = beg; j < end; ++j) at += d.uid[members[j]] < key ? 1u : 0u;
        place(s, at);
    }
    const uint32_t crowded = min(__ldcg(&V.crowded), CROWDED_CAP);
    for (uint32_t e = blockIdx.x; e < crowded; e += gridDim.x) {
        const uint32_t c = __ldcg(&d.scan_tiles[CROWDED_AT + e]);
        uint32_t at = d.cell_start[c];
        for (uint32_t u0 = 0; u0 < np; u0 += BLOCK) {
            const uint32_t u = u0 + threadIdx.x;
            const uint32_t s = u < np ? d.sidx[u] : 0u;
            const bool in = u < np && d.cell[s] == c;
            const uint32_t k = at + block_scan<BLOCK>(in ? 1u : 0u, total);
            if (in) place(s, k);
            at += total;
        }
    }
    stamp_moves(d, first, stride);
    if (first == 0) {
        V.rebuilds += 1u;
        if (__ldcg(&V.movers_overflow)) {
            V.all_rebuild = 1u;
            V.moved = 0.0f;
        }
    }
    if (!grid_barrier(d, bar)) return false;
    if (first == 0) {
        // the flag and the movers, consumed
        d.rebuild[REBUILD_NOW] = 0u;
        d.vs->nmovers = 0u;
        d.vs->movers_overflow = 0u;
    }
    return true;
}

// A launch whose blocks are all on the device together.
template <class T>
struct SameType {
    using type = T;
};
template <class... Args>
inline cudaError_t launch_together(void (*kernel)(Args...), unsigned grid, unsigned block, cudaStream_t st,
                                   typename SameType<Args>::type... args)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.stream = st;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeCooperative;
    attr.val.cooperative = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

}  // namespace sphk

#endif
