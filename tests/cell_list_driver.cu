// Runs the grid barrier and the cell list's kernel by themselves, for
// tests/test_grid_barrier.py: prints one line per check, "ok" or what went wrong.
#include <cstdio>
#include <vector>

#include "cells.cu"

using namespace sphk;

// Rounds of the barrier by the blocks of the grid but those in [0, absent): each
// marks the round, and after the barrier looks for blocks that have not.
__global__ void k_rounds(Dev d, unsigned long long *count, uint32_t *mark, uint32_t *behind, int rounds,
                         uint32_t absent)
{
    if (blockIdx.x < absent) return;
    GridBar bar{count, 0};
    for (int r = 1; r <= rounds; ++r) {
        if (threadIdx.x == 0) __stcg(&mark[blockIdx.x], (uint32_t)r);
        if (!grid_barrier(d, bar)) return;
        for (uint32_t b = threadIdx.x; b < gridDim.x; b += blockDim.x)
            if (__ldcg(&mark[b]) < (uint32_t)r) atomicAdd(behind, 1u);
        if (!grid_barrier(d, bar)) return;
    }
}

static int failures = 0;
static void check(const char *what, bool good)
{
    if (!good) ++failures;
    std::printf("%s: %s\n", what, good ? "ok" : "wrong");
}
static void must(cudaError_t e)
{
    if (e == cudaSuccess) return;
    std::printf("%s\n", cudaGetErrorString(e));
    std::exit(2);
}

template <class T>
static T *filled(const std::vector<T> &v)
{
    T *p = nullptr;
    must(cudaMalloc(&p, v.size() * sizeof(T)));
    must(cudaMemcpy(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice));
    return p;
}
template <class T>
static std::vector<T> fetch(const T *p, size_t n)
{
    std::vector<T> v(n);
    must(cudaMemcpy(v.data(), p, n * sizeof(T), cudaMemcpyDeviceToHost));
    return v;
}

int main()
{
    Dev d{};
    d.status = filled(std::vector<uint32_t>(1, 0u));
    std::vector<unsigned long long> start(1, BARRIER_START);
    uint32_t *mark = filled(std::vector<uint32_t>(1024, 0u)), *behind = filled(std::vector<uint32_t>(1, 0u));
    for (unsigned grid : {1u, 7u, 148u, 296u, 391u, 592u}) {
        unsigned long long *count = filled(start);
        must(cudaMemset(mark, 0, 4096));
        for (int launch = 0; launch < 4; ++launch) {
            launch_together(k_rounds, grid, 64, nullptr, d, count, mark, behind, 40, 0u);
            must(cudaMemset(mark, 0, 4096));
        }
        must(cudaDeviceSynchronize());
        check("arrivals", fetch(count, 1)[0] == BARRIER_START + 4ull * 80ull * grid);
    }
    check("no block ahead", fetch(behind, 1)[0] == 0u && fetch(d.status, 1)[0] == 0u);

    // a grid that the device does not hold at once is refused, and said to be
    const cudaError_t refused = launch_together(k_rounds, 1u << 20, 64, nullptr, d, filled(start), mark, behind, 1, 0u);
    check("too large", refused == cudaErrorCooperativeLaunchTooLarge && cudaGetLastError() == refused);
    const uint32_t most = resident_blocks<k_rebuild, REBUILD_BLOCK>();
    check("resident", most >= sm_count() * REBUILD_BLOCKS_PER_SM && most <= CROWDED_AT);

    // a cell list of 3,000 particles in 10 x 10 x 10 cells, in storage order
    // reversed against their indices
    const uint32_t np = 3000, nc = 1000;
    Params P{};
    P.np = np;
    P.ncells = nc;
    std::vector<uint32_t> uid(np), cell(np);
    std::vector<double4> x(np);
    for (int k = 0; k < 3; ++k) {
        P.num[k] = 10;
        P.L[k] = 1.0;
        P.cellsize[k] = 0.1;
    }
    for (uint32_t s = 0; s < np; ++s) {
        uid[s] = np - 1u - s;
        x[s] = make_double4((s * 37u % 1000u) * 1e-3, (s * 101u % 1000u) * 1e-3, (s * 7u % 1000u) * 1e-3, 1e-3);
    }
    std::vector<uint32_t> none(np, 0u), cells(nc + 2, 0u);
    d.np_all = np;
    d.ncells_all = nc;
    d.ninst = 1;
    d.prm = filled(std::vector<Params>(1, P));
    d.uid = filled(uid);
    d.sidx = filled(uid);
    d.cell = filled(none);
    d.cellorder = filled(none);
    d.pos = filled(none);
    d.xr[0] = filled(x);
    d.xs[0] = filled(std::vector<float4>(np));
    d.xs[1] = filled(std::vector<float4>(np));
    d.cell_start = filled(cells);
    d.cell_fill = filled(cells);
    d.dirty = filled(cells);
    d.scan_tiles = filled(std::vector<uint32_t>(SCAN_TILES, 0u));
    d.alias_any = filled(std::vector<uint32_t>(1, 0u));
    d.rebuild = filled(std::vector<uint32_t>(2, 0u));
    d.vs = filled(std::vector<Verlet>(1));
    auto ordered = [&]() {
        const auto o = fetch(d.cellorder, np), c = fetch(d.cell, np), b = fetch(d.cell_start, nc + 2);
        bool good = b[nc + 1] == np;
        for (uint32_t k = 0; k < np; ++k) {
            good = good && o[k] < np && b[c[o[k]]] <= k && k < b[c[o[k]] + 1];
            if (k > 0) good = good && (c[o[k - 1]] < c[o[k]] ||
                                       (c[o[k - 1]] == c[o[k]] && uid[o[k - 1]] < uid[o[k]]));
        }
        return good;
    };
    launch_epoch_reset(d, nullptr);
    launch_cell_init(d, np, 0, nullptr);
    launch_rebuild(d, np, nc, 0, nullptr);
    must(cudaDeviceSynchronize());
    check("list", ordered() && fetch(d.rebuild, 1)[0] == 0u);

    // a block that never comes: the others give up and say so
    unsigned long long *count = filled(start);
    launch_together(k_rounds, 16, 64, nullptr, d, count, mark, behind, 1, 1u);
    must(cudaDeviceSynchronize());
    check("gives up", fetch(d.status, 1)[0] == ST_TIMEOUT);

    // as a list that was given up after its count leaves it: nothing is made
    // until the upload's reset, then the list is right again
    must(cudaMemset(d.cell_fill, 1, (nc + 1) * 4));
    const Verlet before = fetch(d.vs, 1)[0];
    const auto order = fetch(d.cellorder, np);
    must(cudaMemset(d.rebuild, 1, 4));
    for (int k = 0; k < 3; ++k) launch_rebuild(d, np, nc, 0, nullptr);
    must(cudaDeviceSynchronize());
    const auto fill = fetch(d.cell_fill, nc + 1);
    bool same = fetch(d.vs, 1)[0].rebuilds == before.rebuilds && fetch(d.cellorder, np) == order;
    for (uint32_t f : fill) same = same && f == 0x01010101u;
    check("nothing is made", same);
    must(cudaMemset(d.status, 0, 4));
    must(cudaMemset(d.cell_fill, 0, (nc + 1) * 4));
    must(cudaMemset(d.cellorder, 0, np * 4));
    launch_epoch_reset(d, nullptr);
    launch_rebuild(d, np, nc, 0, nullptr);
    must(cudaDeviceSynchronize());
    check("list after a reset", ordered() && fetch(d.status, 1)[0] == 0u);
    return failures;
}
