// C entry points of barrier_count.h for tests/test_grid_barrier.py.
#include "barrier_count.h"

extern "C" {

uint64_t barrier_start_c() { return sphk::BARRIER_START; }
uint64_t barrier_round_end_c(uint64_t before, uint64_t ticket, uint32_t grid)
{
    return sphk::barrier_round_end(before, ticket, grid);
}
int barrier_open_c(uint64_t count, uint64_t end) { return sphk::barrier_open(count, end) ? 1 : 0; }

}
