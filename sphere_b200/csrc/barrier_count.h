// barrier_count.h -- the arithmetic of a barrier over a whole grid (grid_barrier,
// rebuild.cuh), for the device and for a host check of it.
//
// Every block of every launch that uses a barrier's counter adds 1 to it on
// arriving and waits until the counter reaches the end of its round, the next
// multiple of the grid past BARRIER_START.  The counter has 64 bits and is
// never set back, so a round's end is above every ticket before it: with 32 bits
// a grid of 296 blocks lost count after 4.3e9 arrivals (2.4 million lists),
// because 2^32 is no multiple of it.  It starts 65,536 arrivals below 2^32, so
// that a run's first lists take it past the range of 32 bits.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define BC_HD __host__ __device__ inline
#else
#define BC_HD inline
#endif

namespace sphk {

constexpr uint64_t BARRIER_START = 0xffff0000ull;

// The end of the round of the block that drew `ticket` (the counter before its
// arrival).  before: the end of the block's previous round in this launch, or 0.
// The blocks of a launch meet at the same barriers, so a round ends one grid
// after the one before; the first of a launch is divided out.
BC_HD uint64_t barrier_round_end(uint64_t before, uint64_t ticket, uint32_t grid)
{
    if (before != 0) return before + grid;
    return BARRIER_START + ((ticket - BARRIER_START) / grid + 1) * grid;
}

BC_HD bool barrier_open(uint64_t count, uint64_t end) { return count >= end; }

}  // namespace sphk
