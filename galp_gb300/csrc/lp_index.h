// lp_index.h -- index and counter arithmetic at the ends of its range, shared by the kernels and
// host-side checks.
#pragma once

#include <cstdint>

#if defined(__CUDACC__)
#define GALP_INDEX __host__ __device__ __forceinline__
#else
#define GALP_INDEX inline
#endif

namespace galp {

// Walk of a list of n < 2^31 entries by blocks that take `width` entries per round.  Unsigned: the
// round ahead of the last one begins up to two strides (less than 2^30 each) past the list's end,
// where a signed index of a list of nearly 2^31 entries would be negative and pass for one inside.
struct ListWalk {
    uint32_t base, stride, n;
    GALP_INDEX ListWalk(int block, int blocks, int width, int n_)
        : base((uint32_t)block * (uint32_t)width), stride((uint32_t)blocks * (uint32_t)width), n((uint32_t)n_)
    {
    }
    GALP_INDEX bool more() const { return base < n; }  // this round has entries (block-uniform)
    GALP_INDEX void next() { base += stride; }
    // entry `at` of the round `rounds` ahead of this one (0 or 1), -1 past the end of the list
    GALP_INDEX int entry(int rounds, int at) const
    {
        const uint32_t i = base + (uint32_t)rounds * stride + (uint32_t)at;
        return i < n ? (int)i : -1;
    }
};

// Whether a barrier of `blocks` blocks, the k-th that a run comes to, still waits: `arrived` counts
// every arrival of the run so far.  Both wrap around (152 blocks pass 2^32 arrivals after 14 M
// iterations), and lie within one barrier of each other: the sign of their difference decides.
GALP_INDEX bool barrier_waits(uint32_t arrived, uint32_t k, uint32_t blocks)
{
    return (int32_t)(arrived - k * blocks) < 0;
}

}  // namespace galp
