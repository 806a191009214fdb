// pool_share.cuh -- which points of a batch a warp of the point pool takes.
//
// The batch is runs of `stride` points, as many as all warps hold; in each run
// a warp has one group of 32, so its share spans the whole batch and dense
// parts of it do not fall to a few warps.  From run to run the warps change
// places by `turn`: a grid's rows and a stride near a multiple of them would
// else leave each warp one part of the shape.  In every run the places of all
// warps are a rotation of one another, so each point is in one share, however
// a warp evaluates it: the places must not depend on the points.
// Also compiled for the host, where a test walks it.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define CG_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define CG_HOST_DEVICE inline
#endif

namespace cg {

struct PoolShare {
    uint32_t stride, turn;  // multiples of 32
    uint32_t place;         // of the warp's group in the run that `next` is in
    uint32_t next, end;     // the next point of the share to take, and all of them

    // `first`: the warp's place in the first run (a multiple of 32).
    CG_HOST_DEVICE PoolShare(uint64_t first, uint64_t stride_, uint64_t n)
        : stride((uint32_t)stride_), turn((uint32_t)(stride_ * 618 / 1000) & ~31u),
          place((uint32_t)first), next(0), end((uint32_t)((n + stride_ - 1) / stride_) * 32) {}

    CG_HOST_DEVICE uint32_t turned() const {
        return place < stride - turn ? place + turn : place - (stride - turn);
    }
    // The index of point next + j of the share, j < 32; n or more for one that
    // the last run does not have.
    CG_HOST_DEVICE uint64_t index(uint32_t j) const {
        const uint32_t k = next + j, run = k >> 5;
        return (uint64_t)run * stride + (run == next >> 5 ? place : turned()) + (k & 31);
    }
    // `by` points were taken (at most 32).
    CG_HOST_DEVICE void advance(uint32_t by) {
        if ((next + by) >> 5 != next >> 5) place = turned();
        next += by;
    }
};

}  // namespace cg
