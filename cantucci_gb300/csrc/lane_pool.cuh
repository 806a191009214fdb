// lane_pool.cuh -- estimates one loop step at a time, so that the lanes of a
// warp need not end together.
//
// A warp that gives each lane one point runs until its slowest point is done.
// Points without spatial order (uniform in the cube: 4 steps on average, 15
// inside the bulb) then keep about a quarter of the lanes busy.  warp_pool
// instead walks a warp through a range of points: a lane whose loop has
// ended waits until some lanes have, and those write their results and take
// the range's next points together.
#pragma once

#include <cstdint>

#include "common.cuh"
#include "de.cuh"
#include "point_io.cuh"

namespace cg {

// The loop of mode M's estimator for one point: the same operations, in the
// same order, as eval<M>.
template <int M>
struct DeLoop {
    float px, py, pz;  // the point (polar forms: R^T p)
    float x, y, z, dr;
    float r;           // |z|; MODE_P8: |z|^2; MODE_SPHERE: the distance
    uint32_t it;
    float limit;       // MODE_P8
    bool inside;       // MODE_P8

    __device__ __forceinline__ void start(const ShapeDev& s, float ax, float ay, float az) {
        if (M == MODE_POLAR) rotate_point<false>(s, ax, ay, az, px, py, pz);
        else if (M == MODE_POLAR_FAST) rotate_point<true>(s, ax, ay, az, px, py, pz);
        else px = ax, py = ay, pz = az;
        x = px;
        y = py;
        z = pz;
        dr = 1.0f;
        r = 0.0f;
        it = 0;
        if (M == MODE_P8) limit = p8_limit(s.p8_m2_max, py, pz);
    }
    // A loop whose point, iterate and count were set by hand.
    __device__ __forceinline__ void resume(const ShapeDev& s) {
        if (M == MODE_P8) limit = p8_limit(s.p8_m2_max, py, pz);
    }
    // One step; false when the loop has ended (max_iters >= 1).
    __device__ __forceinline__ bool step(const ShapeDev& s) {
        if (M == MODE_SPHERE) {
            r = sphere_de(s, px, py, pz);
            return false;
        }
        const bool last = ++it >= s.max_iters;
        if (M == MODE_P8) return p8_step(limit, px, py, pz, last, x, y, z, dr, r, inside);
        if (M == MODE_INT) return int_step(s, px, py, pz, last, x, y, z, dr, r);
        if (M == MODE_POLAR) return polar_step(s, px, py, pz, last, x, y, z, dr, r);
        if (M == MODE_P8_FAST) return p8_fast_step(s.bailout, px, py, pz, x, y, z, dr, r) && !last;
        if (M == MODE_INT_POLY)
            return int_poly_step(s.power, (float)s.power, s.bailout, px, py, pz, x, y, z, dr, r) &&
                   !last;
        return polar_step_fast(s, px, py, pz, x, y, z, dr, r) && !last;
    }
    __device__ __forceinline__ float value(const ShapeDev& s) const {
        if (M == MODE_SPHERE) return r;
        if (M == MODE_P8)
            return p8_value(s.max_iters, s.bailout, limit, px, py, pz, r, dr, inside);
        if (M == MODE_INT || M == MODE_POLAR) return de_value(r, dr);
        if (M == MODE_INT_POLY) return x86_nan(0.5f * logf(r) * r / dr);
        return x86_nan(__fdividef(0.5f * __logf(r) * r, dr));
    }
};

// Whether 32 consecutive points lie one beside the other (a grid's rows, a
// scan line's hits): their loops then end at about the same step.  Measured as
// the mean distance (L1) from a point to the next against the bulb's size of
// about 2; uniform points in the cube have 2.4.  Call from all 32 lanes, each
// with its point.
__device__ __forceinline__ bool points_side_by_side(float x, float y, float z) {
    float d = fabsf(x - __shfl_down_sync(0xFFFFFFFFu, x, 1)) +
              fabsf(y - __shfl_down_sync(0xFFFFFFFFu, y, 1)) +
              fabsf(z - __shfl_down_sync(0xFFFFFFFFu, z, 1));
    for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xFFFFFFFFu, d, o);
    return d < 32.0f * 0.25f;
}

__device__ __forceinline__ bool points_side_by_side(const float* __restrict__ pts,
                                                    const WarpWalk& w, uint64_t n) {
    const uint64_t i = min(w.first + (threadIdx.x & 31), n - 1);
    return points_side_by_side(pts[3 * i], pts[3 * i + 1], pts[3 * i + 2]);
}

// Runs `task` over this warp's points, groups of 32 consecutive ones from
// w.first (< n) on, w.stride apart (each warp's share then spans the whole
// batch, so that dense parts of it do not fall to a few warps).  Call from all
// 32 lanes.
//   task.start(i)   begin point i            task.step()  one step, false at the end
//   task.finish(i)  write point i's result   task.steps() the steps of the point
// `wait`: the lanes that wait before results are written and new points taken
// together; 32 keeps the lanes in step, group by group.  Lanes in step also
// agree on the branches inside the trigonometric functions, so where steps are
// alike the pool costs 15 to 25 %.  Points side by side are the caller's to
// tell; points that run most of `max_steps` (on the surface) show here: once a
// warp's worth of points has averaged 0.45 of it, the lanes stay in step.
template <class Task>
__device__ __forceinline__ void warp_pool(const WarpWalk& w, uint64_t n, int wait,
                                          uint32_t max_steps, Task& task) {
    const uint32_t below = (1u << (threadIdx.x & 31)) - 1u;
    // Point k of the warp's share is first + (k / 32) stride + k % 32.
    const uint64_t groups = (n - w.first + w.stride - 1) / w.stride;
    const uint64_t last = n - (w.first + (groups - 1) * w.stride);
    const uint64_t count = (groups - 1) * 32 + (last < 32 ? last : 32);
    uint64_t next = 0, mine = 0;
    uint32_t ended = 0, steps = 0;
    bool have = false, busy = false;
    for (;;) {
        const uint32_t idle = __ballot_sync(0xFFFFFFFFu, !busy);
        const uint32_t done = __ballot_sync(0xFFFFFFFFu, have && !busy);
        // Enough lanes wait for new points or, when there are none, with results.
        const uint32_t waiting = next < count ? idle : done;
        if (__popc(waiting) >= wait || idle == 0xFFFFFFFFu) {
            if (have && !busy) task.finish(mine);
            if (wait < 32) {
                ended += __popc(done);
                steps += __reduce_add_sync(0xFFFFFFFFu, have && !busy ? task.steps() : 0u);
                if (ended >= 32 && (float)steps > 0.45f * (float)ended * (float)max_steps) wait = 32;
            }
            if (!busy) {
                const uint64_t k = next + __popc(idle & below);
                have = busy = k < count;
                mine = w.first + (k >> 5) * w.stride + (k & 31);
                if (have) task.start(mine);
            }
            next += __popc(idle);
            if (!__any_sync(0xFFFFFFFFu, busy)) break;
        }
        if (busy) busy = task.step();
    }
}

// The blocks (of 128 threads) of a pool kernel over n points: four points to a
// lane, and for larger batches up to twice the blocks that fit on the GPU at
// once (blocks then end at different times and the SMs stay full: 209 against
// 253 us for 3M points of a grid).  0 when four points to a lane do not fill
// the GPU, where a pool gains less than the missing warps cost.
template <class Kernel>
unsigned pool_grid(Kernel kernel, uint64_t n) {
    static int per_sm = 0;
    if (!per_sm) {
        int b = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kernel, 128, 0) != cudaSuccess ||
            b < 1)
            b = 1;
        per_sm = b;
    }
    const unsigned g = grid_for((n + 3) / 4, 128, 2 * per_sm);
    return g >= (unsigned)(sm_count() * per_sm) ? g : 0;
}

}  // namespace cg
