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

#include <algorithm>
#include <cstdint>

#include "common.cuh"
#include "de.cuh"
#include "point_io.cuh"
#include "pool_share.cuh"

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

// Runs `task` over this warp's share of the n points (pool_share.cuh; w.first <
// n).  Call from all 32 lanes.
//   task.start(i)   begin point i            task.step()  one step, false at the end
//   task.finish(i)  write point i's result   task.steps() the steps of the point
//   task.whole(i)   all of point i
// `wait`: the lanes that wait before results are written and new points taken
// together.  Lanes in step also agree on the branches inside the trigonometric
// functions, so where steps are alike the pool costs 15 to 25 %: there the
// points are taken whole, group by group.  Points side by side are the caller's
// to tell (wait 32); points that run most of `max_steps` (on the surface) show
// here: if fewer than `wait` of the first 32 have ended after a fifth of it (of
// uniform points in the cube 73 % have after two of 15 steps, of points on the
// surface 4 % after three), or a warp's worth of points has averaged 0.45 of it.
template <class Task>
__device__ __forceinline__ void warp_pool(const WarpWalk& w, uint64_t n, int wait,
                                          uint32_t max_steps, Task& task) {
    const uint32_t below = (1u << (threadIdx.x & 31)) - 1u;
    PoolShare share(w.first, w.stride, n);
    uint64_t mine = 0;
    uint32_t ended = 0, steps = 0;
    const bool alike = wait == 32;
    uint32_t probe = max(max_steps / 5, 1u);
    bool have = false, busy = false;
    while (!alike) {
        const uint32_t idle = __ballot_sync(0xFFFFFFFFu, !busy);
        const uint32_t done = __ballot_sync(0xFFFFFFFFu, have && !busy);
        // Enough lanes wait for new points or, when there are none, with results.
        const uint32_t waiting = share.next < share.end ? idle : done;
        if (__popc(waiting) >= wait || idle == 0xFFFFFFFFu) {
            if (have && !busy) task.finish(mine);
            if (wait == 32) break;  // every lane has ended
            ended += __popc(done);
            steps += __reduce_add_sync(0xFFFFFFFFu, have && !busy ? task.steps() : 0u);
            if (ended >= 32 && (float)steps > 0.45f * (float)ended * (float)max_steps) {
                wait = 32;
                have = have && busy;
                if (!__any_sync(0xFFFFFFFFu, busy)) break;
                continue;
            }
            if (!busy) {
                mine = share.index(__popc(idle & below));
                have = busy = mine < n;
                if (have) task.start(mine);
            }
            share.advance(__popc(idle));
            if (!__any_sync(0xFFFFFFFFu, busy)) break;
        }
        if (busy) busy = task.step();
        if (--probe == 0) wait = share.next == 32 ? 32 : wait;
    }
    for (; share.next < share.end; share.advance(32)) {
        const uint64_t i = share.index(threadIdx.x & 31);
        if (i < n) task.whole(i);
    }
}

// The blocks (of 128 threads) of a pool kernel over n points: 16 points to a
// lane, between two and eight times `per_sm` to an SM (about what fits on it:
// blocks then end at different times and the SMs stay full; 3 M points of a grid
// take 193 us at two times ten, 205 at once).  0 with fewer than 8 points to a
// lane of `per_sm` blocks, where a pool gains less than its uneven end costs (1.1
// M points: uniform 145 -> 115 us, but on the surface 145 -> 154 and of a grid
// 80 -> 88).  A function of n and the estimator alone.
inline unsigned pool_grid(uint32_t per_sm, uint64_t n) {
    const uint64_t resident = (uint64_t)sm_count() * per_sm;
    if (n < 8 * 128 * resident) return 0;
    return (unsigned)std::min(std::max(n / (16 * 128), 2 * resident), 8 * resident);
}

}  // namespace cg
