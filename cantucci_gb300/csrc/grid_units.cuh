// grid_units.cuh -- the corners of a span grid as full warps' work.
//
// A grid has res + 1 corners per axis (res a power of two), so 2x4x4 bricks
// over all of it spend a tenth of their lanes past its end at res 64 (a few
// percent at 256).  For res >= 32 the grid is instead the res^3 corners before
// the last planes, in bricks without remainder, and three faces: the rows
// with x = res or y = res, 32 corners along z (one sign word) at a time, and
// the plane z = res, 32 of its corners at a time.
//   core unit c   the 8 bricks along z of one sign word of 2 x 4 rows
//   face item f   32 corners of a face
#pragma once

#include <cstdint>

#include "common.cuh"
#include "de.cuh"

namespace cg {

constexpr uint32_t kUnitMinRes = 32;

// shift = log2 res.
__host__ __device__ constexpr uint32_t core_bricks(uint32_t shift) { return 1u << (3 * shift - 5); }
__host__ __device__ constexpr uint32_t core_units(uint32_t shift) { return 1u << (3 * shift - 8); }
__host__ __device__ constexpr uint32_t face_row_items(uint32_t shift) {
    return ((2u << shift) + 1u) << (shift - 5);
}
__host__ __device__ constexpr uint32_t face_items(uint32_t shift) {
    const uint32_t n = (1u << shift) + 1u;
    return face_row_items(shift) + (n * n + 31u) / 32u;
}

// The 8 bricks of core unit c; `coord(axis, v)` is a corner's coordinate.
// Each lane writes its 8 distances, and the z-lane-0 thread of each row its
// row's sign word, collected from one ballot per brick.
template <int M, class Coord>
__device__ __forceinline__ void core_unit(const ShapeDev& s, const Coord& coord, uint32_t shift,
                                          uint32_t W, uint32_t c, float* __restrict__ out,
                                          uint32_t* __restrict__ sgn) {
    const uint32_t lane = threadIdx.x & 31, n = (1u << shift) + 1u;
    const uint32_t gz = c & ((1u << (shift - 5)) - 1u), t = c >> (shift - 5);
    const uint32_t x = 2 * (t >> (shift - 2)) + (lane >> 4);
    const uint32_t y = 4 * (t & ((1u << (shift - 2)) - 1u)) + ((lane >> 2) & 3);
    const float px = coord(0, x), py = coord(1, y);
    const uint32_t row = x * n + y;
    [[maybe_unused]] const uint64_t total = (uint64_t)n * n * n;
    uint32_t word = 0;
#pragma unroll 1
    for (uint32_t z0 = 32 * gz; z0 < 32 * gz + 32; z0 += 4) {
        const uint32_t z = z0 + (lane & 3);
        const float d = eval<M>(s, px, py, coord(2, z));
        CG_AT(out, (size_t)row * n + z, total) = d;
        if (sgn) {
            const uint32_t b = __ballot_sync(0xFFFFFFFFu, (__float_as_uint(d) >> 31) == 0u);
            word |= ((b >> (lane & ~3u)) & 0xFu) << (z0 & 31);
        }
    }
    if (sgn && (lane & 3) == 0) CG_AT(sgn, row * W + gz, (uint64_t)n * n * W) = word;
}

template <int M, class Coord>
__device__ __forceinline__ void face_item(const ShapeDev& s, const Coord& coord, uint32_t shift,
                                          uint32_t W, uint32_t f, float* __restrict__ out,
                                          uint32_t* __restrict__ sgn) {
    const uint32_t lane = threadIdx.x & 31, res = 1u << shift, n = res + 1u;
    const uint32_t rows = face_row_items(shift);
    uint32_t x, y, z;
    bool in = true;
    if (f < rows) {
        const uint32_t r = f >> (shift - 5);
        x = r <= res ? res : r - n;
        y = r <= res ? r : res;
        z = 32 * (f & ((1u << (shift - 5)) - 1u)) + lane;
    } else {
        const uint32_t i = (f - rows) * 32 + lane;
        in = i < n * n;
        x = i / n;
        y = i - x * n;
        z = res;
    }
    bool pos = false;
    if (in) {
        const float d = eval<M>(s, coord(0, x), coord(1, y), coord(2, z));
        CG_AT(out, ((size_t)x * n + y) * n + z, (uint64_t)n * n * n) = d;
        pos = (__float_as_uint(d) >> 31) == 0u;
    }
    if (!sgn) return;
    const uint32_t bits = __ballot_sync(0xFFFFFFFFu, pos);
    if (f < rows) {
        if (lane == 0) CG_AT(sgn, (x * n + y) * W + (z >> 5), (uint64_t)n * n * W) = bits;
    } else if (in) {
        CG_AT(sgn, (x * n + y) * W + (res >> 5), (uint64_t)n * n * W) = pos ? 1u : 0u;
    }
}

}  // namespace cg
