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

// Lane `lane`'s corner of face item f; `row_word`: the item is one sign word of
// a row, else part of the plane z = res.
struct FaceCorner {
    uint32_t x, y, z;
    bool in, row_word;
};

__device__ __forceinline__ FaceCorner face_corner(uint32_t shift, uint32_t f, uint32_t lane) {
    const uint32_t res = 1u << shift, n = res + 1u, rows = face_row_items(shift);
    FaceCorner c;
    c.row_word = f < rows;
    if (c.row_word) {
        const uint32_t r = f >> (shift - 5);
        c.x = r <= res ? res : r - n;
        c.y = r <= res ? r : res;
        c.z = 32 * (f & ((1u << (shift - 5)) - 1u)) + lane;
        c.in = true;
    } else {
        const uint32_t i = (f - rows) * 32 + lane;
        c.in = i < n * n;
        c.x = i / n;
        c.y = i - c.x * n;
        c.z = res;
    }
    return c;
}

// The item's signs from its ballot: a row's word whole, or the first bit of
// each row's last word (its only corner).
__device__ __forceinline__ void face_sign(const FaceCorner& c, uint32_t W, uint32_t ballot,
                                          bool pos, uint32_t lane, uint32_t n,
                                          uint32_t* __restrict__ sgn) {
    if (c.row_word ? lane == 0 : c.in)
        CG_AT(sgn, (c.x * n + c.y) * W + (c.z >> 5), (uint64_t)n * n * W) =
            c.row_word ? ballot : (pos ? 1u : 0u);
}

template <int M, class Coord>
__device__ __forceinline__ void face_item(const ShapeDev& s, const Coord& coord, uint32_t shift,
                                          uint32_t W, uint32_t f, float* __restrict__ out,
                                          uint32_t* __restrict__ sgn) {
    const uint32_t lane = threadIdx.x & 31, n = (1u << shift) + 1u;
    const FaceCorner c = face_corner(shift, f, lane);
    bool pos = false;
    if (c.in) {
        const float d = eval<M>(s, coord(0, c.x), coord(1, c.y), coord(2, c.z));
        CG_AT(out, ((size_t)c.x * n + c.y) * n + c.z, (uint64_t)n * n * n) = d;
        pos = (__float_as_uint(d) >> 31) == 0u;
    }
    if (!sgn) return;
    face_sign(c, W, __ballot_sync(0xFFFFFFFFu, pos), pos, lane, n, sgn);
}

}  // namespace cg
