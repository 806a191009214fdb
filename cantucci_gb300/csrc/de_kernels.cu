// de_kernels.cu -- distance-estimator kernels: point batches, span grids,
// contains, loop-state dumps and the get_focii march loop.
#include <cmath>

#include "common.cuh"
#include "de.cuh"
#include "grid_units.cuh"
#include "kernels.cuh"
#include "lane_pool.cuh"
#include "point_io.cuh"

namespace cg {

CG_OOB_READER(de_kernels)

template <int M>
__global__ void __launch_bounds__(256) k_de_points(ShapeDev s, const float* __restrict__ pts,
                                                   uint64_t n, float* __restrict__ out) {
    __shared__ __align__(16) float stage[8][96];
    const WarpWalk w = warp_walk();
    for (uint64_t base = w.first; base < n; base += w.stride) {
        float x = 0.0f, y = 0.0f, z = 0.0f;
        if (load_point_warp(pts, n, base, stage[threadIdx.x >> 5], x, y, z))
            out[base + (threadIdx.x & 31)] = eval<M>(s, x, y, z);
    }
}

// Large batches: each warp takes its points through a lane pool.  MU: the mode
// of points taken whole.
template <int M, int MU>
struct PointTask {
    const ShapeDev& s;
    const float* __restrict__ pts;
    float* __restrict__ out;
    DeLoop<M> de;
    __device__ __forceinline__ void start(uint64_t i) {
        de.start(s, pts[3 * i], pts[3 * i + 1], pts[3 * i + 2]);
    }
    __device__ __forceinline__ bool step() { return de.step(s); }
    __device__ __forceinline__ void finish(uint64_t i) { out[i] = de.value(s); }
    __device__ __forceinline__ uint32_t steps() const { return de.it; }
    __device__ __forceinline__ void whole(uint64_t i) {
        out[i] = eval<MU>(s, pts[3 * i], pts[3 * i + 1], pts[3 * i + 2]);
    }
};

// Lanes that wait in a pool: more where a step is short.
template <int M>
constexpr int kPointFlush = M == MODE_P8 ? 12 : 8;

// Blocks to an SM (pool_grid): 2 M uniform points, polar power 8, 168 us with 8,
// 174 with 10, on the surface 272 and 274, but 1.7 M on it 238 and 229, 5 M 692
// and 653; Mandelbulb<8>, 2 M uniform 76 and 80, 5 M 168 and 164.
template <int M>
constexpr uint32_t kPointBlocks = M == MODE_P8 ? 8 : 10;

template <int M, int MU>
__global__ void __launch_bounds__(128) k_de_points_pool(ShapeDev s, const float* __restrict__ pts,
                                                        uint64_t n, float* __restrict__ out) {
    const WarpWalk w = warp_walk();
    if (w.first >= n) return;
    PointTask<M, MU> task{s, pts, out, {}};
    warp_pool(w, n, points_side_by_side(pts, w, n) ? 32 : kPointFlush<M>, s.max_iters, task);
}

// Corner (x, y, z) of a span grid: p = start + across * (v / res)
// (src/mesh/buffer.rs:79-80).  v / res is exact for a power-of-two res, so it
// is formed as v * inv_res.
__device__ __forceinline__ void grid_point(const GridDev& g, uint32_t i, float& px, float& py,
                                           float& pz) {
    const uint32_t z = i % g.n;
    const uint32_t xy = i / g.n;
    const uint32_t y = xy % g.n;
    const uint32_t x = xy / g.n;
    px = __fadd_rn(g.start[0], __fmul_rn(g.across[0], __fmul_rn((float)x, g.inv_res)));
    py = __fadd_rn(g.start[1], __fmul_rn(g.across[1], __fmul_rn((float)y, g.inv_res)));
    pz = __fadd_rn(g.start[2], __fmul_rn(g.across[2], __fmul_rn((float)z, g.inv_res)));
}

__device__ __forceinline__ float grid_coord(const GridDev& g, int k, uint32_t v) {
    return __fadd_rn(g.start[k], __fmul_rn(g.across[k], __fmul_rn((float)v, g.inv_res)));
}

// Small grids: one corner per thread in linear (GridTable) order.  With
// `sgn`, also sets bit z%32 of sign word (x, y, z/32) for positive corners.
template <int M>
__global__ void __launch_bounds__(256) k_de_grid(ShapeDev s, GridDev g, float* __restrict__ out,
                                                 uint32_t* __restrict__ sgn, uint32_t W,
                                                 const GridDev* __restrict__ gp) {
    if (gp) g = *gp;
    const uint32_t total = g.n * g.n * g.n;
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
        float x, y, z;
        grid_point(g, i, x, y, z);
        const float d = eval<M>(s, x, y, z);
        CG_AT(out, i, total) = d;
        if (sgn && !(__float_as_uint(d) >> 31)) {
            const uint32_t zi = i % g.n, row = i / g.n;
            atomicOr(&CG_AT(sgn, row * W + (zi >> 5), (uint64_t)g.n * g.n * W), 1u << (zi & 31));
        }
    }
}

struct GridCoord {
    const GridDev& g;
    __device__ __forceinline__ float operator()(int k, uint32_t v) const {
        return grid_coord(g, k, v);
    }
};

// Grids of res 32 and 64, one brick or face item to a warp: the lanes of
// k_de_grid_units without its walk, in fewer registers.  A block is a core unit
// (its eight bricks' ballots meet in shared memory as the rows' sign words) or
// eight face items, so every sign word is stored whole.
template <int M>
__global__ void __launch_bounds__(256, 5) k_de_grid_small(ShapeDev s, GridDev g,
                                                          float* __restrict__ out,
                                                          uint32_t* __restrict__ sgn, uint32_t W,
                                                          uint32_t shift,
                                                          const GridDev* __restrict__ gp) {
    __shared__ uint32_t ballots[8];
    if (gp) g = *gp;
    const GridCoord coord{g};
    const uint32_t n = g.n, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t core = core_units(shift);
    if (blockIdx.x >= core) {
        const uint32_t f = 8 * (blockIdx.x - core) + warp;
        if (f < face_items(shift)) face_item<M>(s, coord, shift, W, f, out, sgn);
        return;
    }
    const uint32_t c = blockIdx.x, gz = c & ((1u << (shift - 5)) - 1u), t = c >> (shift - 5);
    const uint32_t x0 = 2 * (t >> (shift - 2)), y0 = 4 * (t & ((1u << (shift - 2)) - 1u));
    const uint32_t x = x0 + (lane >> 4), y = y0 + ((lane >> 2) & 3);
    const uint32_t z = 32 * gz + 4 * warp + (lane & 3);
    const float d = eval<M>(s, coord(0, x), coord(1, y), coord(2, z));
    CG_AT(out, ((size_t)x * n + y) * n + z, (uint64_t)n * n * n) = d;
    if (!sgn) return;
    const uint32_t b = __ballot_sync(0xFFFFFFFFu, (__float_as_uint(d) >> 31) == 0u);
    if (lane == 0) ballots[warp] = b;
    __syncthreads();
    if (threadIdx.x < 8) {  // row k of the unit's 2 x 4: bits 4 k of each ballot
        const uint32_t k = threadIdx.x;
        uint32_t word = 0;
#pragma unroll
        for (uint32_t w = 0; w < 8; ++w) word |= ((ballots[w] >> (4 * k)) & 0xFu) << (4 * w);
        CG_AT(sgn, ((x0 + (k >> 2)) * n + y0 + (k & 3)) * W + gz, (uint64_t)n * n * W) = word;
    }
}

// Large grids: persistent warps take core units, then groups of 8 face items,
// from `queue` (a unit of the bulb's inside costs seven of the outside, so a
// fixed share left warps idle at the end: 309 against 285 us for the 257^3 span)
// or, without one, in strides.  A warp asks for its next unit before it begins
// the one it has.
template <int M>
__global__ void __launch_bounds__(256) k_de_grid_units(ShapeDev s, GridDev g,
                                                       float* __restrict__ out,
                                                       uint32_t* __restrict__ sgn, uint32_t W,
                                                       uint32_t shift,
                                                       uint32_t* __restrict__ queue,
                                                       const GridDev* __restrict__ gp) {
    if (gp) g = *gp;
    const GridCoord coord{g};
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5, core = core_units(shift);
    const uint32_t faces = face_items(shift), units = core + (faces + 7) / 8;
    uint32_t u = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;  // the queue starts at nwarps
    while (u < units) {
        uint32_t next = u + nwarps;
        if (queue && lane == 0) next = nwarps + atomicAdd(queue, 1u);
        if (u < core) {
            // y and z ranges turned by x: a warp's stride is a multiple of the
            // words of a row, and it would else meet the same z range every
            // time (the 513^3 span's mesh 3.03 against 2.9 ms).
            const uint32_t a = shift - 5, b = shift - 2, x = u >> (a + b);
            const uint32_t y = ((u >> a) + 37 * x) & ((1u << b) - 1u);
            const uint32_t z = (u + x) & ((1u << a) - 1u);
            core_unit<M>(s, coord, shift, W, (((x << b) | y) << a) | z, out, sgn);
        } else {
            const uint32_t f0 = 8 * (u - core), f1 = min(f0 + 8, faces);
#pragma unroll 1
            for (uint32_t f = f0; f < f1; ++f) face_item<M>(s, coord, shift, W, f, out, sgn);
        }
        u = queue ? __shfl_sync(0xFFFFFFFFu, next, 0) : next;
    }
}

// Grids between: warps walk 2x4x4 bricks of corners (x, y, z), which keeps the
// escape counts of a warp's lanes close (89% lane efficiency on the 513^3
// span vs 75% for 32 corners along z); 8-brick units would leave SMs idle.
// Each brick's 4 bits per row go into the sign word with atomicOr (sgn zeroed
// first).
template <int M>
__global__ void __launch_bounds__(256) k_de_grid_brick(ShapeDev s, GridDev g,
                                                       float* __restrict__ out,
                                                       uint32_t* __restrict__ sgn, uint32_t W,
                                                       const GridDev* __restrict__ gp) {
    if (gp) g = *gp;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t n = g.n;
    const uint32_t BX = (n + 1) >> 1, B4 = (n + 3) >> 2;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    // Brick (bx, by, bz), advanced by the grid stride in the same mixed radix.
    const uint32_t u0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    uint32_t bz = u0 % B4, by = (u0 / B4) % B4, bx = u0 / (B4 * B4);
    const uint32_t sz = nwarps % B4, sy = (nwarps / B4) % B4, sx = nwarps / (B4 * B4);
    for (; bx < BX;) {
        const uint32_t x = 2 * bx + (lane >> 4), y = 4 * by + ((lane >> 2) & 3),
                       z = 4 * bz + (lane & 3);
        bool pos = false;
        const bool in = x < n && y < n && z < n;
        if (in) {
            const float d =
                eval<M>(s, grid_coord(g, 0, x), grid_coord(g, 1, y), grid_coord(g, 2, z));
            CG_AT(out, ((size_t)x * n + y) * n + z, (uint64_t)n * n * n) = d;
            pos = (__float_as_uint(d) >> 31) == 0u;
        }
        if (sgn) {
            const uint32_t b = __ballot_sync(0xFFFFFFFFu, pos);
            const uint32_t bits = (b >> (lane & ~3u)) & 0xFu;
            if ((lane & 3) == 0 && bits)
                atomicOr(&CG_AT(sgn, (x * n + y) * W + (z >> 5), (uint64_t)n * n * W),
                         bits << (z & 31));
        }
        bz += sz;
        uint32_t carry = 0;
        if (bz >= B4) {
            bz -= B4;
            carry = 1;
        }
        by += sy + carry;
        carry = 0;
        if (by >= B4) {
            by -= B4;
            carry = 1;
        }
        bx += sx + carry;
    }
}

__global__ void __launch_bounds__(256) k_state(ShapeDev s, const float* __restrict__ pts,
                                               uint64_t n, float4* __restrict__ out) {
    __shared__ __align__(16) float stage[8][96];
    const WarpWalk w = warp_walk();
    for (uint64_t base = w.first; base < n; base += w.stride) {
        float x = 0.0f, y = 0.0f, z = 0.0f;
        if (!load_point_warp(pts, n, base, stage[threadIdx.x >> 5], x, y, z)) continue;
        MbState st;
        if (s.power == 8)
            mandelbulb_de<Exact, true>(8, s.max_iters, s.bailout, x, y, z, &st);
        else
            mandelbulb_de<Exact, false>(s.power, s.max_iters, s.bailout, x, y, z, &st);
        out[base + (threadIdx.x & 31)] =
            make_float4(st.r, st.dr, __uint_as_float(st.steps), __uint_as_float(st.escaped));
    }
}

// Shape::contains (src/shape/mod.rs:78-80); Sphere overrides it with
// |c - p|^2 <= r^2 (src/shape/sphere.rs:24-26).
__global__ void __launch_bounds__(256) k_contains(ShapeDev s, const float* __restrict__ pts,
                                                  uint64_t n, uint8_t* __restrict__ out) {
    __shared__ __align__(16) float stage[8][96];
    const WarpWalk w = warp_walk();
    for (uint64_t base = w.first; base < n; base += w.stride) {
        float x = 0.0f, y = 0.0f, z = 0.0f;
        if (!load_point_warp(pts, n, base, stage[threadIdx.x >> 5], x, y, z)) continue;
        const uint64_t i = base + (threadIdx.x & 31);
        bool in;
        if (s.kind == CG_SHAPE_SPHERE) {
            const float dx = __fsub_rn(s.center[0], x), dy = __fsub_rn(s.center[1], y),
                        dz = __fsub_rn(s.center[2], z);
            const float m2 = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)),
                                       __fmul_rn(dz, dz));
            in = m2 <= __fmul_rn(s.radius, s.radius);
        } else {
            in = shape_de(s, x, y, z) < 0.0f;
        }
        out[i] = in ? 1 : 0;
    }
}

// March loop of ShapeMesh::get_focii (src/mesh/mod.rs:229-241).
__global__ void k_march(ShapeDev s, const float* __restrict__ org, const float* __restrict__ dir,
                        uint64_t n, uint32_t max_steps, float eps, float* __restrict__ hits,
                        uint8_t* __restrict__ hit) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        float px = org[3 * i], py = org[3 * i + 1], pz = org[3 * i + 2];
        const float dx = dir[3 * i], dy = dir[3 * i + 1], dz = dir[3 * i + 2];
        uint8_t h = 0;
        for (uint32_t k = 0; k < max_steps; ++k) {
            const float d = shape_de(s, px, py, pz);
            px = __fadd_rn(px, __fmul_rn(dx, d));
            py = __fadd_rn(py, __fmul_rn(dy, d));
            pz = __fadd_rn(pz, __fmul_rn(dz, d));
            if (d < eps) {
                h = 1;
                break;
            }
        }
        hits[3 * i] = px;
        hits[3 * i + 1] = py;
        hits[3 * i + 2] = pz;
        hit[i] = h;
    }
}

// Rotate steps and escapes over a span grid (same loop as k_de_grid).
template <bool P8>
__global__ void __launch_bounds__(256) k_grid_work(ShapeDev s, GridDev g,
                                                   unsigned long long* __restrict__ acc) {
    const uint32_t total = g.n * g.n * g.n;
    unsigned long long steps = 0, esc = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += gridDim.x * blockDim.x) {
        float x, y, z;
        grid_point(g, i, x, y, z);
        MbState st;
        mandelbulb_de<Exact, P8>(s.power, s.max_iters, s.bailout, x, y, z, &st);
        steps += st.steps;
        esc += st.escaped;
    }
    for (int o = 16; o > 0; o >>= 1) {
        steps += __shfl_down_sync(0xFFFFFFFFu, steps, o);
        esc += __shfl_down_sync(0xFFFFFFFFu, esc, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&acc[0], steps);
        atomicAdd(&acc[1], esc);
    }
}

cg_status launch_grid_work(const ShapeDev& s, const GridDev& g, unsigned long long* acc,
                           cudaStream_t st) {
    const uint64_t total = (uint64_t)g.n * g.n * g.n;
    const unsigned B = 256, G = grid_for(total, B, 16);
    if (s.power == 8)
        k_grid_work<true><<<G, B, 0, st>>>(s, g, acc);
    else
        k_grid_work<false><<<G, B, 0, st>>>(s, g, acc);
    CG_CHECK_LAUNCH("k_grid_work");
    return CG_OK;
}


template <int M, int MU = M>
static bool launch_points_pool(const ShapeDev& s, const float* pts, uint64_t n, float* out,
                               cudaStream_t st) {
    const unsigned G = pool_grid(kPointBlocks<M>, n);
    if (G) k_de_points_pool<M, MU><<<G, 128, 0, st>>>(s, pts, n, out);
    return G != 0;
}

// True if the batch is large enough for a pool kernel (and was launched).  The
// exact estimators only: a step of the fast ones is too short for it (9 M points
// on the surface 4 to 8 % slower, 3 M points anywhere no faster).
// In us, the plain kernel -> the pool: polar power 8, 3 M uniform points 383 ->
// 235, 16 M 2008 -> 1061; 3 M on the surface 383 -> 399, 16 M 2008 -> 2014; 9 M
// of a grid 496 -> 506; Mandelbulb<8>, 3 M uniform 115 -> 104, on the surface
// 117 -> 123, a grid 61 -> 57; 1.7 M polar uniform 218 -> 152, on the surface
// 217 -> 229.
static bool launch_points_pool_mode(const ShapeDev& s, const float* pts, uint64_t n, float* out,
                                    uint32_t numerics, cudaStream_t st) {
    if (s.max_iters < 1) return false;
    switch (mode_of(s, numerics)) {
    case MODE_P8:
        return p8_unrolled(s) ? launch_points_pool<MODE_P8, MODE_P8_IT15>(s, pts, n, out, st)
                              : launch_points_pool<MODE_P8>(s, pts, n, out, st);
    case MODE_INT: return launch_points_pool<MODE_INT>(s, pts, n, out, st);
    case MODE_POLAR: return launch_points_pool<MODE_POLAR>(s, pts, n, out, st);
    default: return false;
    }
}

cg_status launch_de_points(const ShapeDev& s, const float* pts, uint64_t n, float* out,
                           uint32_t numerics, cudaStream_t st) {
    if (n == 0) return CG_OK;
    if (launch_points_pool_mode(s, pts, n, out, numerics, st)) {
        CG_CHECK_LAUNCH("k_de_points_pool");
        return CG_OK;
    }
    const unsigned B = 256, G = grid_for(n, B, 16);
    switch (mode_of(s, numerics)) {
    case MODE_P8:
        if (p8_unrolled(s)) k_de_points<MODE_P8_IT15><<<G, B, 0, st>>>(s, pts, n, out);
        else k_de_points<MODE_P8><<<G, B, 0, st>>>(s, pts, n, out);
        break;
    case MODE_INT: k_de_points<MODE_INT><<<G, B, 0, st>>>(s, pts, n, out); break;
    case MODE_POLAR: k_de_points<MODE_POLAR><<<G, B, 0, st>>>(s, pts, n, out); break;
    case MODE_SPHERE: k_de_points<MODE_SPHERE><<<G, B, 0, st>>>(s, pts, n, out); break;
    case MODE_INT_POLY: k_de_points<MODE_INT_POLY><<<G, B, 0, st>>>(s, pts, n, out); break;
    case MODE_POLAR_FAST: k_de_points<MODE_POLAR_FAST><<<G, B, 0, st>>>(s, pts, n, out); break;
    default:
        if (p8_unrolled(s)) k_de_points<MODE_P8_FAST_IT15><<<G, B, 0, st>>>(s, pts, n, out);
        else k_de_points<MODE_P8_FAST><<<G, B, 0, st>>>(s, pts, n, out);
        break;
    }
    CG_CHECK_LAUNCH("k_de_points");
    return CG_OK;
}

// P=8 exact, two corners per thread with packed f32x2 instructions: each
// warp evaluates a 4x4x4 brick, lane (dx, dy, dz) taking corners (x, y, z)
// and (x + 2, y, z).  With `sgn` the four z-lanes of each (x, y) row OR their
// sign bits with two shuffles and one lane sets them with atomicOr (sgn must
// be zeroed first).
__global__ void __launch_bounds__(256) k_de_grid_p8x2(ShapeDev s, GridDev g,
                                                      float* __restrict__ out,
                                                      uint32_t* __restrict__ sgn, uint32_t W,
                                                      const GridDev* __restrict__ gp) {
    if (gp) g = *gp;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t n = g.n;
    const uint32_t B4 = (n + 3) >> 2;
    const uint32_t bricks = B4 * B4 * B4;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t dx = lane >> 4, dy = (lane >> 2) & 3, dz = lane & 3;
    for (uint32_t b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; b < bricks; b += nwarps) {
        const uint32_t bz = b % B4, t = b / B4, by = t % B4, bx = t / B4;
        const uint32_t xA = 4 * bx + dx, xB = xA + 2, y = 4 * by + dy, z = 4 * bz + dz;
        const bool inYZ = y < n && z < n;
        const bool liveA = inYZ && xA < n, liveB = inYZ && xB < n;
        const float py = grid_coord(g, 1, y), pz = grid_coord(g, 2, z);
        float dA = 0.0f, dB = 0.0f;
        // Both lanes always iterate a real corner (an inactive lane repeats
        // the other's), so no code path sees a lane that is known to be idle.
        const float pxA = grid_coord(g, 0, liveA ? xA : xB);
        const float pxB = grid_coord(g, 0, liveB ? xB : xA);
        if (liveA || liveB)
            mandelbulb_p8_x2(s.max_iters, s.bailout, true, true, pxA, py, pz, pxB, py, pz, dA, dB);
        uint32_t bitA = 0, bitB = 0;
        if (liveA) {
            out[((size_t)xA * n + y) * n + z] = dA;
            bitA = (__float_as_uint(dA) >> 31) ? 0u : (1u << (z & 31));
        }
        if (liveB) {
            out[((size_t)xB * n + y) * n + z] = dB;
            bitB = (__float_as_uint(dB) >> 31) ? 0u : (1u << (z & 31));
        }
        if (sgn) {
            bitA |= __shfl_xor_sync(0xFFFFFFFFu, bitA, 1);
            bitA |= __shfl_xor_sync(0xFFFFFFFFu, bitA, 2);
            bitB |= __shfl_xor_sync(0xFFFFFFFFu, bitB, 1);
            bitB |= __shfl_xor_sync(0xFFFFFFFFu, bitB, 2);
            if (dz == 0 && bitA) atomicOr(&sgn[(xA * n + y) * W + (z >> 5)], bitA);
            if (dz == 0 && bitB) atomicOr(&sgn[(xB * n + y) * W + (z >> 5)], bitB);
        }
    }
}

// Kernel choice for step 1 (cg_set_option "de_grid_kernel").
static int g_de_grid_kernel = DE_GRID_AUTO;

int de_grid_kernel_option() { return g_de_grid_kernel; }

int set_de_grid_kernel(int v) {
    if (v < DE_GRID_AUTO || v > DE_GRID_PACKED) return 0;
    g_de_grid_kernel = v;
    return 1;
}

template <int M>
static cg_status launch_grid_mode(const ShapeDev& s, const GridDev& g, float* out, uint32_t* sgn,
                                  uint32_t W, cudaStream_t st, const GridDev* gp) {
    const unsigned B = 256;
    int k = g_de_grid_kernel;
    const bool automatic = k == DE_GRID_AUTO;
    const size_t words = (size_t)g.n * g.n * W;
    // The kernels that set single bits of a sign word want the words zeroed.
    auto clear = [&](uint32_t* p, size_t count) -> cg_status {
        if (sgn) CG_CUDA(cudaMemsetAsync(p, 0, count * sizeof(uint32_t), st));
        return CG_OK;
    };
    // Up to 65^3 corners (res 64, cantucci's leaves) one brick to a warp: the
    // brick walk's 63 registers (4 blocks of 256 threads per SM) would fit the
    // grid in more waves than k_de_grid_small's, and one corner per thread in
    // row order keeps 24 lanes busy against 27 (15.8 against 14.7 us).
    if (automatic) k = g.n > 65 ? DE_GRID_BRICK : DE_GRID_LINEAR;
    uint32_t shift = 0;
    while ((2u << shift) < g.n) ++shift;
    if (automatic && k == DE_GRID_LINEAR && g.n > kUnitMinRes) {
        const uint32_t blocks = core_units(shift) + (face_items(shift) + 7) / 8;
        k_de_grid_small<M><<<blocks, B, 0, st>>>(s, g, out, sgn, W, shift, gp);
    } else if (k == DE_GRID_PACKED && (M == MODE_P8 || M == MODE_P8_IT15)) {
        CG_TRY(clear(sgn, words));
        const uint64_t b4 = (g.n + 3) >> 2;
        k_de_grid_p8x2<<<grid_for(b4 * b4 * b4 * 32, B, 8), B, 0, st>>>(s, g, out, sgn, W, gp);
    } else if (k != DE_GRID_LINEAR) {
        // 8-brick units when they make at least four waves of resident warps
        // (8 blocks of 256 threads per SM), single bricks otherwise.
        const uint64_t rows = (uint64_t)((g.n + 1) >> 1) * ((g.n + 3) >> 2);
        const uint64_t bz = (g.n + 3) >> 2;
        const uint64_t units8 = rows * ((bz + 7) / 8);
        if (units8 >= 4ull * sm_count() * 8 * (B / 32)) {
            const uint64_t units = core_units(shift) + (face_items(shift) + 7) / 8;
            // (A sphere's units are so short that they would wait for the queue:
            // a mesh of 256^3 cells 195 us with it, 155 without.)
            uint32_t* queue = sgn && M != MODE_SPHERE ? sgn + words : nullptr;
            if (queue) CG_TRY(clear(queue, 1));
            k_de_grid_units<M><<<grid_for(units * 32, B, 8), B, 0, st>>>(s, g, out, sgn, W, shift,
                                                                         queue, gp);
        } else {
            CG_TRY(clear(sgn, words));
            k_de_grid_brick<M><<<grid_for(rows * bz * 32, B, 8), B, 0, st>>>(s, g, out, sgn, W, gp);
        }
    } else {
        CG_TRY(clear(sgn, words));
        const uint64_t total = (uint64_t)g.n * g.n * g.n;
        k_de_grid<M><<<grid_for(total, B, 8), B, 0, st>>>(s, g, out, sgn, W, gp);
    }
    return CG_OK;
}

cg_status launch_de_grid(const ShapeDev& s, const GridDev& g, float* out, uint32_t numerics,
                         cudaStream_t st, uint32_t* sgn, uint32_t W, const GridDev* gp) {
    switch (mode_of(s, numerics)) {
    case MODE_P8:
        if (p8_unrolled(s)) CG_TRY(launch_grid_mode<MODE_P8_IT15>(s, g, out, sgn, W, st, gp));
        else CG_TRY(launch_grid_mode<MODE_P8>(s, g, out, sgn, W, st, gp));
        break;
    case MODE_INT: CG_TRY(launch_grid_mode<MODE_INT>(s, g, out, sgn, W, st, gp)); break;
    case MODE_POLAR: CG_TRY(launch_grid_mode<MODE_POLAR>(s, g, out, sgn, W, st, gp)); break;
    case MODE_SPHERE: CG_TRY(launch_grid_mode<MODE_SPHERE>(s, g, out, sgn, W, st, gp)); break;
    case MODE_INT_POLY: CG_TRY(launch_grid_mode<MODE_INT_POLY>(s, g, out, sgn, W, st, gp)); break;
    case MODE_POLAR_FAST: CG_TRY(launch_grid_mode<MODE_POLAR_FAST>(s, g, out, sgn, W, st, gp)); break;
    default:
        if (p8_unrolled(s)) CG_TRY(launch_grid_mode<MODE_P8_FAST_IT15>(s, g, out, sgn, W, st, gp));
        else CG_TRY(launch_grid_mode<MODE_P8_FAST>(s, g, out, sgn, W, st, gp));
        break;
    }
    CG_CHECK_LAUNCH("k_de_grid");
    return CG_OK;
}

cg_status launch_state(const ShapeDev& s, const float* pts, uint64_t n, float* out,
                       cudaStream_t st) {
    if (n == 0) return CG_OK;
    const unsigned B = 256, G = grid_for(n, B, 16);
    k_state<<<G, B, 0, st>>>(s, pts, n, reinterpret_cast<float4*>(out));
    CG_CHECK_LAUNCH("k_state");
    return CG_OK;
}

cg_status launch_contains(const ShapeDev& s, const float* pts, uint64_t n, uint8_t* out,
                          cudaStream_t st) {
    if (n == 0) return CG_OK;
    const unsigned B = 256, G = grid_for(n, B, 16);
    k_contains<<<G, B, 0, st>>>(s, pts, n, out);
    CG_CHECK_LAUNCH("k_contains");
    return CG_OK;
}

cg_status launch_march(const ShapeDev& s, const float* org, const float* dir, uint64_t n,
                       uint32_t max_steps, float eps, float* hits, uint8_t* hit, cudaStream_t st) {
    if (n == 0) return CG_OK;
    const unsigned B = 128, G = grid_for(n, B, 16);
    k_march<<<G, B, 0, st>>>(s, org, dir, n, max_steps, eps, hits, hit);
    CG_CHECK_LAUNCH("k_march");
    return CG_OK;
}

}  // namespace cg
