// trace.cu -- sphere tracing a depth map and its implicit-surface gradient.
//
// The reference's only ray march is ShapeMesh::get_focii
// (src/mesh/mod.rs:229-241: pos += dir * DE, hit when DE < eps); cg_march
// restates it.  Here the same march runs per pixel of a pinhole camera, with
// the hit threshold scaled by the pixel footprint at the ray distance t
// (eps_scale * t * pixel_angle), up to max_steps steps, and returns the depth
// t of every pixel (-1 for a miss).
//
// Backward: at a hit x = o + t d the surface satisfies DE(x; theta) = 0, so
// dt/dtheta = -(dDE/dtheta) / (grad_x DE . d).  The adjoint kernel gives
// both gradients at x; the kernel sums dL/dt * dt/dtheta over pixels for
// theta = (power, three Euler angles).
#include <cmath>
#include <cstring>

#include "adjoint.cuh"
#include "common.cuh"
#include "kernels.cuh"
#include "lane_pool.cuh"
#include "point_io.cuh"

namespace cg {

struct CameraDev {
    float eye[3], right[3], up[3], fwd[3];
    float tan_half, aspect;
    uint32_t width, height;
};

__device__ __forceinline__ void pixel_ray(const CameraDev& c, uint32_t i, float d[3]) {
    const uint32_t px = i % c.width, py = i / c.width;
    const float u = ((px + 0.5f) / c.width * 2.0f - 1.0f) * c.tan_half * c.aspect;
    const float v = (1.0f - (py + 0.5f) / c.height * 2.0f) * c.tan_half;
    float x = c.fwd[0] + u * c.right[0] + v * c.up[0];
    float y = c.fwd[1] + u * c.right[1] + v * c.up[1];
    float z = c.fwd[2] + u * c.right[2] + v * c.up[2];
    const float inv = rsqrtf(x * x + y * y + z * z);
    d[0] = x * inv;
    d[1] = y * inv;
    d[2] = z * inv;
}

template <int M>
__global__ void __launch_bounds__(128) k_trace(ShapeDev s, CameraDev c, uint32_t max_steps,
                                               float eps_scale, float* __restrict__ depth) {
    const uint32_t n = c.width * c.height;
    const float pix = 2.0f * c.tan_half / c.height;  // radians per pixel
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float d[3];
        pixel_ray(c, i, d);
        float t = 0.0f, out = -1.0f;
        for (uint32_t k = 0; k < max_steps; ++k) {
            const float x = c.eye[0] + t * d[0], y = c.eye[1] + t * d[1], z = c.eye[2] + t * d[2];
            const float de = eval<M>(s, x, y, z);
            if (!(de == de)) break;  // NaN: no surface information
            if (de < eps_scale * fmaxf(t, 1e-3f) * pix) {
                out = t;
                break;
            }
            t += de;
            if (t > 10.0f) break;
        }
        depth[i] = out;
    }
}

// One ray of the march: its pixel, direction, parameter, steps, and the loop
// of the estimate it waits for.
template <int M>
struct Ray {
    uint32_t i, k;
    float d[3], t;
    DeLoop<M> de;

    // Estimates so short that a ray waits for a whole one at a time.
    static constexpr bool kWhole = M == MODE_P8_FAST || M == MODE_SPHERE;

    __device__ __forceinline__ void estimate(const ShapeDev& s, const CameraDev& c) {
        de.start(s, c.eye[0] + t * d[0], c.eye[1] + t * d[1], c.eye[2] + t * d[2]);
    }
    __device__ __forceinline__ void start(const ShapeDev& s, const CameraDev& c, uint32_t pixel) {
        i = pixel;
        k = 0;
        pixel_ray(c, i, d);
        t = 0.0f;
        de.start(s, c.eye[0], c.eye[1], c.eye[2]);
    }
    // One step of the estimate's loop and, where it ends, the ray's: false
    // when the ray has ended (its depth is then written).
    __device__ __forceinline__ bool step(const ShapeDev& s, const CameraDev& c, uint32_t max_steps,
                                         float eps_scale, float pix, float* __restrict__ depth) {
        float v;
        if constexpr (kWhole) {
            v = eval<M>(s, de.px, de.py, de.pz);
        } else {
            if (de.step(s)) return true;
            v = de.value(s);
        }
        float out = -1.0f;
        bool fin = false;
        if (!(v == v)) {
            fin = true;  // NaN: no surface information
        } else if (v < eps_scale * fmaxf(t, 1e-3f) * pix) {
            out = t;
            fin = true;
        } else {
            t += v;
            fin = t > 10.0f || ++k >= max_steps;
        }
        if (fin) depth[i] = out;
        else estimate(s, c);
        return !fin;
    }
};

// The same march with the rays of a block in one pool.  A ray ends after 10 to
// 3600 loop steps of its estimates (512 x 512, power 8.3: a tenth of them
// after 570, one in a thousand after 2100), so warps that keep their rays run
// with a third of their lanes, and a long ray waits for the instructions of
// all the others' nearly empty warps.  Here the block's warps step their rays
// kTraceRound times, then meet: while the queue has pixels the ended rays'
// lanes take new ones (up to `share` rays a block: a small image spreads over
// all blocks), and once it is empty the rays still marching move together into
// as few warps as hold them; the last 32 need no one else.  The depths are
// k_trace's, bit for bit; a ray moves with its whole state.  Fast polar form,
// 512 x 512: 1.70 -> 1.05 ms, 64 x 64 0.77 -> 0.49 ms (one queue without the
// pool before); what is left is mostly the longest ray's own chain of
// dependent steps.  Blocks of 512 meet more slowly (1.14 ms with six blocks of
// 256 at 1.12), rounds of 8 too often (1.48 ms).
constexpr unsigned kTraceBlock = 256;
constexpr int kTraceRound = 32, kTraceWholeRound = 4;

template <int M>
__global__ void __launch_bounds__(kTraceBlock) k_trace_pool(ShapeDev s, CameraDev c,
                                                            uint32_t max_steps, float eps_scale,
                                                            float* __restrict__ depth,
                                                            uint32_t* __restrict__ next,
                                                            uint32_t share) {
    constexpr uint32_t kWarps = kTraceBlock / 32;
    __shared__ float sf[11][kTraceBlock];
    __shared__ uint32_t su[3][kTraceBlock];
    __shared__ uint32_t active[kWarps];
    __shared__ uint32_t first;
    const uint32_t n = c.width * c.height;
    const float pix = 2.0f * c.tan_half / c.height;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    Ray<M> ray;
    bool busy = false, more = true;
    for (;;) {
        const uint32_t mask = __ballot_sync(0xFFFFFFFFu, busy);
        if (lane == 0) active[warp] = __popc(mask);
        __syncthreads();
        uint32_t count = 0, before = 0, warps = 0;  // busy lanes: all, of earlier warps
        for (uint32_t w = 0; w < kWarps; ++w) {
            const uint32_t a = active[w];
            before += w < warp ? a : 0u;
            count += a;
            warps += a != 0u;
        }
        const uint32_t below = (1u << lane) - 1u;
        const bool draw = more;
        if (draw) {
            const uint32_t room = share - count;
            if (tid == 0) first = room ? atomicAdd(next, room) : 0u;
            __syncthreads();
            if (room) {
                more = first < n && n - first > room;
                const uint32_t rank = 32 * warp - before + __popc(~mask & below);
                if (!busy && rank < room && first < n && rank < n - first) {
                    if (max_steps == 0) {
                        depth[first + rank] = -1.0f;
                    } else {
                        ray.start(s, c, first + rank);
                        busy = true;
                    }
                }
            }
        } else {
            if (count == 0) break;
            if ((count + 31) / 32 < warps) {
                if (busy) {
                    const uint32_t p = before + __popc(mask & below);
                    sf[0][p] = ray.de.px; sf[1][p] = ray.de.py; sf[2][p] = ray.de.pz;
                    sf[3][p] = ray.de.x; sf[4][p] = ray.de.y; sf[5][p] = ray.de.z;
                    sf[6][p] = ray.de.dr; sf[7][p] = ray.d[0]; sf[8][p] = ray.d[1];
                    sf[9][p] = ray.d[2]; sf[10][p] = ray.t;
                    su[0][p] = ray.de.it; su[1][p] = ray.i; su[2][p] = ray.k;
                }
                __syncthreads();
                busy = tid < count;
                if (busy) {
                    ray.de.px = sf[0][tid]; ray.de.py = sf[1][tid]; ray.de.pz = sf[2][tid];
                    ray.de.x = sf[3][tid]; ray.de.y = sf[4][tid]; ray.de.z = sf[5][tid];
                    ray.de.dr = sf[6][tid]; ray.d[0] = sf[7][tid]; ray.d[1] = sf[8][tid];
                    ray.d[2] = sf[9][tid]; ray.t = sf[10][tid];
                    ray.de.it = su[0][tid]; ray.i = su[1][tid]; ray.k = su[2][tid];
                    ray.de.resume(s);
                }
            }
        }
        if (!draw && count <= 32) {
            // The block's last rays are in one warp now: they need no one else.
            while (busy) busy = ray.step(s, c, max_steps, eps_scale, pix, depth);
            return;
        }
        constexpr int kRound = Ray<M>::kWhole ? kTraceWholeRound : kTraceRound;
        for (int round = 0; round < kRound && __any_sync(0xFFFFFFFFu, busy); ++round)
            if (busy) busy = ray.step(s, c, max_steps, eps_scale, pix, depth);
        __syncthreads();  // `active` and `first` have been read
    }
}

// Sum over hit pixels of g[i] * dt_i/dtheta; with cap > 0, pixels whose
// |dt_i/dtheta_k| exceeds cap for some k are left out.
template <bool LONG>
__global__ void __launch_bounds__(128) k_trace_backward(ShapeDev s, CameraDev c, Dm3 dm,
                                                        const float* __restrict__ depth,
                                                        const float* __restrict__ g, float cap,
                                                        double* __restrict__ params) {
    extern __shared__ __align__(16) float4 adj_smem[];
    __shared__ uint32_t slot;
    const uint32_t columns = long_tape_columns(s.max_iters);
    LongTape tape;
    if constexpr (LONG) tape = long_tape_open(reinterpret_cast<float*>(adj_smem), &slot, columns);
    const uint32_t n = c.width * c.height;
    const WarpWalk walk = warp_walk();
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    for (uint64_t base = walk.first; base < n; base += walk.stride) {
        const uint32_t i = (uint32_t)base + (threadIdx.x & 31);
        const bool in = base + (threadIdx.x & 31) < n;
        const float t = in ? depth[i] : 0.0f, gi = in ? g[i] : 0.0f;
        const bool hit = t > 0.0f && gi != 0.0f;
        if (!__any_sync(0xFFFFFFFFu, hit)) continue;
        float d[3];
        pixel_ray(c, i, d);
        float o[8];
        const float x = c.eye[0] + t * d[0], y = c.eye[1] + t * d[1], z = c.eye[2] + t * d[2];
        if constexpr (LONG)
            polar_de_grad_long(s, dm.m, hit, x, y, z, tape, o);
        else if (hit)
            polar_de_grad<ADJ_CK>(s, dm.m, x, y, z, adj_tape(adj_smem, s.max_iters, ADJ_CK), o);
        if (!hit) continue;
        const float dn = o[1] * d[0] + o[2] * d[1] + o[3] * d[2];
        if (!(fabsf(dn) > 1e-6f)) continue;  // grazing ray: no stable depth derivative
        float dt[4];
        bool keep = true;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            dt[k] = -o[4 + k] / dn;
            if (cap > 0.0f && !(fabsf(dt[k]) <= cap)) keep = false;
        }
        if (!keep) continue;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float v = gi * dt[k];
            if (v == v && fabsf(v) < 1e30f) acc[k] += v;
        }
    }
    if constexpr (LONG) long_tape_close(&slot, columns);
    block_sums(acc, params);  // the blocks' are added up by k_sum_partials4
}

static CameraDev make_camera(const cg_camera& cam) {
    CameraDev c;
    for (int k = 0; k < 3; ++k) {
        c.eye[k] = cam.eye[k];
    }
    // forward = normalize(target - eye); right = normalize(forward x up); up' = right x forward
    double f[3] = {cam.target[0] - cam.eye[0], cam.target[1] - cam.eye[1],
                   cam.target[2] - cam.eye[2]};
    double fl = sqrt(f[0] * f[0] + f[1] * f[1] + f[2] * f[2]);
    for (double& v : f) v /= fl;
    double r[3] = {f[1] * cam.up[2] - f[2] * cam.up[1], f[2] * cam.up[0] - f[0] * cam.up[2],
                   f[0] * cam.up[1] - f[1] * cam.up[0]};
    double rl = sqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2]);
    for (double& v : r) v /= rl;
    double u[3] = {r[1] * f[2] - r[2] * f[1], r[2] * f[0] - r[0] * f[2], r[0] * f[1] - r[1] * f[0]};
    for (int k = 0; k < 3; ++k) {
        c.fwd[k] = (float)f[k];
        c.right[k] = (float)r[k];
        c.up[k] = (float)u[k];
    }
    c.tan_half = (float)tan(0.5 * (double)cam.fov_y);
    c.width = cam.width;
    c.height = cam.height;
    c.aspect = (float)cam.width / (float)cam.height;
    return c;
}

// "trace_kernel": 1 (default) the pooled march, 0 one pixel per thread.
static int g_trace_kernel = 1;

int set_trace_option(const char* name, int64_t v) {
    if (strcmp(name, "trace_kernel") || v < 0 || v > 1) return 0;
    g_trace_kernel = (int)v;
    return 1;
}

template <int M>
static void launch_trace_pool(const ShapeDev& s, const CameraDev& c, uint32_t max_steps,
                              float eps_scale, float* depth, uint32_t* next, cudaStream_t st) {
    static int per_sm = 0;
    if (!per_sm) {
        int b = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_trace_pool<M>, kTraceBlock, 0) !=
                cudaSuccess ||
            b < 1)
            b = 1;
        per_sm = b;
    }
    const uint64_t n = (uint64_t)c.width * c.height;
    // Four blocks (32 warps) per SM already keep it busy, and a long ray then
    // shares it with fewer others: 1.05 against 1.13 ms with six (fast polar
    // form, 512 x 512), 1.12 with two.
    const unsigned G = grid_for(n, 1, per_sm < 4 ? per_sm : 4);
    const uint64_t share = (n + G - 1) / G;
    k_trace_pool<M><<<G, kTraceBlock, 0, st>>>(s, c, max_steps, eps_scale, depth, next,
                                               (uint32_t)(share < kTraceBlock ? share : kTraceBlock));
}

static cg_status check_camera(const cg_camera* cam) {
    if (!cam || cam->width == 0 || cam->height == 0 || !(cam->fov_y > 0.0f && cam->fov_y < 3.1f) ||
        (uint64_t)cam->width * cam->height > (1ull << 31)) {
        set_error("bad camera");
        return CG_EINVAL;
    }
    return CG_OK;
}

}  // namespace cg

using namespace cg;

extern "C" {

cg_status cg_trace_depth(const cg_shape* shape, const cg_camera* camera, uint32_t max_steps,
                         float eps_scale, uint32_t numerics, float* depth, void* stream) {
    if (!shape || !depth) {
        set_error("NULL argument");
        return CG_EINVAL;
    }
    CG_TRY(check_camera(camera));
    const ShapeDev s = make_shape_dev(*shape);
    const CameraDev c = make_camera(*camera);
    const uint64_t n = (uint64_t)c.width * c.height;
    cudaStream_t st = (cudaStream_t)stream;
    // (no steps, no loop for the pool to step; the polar forms take one)
    if (g_trace_kernel == 0 || (s.max_iters < 1 && s.kind == CG_SHAPE_MANDELBULB)) {
        const unsigned G = grid_for(n, 128, 16);
        switch (mode_of(s, numerics)) {
        case MODE_P8: k_trace<MODE_P8><<<G, 128, 0, st>>>(s, c, max_steps, eps_scale, depth); break;
        case MODE_INT: k_trace<MODE_INT><<<G, 128, 0, st>>>(s, c, max_steps, eps_scale, depth); break;
        case MODE_POLAR: k_trace<MODE_POLAR><<<G, 128, 0, st>>>(s, c, max_steps, eps_scale, depth); break;
        case MODE_POLAR_FAST:
            k_trace<MODE_POLAR_FAST><<<G, 128, 0, st>>>(s, c, max_steps, eps_scale, depth);
            break;
        case MODE_P8_FAST:
            k_trace<MODE_P8_FAST><<<G, 128, 0, st>>>(s, c, max_steps, eps_scale, depth);
            break;
        case MODE_INT_POLY:
            k_trace<MODE_INT_POLY><<<G, 128, 0, st>>>(s, c, max_steps, eps_scale, depth);
            break;
        default: k_trace<MODE_SPHERE><<<G, 128, 0, st>>>(s, c, max_steps, eps_scale, depth); break;
        }
        CG_CHECK_LAUNCH("k_trace");
        return CG_OK;
    }
    // the work queue's counter: the first word of the thread's scratch buffer
    float* scratch = nullptr;
    CG_TRY(acquire_partials(4, st, &scratch));
    uint32_t* next = reinterpret_cast<uint32_t*>(scratch);
    const cudaError_t ze = cudaMemsetAsync(next, 0, sizeof(uint32_t), st);
    if (ze != cudaSuccess) {  // give the scratch buffer back before reporting
        const cg_status rr = release_partials(scratch, st);
        CG_CUDA(ze);
        return rr;
    }
    switch (mode_of(s, numerics)) {
    case MODE_P8: launch_trace_pool<MODE_P8>(s, c, max_steps, eps_scale, depth, next, st); break;
    case MODE_INT: launch_trace_pool<MODE_INT>(s, c, max_steps, eps_scale, depth, next, st); break;
    case MODE_POLAR: launch_trace_pool<MODE_POLAR>(s, c, max_steps, eps_scale, depth, next, st); break;
    case MODE_POLAR_FAST:
        launch_trace_pool<MODE_POLAR_FAST>(s, c, max_steps, eps_scale, depth, next, st);
        break;
    case MODE_P8_FAST:
        launch_trace_pool<MODE_P8_FAST>(s, c, max_steps, eps_scale, depth, next, st);
        break;
    case MODE_INT_POLY:
        launch_trace_pool<MODE_INT_POLY>(s, c, max_steps, eps_scale, depth, next, st);
        break;
    default: launch_trace_pool<MODE_SPHERE>(s, c, max_steps, eps_scale, depth, next, st); break;
    }
    const cudaError_t le = cudaGetLastError();
    CG_TRY(release_partials(scratch, st));
    CG_CUDA(le);
    return CG_OK;
}

cg_status cg_trace_backward_capped(const cg_shape* shape, const cg_camera* camera,
                                   const float* depth, const float* grad_depth, float cap,
                                   float* grad_params, void* stream);

cg_status cg_trace_backward(const cg_shape* shape, const cg_camera* camera, const float* depth,
                            const float* grad_depth, float* grad_params, void* stream) {
    return cg_trace_backward_capped(shape, camera, depth, grad_depth, 0.0f, grad_params, stream);
}

cg_status cg_trace_backward_capped(const cg_shape* shape, const cg_camera* camera,
                                   const float* depth, const float* grad_depth, float cap,
                                   float* grad_params, void* stream) {
    if (!shape || shape->kind != CG_SHAPE_MANDELBULB_POLAR || !depth || !grad_depth ||
        !grad_params) {
        set_error("cg_trace_backward needs the polar shape and device buffers");
        return CG_EINVAL;
    }
    if (shape->max_iters < 1 || shape->max_iters > ADJ_MAX_ITERS) {
        set_error("cg_trace_backward supports 1 <= max_iters <= %d", ADJ_MAX_ITERS);
        return CG_EINVAL;
    }
    if (!(cap >= 0.0f)) {
        set_error("cg_trace_backward_capped: cap must be >= 0 (0: no cap)");
        return CG_EINVAL;
    }
    CG_TRY(check_camera(camera));
    const ShapeDev s = make_shape_dev(*shape);
    const CameraDev c = make_camera(*camera);
    const Dm3 dm = rotation_derivatives(*shape);
    cudaStream_t st = (cudaStream_t)stream;
    const uint64_t n = (uint64_t)c.width * c.height;
    const bool lng = takes_long_tape(shape->max_iters);
    size_t smem = adj_tape_bytes(shape->max_iters, ADJ_CK, ADJ_BLOCK);
    auto kernel = lng ? k_trace_backward<true> : k_trace_backward<false>;
    unsigned G = 0;
    CG_TRY(lng ? long_launch_shape(kernel, shape->max_iters, n, &smem, &G)
               : adj_launch_shape(kernel, ADJ_BLOCK, smem, n, &G));
    float* partial = nullptr;
    CG_TRY(acquire_partials((size_t)G * 8, st, &partial));
    kernel<<<G, ADJ_BLOCK, smem, st>>>(s, c, dm, depth, grad_depth, cap,
                               reinterpret_cast<double*>(partial));
    cg_status rs = cuda_status(cudaGetLastError(), "k_trace_backward", __FILE__, __LINE__);
    if (rs == CG_OK) rs = launch_sum_partials4(partial, G, grad_params, st);
    const cg_status rr = release_partials(partial, st);
    return rs == CG_OK ? rr : rs;
}

}  // extern "C"
