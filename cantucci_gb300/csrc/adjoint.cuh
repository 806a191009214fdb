// adjoint.cuh -- reverse-mode gradient of the real-power polar estimator
// (src/shape/mandelbulb.frag:1-39, rotated), shared by the point kernels
// (adjoint.cu) and the depth-map backward (trace.cu); and its forward-mode
// twin polar_de_tangent (end of file), also used for analytic mesh normals
// (mesh_rows.cuh).
//
// For the polar loop one thread returns, per point,
//   DE, dDE/dp (3), dDE/dpower, dDE/d(euler angles) (3).
// It is the adjoint of the forward loop, not a finite difference: the
// forward pass keeps every step's record in a per-thread tape in shared and
// tensor memory (loops of up to ADJ_LONG_MAX steps), or a checkpoint of (z, dr)
// every CK steps and the records of its last segment in shared memory; never
// in HBM or local memory.  With checkpoints the backward pass walks the
// segments from last to first, recomputes each earlier segment's iterates and
// back-propagates through them: one forward pass, the recompute of all steps
// but the last segment's, and one backward pass.
//
// Per step k (z_k -> z_{k+1} = r^P u(P theta, P phi) + q, dr_{k+1} =
// r^(P-1) P dr_k + 1, r = |z_k|, theta = acos(z_z / r), phi = atan2(y, x)):
//   q_bar     += z_bar
//   g_zr       = z_bar . u,   g_th = zr (z_bar . du/dtheta'),  g_ph = zr (z_bar . du/dphi')
//   r_bar     += g_zr P zr / r + dr_bar P dr (P - 1) r^(P-1) / r
//   P_bar     += g_zr zr ln r + g_th theta + g_ph phi + dr_bar dr r^(P-1) (1 + P ln r)
//   dr_bar     = dr_bar P r^(P-1)
//   z_bar      = r_bar z / r + P g_th grad(theta) + P g_ph grad(phi)
// The final DE = 0.5 r ln r / dr seeds r_bar = 0.5 (ln r + 1) / dr and
// dr_bar = -DE / dr on the z whose |z| is the returned r (the escaping
// iterate, or the stale one of the last step when the loop runs out).
#pragma once

#include <cmath>

#include "common.cuh"
#include "de.cuh"

namespace cg {

constexpr int ADJ_CK = 5;          // default checkpoint interval (steps)
constexpr int ADJ_MAX_ITERS = 64;  // the longest loop a tape is sized for

// dR/d(angle k) for k = a, b, c, row-major, 3 x 9 floats.
struct Dm3 {
    float m[27];
};
Dm3 rotation_derivatives(const cg_shape& c);

struct StepState {
    float x, y, z, dr;
};

// A step's input and the values its forward computation produces.
struct StepDeriv {
    float x, y, z, dr;       // z_k, dr_k
    float r, theta, phi;     // |z_k|, acos(z/r), atan2(y, x)
    float t1, zr;            // r^(P-1), r^P
    float sn, cs, sp, cp;    // sin/cos of P theta and P phi
};
constexpr int STEP_FIELDS = 13;

// The step from `st` with |z| = r and z / r = c (not an escape), recorded
// into `d`: the same operations as polar_step, so the iterate is
// bit-identical.  `last`: the loop ends here and z stays; nothing flows back
// into the z that is not formed, so the record's angles and r^P are 0.
__device__ __forceinline__ void polar_step_rec(const ShapeDev& s, float qx, float qy, float qz,
                                               float r, float c, StepState& st, StepDeriv& d,
                                               bool last) {
    d.x = st.x;
    d.y = st.y;
    d.z = st.z;
    d.dr = st.dr;
    d.r = r;
    const float P = s.power_f;
    d.t1 = powf(r, __fsub_rn(P, 1.0f));
    st.dr = __fadd_rn(__fmul_rn(__fmul_rn(d.t1, P), st.dr), 1.0f);
    if (last) {
        d.theta = d.phi = d.zr = d.sn = d.cs = d.sp = d.cp = 0.0f;
        return;
    }
    d.theta = acosf(c);
    d.phi = atan2f(st.y, st.x);
    d.zr = powf(r, P);
    sincosf(__fmul_rn(d.theta, P), &d.sn, &d.cs);
    sincosf(__fmul_rn(d.phi, P), &d.sp, &d.cp);
    st.x = __fadd_rn(__fmul_rn(d.zr, __fmul_rn(d.sn, d.cp)), qx);
    st.y = __fadd_rn(__fmul_rn(d.zr, __fmul_rn(d.sp, d.sn)), qy);
    st.z = __fadd_rn(__fmul_rn(d.zr, d.cs), qz);
}

// The same step in the fast polar arithmetic (polar_step_fast: one
// branch-free arctangent per angle, SFU powers and sin/cos), recorded.  For
// recomputing a segment from an exact checkpoint: its iterates stay within
// the fast arithmetic's error of the exact ones over the few steps of a
// segment.
__device__ __forceinline__ void polar_step_rec_fast(float P, float qx, float qy, float qz,
                                                    StepState& st, StepDeriv& d) {
    d.x = st.x;
    d.y = st.y;
    d.z = st.z;
    d.dr = st.dr;
    const float rho2 = fmaf(st.x, st.x, st.y * st.y);
    d.r = sqrtf(fmaf(st.z, st.z, rho2));
    d.theta = atan2_fast(sqrtf(rho2), st.z);
    d.phi = atan2_fast(st.y, st.x);
    const float lr = __log2f(d.r);
    d.zr = exp2f(P * lr);
    d.t1 = exp2f((P - 1.0f) * lr);
    st.dr = fmaf(d.t1 * P, st.dr, 1.0f);
    sincos_fast(d.theta * P, &d.sn, &d.cs);
    sincos_fast(d.phi * P, &d.sp, &d.cp);
    st.x = fmaf(d.zr, d.sn * d.cp, qx);
    st.y = fmaf(d.zr, d.sp * d.sn, qy);
    st.z = fmaf(d.zr, d.cs, qz);
}

// 1/x from the hardware estimate and one Newton step (within an ulp).
__device__ __forceinline__ float rcp_nr(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return fmaf(fmaf(-x, y, 1.0f), y, y);
}

// A thread's tape in shared memory: the (z, dr) checkpoint of every CK-th
// step and the records of one segment of CK steps, field-major
// ([slot][field][thread]) so that a warp's accesses fall in distinct banks.
// Shared memory takes run-time slot indices without spilling to local
// memory.  Bytes per block: adj_tape_bytes.
struct AdjTape {
    float4* ck;
    float* seg;
    uint32_t tid, nth;
};

__host__ __device__ constexpr size_t adj_tape_bytes(uint32_t max_iters, int ck, uint32_t nth) {
    return ((size_t)((max_iters + ck - 1) / ck) * 16u + (size_t)STEP_FIELDS * ck * 4u) * nth;
}

__device__ __forceinline__ AdjTape adj_tape(void* smem, uint32_t max_iters, int ck) {
    AdjTape t;
    t.tid = threadIdx.x;
    t.nth = blockDim.x;
    t.ck = reinterpret_cast<float4*>(smem);
    t.seg = reinterpret_cast<float*>(t.ck + (size_t)((max_iters + ck - 1) / ck) * blockDim.x);
    return t;
}

__device__ __forceinline__ void tape_put_ck(const AdjTape& t, uint32_t j, const StepState& st) {
    t.ck[(size_t)j * t.nth + t.tid] = make_float4(st.x, st.y, st.z, st.dr);
}

__device__ __forceinline__ StepState tape_get_ck(const AdjTape& t, uint32_t j) {
    const float4 v = t.ck[(size_t)j * t.nth + t.tid];
    return StepState{v.x, v.y, v.z, v.w};
}

__device__ __forceinline__ void tape_put(const AdjTape& t, uint32_t slot, const StepDeriv& d) {
    float* b = t.seg + (size_t)slot * STEP_FIELDS * t.nth + t.tid;
    const uint32_t n = t.nth;
    b[0] = d.x; b[n] = d.y; b[2 * n] = d.z; b[3 * n] = d.dr; b[4 * n] = d.r;
    b[5 * n] = d.theta; b[6 * n] = d.phi; b[7 * n] = d.t1; b[8 * n] = d.zr;
    b[9 * n] = d.sn; b[10 * n] = d.cs; b[11 * n] = d.sp; b[12 * n] = d.cp;
}

__device__ __forceinline__ StepDeriv tape_get(const AdjTape& t, uint32_t slot) {
    const float* b = t.seg + (size_t)slot * STEP_FIELDS * t.nth + t.tid;
    const uint32_t n = t.nth;
    return StepDeriv{b[0], b[n], b[2 * n], b[3 * n], b[4 * n], b[5 * n], b[6 * n],
                     b[7 * n], b[8 * n], b[9 * n], b[10 * n], b[11 * n], b[12 * n]};
}

// The long tape: of every step what the backward sweep cannot form again from
// its neighbours -- dr, r^(P-1), the two angles and r^P in shared memory, the
// sines and cosines in tensor memory (z_k follows from step k - 1's record and
// q by the step's own operations, r from z_k).  The last step the loop allows
// needs the first two only.  No checkpoints and no recomputed segments.
//
// Tensor memory is 256 KB per SM that nothing else here uses: a thread's row of
// it (its lane in its warp's quarter) holds four columns per step.  With all
// nine values in shared memory 12 warps fit an SM at 15 steps and the kernels
// issued 65 % of the time; with five, 24 do, 80 %.  Gradients of 2 M points near
// the surface at 15 steps 555 -> 430 us, at 10 steps 328 -> 285; batch products
// with their sums, 1 M points, 285 -> 235; the depth map's backward pass,
// 512 x 512, 77 -> 64; up to 20 K points the same (latency).
constexpr int LONG_FIELDS = 5;
// The longest loop that takes it: the last with three blocks per SM (1 M points
// at 30 steps, checkpoints 779 us, long tape 530; at 21, 571 and 338).
constexpr uint32_t ADJ_LONG_MAX = 30;

// (Up to ADJ_CK steps the checkpointed tape holds them all too and needs no
// tensor memory: a 256 x 256 backward pass of 5 steps 21 against 25 us.  At 6
// steps the long tape is ahead, 1 M points 175 -> 92.)
__host__ __device__ constexpr bool takes_long_tape(uint32_t max_iters) {
    return max_iters > (uint32_t)ADJ_CK && max_iters <= ADJ_LONG_MAX;
}

// Columns for the sines and cosines of max_iters - 1 steps: a power of two.
__host__ __device__ constexpr uint32_t long_tape_columns(uint32_t max_iters) {
    return max_iters <= 9 ? 32u : (max_iters <= 17 ? 64u : 128u);
}

constexpr unsigned ADJ_BLOCK = 128;  // threads per block: a warp per quarter of tensor memory

constexpr unsigned LONG_BLOCKS = 7;  // most blocks per SM: 72 registers a thread
// Blocks launched for each that fits: the SMs even out what one of them is late
// (2 M points: 467 us at 1, 444 at 2, 430 at 4 and 425 at 16, but 16 times the
// partial sums cost the sums 17 us more).
constexpr unsigned LONG_WAVES = 4;

// Dynamic shared memory of a block; never so little that more than LONG_BLOCKS
// blocks (at more than 64 columns 4) share an SM's 228 KB, of which every block
// takes 1 KB more, since a block that finds its SM's 512 columns taken waits
// for another to end.
__host__ __device__ constexpr size_t long_tape_bytes(uint32_t max_iters) {
    const size_t b = ((size_t)LONG_FIELDS * (max_iters - 1) + 2u) * 4u * ADJ_BLOCK;
    const size_t least = long_tape_columns(max_iters) > 64u ? 46u * 1024u : 30u * 1024u;
    return b < least ? least : b;
}

struct LongTape {
    float* smem;    // this thread's first word; fields ADJ_BLOCK apart
    uint32_t tmem;  // this warp's tensor memory address
};

// Allocates the block's columns (all its threads call, once).
__device__ __forceinline__ LongTape long_tape_open(float* smem, uint32_t* slot, uint32_t columns) {
    const uint32_t warp = threadIdx.x >> 5;
    if (warp == 0) {
        const uint32_t at = (uint32_t)__cvta_generic_to_shared(slot);
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(at),
                     "r"(columns)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    return {smem + threadIdx.x, *slot + (warp << 21)};  // lanes 32 w of the block's columns
}

__device__ __forceinline__ void long_tape_close(const uint32_t* slot, uint32_t columns) {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (threadIdx.x < 32)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(*slot),
                     "r"(columns));
}

// Four columns of every lane's row; all lanes of the warp together.
__device__ __forceinline__ void tmem_put4(uint32_t at, float a, float b, float c, float d) {
    __syncwarp();
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at),
                 "r"(__float_as_uint(a)), "r"(__float_as_uint(b)), "r"(__float_as_uint(c)),
                 "r"(__float_as_uint(d))
                 : "memory");
}

__device__ __forceinline__ void tmem_put_done() {
    __syncwarp();
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_get4(uint32_t at, float& a, float& b, float& c, float& d) {
    uint32_t u[4];
    __syncwarp();
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3])
                 : "r"(at));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    a = __uint_as_float(u[0]);
    b = __uint_as_float(u[1]);
    c = __uint_as_float(u[2]);
    d = __uint_as_float(u[3]);
}

// Launch shape of a kernel with a per-thread tape in dynamic shared memory
// (opting in above 48 KB): a grid of the blocks that fit on the GPU at once
// (the kernels walk their points grid-stride).
template <class Kernel>
cg_status adj_launch_shape(Kernel kernel, unsigned block, size_t smem, uint64_t n,
                           unsigned* grid) {
    if (smem > 48 * 1024)
        CG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)smem));
    int per_sm = 0;
    CG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, (int)block, smem));
    *grid = grid_for(n, block, (unsigned)(per_sm > 0 ? per_sm : 1));
    return CG_OK;
}

// The same for a kernel with the long tape.  (The occupancy query counts one
// block per SM for any kernel that allocates tensor memory: measured, 7 run.)
template <class Kernel>
cg_status long_launch_shape(Kernel kernel, uint32_t max_iters, uint64_t n, size_t* smem,
                            unsigned* grid) {
    *smem = long_tape_bytes(max_iters);
    if (*smem > 47 * 1024)
        CG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)*smem));
    *grid = grid_for(n, ADJ_BLOCK, LONG_WAVES * (unsigned)(228u * 1024u / (*smem + 1024u)));
    return CG_OK;
}

// The sum over a warp of v[k] in lane k * (32 / M), in a fixed order: with each
// exchange a lane gives half of its values away, so M values take M - 1 + log2(32
// / M) additions instead of 5 M.  An SM adds about two doubles a clock, so a
// warp's addition takes some 16: with 20 of them for four values the sums were a
// tenth of a short pass (a depth map's backward pass of 5 steps, 256 x 256: 19.3
// -> 17.3 us, 512 x 512: 33.7 -> 31.6; the surface term's six values, 100 K points
// of 5 steps: 27.5 -> 23.5).
template <int M>
__device__ __forceinline__ double warp_sums(double (&v)[M]) {
    const uint32_t lane = threadIdx.x & 31;
    int o = 16;
#pragma unroll
    for (int half = M / 2; half >= 1; half /= 2, o /= 2) {
        const bool upper = lane & o;
#pragma unroll
        for (int k = 0; k < half; ++k) {
            const double give = upper ? v[k] : v[k + half];
            v[k] = (upper ? v[k + half] : v[k]) + __shfl_xor_sync(0xFFFFFFFFu, give, o);
        }
    }
#pragma unroll
    for (; o > 0; o /= 2) v[0] += __shfl_xor_sync(0xFFFFFFFFu, v[0], o);
    return v[0];
}

// out[N b + k] = block b's sum of acc[k], in a fixed order; with `whole` (a grid
// of one block) whole[k] instead, rounded.
template <int N>
__device__ __forceinline__ void block_sums(const double (&acc)[N], double* __restrict__ out,
                                           float* __restrict__ whole = nullptr) {
    constexpr int M = N <= 4 ? 4 : 8;
    __shared__ double sums[ADJ_BLOCK / 32][M];
    double v[M];
#pragma unroll
    for (int k = 0; k < M; ++k) v[k] = k < N ? acc[k] : 0.0;
    const double sum = warp_sums<M>(v);
    const uint32_t lane = threadIdx.x & 31;
    if (lane % (32 / M) == 0) sums[threadIdx.x >> 5][lane / (32 / M)] = sum;
    __syncthreads();
    if (threadIdx.x < N) {
        double t = 0.0;
        for (unsigned w = 0; w < ADJ_BLOCK / 32; ++w) t += sums[w][threadIdx.x];
        if (whole) whole[threadIdx.x] = (float)t;
        else out[(size_t)blockIdx.x * N + threadIdx.x] = t;
    }
}

// Backward through one recorded step (the step formulas at the top of this
// file).  `stale` adds the seed of the returned r when the loop ran out and
// this is its last step.  Every FMA is written out, so that the sweep rounds
// alike wherever it is compiled.
__device__ __forceinline__ void polar_back_step(float P, const StepDeriv& z, bool stale,
                                                float r_seed, float& zbx, float& zby, float& zbz,
                                                float& drb, float& qbx, float& qby, float& qbz,
                                                float& Pb) {
    qbx += zbx;  // the "+ q" of this step
    qby += zby;
    qbz += zbz;
    const float inv_r = rcp_nr(z.r);
    const float rho2 = fmaf(z.x, z.x, z.y * z.y);
    const float lnr = __logf(z.r);
    const float g_zr = fmaf(zbz, z.cs, fmaf(zby, z.sn * z.sp, zbx * (z.sn * z.cp)));
    const float g_th = z.zr * fmaf(-zbz, z.sn, fmaf(zby, z.cs * z.sp, zbx * (z.cs * z.cp)));
    const float g_ph = z.zr * z.sn * fmaf(zby, z.cp, -(zbx * z.sp));
    float rb = fmaf(drb * P * z.dr * (P - 1.0f) * z.t1, inv_r, g_zr * P * z.t1);
    if (stale) rb += r_seed;
    Pb += fmaf(drb * z.dr * z.t1, fmaf(P, lnr, 1.0f),
               fmaf(g_ph, z.phi, fmaf(g_zr * z.zr, lnr, g_th * z.theta)));
    drb = drb * P * z.t1;
    const float thb = P * g_th, phb = P * g_ph;
    const float rbr = rb * inv_r;
    zbx = __fmul_rn(rbr, z.x);
    zby = __fmul_rn(rbr, z.y);
    zbz = __fmul_rn(rbr, z.z);
    if (rho2 > 1e-30f) {
        const float inv_rho = rsqrtf(rho2);
        const float rho = rho2 * inv_rho;
        const float inv_rho2 = inv_rho * inv_rho;
        const float inv_r2 = inv_r * inv_r;
        const float k = thb * z.z * inv_r2 * inv_rho;
        zbx = __fadd_rn(zbx, fmaf(k, z.x, -(phb * z.y * inv_rho2)));
        zby = __fadd_rn(zby, fmaf(k, z.y, phb * z.x * inv_rho2));
        zbz = fmaf(-thb * rho, inv_r2, zbz);
    }
}

// out[0..7] from the swept adjoints of z_0 and q: dDE/dp = R q_bar (q = R^T p)
// and, per angle, q_bar . (dR/d(angle))^T p.
__device__ __forceinline__ void grad_outputs(const ShapeDev& s, const float* __restrict__ dm,
                                             float px, float py, float pz, float de, float zbx,
                                             float zby, float zbz, float qbx, float qby, float qbz,
                                             float Pb, float* out) {
    qbx += zbx;  // z_0 = q
    qby += zby;
    qbz += zbz;
    out[0] = x86_nan(de);
    out[1] = fmaf(s.m[2], qbz, fmaf(s.m[1], qby, s.m[0] * qbx));
    out[2] = fmaf(s.m[5], qbz, fmaf(s.m[4], qby, s.m[3] * qbx));
    out[3] = fmaf(s.m[8], qbz, fmaf(s.m[7], qby, s.m[6] * qbx));
    out[4] = Pb;
    for (int a = 0; a < 3; ++a) {
        const float* d = dm + 9 * a;
        const float dqx = fmaf(d[6], pz, fmaf(d[0], px, d[3] * py));
        const float dqy = fmaf(d[7], pz, fmaf(d[1], px, d[4] * py));
        const float dqz = fmaf(d[8], pz, fmaf(d[2], px, d[5] * py));
        out[5 + a] = fmaf(qbz, dqz, fmaf(qbx, dqx, qby * dqy));
    }
}

// DE and its gradient with respect to p, the power and the Euler angles
// (out[0..7]) by reverse mode over `tape` (adj_tape, sized for
// s.max_iters <= ADJ_MAX_ITERS).  The forward pass keeps a checkpoint every
// CK steps and the records of its last segment; the backward pass walks the
// segments from last to first, recomputing every segment but the last from
// its checkpoint (FASTREC: in the fast polar arithmetic).
template <int CK = ADJ_CK, bool FASTREC = false>
__device__ __forceinline__ void polar_de_grad(const ShapeDev& s, const float* __restrict__ dm,
                                              float px, float py, float pz, const AdjTape& tape,
                                              float* out) {
    float qx, qy, qz;
    rotate_point(s, px, py, pz, qx, qy, qz);
    const float P = s.power_f;
    const uint32_t N = s.max_iters;

    // Forward: checkpoints, and every step recorded in its segment slot.
    StepState st = {qx, qy, qz, 1.0f};
    float r = 0.0f;
    uint32_t K = 0;
    bool escaped = false;
    for (uint32_t i = 0; i < N; ++i) {
        if (i % CK == 0) tape_put_ck(tape, i / CK, st);
        const float m2 = magnitude2(st.x, st.y, st.z);
        float c;
        if (FASTREC) {
            // polar_radius with the IEEE operations alone: beside the fast
            // segments the shorter ones cost more than they save (1 M points of 15
            // steps 283 against 287 us).
            r = __fsqrt_rn(m2);
            c = __fdiv_rn(st.z, r);
            escaped = r > s.bailout;
        } else {
            escaped = !polar_radius(s, m2, st.z, r, c);
        }
        if (escaped) break;
        StepDeriv d;
        polar_step_rec(s, qx, qy, qz, r, c, st, d, i + 1 == N);
        tape_put(tape, i % CK, d);
        ++K;
    }
    // st = z_K (escaped) or z_N; r = |z_K| (escaped) or |z_{N-1}| (stale).
    const float dr_fin = st.dr;
    const float ln_r = logf(r);
    const float de = __fdiv_rn(__fmul_rn(0.5f, __fmul_rn(ln_r, r)), dr_fin);
    float r_seed = 0.5f * (ln_r + 1.0f) / dr_fin;
    float drb = -de / dr_fin;
    float zbx = 0.0f, zby = 0.0f, zbz = 0.0f;
    if (escaped && r > 0.0f) {
        const float k = r_seed / r;
        zbx = k * st.x;
        zby = k * st.y;
        zbz = k * st.z;
        r_seed = 0.0f;
    }
    float qbx = 0.0f, qby = 0.0f, qbz = 0.0f, Pb = 0.0f;

    // Backward, segment by segment; the last segment's records are the
    // forward pass's own.
    if (K > 0) {
        const uint32_t last = (K - 1) / CK;
        for (int j = (int)last; j >= 0; --j) {
            const uint32_t k0 = (uint32_t)j * CK;
            const uint32_t k1 = min(k0 + CK, K);
            if ((uint32_t)j != last) {
                StepState t = tape_get_ck(tape, (uint32_t)j);
                for (uint32_t k = k0; k < k1; ++k) {
                    StepDeriv d;
                    if (FASTREC) {
                        polar_step_rec_fast(P, qx, qy, qz, t, d);
                    } else {
                        float rk, c;
                        polar_radius(s, magnitude2(t.x, t.y, t.z), t.z, rk, c);
                        polar_step_rec(s, qx, qy, qz, rk, c, t, d, false);
                    }
                    tape_put(tape, k - k0, d);
                }
            }
            for (int k = (int)k1 - 1; k >= (int)k0; --k) {
                const StepDeriv d = tape_get(tape, (uint32_t)k - k0);
                polar_back_step(P, d, !escaped && (uint32_t)k + 1 == N, r_seed, zbx, zby, zbz,
                                drb, qbx, qby, qbz, Pb);
            }
        }
    }
    grad_outputs(s, dm, px, py, pz, de, zbx, zby, zbz, qbx, qby, qbz, Pb, out);
}

// polar_de_grad over the long tape: the same operations and the same records,
// each formed once.  All 32 lanes of a warp call it (`valid`: the lane has a
// point) and go through the steps together, since tensor memory is read and
// written by whole warps; a lane that has ended writes columns it never reads.
__device__ __forceinline__ void polar_de_grad_long(const ShapeDev& s, const float* __restrict__ dm,
                                                   bool valid, float px, float py, float pz,
                                                   const LongTape& tape, float* out) {
    float qx, qy, qz;
    rotate_point(s, px, py, pz, qx, qy, qz);
    const float P = s.power_f;
    const uint32_t N = s.max_iters;
    constexpr uint32_t n = ADJ_BLOCK;
    float x = qx, y = qy, z = qz, dr = 1.0f, r = 0.0f;
    uint32_t K = 0;
    bool escaped = false, live = valid;
    for (uint32_t k = 0; k < N; ++k) {
        float zr = 0.0f, sn = 0.0f, cs = 0.0f, sp = 0.0f, cp = 0.0f;
        if (live) {
            float c;
            float* b = tape.smem + k * (LONG_FIELDS * n);
            if (!polar_radius(s, magnitude2(x, y, z), z, r, c)) {
                escaped = true;
                live = false;
            } else {
                const float t1 = powf(r, __fsub_rn(P, 1.0f));
                b[0] = dr;
                b[n] = t1;
                dr = __fadd_rn(__fmul_rn(__fmul_rn(t1, P), dr), 1.0f);
                ++K;
                live = k + 1 < N;
            }
            if (live) {
                const float theta = acosf(c), phi = atan2f(y, x);
                zr = powf(r, P);
                sincosf(__fmul_rn(theta, P), &sn, &cs);
                sincosf(__fmul_rn(phi, P), &sp, &cp);
                b[2 * n] = theta;
                b[3 * n] = phi;
                b[4 * n] = zr;
            }
        }
        if (!__any_sync(0xFFFFFFFFu, live)) break;
        tmem_put4(tape.tmem + 4 * k, sn, cs, sp, cp);
        if (live) {
            x = __fadd_rn(__fmul_rn(zr, __fmul_rn(sn, cp)), qx);
            y = __fadd_rn(__fmul_rn(zr, __fmul_rn(sp, sn)), qy);
            z = __fadd_rn(__fmul_rn(zr, cs), qz);
        }
    }
    tmem_put_done();
    const float ln_r = logf(r);
    const float de = __fdiv_rn(__fmul_rn(0.5f, __fmul_rn(ln_r, r)), dr);
    float r_seed = 0.5f * (ln_r + 1.0f) / dr;
    float drb = -de / dr;
    float zbx = 0.0f, zby = 0.0f, zbz = 0.0f;
    if (escaped && r > 0.0f) {
        const float k = r_seed / r;
        zbx = k * x;
        zby = k * y;
        zbz = k * z;
        r_seed = 0.0f;
    }
    float qbx = 0.0f, qby = 0.0f, qbz = 0.0f, Pb = 0.0f;
    const uint32_t top = __reduce_max_sync(0xFFFFFFFFu, K);
    StepDeriv d = {};
    // Step top - 1's sines and cosines (a loop's last step has none: 0).
    if (top > 0 && top < N) tmem_get4(tape.tmem + 4 * (top - 1), d.sn, d.cs, d.sp, d.cp);
    for (uint32_t k = top; k-- > 0;) {
        float sn = 0.0f, cs = 0.0f, sp = 0.0f, cp = 0.0f;  // step k - 1's
        if (k > 0) tmem_get4(tape.tmem + 4 * (k - 1), sn, cs, sp, cp);
        if (k < K) {
            const float* b = tape.smem + k * (LONG_FIELDS * n);
            const bool stale = !escaped && k + 1 == N;
            d.dr = b[0];
            d.t1 = b[n];
            d.theta = stale ? 0.0f : b[2 * n];
            d.phi = stale ? 0.0f : b[3 * n];
            d.zr = stale ? 0.0f : b[4 * n];
            if (k > 0) {  // z_k, by the operations that formed it
                const float zr = *(b - n);  // r^P of step k - 1
                d.x = __fadd_rn(__fmul_rn(zr, __fmul_rn(sn, cp)), qx);
                d.y = __fadd_rn(__fmul_rn(zr, __fmul_rn(sp, sn)), qy);
                d.z = __fadd_rn(__fmul_rn(zr, cs), qz);
            } else {
                d.x = qx;
                d.y = qy;
                d.z = qz;
            }
            float c;
            polar_radius(s, magnitude2(d.x, d.y, d.z), d.z, d.r, c);
            polar_back_step(P, d, stale, r_seed, zbx, zby, zbz, drb, qbx, qby, qbz, Pb);
        }
        d.sn = sn;
        d.cs = cs;
        d.sp = sp;
        d.cp = cp;
    }
    grad_outputs(s, dm, px, py, pz, de, zbx, zby, zbz, qbx, qby, qbz, Pb, out);
}

// Forward (tangent) mode of the same loop: one pass carries the derivative
// of (z, dr) along T directions next to the iterate -- dq = e_x, e_y, e_z
// and, with T = 4, d(power) -- so nothing is stored or recomputed.  The
// loop state and DE are those of polar_de (same exact operations); the
// tangent updates use contracted arithmetic.  Per step and direction:
//   r'   = (z . z') / r
//   th'  = (z_z (x x' + y y') / rho - rho z_z') / r^2,  ph' = (x y' - y x') / rho^2
//   zr'  = P r^(P-1) r' (+ r^P ln r P')
//   Z'   = zr' u + zr ((P th' + th P') du/dTh + (P ph' + ph P') du/dPh) + q'
//   dr'' = P (P-1) r^(P-2) dr r' + P r^(P-1) dr' (+ r^(P-1) dr (1 + P ln r) P')
// and at the end DE' = 0.5 (ln r + 1) r' / dr - DE dr' / dr (the quotient
// rule on DE = 0.5 r ln r / dr).  Outputs as polar_de_grad; with T = 3 there
// is no power direction and out[4] = 0 (the rotation derivatives need only
// the three point directions).  Work: one forward pass plus T tangent
// updates of ~30 operations per step, against polar_de_grad's two forward
// passes plus one backward step.
template <int T, bool Rot = true, bool FAST = false>
__device__ __forceinline__ void polar_de_tangent(const ShapeDev& s, const float* __restrict__ dm,
                                                 float px, float py, float pz, float* out) {
    float qx, qy, qz;
    rotate_point<FAST>(s, px, py, pz, qx, qy, qz);
    const float P = s.power_f;
    float zx = qx, zy = qy, zz = qz, dr = 1.0f, r = 0.0f;
    // tangents: direction k has (tx, ty, tz, tdr); dq_k = e_k for k < 3
    float tx[T], ty[T], tz[T], tdr[T], tr[T];
#pragma unroll
    for (int k = 0; k < T; ++k) {
        tx[k] = k == 0 ? 1.0f : 0.0f;
        ty[k] = k == 1 ? 1.0f : 0.0f;
        tz[k] = k == 2 ? 1.0f : 0.0f;
        tdr[k] = 0.0f;
        tr[k] = 0.0f;
    }
    for (uint32_t i = 0; i < s.max_iters;) {
        // One test finds rho, r and their squares normal: the roots,
        // reciprocals and the quotient z / r then need none of their own (the
        // same bits either way).  It takes in the iterates that escape, so
        // that a warp seldom runs both forms (1.5 M points on the surface 315
        // -> 297 us).
        const float rho2 = zx * zx + zy * zy;
        const float m2 = FAST ? fmaf(zz, zz, rho2) : magnitude2(zx, zy, zz);
        const bool normal = m2 <= s.m2_wide && rho2 >= kPolarMinM2;
        float inv_r, rho, inv_rho, inv_rho2, c;
        if (normal) {
            r = sqrt_rn_normal(m2);
            inv_r = rcp_rn_normal(r);
            rho = sqrt_rn_normal(rho2);
            inv_rho = rcp_rn_normal(rho);
            inv_rho2 = rcp_rn_normal(rho2);
            c = FAST ? 0.0f : div_rn_normal(zz, r);
        } else {
            r = sqrtf(m2);
            inv_r = 1.0f / r;
            rho = sqrtf(rho2);
            const bool off_axis = rho > 1e-30f;
            inv_rho = off_axis ? 1.0f / rho : 0.0f;
            inv_rho2 = off_axis ? 1.0f / rho2 : 0.0f;
            c = FAST ? 0.0f : __fdiv_rn(zz, r);
        }
#pragma unroll
        for (int k = 0; k < T; ++k) tr[k] = (zx * tx[k] + zy * ty[k] + zz * tz[k]) * inv_r;
        if (normal ? m2 > s.m2_max : r > s.bailout) break;
        const float lr = FAST ? __log2f(r) : 0.0f;
        const float t1 = FAST ? exp2f((P - 1.0f) * lr) : powf(r, __fsub_rn(P, 1.0f));
        const float Pt1 = P * t1;
        const float k_dr = Pt1 * (P - 1.0f) * inv_r * dr;  // d(dr')/dr
        float lnr = 0.0f;
        if (T == 4) lnr = FAST ? __logf(r) : logf(r);
#pragma unroll
        for (int k = 0; k < T; ++k) {
            tdr[k] = k_dr * tr[k] + Pt1 * tdr[k];
            if (T == 4 && k == 3) tdr[k] += t1 * dr * (1.0f + P * lnr);  // the power direction
        }
        dr = FAST ? fmaf(t1 * P, dr, 1.0f)
                  : __fadd_rn(__fmul_rn(__fmul_rn(t1, P), dr), 1.0f);
        if (++i == s.max_iters) break;  // nobody reads the last z or its tangents
        float theta, phi, zr, sn, cs, sp, cp;
        if (FAST) {  // polar_step_fast's arithmetic
            theta = atan2_fast(rho, zz);
            phi = atan2_fast(zy, zx);
            zr = exp2f(P * lr);
            sincos_fast(theta * P, &sn, &cs);
            sincos_fast(phi * P, &sp, &cp);
        } else {
            theta = acosf(c);
            phi = atan2f(zy, zx);
            zr = powf(r, P);
            sincosf(__fmul_rn(theta, P), &sn, &cs);
            sincosf(__fmul_rn(phi, P), &sp, &cp);
        }
        // shared factors of the tangent step: u and its derivatives, scaled
        // by zr
        const float inv_r2 = inv_r * inv_r;
        const float ux = sn * cp, uy = sp * sn, uz = cs;
        const float ax = zr * cs * cp, ay = zr * sp * cs, az = -zr * sn;  // zr du/dTh
        const float bx = -zr * sn * sp, by = zr * cp * sn;                // zr du/dPh
#pragma unroll
        for (int k = 0; k < T; ++k) {
            const float th_t = (zz * (zx * tx[k] + zy * ty[k]) * inv_rho - rho * tz[k]) * inv_r2;
            const float ph_t = (zx * ty[k] - zy * tx[k]) * inv_rho2;
            float zr_t = Pt1 * tr[k];
            float Th_t = P * th_t, Ph_t = P * ph_t;
            if (T == 4 && k == 3) {  // the power direction
                zr_t += zr * lnr;
                Th_t += theta;
                Ph_t += phi;
            }
            tx[k] = zr_t * ux + Th_t * ax + Ph_t * bx + (k == 0 ? 1.0f : 0.0f);
            ty[k] = zr_t * uy + Th_t * ay + Ph_t * by + (k == 1 ? 1.0f : 0.0f);
            tz[k] = zr_t * uz + Th_t * az + (k == 2 ? 1.0f : 0.0f);
        }
        if (FAST) {
            zx = fmaf(zr, sn * cp, qx);
            zy = fmaf(zr, sp * sn, qy);
            zz = fmaf(zr, cs, qz);
        } else {
            zx = __fadd_rn(__fmul_rn(zr, __fmul_rn(sn, cp)), qx);
            zy = __fadd_rn(__fmul_rn(zr, __fmul_rn(sp, sn)), qy);
            zz = __fadd_rn(__fmul_rn(zr, cs), qz);
        }
    }
    // tr holds r' of the returned r: the escaping iterate's, or the stale
    // one of the last step when the loop runs out (tdr is then dr_N's).
    const float ln_r = FAST ? __logf(r) : logf(r);
    const float de = FAST ? __fdividef(0.5f * ln_r * r, dr)
                          : __fdiv_rn(__fmul_rn(0.5f, __fmul_rn(ln_r, r)), dr);
    const float c_r = 0.5f * (ln_r + 1.0f) / dr, c_dr = -de / dr;
    float g[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int k = 0; k < T; ++k) g[k] = c_r * tr[k] + c_dr * tdr[k];
    out[0] = x86_nan(de);
    out[1] = s.m[0] * g[0] + s.m[1] * g[1] + s.m[2] * g[2];
    out[2] = s.m[3] * g[0] + s.m[4] * g[1] + s.m[5] * g[2];
    out[3] = s.m[6] * g[0] + s.m[7] * g[1] + s.m[8] * g[2];
    out[4] = g[3];
    if constexpr (Rot) {  // without Rot: out[0..4] only (dm unused)
        for (int a = 0; a < 3; ++a) {
            const float* d = dm + 9 * a;
            const float dqx = d[0] * px + d[3] * py + d[6] * pz;
            const float dqy = d[1] * px + d[4] * py + d[7] * pz;
            const float dqz = d[2] * px + d[5] * py + d[8] * pz;
            out[5 + a] = g[0] * dqx + g[1] * dqy + g[2] * dqz;
        }
    }
}

}  // namespace cg
