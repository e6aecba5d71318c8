// pbd_device.cuh -- device-side parameter block and the per-pair arithmetic of the step.
//
// Everything here restates the reference's device helpers in our own code:
//   Morton hashing          kernel/Hash.h:10-34
//   poly6 / spiky kernels   kernel/Density.h:14-42
//   wall confinement        kernel/Forces.h:19-59
// The parameter block replaces `__constant__ SimulationParameters params`
// (kernel/Globals.h:50-77): it is passed by value to every kernel (kernel parameters live
// in the constant bank), so separate simulations never share a global.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace pbd {

constexpr uint32_t kEmptyCell = 0xFFFFFFFFu;   // UINT_MAX start = empty cell (SortReorder.h:146)

// Per-scene values of the batched form (one simulation holding many independent scenes).
struct SceneParams {
    float rho0;            // Density.restDensity of this scene
    float gravity;         // Forces.gravity of this scene
    float bmin[3], bmax[3];
    uint32_t base;         // first entry of the scene's slice of the cell tables
    uint32_t cells;        // the slice's size: the Morton cube (power-of-two side) that holds its walls
};

struct DevParams {
    uint32_t N;            // numberOfParticles this frame
    uint32_t G;            // maxGrid (cells addressable by the tables)
    uint32_t M;            // maxNeighboursPerParticle (list cap)
    uint32_t K;            // kernelWidthNeighbours (cell shells)
    uint32_t active;       // PBD_ACTIVE_* bits
    uint32_t flags;        // PBD_FLAG_* bits
    int32_t  n_scorr;
    uint32_t far_pairs_zero;  // 1 when pairs beyond every kernel support contribute exactly 0
    float d;               // particleDiameter = 2 r
    float dt, gravity;
    float inv_dt;          // 1 / dt: v = (p - x) / dt as a multiply (Update.h:22)
    float rho0;
    float hs, hp;          // spiky width (x diameter already applied), poly width
    float hp2;             // hp*hp
    float hp_lim;          // hp - 0.001 (poly6's upper bound, Density.h:19)
    float k_scorr;
    float c_visc, e_vort;
    float stiffness, one_minus_stiffness;
    float pos_damp, vel_damp;
    float lambda_eps;
    float bmin[3], bmax[3];
    float poly_inv_den;    // 1 / (0.001 + 64 pi hp^9)   (Density.h:21, double there)
    float spiky_den;       // pi * hs^6                  (Density.h:37)
    float wq;              // poly6(q), the s_corr reference value (Density.h:138)
    float inv_wq;          // 1 / wq
    float inv_spiky_den;   // 1 / spiky_den
    float cut2;            // max(hp, hs, d)^2: beyond it no kernel and no contact is non-zero
    // batched form: scene of each particle (sorted order), each scene's [start, end) in the sorted
    // arrays and its parameters; cells of scene s live at s * G + morton in the tables
    uint32_t batched;
    uint32_t nscenes;
    uint32_t table_size;   // cells in the tables: G, or nscenes * G in the batched form
    const SceneParams* scenes;
    uint32_t* scene_of;
    uint32_t* scene_range;
    // an adjoint's taped frame: the vorticity pass also stores each particle's eta (its
    // sum_j |omega_j - omega_i| / (p_j - p_i + 1e-8)) here; null in every other frame
    float4* eta_tape;
    // every predicted position's w is 1 for the whole frame: applyForces sets it (Forces.h:94), and with
    // collisionType 0 and the frame's own corrections nothing but a 0 is ever added to it (collisionType 1
    // writes 0 there, and corrections that an earlier frame stored may hold what came of that)
    uint32_t unit_w;
    // the predicted positions in steps of 1/512 cell (coarse_pos), kept by every kernel that writes them
    // in a frame whose passes filter lists by them, else null; near_coarse: coarse_near's limit
    uint2* coarse;
    uint32_t near_coarse;
};

// A position in steps of 1/512 cell, clamped to the 128 cells the enclosure's limits leave (x | y << 16,
// z); a coordinate that is not a number goes to the far end, and the sums leave such an entry out.  Two
// positions closer than the cut are also near by coarse_near: rounding moves a difference by at most 1.01 steps
// per axis (clamping by none), coarse_near's packed subtraction another one in x, together 2.5 steps.
__device__ __forceinline__ uint32_t coarse_axis(float c) {
    const float q = c * 512.0f;
    return __float2uint_rn(q == q ? fminf(fmaxf(q, 0.0f), 65535.0f) : 65535.0f);
}
__device__ __forceinline__ uint2 coarse_pos(float4 p) {
    return make_uint2(coarse_axis(p.x) | (coarse_axis(p.y) << 16), coarse_axis(p.z));
}
// Whether two coarse positions may be within the cut (limit = near_coarse; 0: never).  Differences beyond
// 64 cells (the cell-end range) wrap around, in x and y to a smaller one and in the sum of squares modulo
// 2^32: such a pair may count as near, which costs an entry and nothing else.
__host__ __device__ __forceinline__ bool coarse_near(uint2 a, uint2 b, uint32_t limit) {
    const uint32_t d = a.x - b.x, dz = a.y - b.y;
    const int dx = (int)d >> 16, dy = (int)(int16_t)(d & 0xFFFFu);
    return (uint32_t)(dx * dx) + (uint32_t)(dy * dy) + dz * dz < limit;
}

// The scene a particle belongs to, as the walk and the per-scene constants see it.
struct SceneCtx {
    uint32_t base;   // first table entry of the scene's cells
    uint32_t end;    // one past the scene's last particle in the sorted arrays
    uint32_t n;      // particles in the scene (the reference's numberOfParticles)
    float rho0;
    uint32_t cells;  // cells of the scene's slice (Morton keys below it are in the tables)
};

__device__ __forceinline__ SceneCtx scene_ctx(const DevParams& P, uint32_t i) {
    if (!P.batched) return SceneCtx{0u, P.N, P.N, P.rho0, P.G};
    const uint32_t sc = P.scene_of[i];
    const uint32_t s = P.scene_range[2 * sc], e = P.scene_range[2 * sc + 1];
    return SceneCtx{P.scenes[sc].base, e, e - s, P.scenes[sc].rho0, P.scenes[sc].cells};
}

// The scene whose slice holds table entry `key` (slices are in scene order): binary search.
__device__ __forceinline__ uint32_t scene_of_key(const DevParams& P, uint32_t key) {
    uint32_t lo = 0, hi = P.nscenes;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (P.scenes[mid].base <= key) lo = mid; else hi = mid;
    }
    return lo;
}

// ---------------------------------------------------------------- Morton (Hash.h) -----
__device__ __forceinline__ uint32_t expand_bits(uint32_t v) {
    v = (v * 0x00010001u) & 0xFF0000FFu;
    v = (v * 0x00000101u) & 0x0F00F00Fu;
    v = (v * 0x00000011u) & 0xC30C30C3u;
    v = (v * 0x00000005u) & 0x49249249u;
    return v;
}

// Per-axis part of mortonCode: clamp to [0, 1023], truncate, spread.
__device__ __forceinline__ uint32_t morton_axis(float c) {
    c = fminf(fmaxf(c, 0.0f), 1023.0f);
    return expand_bits((uint32_t)c);
}

__device__ __forceinline__ uint32_t morton(float x, float y, float z) {
    return (morton_axis(x) << 2) + (morton_axis(y) << 1) + morton_axis(z);
}

// |r|^2 over xyz with explicit rounding: x*x, then + y*y and + z*z as fused multiply-adds, in that
// order.  The compiler may contract a plain x*x + y*y + z*z differently from one kernel to
// another; this spelling gives every walker (cells, lists, staged copies) the same bits.
__device__ __forceinline__ float dist2(float rx, float ry, float rz) {
    return __fmaf_rn(rz, rz, __fmaf_rn(ry, ry, __fmul_rn(rx, rx)));
}

// Square root, its reciprocal and the reciprocal as one instruction each.  Without .ftz the compiler
// wraps every one in the scaling of denormal inputs (~4 instructions); all normal inputs give the
// same bits either way (checked over all of them), and a denormal squared distance is below every
// kernel's lower limit (0.0001), scaled or flushed.
__device__ __forceinline__ float sqrt_fast(float x) {
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float rsqrt_fast(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float rcp_fast(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Two floats as one operand: an instruction does the arithmetic of two pairs of particles, each half
// rounded as the scalar instruction rounds it.
struct F2 { unsigned long long v; };
__device__ __forceinline__ F2 f2(float a, float b) { F2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ void f2_split(F2 a, float& x, float& y) { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v)); }
__device__ __forceinline__ F2 mul2(F2 a, F2 b) { F2 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v)); return r; }
__device__ __forceinline__ F2 sub2(F2 a, F2 b) {   // a - b = b * (-1) + a, rounded once
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(b.v), "l"(f2(-1.0f, -1.0f).v), "l"(a.v));
    return r;
}

// ---------------------------------------------------------- pair kernels (Density.h) --
// poly6Viscosity: W = 315 t^3 t^3 / den, t = hp^2 - d^2, for 0.001 < d < hp - 0.001.  Selected, not
// branched: the lanes of a warp disagree on the range.
__device__ __forceinline__ float poly6(const DevParams& P, float dist) {
    const float t = __fsub_rn(P.hp2, __fmul_rn(dist, dist));
    const float t3 = t * t * t;
    const float w = (315.0f * t3 * t3) * P.poly_inv_den;
    return (dist > 0.001f && dist < P.hp_lim) ? w : 0.0f;
}

// Scalar part of spiky: 15 (hs - d)^2 / (pi hs^6) / |r|_4, so that grad = s * r (r = pi - pj,
// normalised over all four lanes as the float4 normalize of the reference does).
__device__ __forceinline__ float spiky_scale(const DevParams& P, float dist, float r2w) {
    const float a = P.hs - dist;
    const float s = 15.0f * (a * a * P.inv_spiky_den) * rsqrt_fast(r2w);
    return (dist > 0.0001f && a > 0.0001f) ? s : 0.0f;
}

// poly6 and spiky_scale of two pairs without their ranges (the caller tests them), the same products in
// the same order.
__device__ __forceinline__ F2 poly6_open(const DevParams& P, F2 dist) {
    const F2 t = sub2(f2(P.hp2, P.hp2), mul2(dist, dist));
    const F2 t3 = mul2(mul2(t, t), t);
    return mul2(mul2(mul2(f2(315.0f, 315.0f), t3), t3), f2(P.poly_inv_den, P.poly_inv_den));
}
__device__ __forceinline__ F2 spiky_open(const DevParams& P, F2 a, F2 inv_r) {   // a = hs - |r|
    return mul2(mul2(f2(15.0f, 15.0f), mul2(mul2(a, a), f2(P.inv_spiky_den, P.inv_spiky_den))), inv_r);
}

// Integer power by repeated multiplication (the reference's pow(float, int)): r = 1, then
// r *= x |n| times.  The usual exponents are spelled out with the same products in the same
// order (1 * x = x exactly), without the loop.
__device__ __forceinline__ float powi(float x, int n) {
    if (n == 4) return ((x * x) * x) * x;   // config.txt's nSCorr: one test before the others
    switch (n) {
        case 0: return 1.0f;
        case 1: return x;
        case 2: return x * x;
        case 3: return (x * x) * x;
        default: break;
    }
    int m = n < 0 ? -n : n;
    float r = 1.0f;
    for (int k = 0; k < m; ++k) r *= x;
    return n < 0 ? 1.0f / r : r;
}

}  // namespace pbd
