// shifted_math.cuh -- storage access and arithmetic of the shifted-storage
// kernels (g_k = f_k - w_k in FP32 or FP16, collision in FP32).
#pragma once
#include "lbm_device.cuh"

namespace lbm {

template <typename T> struct SV;
// rnd: the value as the storage type would hold it. Pre-collision values that
// are computed rather than loaded (bounce-back interpolation, edge BCs) are
// rounded to the storage type before the collision, so a run split into
// chunks (whose boundaries store and reload them) gives the same bits.
// ld2 / st2: two adjacent nodes of one row (an even column: the pair is 8- or
// 4-byte aligned because the pitch and the planes are multiples of 64 nodes).
template <> struct SV<float> {
    static __device__ __forceinline__ float ld(const float *p) { return __ldg(p); }
    static __device__ __forceinline__ float ld_plain(const float *p) { return *p; }
    static __device__ __forceinline__ void st(float *p, float v) { *p = v; }
    static __device__ __forceinline__ float rnd(float v) { return v; }
    static __device__ __forceinline__ float2 ld2(const float *p) { return __ldg((const float2 *)p); }
    static __device__ __forceinline__ float2 ld2_plain(const float *p) { return *(const float2 *)p; }
    static __device__ __forceinline__ void st2(float *p, float2 v) { *(float2 *)p = v; }
};
template <> struct SV<__half> {
    static __device__ __forceinline__ float ld(const __half *p) { return __half2float(__ldg(p)); }
    static __device__ __forceinline__ float ld_plain(const __half *p) { return __half2float(*p); }
    static __device__ __forceinline__ void st(__half *p, float v) { *p = __float2half_rn(v); }
    static __device__ __forceinline__ float rnd(float v) { return __half2float(__float2half_rn(v)); }
    static __device__ __forceinline__ float2 ld2(const __half *p) { return __half22float2(__ldg((const __half2 *)p)); }
    static __device__ __forceinline__ float2 ld2_plain(const __half *p) { return __half22float2(*(const __half2 *)p); }
    static __device__ __forceinline__ void st2(__half *p, float2 v) { *(__half2 *)p = __float22half2_rn(v); }
};

// Loads of the populations a step pulls from. RO: nobody writes them while the
// kernel's grid is resident, so the read-only path may serve them. Not so in a
// chain of programmatic followers (kernels_near.cu), whose grid is resident while
// the one before it still writes what it reads after pdl_wait().
template <typename T, bool RO> __device__ __forceinline__ float ld_src(const T *p) {
    return RO ? SV<T>::ld(p) : SV<T>::ld_plain(p);
}
template <typename T, bool RO> __device__ __forceinline__ float2 ld2_src(const T *p) {
    return RO ? SV<T>::ld2(p) : SV<T>::ld2_plain(p);
}

// ---------------------------------------------------------------- lane math
// The arithmetic of one node (float) or of two adjacent nodes at once (float2,
// Blackwell's packed FP32 instructions). Every operation is one correctly
// rounded IEEE operation with no contraction left to the compiler, so a node
// gets the same bits whichever form, kernel or launch shape computed it.
__device__ __forceinline__ float v_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float v_sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float v_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float v_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
// The hardware's estimate of 1/a, a >= 2^-126, and max and min that keep a NaN.
__device__ __forceinline__ float v_rcp_seed(float a) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
    return r;
}
__device__ __forceinline__ float v_max_nan(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float v_min_nan(float a, float b) {
    float r;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 v_add(float2 a, float2 b) { return __fadd2_rn(a, b); }
// a - b rounded once: b * (-1) is exact.
__device__ __forceinline__ float2 v_sub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
__device__ __forceinline__ float2 v_mul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 v_fma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
// A product that an addition follows. ptxas 13.0 contracts a packed multiply
// and add into one multiply-add although both are written with their own
// rounding (seen in one of the forced kernels: one ulp off in a node of 10^5),
// so the packed product is a multiply-add of -0, which it does not know: 0x8000'0000
// plus a block depth of one less one. (Every block is one deep: launch_follower
// refuses others, the pass kernels are launched with one number. -0 from constant
// memory instead: lid 129 x 129 3.91 -> 4.17 us per step.)
__device__ __forceinline__ float v_mul_alone(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float2 v_mul_alone(float2 a, float2 b) {
    const float nz = __uint_as_float(0x80000000u + (blockDim.z - 1u));
    return __ffma2_rn(a, b, make_float2(nz, nz));
}
__device__ __forceinline__ float2 v_rcp_seed(float2 a) { return make_float2(v_rcp_seed(a.x), v_rcp_seed(a.y)); }
__device__ __forceinline__ float2 v_max_nan(float2 a, float2 b) {
    return make_float2(v_max_nan(a.x, b.x), v_max_nan(a.y, b.y));
}
__device__ __forceinline__ float2 v_min_nan(float2 a, float2 b) {
    return make_float2(v_min_nan(a.x, b.x), v_min_nan(a.y, b.y));
}
__device__ __forceinline__ float2 v_neg(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float v_neg(float a) { return -a; }
template <class V> __device__ __forceinline__ V v_splat(float x);
template <> __device__ __forceinline__ float v_splat<float>(float x) { return x; }
template <> __device__ __forceinline__ float2 v_splat<float2>(float x) { return make_float2(x, x); }

// 8/rho, rho = 1 + dr with lbc's floor (compute_macroscopic_fields.c:27): an
// eighth of it is 1/rho as __frcp_rn rounds it. The hardware's estimate of the
// reciprocal and one Newton step (that intrinsic has a branch, which keeps the
// compiler from interleaving the steps of kernels_multi.cu), both on rho / 8, whose
// reciprocal is a normal number for every finite density; 0 for an infinite one.
// NaN stays NaN.
template <class V> __device__ __forceinline__ V eight_over_density(V dr) {
    const V eighth = v_splat<V>(0.125f);
    const V a = v_max_nan(v_fma(dr, eighth, eighth), v_splat<V>(0.125f * 1e-16f));
    const V r = v_rcp_seed(a);
    return v_fma(r, v_fma(v_neg(v_min_nan(a, v_splat<V>(0x1p125f))), r, v_splat<V>(1.0f)), r);
}

// h1 = fl(3 w1), h5 = (1 - 2 h1) / 4, as the host computes them.
__device__ __forceinline__ void shifted_h(float w1, float &h1, float &h5) {
    h1 = __fmul_rn(3.0f, w1);
    h5 = __fmul_rn(__fsub_rn(1.0f, __fmul_rn(2.0f, h1)), 0.25f);
}

// Shifted moments: delta rho = sum g, j = sum c g (sum c w = 0). Jx, Jy are the
// momentum including half the body force (rho u of lbc); jx, jy without it. u8x,
// u8y: eight times the velocity (eight_over_density); the factor goes into the
// constants of collide_v, and powers of two change no bits.
template <class V>
__device__ __forceinline__ void moments_v(const V g[9], V hFx, V hFy, V &dr, V &u8x, V &u8y, V &Jx, V &Jy, V &jx,
                                          V &jy) {
    dr = v_add(v_add(v_add(v_add(g[0], g[1]), v_add(g[2], g[3])), v_add(v_add(g[4], g[5]), v_add(g[6], g[7]))),
               g[8]);
    jx = v_add(v_add(v_sub(g[1], g[3]), v_sub(g[5], g[6])), v_sub(g[8], g[7]));
    jy = v_sub(v_add(v_sub(g[2], g[4]), v_add(g[5], g[6])), v_add(g[7], g[8]));
    const V inv8 = eight_over_density(dr);
    Jx = v_add(jx, hFx);
    Jy = v_add(jy, hFy);
    u8x = v_mul_alone(Jx, inv8);
    u8y = v_mul_alone(Jy, inv8);
}

// One pair of directions (k, opposite) of the equilibrium (c8: 8 c.u): X = w (dr + 4.5 J c
// - rt) is the even part, h o the odd part, added to X with one rounding
// (X +- h o as FMAs: rounding h o first doubles the FP32 velocity error of a
// Taylor-Green run against FP64). The odd part takes the momentum without
// the half force, o = c.j; the force enters the odd part separately (see
// collide_v).
template <class V>
__device__ __forceinline__ void geq_pair(float w, float h, V dr, V c8, V J, V o, V nrt, V &a, V &b) {
    const V X = v_mul(v_splat<V>(w), v_add(dr, v_fma(v_mul(v_splat<V>(4.5f / 8), J), c8, nrt)));
    a = v_fma(v_splat<V>(h), o, X);
    b = v_fma(v_splat<V>(-h), o, X);
}

// BGK + Guo on shifted populations, g' = g + om (geq - g) + (1 - om/2) F_k,
// with geq_k = w_k (drho + rho (3 c.u + 4.5 (c.u)^2 - 1.5 u.u)) built so that
// its mass and momentum are the node's own by construction: the odd part of
// each pair is h (c.J) with FP32 coefficients h1 = fl(3 w1) and
// h5 = (1 - 2 h1) / 4 whose sum rule 2 h1 + 4 h5 = 1 holds exactly, the linear
// term uses J = rho u directly (no division), and the rest population closes
// the mass. Rounded weights would otherwise bias every collision's momentum by
// ~1e-8 in the same direction, an error that grows linearly with the steps.
//
// With a body force, J = j + F/2 would round F/2 (~1e-7) against j: an error of
// the same sign every step, which drove a forced channel 6.6e-5 away from FP64
// in 20,000 steps. Instead the odd part relaxes towards h (c.j) and the whole
// odd forcing, om h c.F/2 + (1 - om/2) 3 w c.F = h c.F (h = 3 w), is added as
// one small term; the even forcing is (1 - om/2) w S, S = 9 (c.u)(c.F) - 3 u.F.
// The relaxation and the forcing are summed first (one FMA) and added to g with
// a single rounding. Channel 256 x 64 against FP64 after 20,000 steps: u L2
// error 5.0e-7 (6.6e-5 before).
template <class V, bool FORCE>
__device__ __forceinline__ void collide_v(V g[9], const float w[9], float h1, float h5, V dr, V u8x, V u8y,
                                          V Jx, V Jy, V jx, V jy, V om, bool force, float Fx, float Fy) {
    const V nrt = v_mul(v_splat<V>(-1.5f / 8), v_fma(Jx, u8x, v_mul(Jy, u8y)));  // -rho * 1.5 u.u
    // Without a body force j = J exactly: one set of momenta stays live.
    const bool forced = FORCE && force;
    if (!FORCE) {
        jx = Jx;
        jy = Jy;
    }
    V geq[9];
    geq_pair(w[1], h1, dr, u8x, Jx, jx, nrt, geq[1], geq[3]);
    geq_pair(w[2], h1, dr, u8y, Jy, jy, nrt, geq[2], geq[4]);
    geq_pair(w[5], h5, dr, v_add(u8x, u8y), v_add(Jx, Jy), v_add(jx, jy), nrt, geq[5], geq[7]);
    geq_pair(w[6], h5, dr, v_sub(u8y, u8x), v_sub(Jy, Jx), v_sub(jy, jx), nrt, geq[6], geq[8]);
    geq[0] = v_sub(dr, v_add(v_add(v_add(geq[1], geq[3]), v_add(geq[2], geq[4])),
                             v_add(v_add(geq[5], geq[7]), v_add(geq[6], geq[8]))));
    if (!forced) {
        // A force-free case: one FMA per population. Kernels that may see
        // forced cases (FORCE) take this branch per case at run time, so a
        // case gets the same bits alone and in any batch.
#pragma unroll
        for (int k = 0; k < 9; k++) g[k] = v_fma(om, v_sub(geq[k], g[k]), g[k]);
        return;
    }
    const V Fxv = v_splat<V>(Fx), Fyv = v_splat<V>(Fy);
    const V gf = v_fma(v_splat<V>(-0.5f), om, v_splat<V>(1.0f));
    const V n3uF = v_mul(v_splat<V>(-3.0f / 8), v_fma(u8x, Fxv, v_mul(u8y, Fyv)));  // -3 u.F
    g[0] = v_add(g[0], v_fma(om, v_sub(geq[0], g[0]), v_mul(gf, v_mul(v_splat<V>(w[0]), n3uF))));
    const V c8u[4] = {u8x, u8y, v_add(u8x, u8y), v_sub(u8y, u8x)};
    const float cFs[4] = {Fx, Fy, Fx + Fy, Fy - Fx};
    const float hs[4] = {h1, h1, h5, h5};
    const int ka[4] = {1, 2, 5, 6}, kb[4] = {3, 4, 7, 8};
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const V cF = v_splat<V>(cFs[q]);
        const V S = v_fma(v_mul(v_splat<V>(9.0f / 8), c8u[q]), cF, n3uF);
        const V E = v_mul_alone(gf, v_mul(v_splat<V>(w[ka[q]]), S));
        const V O = v_splat<V>(hs[q] * cFs[q]);
        const int a = ka[q], b = kb[q];
        g[a] = v_add(g[a], v_fma(om, v_sub(geq[a], g[a]), v_add(E, O)));
        g[b] = v_add(g[b], v_fma(om, v_sub(geq[b], g[b]), v_sub(E, O)));
    }
}

}  // namespace lbm
