// shifted_node.cuh -- one node or one pair of nodes of a step in shifted storage,
// shared by the kernels that step them (kernels_shifted.cu, kernels_near.cu).
#pragma once
#include "bc_shifted.cuh"
#include "kernels.h"
#include "lbm_device.cuh"
#include "shifted_math.cuh"

namespace lbm {

// Scalar entry points used by the per-node paths.
__device__ __forceinline__ void moments_shifted(const float g[9], float hFx, float hFy, float &dr,
                                                float &u8x, float &u8y, float &Jx, float &Jy, float &jx, float &jy) {
    moments_v<float>(g, hFx, hFy, dr, u8x, u8y, Jx, Jy, jx, jy);
}

// Rare per-node outputs, kept out of line so the compiler cannot hoist their
// FP64 conversions into every thread's path (FP64 issue is slow on GB300).
template <typename T>
static __device__ __noinline__ void solid_node_outputs(const StepParams &p, int slot, long long node, size_t dn,
                                                uint16_t fl) {
    if (p.write_macro) { p.rho[dn] = NAN; p.ux[dn] = NAN; p.uy[dn] = NAN; }
    if (fl & NF_BAND) {
        // A BC may read a solid neighbour: lbc sees the untouched buffer
        // content and NaN moments there.
        const T *Old = (const T *)p.stale;
#pragma unroll
        for (int k = 0; k < 9; k++) p.bandg[(size_t)k * p.nslots + slot] = SV<T>::ld_plain(Old + k * p.plane + node);
        p.bandm_next[slot] = NAN;
        p.bandm_next[(size_t)p.nslots + slot] = NAN;
        p.bandm_next[2 * (size_t)p.nslots + slot] = NAN;
    }
}


// A solid node off the edge band (kSpecialSolid entries): NaN moments on steps
// that write the fields, as solid_node_outputs writes them.
__device__ __forceinline__ void solid_nan(const StepParams &p, int i, int j) {
    if (!p.write_macro) return;
    const size_t dn = (size_t)j * (size_t)p.Nx + (size_t)i;
    p.rho[dn] = NAN;
    p.ux[dn] = NAN;
    p.uy[dn] = NAN;
}

static __device__ __noinline__ void macro_store(const StepParams &p, size_t dn, int slot, float dr, float ux,
                                         float uy) {
    if (p.write_macro) { p.rho[dn] = 1.0 + (double)dr; p.ux[dn] = ux; p.uy[dn] = uy; }
    if (slot >= 0) {
        p.bandm_next[slot] = 1.0 + (double)dr;
        p.bandm_next[(size_t)p.nslots + slot] = ux;
        p.bandm_next[2 * (size_t)p.nslots + slot] = uy;
    }
}

static __device__ __noinline__ void macro_store_pair(const StepParams &p, size_t dn, float2 dr, float2 ux, float2 uy) {
    p.rho[dn] = 1.0 + (double)dr.x;
    p.rho[dn + 1] = 1.0 + (double)dr.y;
    p.ux[dn] = ux.x;
    p.ux[dn + 1] = ux.y;
    p.uy[dn] = uy.x;
    p.uy[dn + 1] = uy.y;
}

static __device__ __noinline__ float2 omega_pair(const double *omega, size_t dn) {
    return make_float2((float)omega[dn], (float)omega[dn + 1]);
}

// One node of the fused step in shifted storage (solids, bounce-back links,
// stale slots, edge-BC band: everything). I is the element-offset type: int
// whenever all nine planes fit in 2^31 elements (fewer address instructions),
// long long otherwise. LINKS = false: no case of the launch has cut-link
// records (plain bounce-back on every solid link), and the record path is
// left out (measured: 116 -> 64 registers for the batched special-node
// kernel, twice the resident warps).
template <typename T, typename I, bool FLAGS, bool COLLIDE, bool FORCE, bool LINKS = true, bool RO = true>
__device__ __forceinline__ void step_node_shifted(const FastStepParams &fp, int i, int j,
                                                  float &mfx, float &mfy, bool &link) {
    const StepParams &p = fp.s;
    const I node = (I)j * (I)p.pitch + (I)i;
    const size_t dn = (size_t)j * (size_t)p.Nx + (size_t)i;
    const T *S = (const T *)p.src;
    T *Dst = (T *)p.dst;
    const T *Old = (const T *)p.stale;
    const I pl = (I)p.plane;
    // The loads come in three waves of independent loads, not one chain: (1)
    // the flag word, the nine pulled populations, the node's eight own
    // opposite populations, its cut-link offset, its band bases and (without
    // cut-link records) the stale slots of off-grid sources, which the
    // position alone decides; (2) the cut-link records of its flagged
    // directions; (3) the populations behind interpolated links (and the
    // stale slots, with records). Source neighbours are wrapped on periodic axes and
    // clamped otherwise, so that every load of wave 1 is in bounds whatever
    // the flags say. (Measured: the own populations loaded in wave 2, for
    // flagged directions only, cost the channel and the cylinder 2-4 %.)
    int im = i - 1, ip = i + 1, jm = j - 1, jp = j + 1;
    if (p.px) { if (im < 0) im += p.Nx; if (ip >= p.Nx) ip -= p.Nx; }
    else { im = max(im, 0); ip = min(ip, p.Nx - 1); }
    if (p.py) { if (jm < 0) jm += p.Ny; if (jp >= p.Ny) jp -= p.Ny; }
    else { jm = max(jm, 0); jp = min(jp, p.Ny - 1); }
    const I r0 = (I)j * (I)p.pitch, rm = (I)jm * (I)p.pitch, rp = (I)jp * (I)p.pitch;
    const I so[9] = {r0 + i, r0 + im, rm + i, r0 + ip, rp + i, rm + im, rm + ip, rp + ip, rp + im};
    const uint16_t fl = FLAGS ? p.flags[node] : (uint16_t)0;
    float g[9];
#pragma unroll
    for (int k = 0; k < 9; k++) g[k] = ld_src<T, RO>(S + (I)k * pl + so[k]);
    int lo = 0, cb = -1, rb = -1;
    float own[9];
    bool off[9];
    if (FLAGS) {
#pragma unroll
        for (int k = 1; k < 9; k++) own[k] = ld_src<T, RO>(S + (I)oppk(k) * pl + node);
        if (LINKS && p.link_off) lo = p.link_off[node];
        // Without cut-link records, also the band bases and the stale slots
        // of off-grid sources (this node's own destination slots, written by
        // no other thread). With records they stay in the later waves: their
        // registers (96 -> 116 for the per-case kernel) cost more than the
        // latency saved.
        if (!LINKS && p.colbase) { cb = p.colbase[i]; rb = p.rowbase[j]; }
        if (!LINKS) {
#pragma unroll
            for (int k = 1; k < 9; k++) {
                const int si = i - cxk(k), sj = j - cyk(k);
                off[k] = (!p.px && (si < 0 || si >= p.Nx)) || (!p.py && (sj < 0 || sj >= p.Ny));
                if (off[k]) g[k] = SV<T>::ld_plain(Old + (I)k * pl + node);
            }
        }
    }
    int slot = -1;
    if (FLAGS && (fl & NF_BAND)) slot = LINKS ? band_slot(p.colbase, p.rowbase, i, j) : (cb >= 0 ? cb + j : rb + i);
    if (FLAGS && (fl & NF_SOLID)) {
        solid_node_outputs<T>(p, slot, (long long)node, dn, fl);
        return;
    }
    if (FLAGS && (fl & NF_SPECIAL_MASK)) {
        const bool has_links = LINKS && (fl & NF_LINKS) != 0;
        Link L[9];
        int m = 0;
#pragma unroll
        for (int k = 1; k < 9; k++) {
            if (LINKS) {
                const int si = i - cxk(k), sj = j - cyk(k);
                off[k] = (!p.px && (si < 0 || si >= p.Nx)) || (!p.py && (sj < 0 || sj >= p.Ny));
            }
            // link records in direction order, one per flagged on-grid direction
            if ((fl & (1u << k)) && !off[k] && has_links) L[k] = p.links[lo + m++];
        }
        float behind[9];
#pragma unroll
        for (int k = 1; k < 9; k++) {
            behind[k] = 0.f;
            if (!(fl & (1u << k))) continue;
            if (off[k]) {
                if (LINKS) g[k] = SV<T>::ld_plain(Old + (I)k * pl + node);
            } else if (has_links) {
                if (L[k].mode == LINK_IBB_LO) behind[k] = ld_src<T, RO>(S + (I)oppk(k) * pl + (I)L[k].behind);
                else if (L[k].mode == LINK_IBB_HI) behind[k] = ld_src<T, RO>(S + (I)k * pl + (I)L[k].behind);
            }
        }
#pragma unroll
        for (int k = 1; k < 9; k++) {
            if (!(fl & (1u << k)) || off[k]) continue;
            float val = own[k];
            if (has_links) {
                if (L[k].mode == LINK_IBB_LO || L[k].mode == LINK_IBB_HI)
                    val = (float)L[k].c1 * own[k] + (float)L[k].c2 * behind[k];
                else if (L[k].mode == LINK_MOVING)
                    val = own[k] - (float)L[k].c2;
            }
            g[k] = SV<T>::rnd(val);
            // Per-node link sum in FP32 (a few terms); chunk and case sums are FP64.
            const float df = (own[k] + val) + 2.0f * fp.wf[k];
            mfx -= df * cxk(k);
            mfy -= df * cyk(k);
            link = true;
        }
    }
    if (FLAGS && (fl & NF_BAND)) {
#pragma unroll
        for (int k = 0; k < 9; k++) p.bandg[(size_t)k * p.nslots + slot] = g[k];
    }
    if (FLAGS && (fl & NF_BCW)) return;
    float dr, u8x, u8y, Jx, Jy, jx, jy;
    moments_v<float>(g, fp.hFxf, fp.hFyf, dr, u8x, u8y, Jx, Jy, jx, jy);
    if (p.write_macro || slot >= 0) macro_store(p, dn, slot, dr, 0.125f * u8x, 0.125f * u8y);
    if (COLLIDE) {
        const float om = p.omega ? (float)p.omega[dn] : fp.omega0f;
        collide_v<float, FORCE>(g, fp.wf, fp.h1f, fp.h5f, dr, u8x, u8y, Jx, Jy, jx, jy, om, p.has_force != 0,
                                fp.Fxf, fp.Fyf);
    }
#pragma unroll
    for (int k = 0; k < 9; k++) SV<T>::st(Dst + (I)k * pl + node, g[k]);
}

// Two adjacent nodes (i0, i0 + 1) of one row, neither of them special (no
// solid, link, stale slot, band or BC node): pair loads where the pull sources
// are adjacent (c_x = 0), a pair and a single load otherwise (c_x = +-1), packed
// FP32 arithmetic, pair stores. im = source column of i0 - 1, ip2 of i0 + 2
// (wrapped or clamped like the per-node path), so every load is in bounds
// whatever the nodes' flags say.
template <typename T, typename I, bool RO = true>
__device__ __forceinline__ void load_pair_shifted(const StepParams &p, int i0, int j, int im, int ip2, int jm,
                                                  int jp, float2 g[9]) {
    const T *S = (const T *)p.src;
    const I pl = (I)p.plane;
    const I r0 = (I)j * (I)p.pitch + (I)i0, rm = (I)jm * (I)p.pitch, rp = (I)jp * (I)p.pitch;
    const I m0 = rm + (I)i0, p0 = rp + (I)i0;
    float2 a;
    g[0] = ld2_src<T, RO>(S + r0);
    a = ld2_src<T, RO>(S + pl + r0);
    g[1] = make_float2(ld_src<T, RO>(S + pl + (r0 - (I)i0 + (I)im)), a.x);
    g[2] = ld2_src<T, RO>(S + 2 * pl + m0);
    a = ld2_src<T, RO>(S + 3 * pl + r0);
    g[3] = make_float2(a.y, ld_src<T, RO>(S + 3 * pl + (r0 - (I)i0 + (I)ip2)));
    g[4] = ld2_src<T, RO>(S + 4 * pl + p0);
    a = ld2_src<T, RO>(S + 5 * pl + m0);
    g[5] = make_float2(ld_src<T, RO>(S + 5 * pl + rm + (I)im), a.x);
    a = ld2_src<T, RO>(S + 6 * pl + m0);
    g[6] = make_float2(a.y, ld_src<T, RO>(S + 6 * pl + rm + (I)ip2));
    a = ld2_src<T, RO>(S + 7 * pl + p0);
    g[7] = make_float2(a.y, ld_src<T, RO>(S + 7 * pl + rp + (I)ip2));
    a = ld2_src<T, RO>(S + 8 * pl + p0);
    g[8] = make_float2(ld_src<T, RO>(S + 8 * pl + rp + (I)im), a.x);
}

template <typename T, typename I, bool COLLIDE, bool FORCE>
__device__ __forceinline__ void collide_store_pair_shifted(const FastStepParams &fp, int i0, int j, float2 g[9]) {
    const StepParams &p = fp.s;
    T *Dst = (T *)p.dst;
    const I pl = (I)p.plane;
    const I r0 = (I)j * (I)p.pitch + (I)i0;
    float2 dr, u8x, u8y, Jx, Jy, jx, jy;
    moments_v<float2>(g, v_splat<float2>(fp.hFxf), v_splat<float2>(fp.hFyf), dr, u8x, u8y, Jx, Jy, jx, jy);
    const size_t dn = (size_t)j * (size_t)p.Nx + (size_t)i0;
    if (p.write_macro)
        macro_store_pair(p, dn, dr, make_float2(0.125f * u8x.x, 0.125f * u8x.y), make_float2(0.125f * u8y.x, 0.125f * u8y.y));
    if (COLLIDE) {
        const float2 om = p.omega ? omega_pair(p.omega, dn) : v_splat<float2>(fp.omega0f);
        collide_v<float2, FORCE>(g, fp.wf, fp.h1f, fp.h5f, dr, u8x, u8y, Jx, Jy, jx, jy, om, p.has_force != 0,
                                 fp.Fxf, fp.Fyf);
    }
#pragma unroll
    for (int k = 0; k < 9; k++) SV<T>::st2(Dst + (I)k * pl + r0, g[k]);
}

// Moments and collision of a node that an edge BC wrote: pre-collision
// populations f (rounded to the storage type here).
template <typename T, bool COLLIDE>
__device__ __forceinline__ void finish_pops_shifted(const FinishParams &p, int2 ij, int slot, const float f[9]) {
    float g[9], wf[9];
#pragma unroll
    for (int k = 0; k < 9; k++) {
        g[k] = SV<T>::rnd(f[k]);
        wf[k] = p.wf[k];
    }
    float dr, u8x, u8y, Jx, Jy, jx, jy;
    moments_shifted(g, p.hFxf, p.hFyf, dr, u8x, u8y, Jx, Jy, jx, jy);
    const size_t dn = (size_t)ij.y * p.Nx + ij.x;
    const float ux = 0.125f * u8x, uy = 0.125f * u8y;
    if (p.write_macro) { p.rho[dn] = 1.0 + (double)dr; p.ux[dn] = ux; p.uy[dn] = uy; }
    p.bandm_next[slot] = 1.0 + (double)dr;
    p.bandm_next[(size_t)p.nslots + slot] = ux;
    p.bandm_next[2 * (size_t)p.nslots + slot] = uy;
    if (COLLIDE) {
        const float om = p.omega ? (float)p.omega[dn] : p.omega0f;
        float h1, h5;
        shifted_h(wf[1], h1, h5);
        if (p.has_force) collide_v<float, true>(g, wf, h1, h5, dr, u8x, u8y, Jx, Jy, jx, jy, om, true, p.Fxf, p.Fyf);
        else collide_v<float, false>(g, wf, h1, h5, dr, u8x, u8y, Jx, Jy, jx, jy, om, false, 0.f, 0.f);
    }
    T *D = (T *)p.dst;
    const long long node = (long long)ij.y * p.pitch + ij.x;
#pragma unroll
    for (int k = 0; k < 9; k++) SV<T>::st(D + k * p.plane + node, g[k]);
}

}  // namespace lbm
