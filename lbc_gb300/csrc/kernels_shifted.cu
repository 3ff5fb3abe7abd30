// kernels_shifted.cu -- fused step with populations stored as shifted deviations
// g_k = f_k - w_k in FP32 or FP16 and the collision done in FP32.
//
// Same pull structure as the exact FP64 step (kernels_exact.cu): stream, halfway /
// interpolated / moving-wall bounce-back, stale slots off non-periodic edges, MEM
// force, moments, BGK + Guo collision. Storing g instead of f keeps the relative
// precision of the small deviations from the rest state; FP64 is used only for the
// force reduction and the band values handed to the edge BCs.
#include <algorithm>
#include <cmath>

#include "bc_shifted.cuh"
#include "kernels.h"
#include "lbm_device.cuh"
#include "pdl.cuh"
#include "reduce.cuh"
#include "shifted_node.cuh"

namespace lbm {

// Flag bits that take a node off the pair path: a solid or off-grid pull
// source, solid, edge-BC band or BC-written, cut links.
constexpr uint32_t kSpecialFlags = NF_SPECIAL_MASK | NF_SOLID | NF_BAND | NF_BCW | NF_LINKS;

// The pair (i0, i0 + 1) of row j when both nodes exist and neither is
// special; nothing otherwise (those nodes are on the case's special-node
// list). A bit per 64-node row segment (one warp's pairs) says the whole
// segment is clean; only other segments read their flag words, issued
// together with the pair's loads (measured: 64 ducts 58.5 -> 62.0 GLUPS,
// channels +1-2 %).
template <typename T, typename I, bool FLAGS, bool COLLIDE, bool FORCE>
__device__ __forceinline__ void step_pair_clean(const FastStepParams &fp, int i0, int j) {
    const StepParams &p = fp.s;
    if (i0 + 1 >= p.Nx) return;
    uint32_t f2 = 0;
    bool clean = !FLAGS;
    if (FLAGS) {
        const uint32_t wrd = __ldg(p.seg_clean + (size_t)j * p.seg_words + (i0 >> 11));
        clean = (wrd >> ((i0 >> 6) & 31)) & 1u;
        if (!clean) f2 = *(const uint32_t *)(p.flags + ((I)j * (I)p.pitch + (I)i0));
    }
    int im = i0 - 1, ip2 = i0 + 2, jm = j - 1, jp = j + 1;
    if (p.px) { if (im < 0) im += p.Nx; if (ip2 >= p.Nx) ip2 -= p.Nx; }
    else { im = max(im, 0); ip2 = min(ip2, p.Nx - 1); }
    if (p.py) { if (jm < 0) jm += p.Ny; if (jp >= p.Ny) jp -= p.Ny; }
    else { jm = max(jm, 0); jp = min(jp, p.Ny - 1); }
    float2 g[9];
    load_pair_shifted<T, I>(p, i0, j, im, ip2, jm, jp, g);
    if (FLAGS && !clean && ((f2 | (f2 >> 16)) & kSpecialFlags) != 0) return;
    collide_store_pair_shifted<T, I, COLLIDE, FORCE>(fp, i0, j, g);
}

// Fully periodic grid without solids or edge BCs: no flag word. Each thread
// steps two adjacent nodes; the last column of an odd-width grid takes the
// per-node path. Five resident blocks per SM (48 registers, no spills) keep
// more loads in flight than the unconstrained 64 registers (measured: FP16
// 135 -> 147 GLUPS on 4096^2).
template <typename T, typename I, bool COLLIDE, bool FORCE>
__global__ void __launch_bounds__(256, 5) k_step_shifted_plain(const FastStepParams fp) {
    pdl_launch_dependents();
    const int i0 = 2 * (blockIdx.x * blockDim.x + threadIdx.x);
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i0 >= fp.s.Nx || j >= fp.s.Ny) return;
    if (i0 + 1 < fp.s.Nx) {
        step_pair_clean<T, I, false, COLLIDE, FORCE>(fp, i0, j);
    } else {
        float mx = 0.f, my = 0.f;
        bool l = false;
        step_node_shifted<T, I, false, COLLIDE, FORCE>(fp, i0, j, mx, my, l);
    }
}

// General geometry (flag word per node): the clean pairs only. The per-node
// path is in k_step_special_shifted, over the case's list of special nodes
// (every node of a pair with a special node, and an odd last column); kept
// out of this kernel, it costs the common path no registers, spills or
// instruction-cache space (measured: cylinder 2048x512 step 21.3 -> 14.2 us
// with the special nodes left out).
template <typename T, typename I, bool COLLIDE, bool FORCE>
__global__ void __launch_bounds__(256, 5) k_step_shifted_geo(const FastStepParams fp) {
    pdl_launch_dependents();
    const int i0 = 2 * (blockIdx.x * blockDim.x + threadIdx.x);
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i0 < fp.s.Nx && j < fp.s.Ny) step_pair_clean<T, I, true, COLLIDE, FORCE>(fp, i0, j);
}

// The special nodes of a case, one per thread, on the per-node path (same
// arithmetic as the pair path, so a node's bits do not depend on which path
// steps it). Wall-link force terms are summed per 32-entry chunk of the list.
// It reads and writes nothing the clean-pair kernel touches: a case alone
// launches it first, as an ordinary launch, with the clean pairs as its
// programmatic follower (pdl.cuh), so their blocks fill the SMs around its
// latency-bound ones; the launch after both is ordinary and, in a graph, has an
// edge from each (Solver::join). (The trigger at the
// start lets the follower launch at once; the wait at the end is then a
// no-op.)
template <typename T, typename I, bool FLAGS, bool COLLIDE, bool FORCE, bool LINKS>
__global__ void __launch_bounds__(128) k_step_special_shifted(const FastStepParams fp,
                                                              const int2 *__restrict__ nodes, int n) {
    pdl_launch_dependents();
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    float mx = 0.f, my = 0.f;
    bool link = false;
    if (q < n) {
        const int2 ij = nodes[q];
        if (ij.x & kSpecialSolid) solid_nan(fp.s, ij.x & ~kSpecialSolid, ij.y);
        else step_node_shifted<T, I, FLAGS, COLLIDE, FORCE, LINKS>(fp, ij.x, ij.y, mx, my, link);
    }
    if (fp.s.mem_partials)
        chunk_reduce2_store((double)mx, (double)my, link, q >> 5, fp.s.chunk_slot, fp.s.mem_partials);
    pdl_wait();
}

// Batched form (see k_step_batch_exact in kernels_exact.cu): tiles of
// 2^(tws + 1) x 2^(8 - tws) nodes, two adjacent nodes per thread, clean pairs
// only (the special nodes of all cases are k_step_batch_special_shifted's:
// blocks of them spread through this kernel's tile list, on 64 liner ducts
// without cut links, measured 57.4 vs 67.7 GLUPS). Blocks stride through the
// tile list, so the tiles in flight at any moment are neighbours in memory
// (sequential DRAM streams, halo rows shared through L2).
template <typename T, typename I, bool FORCE, bool ALLFLAGS>
__global__ void __launch_bounds__(256, 4) k_step_batch_shifted(const FastStepParams *__restrict__ sp,
                                                            const int4 *__restrict__ tiles,
                                                            int ntiles, int sel, int tws) {
    pdl_launch_dependents();
    const int tx = threadIdx.x & ((1 << tws) - 1), ty = threadIdx.x >> tws;
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const int4 td = tiles[t];
        const FastStepParams &fp = sp[2 * td.x + sel];
        const int i0 = td.y + 2 * tx, j = td.z + ty;
        // FORCE: some case of the batch has a body force; force-free cases
        // still take their own (force-free) arithmetic per case (collide_v).
        // ALLFLAGS: every case has a flag word, and the flag-free form of the
        // pair step is left out (measured on 64 ducts: 54.4 -> 57.8 GLUPS,
        // from 72 to 12 bytes of spills).
        if (i0 < fp.s.Nx && j < fp.s.Ny) {
            if (ALLFLAGS || fp.s.flags) step_pair_clean<T, I, true, true, FORCE>(fp, i0, j);
            else step_pair_clean<T, I, false, true, FORCE>(fp, i0, j);
        }
    }
}

// The special nodes of every case of a batch: nodes[q] = (case, i, j, chunk),
// each case's list padded to a multiple of 32 entries (padding: i = -1), so
// that a warp holds one chunk of one case and the force partials are those of
// the case alone. LINKS: some case of the batch has cut-link records.
template <typename T, typename I, bool FORCE, bool LINKS>
__global__ void __launch_bounds__(128) k_step_batch_special_shifted(const FastStepParams *__restrict__ sp,
                                                                    const int4 *__restrict__ nodes, int n,
                                                                    int sel) {
    pdl_launch_dependents();
    const int q = (int)blockIdx.x * (int)blockDim.x + (int)threadIdx.x;
    if (q < n) {  // n is a multiple of 32: whole warps
        const int4 e = nodes[q];
        const FastStepParams &fp = sp[2 * e.x + sel];
        float mx = 0.f, my = 0.f;
        bool link = false;
        if (e.y & kSpecialSolid) solid_nan(fp.s, e.y & ~kSpecialSolid, e.z);
        else if (e.y >= 0) {
            if (fp.s.flags) step_node_shifted<T, I, true, true, FORCE, LINKS>(fp, e.y, e.z, mx, my, link);
            else step_node_shifted<T, I, false, true, FORCE, LINKS>(fp, e.y, e.z, mx, my, link);
        }
        if (fp.s.mem_partials)
            chunk_reduce2_store((double)mx, (double)my, link, e.w, fp.s.chunk_slot, fp.s.mem_partials);
    }
    pdl_wait();
}

// finish_pops_shifted from the band, read at L2 (__ldcg), never from a possibly
// stale L1 line.
template <typename T, bool COLLIDE>
__device__ __forceinline__ void finish_node_shifted(const FinishParams &p, int2 ij, int slot) {
    float f[9];
#pragma unroll
    for (int k = 0; k < 9; k++) f[k] = __ldcg(p.bandg + (size_t)k * p.nslots + slot);
    finish_pops_shifted<T, COLLIDE>(p, ij, slot, f);
}

// In-place collision of shifted populations with the stored (FP64) rho/u/v:
// the first step of a run (src/core/collision.c:18-40).
template <typename T>
__global__ void k_collide_shifted(const CollideParams p) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= p.Nx || j >= p.Ny) return;
    const long long node = (long long)j * p.pitch + i;
    if (p.flags && (p.flags[node] & NF_SOLID)) return;
    const size_t dn = (size_t)j * p.Nx + i;
    T *F = (T *)p.f;
    float g[9], wf[9];
#pragma unroll
    for (int k = 0; k < 9; k++) { g[k] = SV<T>::ld_plain(F + k * p.plane + node); wf[k] = (float)p.w[k]; }
    const float om = p.omega ? (float)p.omega[dn] : (float)p.omega0;
    float dr, u8x, u8y, Jx, Jy, jx, jy;
    if (p.from_pops) {
        moments_shifted(g, (float)(0.5 * p.Fx), (float)(0.5 * p.Fy), dr, u8x, u8y, Jx, Jy, jx, jy);
    } else {
        // the stored fields: rho, u = (j + F/2) / rho
        dr = (float)(p.rho[dn] - 1.0);
        u8x = 8.0f * (float)p.ux[dn];
        u8y = 8.0f * (float)p.uy[dn];
        Jx = (float)(p.rho[dn] * p.ux[dn]);
        Jy = (float)(p.rho[dn] * p.uy[dn]);
        jx = (float)(p.rho[dn] * p.ux[dn] - 0.5 * p.Fx);
        jy = (float)(p.rho[dn] * p.uy[dn] - 0.5 * p.Fy);
    }
    float h1, h5;
    shifted_h(wf[1], h1, h5);
    if (p.has_force) collide_v<float, true>(g, wf, h1, h5, dr, u8x, u8y, Jx, Jy, jx, jy, om, true, (float)p.Fx,
                                            (float)p.Fy);
    else collide_v<float, false>(g, wf, h1, h5, dr, u8x, u8y, Jx, Jy, jx, jy, om, false, 0.f, 0.f);
#pragma unroll
    for (int k = 0; k < 9; k++) SV<T>::st(F + k * p.plane + node, g[k]);
}

// ---------------------------------------------------------------- edge BCs
// The Boundary list on the band in FP32 (bc_shifted.cuh): band populations are
// g, previous-step moments come from the FP64 band moments (rho - 1 formed in
// FP64). The impedance wall's mass-spring-damper state and DFT stay FP64.
template <typename T> struct BandAccessorS {
    const StageParams &p;
    const StagePre &c;
    __device__ int slot(int i, int j) const {
        if (i == c.ij.x && j == c.ij.y) return c.slot;
        if (i == c.nij.x && j == c.nij.y) return c.nslot;
        return band_slot(p.colbase, p.rowbase, i, j);
    }
    __device__ bool nb(int i, int j) const { return i == c.nij.x && j == c.nij.y; }
    __device__ double m(int q, int i, int j) const { return p.bandm_prev[(size_t)q * p.nslots + slot(i, j)]; }
    __device__ float get(int i, int j, int k) const { return __ldcg(p.bandg + (size_t)k * p.nslots + slot(i, j)); }
    __device__ void set(int i, int j, int k, float v) const {
        p.bandg[(size_t)k * p.nslots + slot(i, j)] = v;
    }
    __device__ float drho(int i, int j) const { return (float)((nb(i, j) ? c.nrho : m(0, i, j)) - 1.0); }
    __device__ float ux(int i, int j) const { return (float)(nb(i, j) ? c.nux : m(1, i, j)); }
    __device__ float uy(int i, int j) const { return (float)(nb(i, j) ? c.nuy : m(2, i, j)); }
    __device__ float post(int i, int j, int k) const {
        return SV<T>::ld_plain((const T *)p.src + k * p.plane + (long long)j * p.pitch + i);
    }
    __device__ bool solid(int i, int j) const {
        if (i == c.ij.x && j == c.ij.y) return c.solid;
        return (p.flags[(long long)j * p.pitch + i] & NF_SOLID) != 0;
    }
};

// One point of one Boundary entry (src/core/main_lbm.c:49-58) after its
// preload, as stage_point in kernels_exact.cu.
template <typename T>
__device__ __forceinline__ void stage_point_s(const StageParams &p, const StagePre &c, int t, int kind) {
    BandAccessorS<T> a{p, c};
    float w[9];
#pragma unroll
    for (int k = 0; k < 9; k++) w[k] = p.wf[k];
    if (kind == BC_VEL_BOT_REG && c.imp) {
        bc_regularized_s(a, w, t, p.index, t, p.index + 1, false, (float)c.v1, (float)c.v2);
        return;
    }
    bc_apply_s(a, w, kind, p.Nx, p.Ny, p.index, t, c.v1, c.v2);
}

// One stage thread, specialised on the entry's kind (each kind one short
// region of code): preload, wait for the kernels before it, the BC, the
// finish. (Alone, the edge launch is an ordinary launch behind the special
// nodes and the clean pairs; in a batch it follows the special nodes.) An
// instruction-cache warm-up pass before the wait, the same code without its
// stores, paid off while the edge launch overlapped the clean pairs' last
// wave; measured without it: cylinder 2048x512 17.96 -> 16.42 us per step
// in the current order, 64 liner ducts 186.3 -> 184.7 us.
template <typename T, bool COLLIDE, int KIND>
__device__ __forceinline__ void stage_thread_s(const StageParams &p, const FinishParams &f, int t) {
    StagePre c = stage_preload<true>(p, t, KIND);
    pdl_wait();
    stage_point_s<T>(p, c, t, KIND);
    if (c.fin) finish_node_shifted<T, COLLIDE>(f, c.ij, c.slot);
}

template <typename T, bool COLLIDE>
__device__ __forceinline__ void stage_dispatch_s(const StageParams &p, const FinishParams &f, int t) {
    switch (p.kind) {
#define LBM_STAGE_KIND(K) \
    case K: stage_thread_s<T, COLLIDE, K>(p, f, t); break;
    LBM_STAGE_KIND(BC_VEL_IN_ZH) LBM_STAGE_KIND(BC_VEL_OUT_ZH) LBM_STAGE_KIND(BC_VEL_TOP_ZH)
    LBM_STAGE_KIND(BC_VEL_BOT_ZH) LBM_STAGE_KIND(BC_PRES_IN_ZH) LBM_STAGE_KIND(BC_PRES_OUT_ZH)
    LBM_STAGE_KIND(BC_CONV_IN) LBM_STAGE_KIND(BC_CONV_OUT) LBM_STAGE_KIND(BC_PERIODIC_X)
    LBM_STAGE_KIND(BC_PERIODIC_Y) LBM_STAGE_KIND(BC_VEL_IN_REG) LBM_STAGE_KIND(BC_VEL_OUT_REG)
    LBM_STAGE_KIND(BC_VEL_TOP_REG) LBM_STAGE_KIND(BC_VEL_BOT_REG) LBM_STAGE_KIND(BC_PRES_IN_REG)
    LBM_STAGE_KIND(BC_PRES_OUT_REG) LBM_STAGE_KIND(BC_PRES_TOP_REG) LBM_STAGE_KIND(BC_PRES_BOT_REG)
    LBM_STAGE_KIND(BC_VEL_BOT_ZH_FIX)
#undef LBM_STAGE_KIND
    default: pdl_wait(); break;
    }
}

// As k_stage_group / k_stage_batch in kernels_exact.cu.
template <typename T, bool COLLIDE>
__global__ void k_stage_group_shifted(const StageGroup g) {
    if ((int)blockIdx.y >= g.n) {
        pdl_wait();
        if (blockIdx.x == 0 && threadIdx.x < 32) force_reduce_warp(*g.fs, (int)threadIdx.x);
        return;
    }
    const StageParams &p = g.p[blockIdx.y];
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= p.along) return;
    stage_dispatch_s<T, COLLIDE>(p, g.fin, t);
}

template <typename T>
__global__ void k_stage_batch_shifted(const StageParams *__restrict__ list,
                                      const int2 *__restrict__ blk, int sel, int n,
                                      const ForceSlot *__restrict__ fs) {
    const int2 b = blk[blockIdx.x];
    const int e = b.x;
    if (e >= n) {
        pdl_wait();
        if (threadIdx.x < 32) force_reduce_warp(fs[e - n], (int)threadIdx.x);
        return;
    }
    const StageParams &p = list[2 * e + sel];
    const int t = b.y + (int)threadIdx.x;
    if (t >= p.along) return;
    stage_dispatch_s<T, true>(p, *p.fin, t);
}

namespace launch {

cudaError_t stage_group_shifted(const StageGroup &g, int store, bool collide, bool after_bulk, cudaStream_t s) {
    const dim3 grid((g.max_along + 63) / 64, g.n + (g.nfs ? 1 : 0)), b(64);
    if (store == STORE_F32) {
        if (collide) return launch_follower(after_bulk, k_stage_group_shifted<float, true>, grid, b, s, g);
        return launch_follower(after_bulk, k_stage_group_shifted<float, false>, grid, b, s, g);
    }
    if (collide) return launch_follower(after_bulk, k_stage_group_shifted<__half, true>, grid, b, s, g);
    return launch_follower(after_bulk, k_stage_group_shifted<__half, false>, grid, b, s, g);
}

cudaError_t stage_batch_shifted(const StageParams *list, int n, const int2 *blocks, int nblocks,
                                int store, int sel, const ForceSlot *fs, bool after_bulk, cudaStream_t s) {
    if (nblocks == 0) return cudaSuccess;
    const dim3 g(nblocks), b(kStageBatchPoints);
    if (store == STORE_F32)
        return launch_follower(after_bulk, k_stage_batch_shifted<float>, g, b, s, list, blocks, sel, n, fs);
    return launch_follower(after_bulk, k_stage_batch_shifted<__half>, g, b, s, list, blocks, sel, n, fs);
}

cudaError_t collide_shifted(const CollideParams &p, int store, cudaStream_t s) {
    const dim3 b(64, 4);
    const dim3 g((p.Nx + 63) / 64, (p.Ny + 3) / 4);
    if (store == STORE_F32) k_collide_shifted<float><<<g, b, 0, s>>>(p);
    else k_collide_shifted<__half><<<g, b, 0, s>>>(p);
    return cudaGetLastError();
}


template <typename T, typename I, bool FORCE>
static cudaError_t step_shifted_tif(const FastStepParams &p, bool flags, bool collide, bool after, dim3 g, dim3 b,
                                    cudaStream_t s) {
    if (flags) {
        if (collide) return launch_follower(after, k_step_shifted_geo<T, I, true, FORCE>, g, b, s, p);
        return launch_follower(after, k_step_shifted_geo<T, I, false, FORCE>, g, b, s, p);
    }
    if (collide) return launch_follower(after, k_step_shifted_plain<T, I, true, FORCE>, g, b, s, p);
    return launch_follower(after, k_step_shifted_plain<T, I, false, FORCE>, g, b, s, p);
}

// The body force is a template parameter: force-free kernels carry no forcing
// code (fewer registers).
template <typename T, typename I>
static cudaError_t step_shifted_ti(const FastStepParams &p, bool flags, bool collide, bool after, dim3 g, dim3 b,
                                   cudaStream_t s) {
    if (p.s.has_force) return step_shifted_tif<T, I, true>(p, flags, collide, after, g, b, s);
    return step_shifted_tif<T, I, false>(p, flags, collide, after, g, b, s);
}

template <typename T>
static cudaError_t step_shifted_t(const FastStepParams &p, bool flags, bool collide, bool after, dim3 g, dim3 b,
                                  cudaStream_t s) {
    // 32-bit element offsets whenever all nine planes fit.
    if (9LL * p.s.plane < (1LL << 31)) return step_shifted_ti<T, int>(p, flags, collide, after, g, b, s);
    return step_shifted_ti<T, long long>(p, flags, collide, after, g, b, s);
}

cudaError_t step_shifted(const FastStepParams &p, int store, bool flags, bool collide, dim3 block,
                         cudaStream_t s, bool after) {
    // Two nodes per thread along x. after: the programmatic follower of the
    // special-node kernel launched just before it (the two touch disjoint
    // nodes, so it needs no wait).
    const dim3 g((p.s.Nx + 2 * block.x - 1) / (2 * block.x), (p.s.Ny + block.y - 1) / block.y);
    if (store == STORE_F32) return step_shifted_t<float>(p, flags, collide, after, g, block, s);
    return step_shifted_t<__half>(p, flags, collide, after, g, block, s);
}

template <typename T, typename I, bool FORCE, bool LINKS>
static cudaError_t special_shifted_tifl(const FastStepParams &p, const int2 *nodes, int n, bool flags, bool collide,
                                        bool after_bulk, cudaStream_t s) {
    const dim3 g((n + 127) / 128), b(128);
    if (flags) {
        if (collide)
            return launch_follower(after_bulk, k_step_special_shifted<T, I, true, true, FORCE, LINKS>, g, b, s, p,
                                   nodes, n);
        return launch_follower(after_bulk, k_step_special_shifted<T, I, true, false, FORCE, LINKS>, g, b, s, p, nodes,
                               n);
    }
    if (collide)
        return launch_follower(after_bulk, k_step_special_shifted<T, I, false, true, FORCE, LINKS>, g, b, s, p, nodes,
                               n);
    return launch_follower(after_bulk, k_step_special_shifted<T, I, false, false, FORCE, LINKS>, g, b, s, p, nodes, n);
}

template <typename T, typename I, bool FORCE>
static cudaError_t special_shifted_tif(const FastStepParams &p, const int2 *nodes, int n, bool flags, bool collide,
                                       bool after_bulk, cudaStream_t s) {
    if (p.s.links) return special_shifted_tifl<T, I, FORCE, true>(p, nodes, n, flags, collide, after_bulk, s);
    return special_shifted_tifl<T, I, FORCE, false>(p, nodes, n, flags, collide, after_bulk, s);
}

template <typename T>
static cudaError_t special_shifted_t(const FastStepParams &p, const int2 *nodes, int n, bool flags, bool collide,
                                     bool after_bulk, cudaStream_t s) {
    const bool wide = 9LL * p.s.plane >= (1LL << 31);
    if (p.s.has_force) {
        if (wide) return special_shifted_tif<T, long long, true>(p, nodes, n, flags, collide, after_bulk, s);
        return special_shifted_tif<T, int, true>(p, nodes, n, flags, collide, after_bulk, s);
    }
    if (wide) return special_shifted_tif<T, long long, false>(p, nodes, n, flags, collide, after_bulk, s);
    return special_shifted_tif<T, int, false>(p, nodes, n, flags, collide, after_bulk, s);
}

cudaError_t special_shifted(const FastStepParams &p, const int2 *nodes, int n, int store, bool flags, bool collide,
                            bool after_bulk, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    if (store == STORE_F32) return special_shifted_t<float>(p, nodes, n, flags, collide, after_bulk, s);
    return special_shifted_t<__half>(p, nodes, n, flags, collide, after_bulk, s);
}

template <typename T, bool FORCE, bool LINKS>
static cudaError_t special_batch_shifted_tfl(const FastStepParams *sp, const int4 *nodes, int n,
                                             int sel, bool wide, bool after, cudaStream_t s) {
    const dim3 g((n + 127) / 128), b(128);
    if (wide)
        return launch_follower(after, k_step_batch_special_shifted<T, long long, FORCE, LINKS>, g, b, s, sp, nodes,
                               n, sel);
    return launch_follower(after, k_step_batch_special_shifted<T, int, FORCE, LINKS>, g, b, s, sp, nodes, n, sel);
}

template <typename T>
static cudaError_t special_batch_shifted_t(const FastStepParams *sp, const int4 *nodes, int n,
                                           int sel, bool wide, bool force, bool links, bool after, cudaStream_t s) {
    if (force) {
        if (links) return special_batch_shifted_tfl<T, true, true>(sp, nodes, n, sel, wide, after, s);
        return special_batch_shifted_tfl<T, true, false>(sp, nodes, n, sel, wide, after, s);
    }
    if (links) return special_batch_shifted_tfl<T, false, true>(sp, nodes, n, sel, wide, after, s);
    return special_batch_shifted_tfl<T, false, false>(sp, nodes, n, sel, wide, after, s);
}

cudaError_t special_batch_shifted(const FastStepParams *sp, const int4 *nodes, int n, int sel,
                                  int store, bool wide, bool force, bool links, bool after, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    if (n % 32) return cudaErrorInvalidValue;
    if (store == STORE_F32) return special_batch_shifted_t<float>(sp, nodes, n, sel, wide, force, links, after, s);
    return special_batch_shifted_t<__half>(sp, nodes, n, sel, wide, force, links, after, s);
}

template <typename T, bool FORCE, bool ALLFLAGS>
static cudaError_t step_batch_shifted_tfa(const FastStepParams *sp, const int4 *tiles, int ntiles,
                                          int sel, int tws, bool wide, int grid, bool after, cudaStream_t s) {
    if (wide)
        return launch_follower(after, k_step_batch_shifted<T, long long, FORCE, ALLFLAGS>, dim3(grid), dim3(256), s,
                               sp, tiles, ntiles, sel, tws);
    return launch_follower(after, k_step_batch_shifted<T, int, FORCE, ALLFLAGS>, dim3(grid), dim3(256), s, sp, tiles,
                           ntiles, sel, tws);
}

template <typename T, bool FORCE>
static cudaError_t step_batch_shifted_tf(const FastStepParams *sp, const int4 *tiles, int ntiles,
                                         int sel, int tws, bool wide, bool all_flags, int grid, bool after,
                                         cudaStream_t s) {
    if (all_flags) return step_batch_shifted_tfa<T, FORCE, true>(sp, tiles, ntiles, sel, tws, wide, grid, after, s);
    return step_batch_shifted_tfa<T, FORCE, false>(sp, tiles, ntiles, sel, tws, wide, grid, after, s);
}

cudaError_t step_batch_shifted(const FastStepParams *sp, const int4 *tiles,
                               int ntiles, int sel, int tws, int store, bool wide, bool force, bool all_flags,
                               int grid, cudaStream_t s) {
    const bool after_special = false;  // an ordinary launch
    if (ntiles == 0) return cudaSuccess;
    if (tws < 5 || tws > 8) return cudaErrorInvalidValue;
    if (store == STORE_F32) {
        if (force)
            return step_batch_shifted_tf<float, true>(sp, tiles, ntiles, sel, tws, wide, all_flags, grid,
                                                      after_special, s);
        return step_batch_shifted_tf<float, false>(sp, tiles, ntiles, sel, tws, wide, all_flags, grid,
                                                   after_special, s);
    }
    if (force)
        return step_batch_shifted_tf<__half, true>(sp, tiles, ntiles, sel, tws, wide, all_flags, grid,
                                                   after_special, s);
    return step_batch_shifted_tf<__half, false>(sp, tiles, ntiles, sel, tws, wide, all_flags, grid,
                                                after_special, s);
}

int sm_count() {
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    return nsm > 0 ? nsm : 1;
}

int step_batch_shifted_grid(int store) {
    int nb = 0, dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    if (store == STORE_F32) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_step_batch_shifted<float, int, true, false>, 256, 0);
    else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_step_batch_shifted<__half, int, true, false>, 256, 0);
    return nsm * (nb > 0 ? nb : 1);
}

}  // namespace launch
}  // namespace lbm
