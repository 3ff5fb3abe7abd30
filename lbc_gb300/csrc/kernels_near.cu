// kernels_near.cu -- a step's special nodes, its Boundary list and, in passes of
// several steps, the clean pairs near them, in one launch (shifted storage).
//
// Force-free cases take the forced kernels' force-free branch, and grids whose
// nine planes pass 2^31 elements keep the separate launches: eight kernels with
// every BC kind in them are enough to compile.
#include "pdl.cuh"
#include "reduce.cuh"
#include "shifted_node.cuh"

namespace lbm {

// ---- a step's special nodes and its edges in one launch
//
// When the whole Boundary list is one group (no entry reads or writes a node
// that another writes), an entry's thread need not wait for the band: it pulls
// the node that its BC reads itself (its own for Zou-He, the interior
// neighbour's for the others), and edges run beside the special nodes. That
// takes the edge launch, and what it waits for, off every step: cylinder
// 2048 x 512 16.5 -> 11.9 us, 256 x 64 12.4 -> 8.3, liner duct 1500 x 200 13.4 ->
// 7.3.

// The pre-collision populations of one node: what step_node_shifted leaves in
// the band for it.
template <typename T, bool LINKS>
__device__ __forceinline__ void pull_node(const StepParams &p, int i, int j, float g[9]) {
    const T *S = (const T *)p.src, *Old = (const T *)p.stale;
    const int pl = (int)p.plane, node = (int)j * (int)p.pitch + (int)i;
    int im = i - 1, ip = i + 1, jm = j - 1, jp = j + 1;
    if (p.px) { if (im < 0) im += p.Nx; if (ip >= p.Nx) ip -= p.Nx; }
    else { im = max(im, 0); ip = min(ip, p.Nx - 1); }
    if (p.py) { if (jm < 0) jm += p.Ny; if (jp >= p.Ny) jp -= p.Ny; }
    else { jm = max(jm, 0); jp = min(jp, p.Ny - 1); }
    const int r0 = (int)j * (int)p.pitch, rm = (int)jm * (int)p.pitch, rp = (int)jp * (int)p.pitch;
    const int so[9] = {r0 + i, r0 + im, rm + i, r0 + ip, rp + i, rm + im, rm + ip, rp + ip, rp + im};
    const uint16_t fl = p.flags[node];
#pragma unroll
    for (int k = 0; k < 9; k++) g[k] = ld_src<T, false>(S + (int)k * pl + so[k]);
    if (!(fl & (NF_SPECIAL_MASK | NF_SOLID))) return;
    if (fl & NF_SOLID) {
#pragma unroll
        for (int k = 0; k < 9; k++) g[k] = SV<T>::ld_plain(Old + (int)k * pl + node);
        return;
    }
    const Link *lk = LINKS && (fl & NF_LINKS) ? p.links + p.link_off[node] : nullptr;
#pragma unroll
    for (int k = 1; k < 9; k++) {
        if (!(fl & (1u << k))) continue;
        const int si = i - cxk(k), sj = j - cyk(k);
        if ((!p.px && (si < 0 || si >= p.Nx)) || (!p.py && (sj < 0 || sj >= p.Ny))) {
            g[k] = SV<T>::ld_plain(Old + (int)k * pl + node);
            continue;
        }
        const float own = ld_src<T, false>(S + (int)oppk(k) * pl + node);
        float val = own;
        if (lk) {
            const Link L = *lk++;
            if (L.mode == LINK_IBB_LO) val = (float)L.c1 * own + (float)L.c2 * ld_src<T, false>(S + (int)oppk(k) * pl + (int)L.behind);
            else if (L.mode == LINK_IBB_HI) val = (float)L.c1 * own + (float)L.c2 * ld_src<T, false>(S + (int)k * pl + (int)L.behind);
            else if (L.mode == LINK_MOVING) val = own - (float)L.c2;
        }
        g[k] = SV<T>::rnd(val);
    }
}

struct EdgeAccessor {
    const StagePre &c;
    const float *g;   // the node that the entry reads
    float *out;       // the node that it writes
    __device__ float get(int, int, int k) const { return g[k]; }
    __device__ void set(int, int, int k, float v) const { out[k] = v; }
    __device__ float drho(int, int) const { return (float)(c.nrho - 1.0); }
    __device__ float ux(int, int) const { return (float)c.nux; }
    __device__ float uy(int, int) const { return (float)c.nuy; }
    __device__ float post(int, int, int) const { return 0.f; }  // periodic entries: not here
    __device__ bool solid(int, int) const { return c.solid; }
};

template <typename T, bool LINKS, int KIND>
__device__ __forceinline__ void edge_thread(const StepParams &sp, const StageParams &p, const FinishParams &f, int t) {
    const StagePre c = stage_preload<true>(p, t, KIND);
    if (c.solid) return;
    float g[9], out[9], w[9];
    const int2 at = edge_reads_neighbour(KIND) ? c.nij : c.ij;
    pull_node<T, LINKS>(sp, at.x, at.y, g);
#pragma unroll
    for (int k = 0; k < 9; k++) {
        out[k] = g[k];
        w[k] = p.wf[k];
    }
    EdgeAccessor a{c, g, out};
    if (KIND == BC_VEL_BOT_REG && c.imp)
        bc_regularized_s(a, w, t, p.index, t, p.index + 1, false, (float)c.v1, (float)c.v2);
    else
        bc_apply_s(a, w, KIND, p.Nx, p.Ny, p.index, t, c.v1, c.v2);
    finish_pops_shifted<T, true>(f, c.ij, c.slot, out);
}

template <typename T, bool LINKS>
__device__ __forceinline__ void edge_dispatch(const StepParams &sp, const StageParams &p, const FinishParams &f, int t) {
    switch (p.kind) {
#define LBM_EDGE_KIND(K) \
    case K: edge_thread<T, LINKS, K>(sp, p, f, t); break;
    LBM_EDGE_KIND(BC_VEL_IN_ZH) LBM_EDGE_KIND(BC_VEL_OUT_ZH) LBM_EDGE_KIND(BC_VEL_TOP_ZH)
    LBM_EDGE_KIND(BC_VEL_BOT_ZH) LBM_EDGE_KIND(BC_PRES_IN_ZH) LBM_EDGE_KIND(BC_PRES_OUT_ZH)
    LBM_EDGE_KIND(BC_CONV_IN) LBM_EDGE_KIND(BC_CONV_OUT)
    LBM_EDGE_KIND(BC_VEL_IN_REG) LBM_EDGE_KIND(BC_VEL_OUT_REG)
    LBM_EDGE_KIND(BC_VEL_TOP_REG) LBM_EDGE_KIND(BC_VEL_BOT_REG) LBM_EDGE_KIND(BC_PRES_IN_REG)
    LBM_EDGE_KIND(BC_PRES_OUT_REG) LBM_EDGE_KIND(BC_PRES_TOP_REG) LBM_EDGE_KIND(BC_PRES_BOT_REG)
    LBM_EDGE_KIND(BC_VEL_BOT_ZH_FIX)
#undef LBM_EDGE_KIND
    default: break;
    }
}

// A warp's clean pairs of a 64-column segment of one row: mask bit l is the pair
// of lane l.
template <typename T>
__device__ __forceinline__ void step_segment(const FastStepParams &fp, int j, int seg0, uint32_t mask) {
    const StepParams &p = fp.s;
    const int lane = (int)(threadIdx.x & 31), i0 = seg0 + 2 * lane;
    if (!((mask >> lane) & 1u)) return;
    int im = i0 - 1, ip2 = i0 + 2, jm = j - 1, jp = j + 1;
    if (p.px) { if (im < 0) im += p.Nx; if (ip2 >= p.Nx) ip2 -= p.Nx; }
    else { im = max(im, 0); ip2 = min(ip2, p.Nx - 1); }
    if (p.py) { if (jm < 0) jm += p.Ny; if (jp >= p.Ny) jp -= p.Ny; }
    else { jm = max(jm, 0); jp = min(jp, p.Ny - 1); }
    float2 g[9];
    load_pair_shifted<T, int, false>(p, i0, j, im, ip2, jm, jp, g);
    collide_store_pair_shifted<T, int, true, true>(fp, i0, j, g);
}

// Blocks [0, g.n * per): `per` blocks of each Boundary entry; then the special
// nodes, as k_step_special_shifted; then the segments (case, row, first column,
// mask), a warp each. The wait at the start lets it follow the same kernel of
// the step before.
template <typename T, bool LINKS>
__global__ void __launch_bounds__(128) k_near_shifted(const FastStepParams fp, const int2 *__restrict__ nodes, int n,
                                                      const int4 *__restrict__ segs, int nseg, int per,
                                                      const StageGroup g) {
    pdl_launch_dependents();
    pdl_wait();
    const int eb = g.n * per;
    if ((int)blockIdx.x < eb) {
        const StageParams &p = g.p[blockIdx.x / per];
        const int t = (int)(blockIdx.x % per) * 128 + (int)threadIdx.x;
        if (t < p.along) edge_dispatch<T, LINKS>(fp.s, p, g.fin, t);
        return;
    }
    const int sb = eb + (n + 127) / 128;
    if ((int)blockIdx.x >= sb) {
        const int q = ((int)blockIdx.x - sb) * 4 + (int)(threadIdx.x >> 5);
        if (q < nseg) {
            const int4 e = segs[q];
            step_segment<T>(fp, e.y, e.z, (uint32_t)e.w);
        }
        return;
    }
    const int q = ((int)blockIdx.x - eb) * 128 + (int)threadIdx.x;
    float mx = 0.f, my = 0.f;
    bool link = false;
    if (q < n) {
        const int2 ij = nodes[q];
        if (!(ij.x & kSpecialSolid)) step_node_shifted<T, int, true, true, true, LINKS, false>(fp, ij.x, ij.y, mx, my, link);
    }
    if (fp.s.mem_partials)
        chunk_reduce2_store((double)mx, (double)my, link, q >> 5, fp.s.chunk_slot, fp.s.mem_partials);
}

// The same for every case of a batch in one of `nsets` parameter sets per case:
// eblocks[0 .. neb) are the edge lists' runs of 64 points (entry, first point),
// two per block; nodes as k_step_batch_special_shifted's.
template <typename T, bool LINKS>
__global__ void __launch_bounds__(128) k_near_batch_shifted(const FastStepParams *__restrict__ sp, int nsp, int sel,
                                                            const StageParams *__restrict__ list, int nst,
                                                            const int2 *__restrict__ eblocks, int neb,
                                                            const int4 *__restrict__ nodes, int n,
                                                            const int4 *__restrict__ segs, int nseg) {
    pdl_launch_dependents();
    pdl_wait();
    const int eb = (neb + 1) / 2, sb = eb + (n + 127) / 128;
    if ((int)blockIdx.x < eb) {
        const int q = 2 * (int)blockIdx.x + (int)(threadIdx.x >> 6);
        if (q >= neb) return;
        const int2 b = eblocks[q];
        const StageParams &p = list[nst * b.x + sel];
        const int t = b.y + (int)(threadIdx.x & 63);
        if (t < p.along) edge_dispatch<T, LINKS>(*p.step, p, *p.fin, t);
        return;
    }
    if ((int)blockIdx.x >= sb) {
        const int q = ((int)blockIdx.x - sb) * 4 + (int)(threadIdx.x >> 5);
        if (q < nseg) {
            const int4 e = segs[q];
            step_segment<T>(sp[nsp * e.x + sel], e.y, e.z, (uint32_t)e.w);
        }
        return;
    }
    const int q = ((int)blockIdx.x - eb) * 128 + (int)threadIdx.x;
    if (q >= n) return;  // n is a multiple of 32: whole warps
    const int4 e = nodes[q];
    const FastStepParams &fp = sp[nsp * e.x + sel];
    float mx = 0.f, my = 0.f;
    bool link = false;
    if (e.y >= 0 && !(e.y & kSpecialSolid)) {
        if (fp.s.flags) step_node_shifted<T, int, true, true, true, LINKS, false>(fp, e.y, e.z, mx, my, link);
        else step_node_shifted<T, int, false, true, true, LINKS, false>(fp, e.y, e.z, mx, my, link);
    }
}

namespace launch {

template <typename T>
static cudaError_t near_shifted_t(const FastStepParams &p, const int2 *nodes, int n, const int4 *segs, int nseg,
                                  const StageGroup &g, bool after, cudaStream_t s) {
    const int per = (g.max_along + 127) / 128;
    const dim3 grid(g.n * per + (n + 127) / 128 + (nseg + 3) / 4), b(128);
    if (p.s.links) return launch_follower(after, k_near_shifted<T, true>, grid, b, s, p, nodes, n, segs, nseg, per, g);
    return launch_follower(after, k_near_shifted<T, false>, grid, b, s, p, nodes, n, segs, nseg, per, g);
}

cudaError_t near_shifted(const FastStepParams &p, const int2 *nodes, int n, const int4 *segs, int nseg, int store,
                         const StageGroup &g, bool after, cudaStream_t s) {
    if (n == 0 && g.n == 0 && nseg == 0) return cudaSuccess;
    if (9LL * p.s.plane >= (1LL << 31)) return cudaErrorInvalidValue;
    if (store == STORE_F32) return near_shifted_t<float>(p, nodes, n, segs, nseg, g, after, s);
    return near_shifted_t<__half>(p, nodes, n, segs, nseg, g, after, s);
}

template <typename T, bool LINKS>
static cudaError_t near_batch_shifted_tl(const NearBatch &b, bool after, cudaStream_t s) {
    const dim3 grid((b.neb + 1) / 2 + (b.n + 127) / 128 + (b.nseg + 3) / 4), blk(128);
    return launch_follower(after, k_near_batch_shifted<T, LINKS>, grid, blk, s, b.sp, b.nsp, b.sel, b.list, b.nst,
                           b.eblocks, b.neb, b.nodes, b.n, b.segs, b.nseg);
}

cudaError_t near_batch_shifted(const NearBatch &b, int store, bool links, bool after, cudaStream_t s) {
    if (b.neb + b.n + b.nseg == 0) return cudaSuccess;
    if (b.n % 32) return cudaErrorInvalidValue;
    if (store == STORE_F32)
        return links ? near_batch_shifted_tl<float, true>(b, after, s) : near_batch_shifted_tl<float, false>(b, after, s);
    return links ? near_batch_shifted_tl<__half, true>(b, after, s) : near_batch_shifted_tl<__half, false>(b, after, s);
}

}  // namespace launch
}  // namespace lbm
