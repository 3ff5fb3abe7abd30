// kernels_multi.cu -- several time steps per pass over memory (shifted storage).
//
// The one-step kernels read and write every population once per step, and the
// periodic FP32 step runs at the copy bandwidth of the device. Here a warp
// takes a strip of 64 columns, two adjacent nodes per lane, and walks it row by
// row with LV time steps in flight: the row it loads gives level 1 at row r,
// and level t at row r - (t - 1) pulls from the rows of level t - 1 that are
// still in registers (populations with c_y = -1 from the row just made, c_y = 0
// from the one before, c_y = 1 from the one before that), the neighbouring
// columns by warp shuffles. Only the last level is stored. No shared memory, no
// barriers: warps are independent. A level's values next to the strip's ends
// are wrong one column further in per level, so strips overlap by those columns
// (60 of 64 columns are kept with two levels, 56 with three or four) and chunks
// of rows by 2 (LV - 1) rows.
//
// The arithmetic of a node is that of the one-step kernels (shifted_math.cuh),
// with intermediate levels rounded to the storage type as a store would, so
// the populations are the same bits.
//
// 4096^2 FP32: 173.5 us per step one at a time (1.0 of the copy bandwidth, 72
// bytes per node and step), 111.5 with two levels (still bound by memory, 36
// bytes), 71.4 with four: 235 GLUPS, 18 bytes, 4.2 TB/s, bound by the FP32 pipe
// (about 65 % busy) and the latency of a warp's chain of collisions, three
// warps per SM sub-partition at 153 registers. FP16: 112.5 -> 80.4 us. Rows
// fetched three ahead by cp.async through shared memory: FP32 within 3 % either
// way, FP16 6 % slower than the one row ahead in registers.
#include <algorithm>

#include "kernels.h"
#include "lbm_device.cuh"
#include "pdl.cuh"
#include "shifted_math.cuh"

namespace lbm {

// Two adjacent nodes of one population as the storage holds them, in registers.
template <typename T> struct PairOf;
template <> struct PairOf<float> {
    using P = float2;
    static __device__ __forceinline__ P load(const float *p) { return __ldg((const float2 *)p); }
    static __device__ __forceinline__ P load1(const float *a, const float *b) { return make_float2(__ldg(a), __ldg(b)); }
    static __device__ __forceinline__ void store(float *p, P v) { *(float2 *)p = v; }
    static __device__ __forceinline__ void store1(float *p, P v, int h) { *p = h ? v.y : v.x; }
    static __device__ __forceinline__ P pack(float2 v) { return v; }
    static __device__ __forceinline__ float2 value(P v) { return v; }
    // the pair one column to the left: (left lane's second, own first)
    static __device__ __forceinline__ P from_left(P v) {
        return make_float2(__shfl_up_sync(0xffffffffu, v.y, 1), v.x);
    }
    static __device__ __forceinline__ P from_right(P v) {
        return make_float2(v.y, __shfl_down_sync(0xffffffffu, v.x, 1));
    }
};
template <> struct PairOf<__half> {
    using P = uint32_t;
    static __device__ __forceinline__ P load(const __half *p) { return __ldg((const unsigned int *)p); }
    static __device__ __forceinline__ P load1(const __half *a, const __half *b) {
        return (uint32_t)__ldg((const unsigned short *)a) | (uint32_t)__ldg((const unsigned short *)b) << 16;
    }
    static __device__ __forceinline__ void store(__half *p, P v) { *(uint32_t *)p = v; }
    static __device__ __forceinline__ void store1(__half *p, P v, int h) {
        *(unsigned short *)p = (unsigned short)(h ? v >> 16 : v);
    }
    static __device__ __forceinline__ P pack(float2 v) {
        const __half2 h = __float22half2_rn(v);
        return *(const uint32_t *)&h;
    }
    static __device__ __forceinline__ float2 value(P v) { return __half22float2(*(const __half2 *)&v); }
    static __device__ __forceinline__ P from_left(P v) {
        return __byte_perm(__shfl_up_sync(0xffffffffu, v, 1), v, 0x5432);
    }
    static __device__ __forceinline__ P from_right(P v) {
        return __byte_perm(v, __shfl_down_sync(0xffffffffu, v, 1), 0x5432);
    }
};

// Collides two nodes and returns their populations as stored.
template <typename T, bool FORCE>
__device__ __forceinline__ void collide_pair(const FastStepParams &fp, float2 g[9], typename PairOf<T>::P out[9]) {
    float2 dr, u8x, u8y, Jx, Jy, jx, jy;
    moments_v<float2>(g, v_splat<float2>(fp.hFxf), v_splat<float2>(fp.hFyf), dr, u8x, u8y, Jx, Jy, jx, jy);
    collide_v<float2, FORCE>(g, fp.wf, fp.h1f, fp.h5f, dr, u8x, u8y, Jx, Jy, jx, jy, v_splat<float2>(fp.omega0f),
                             fp.s.has_force != 0, fp.Fxf, fp.Fyf);
#pragma unroll
    for (int k = 0; k < 9; k++) out[k] = PairOf<T>::pack(g[k]);
}

// A level's rows still in registers, already shifted to the columns that pull
// them: populations with c_y = 0 of the last row, c_y = 1 of the last two.
template <typename T> struct Rows {
    using P = typename PairOf<T>::P;
    P mid[3];     // 0, 1, 3 of the row before
    P up[3];      // 2, 5, 6 of the row before
    P up2[3];     // 2, 5, 6 of the row before that
};

// deep: null, or a word per row whose bit l says that lane l's pair is stored
// (a case with a flag word; the others are garbage near special nodes).
template <typename T, int LV, bool FORCE, bool EDGE, bool DEEP>
__device__ __forceinline__ void walk_strip(const FastStepParams &fp, const uint32_t *deep, int cb, int keep0, int keep1,
                                           int y0, int y1) {
    using PO = PairOf<T>;
    using P = typename PO::P;
    const StepParams &p = fp.s;
    const T *S = (const T *)p.src;
    T *D = (T *)p.dst;
    const size_t pl = (size_t)p.plane;
    const int lane = (int)(threadIdx.x & 31);
    const int v0 = cb + 2 * lane;  // this lane's columns v0, v0 + 1, before wrapping
    int c0 = v0, c1 = v0 + 1;
    // Wrapped on periodic axes; clamped otherwise, where the values loaded
    // reach no node that is stored.
    if (EDGE && p.px) {
        c0 = (c0 + p.Nx) % p.Nx;
        c1 = (c1 + p.Nx) % p.Nx;
    } else if (EDGE) {
        c0 = min(max(c0, 0), p.Nx - 1);
        c1 = min(max(c1, 0), p.Nx - 1);
    }
    const bool st0 = v0 >= keep0 && v0 < keep1, st1 = v0 + 1 >= keep0 && v0 + 1 < keep1;

    auto row_of = [&](int r) {
        if (DEEP && !p.py) return (uint32_t)min(max(r, 0), p.Ny - 1) * (uint32_t)p.pitch;
        r = r < 0 ? r + p.Ny : r;
        return (uint32_t)(r >= p.Ny ? r - p.Ny : r) * (uint32_t)p.pitch;
    };
    auto load = [&](int r, P q[9]) {
        const uint32_t rm = row_of(r - 1), r0 = row_of(r), rp = row_of(r + 1);
#pragma unroll
        for (int k = 0; k < 9; k++) {
            const uint32_t ro = cyk(k) == 0 ? r0 : cyk(k) > 0 ? rm : rp;
            if (EDGE) q[k] = PO::load1(S + k * pl + (ro + (uint32_t)c0), S + k * pl + (ro + (uint32_t)c1));
            else q[k] = PO::load(S + k * pl + (ro + (uint32_t)c0));
        }
    };
    auto shifted = [&](int k, P v) { return cxk(k) == 0 ? v : cxk(k) > 0 ? PO::from_left(v) : PO::from_right(v); };

    Rows<T> lv[LV > 1 ? LV - 1 : 1];
#pragma unroll
    for (int t = 0; t < LV - 1; t++) {
#pragma unroll
        for (int q = 0; q < 3; q++) lv[t].mid[q] = lv[t].up[q] = lv[t].up2[q] = P{};
    }
    P next[9];
    const int first = y0 - (LV - 1), last = y1 + (LV - 1);
    load(first, next);
#pragma unroll 2
    for (int r = first; r < last; r++) {
        float2 g[9];
#pragma unroll
        for (int k = 0; k < 9; k++) g[k] = PO::value(shifted(k, next[k]));
        if (r + 1 < last) load(r + 1, next);
        P f[9];
        collide_pair<T, FORCE>(fp, g, f);
#pragma unroll
        for (int t = 0; t < LV - 1; t++) {
            // level t + 2 at row r - t - 1
            Rows<T> &w = lv[t];
            const int mid[3] = {0, 1, 3}, up[3] = {2, 5, 6}, dn[3] = {4, 7, 8};
#pragma unroll
            for (int q = 0; q < 3; q++) {
                g[mid[q]] = PO::value(w.mid[q]);
                g[up[q]] = PO::value(w.up2[q]);
                g[dn[q]] = PO::value(shifted(dn[q], f[dn[q]]));
                w.mid[q] = shifted(mid[q], f[mid[q]]);
                w.up2[q] = w.up[q];
                w.up[q] = shifted(up[q], f[up[q]]);
            }
            collide_pair<T, FORCE>(fp, g, f);
        }
        const int row = r - (LV - 1);
        if (row >= y0) {
            const size_t o = (size_t)row * (size_t)p.pitch;
            const bool pair = DEEP ? (__ldg(deep + row) >> lane) & 1u : st0;
#pragma unroll
            for (int k = 0; k < 9; k++) {
                T *d = D + k * pl + o;
                if (DEEP) {
                    if (pair) PO::store(d + v0, f[k]);
                } else if (EDGE) {
                    if (st0) PO::store1(d + v0, f[k], 0);
                    if (st1) PO::store1(d + v0 + 1, f[k], 1);
                } else if (pair) {
                    PO::store(d + v0, f[k]);
                }
            }
        }
    }
}

// Fully periodic grid, no flag word, one omega. Warp = strip x chunk of rows.
template <typename T, int LV, bool FORCE>
__global__ void __launch_bounds__(kMultiThreads) k_multi_plain(const FastStepParams fp, int strips, int height) {
    const int w = (int)(blockIdx.x * (kMultiThreads / 32) + threadIdx.x / 32);
    const int chunk = w / strips, strip = w - chunk * strips;
    const int y0 = chunk * height, y1 = min(y0 + height, fp.s.Ny);
    if (y0 >= y1) return;
    const int halo = multi_halo(LV), width = 64 - 2 * halo;
    const int keep0 = strip * width, keep1 = min(keep0 + width, fp.s.Nx), cb = keep0 - halo;
    if (cb >= 0 && cb + 64 <= fp.s.Nx) walk_strip<T, LV, FORCE, false, false>(fp, nullptr, cb, keep0, keep1, y0, y1);
    else walk_strip<T, LV, FORCE, true, false>(fp, nullptr, cb, keep0, keep1, y0, y1);
}

// A case with a flag word and one omega: the nodes at least LV nodes away from
// any special node (the others are the list kernels', which run beside it:
// its blocks leave registers free on every SM). Cavity 4096^2: 184 us per step
// one at a time, 85 with four levels; 2048^2 50.4 -> 25.6.
template <typename T, int LV, bool FORCE>
__global__ void __launch_bounds__(kMultiThreads) k_multi_geo(const FastStepParams fp, const uint32_t *deep, int strips,
                                                             int height) {
    const int w = (int)(blockIdx.x * (kMultiThreads / 32) + threadIdx.x / 32);
    const int chunk = w / strips, strip = w - chunk * strips;
    const int y0 = chunk * height, y1 = min(y0 + height, fp.s.Ny);
    if (y0 >= y1) return;
    const int halo = multi_halo(LV), width = 64 - 2 * halo;
    const int keep0 = strip * width, keep1 = min(keep0 + width, fp.s.Nx), cb = keep0 - halo;
    deep += (size_t)strip * (size_t)fp.s.Ny;
    if (cb >= 0 && cb + 64 <= fp.s.Nx) walk_strip<T, LV, FORCE, false, true>(fp, deep, cb, keep0, keep1, y0, y1);
    else walk_strip<T, LV, FORCE, true, true>(fp, deep, cb, keep0, keep1, y0, y1);
}

// Every case of a batch: a warp per task.
template <typename T, int LV, bool FORCE>
__global__ void __launch_bounds__(kMultiThreads) k_multi_batch(const FastStepParams *__restrict__ sp, int nsp, int sel,
                                                               const MultiTask *__restrict__ tasks, int ntasks,
                                                               const uint32_t *__restrict__ deep) {
    const int w = (int)(blockIdx.x * (kMultiThreads / 32) + threadIdx.x / 32);
    if (w >= ntasks) return;
    const MultiTask t = tasks[w];
    const FastStepParams &fp = sp[nsp * t.cs + sel];
    const int halo = multi_halo(LV), width = 64 - 2 * halo;
    const int keep0 = t.strip * width, keep1 = min(keep0 + width, fp.s.Nx), cb = keep0 - halo;
    const uint32_t *d = deep + t.deep + (size_t)t.strip * (size_t)fp.s.Ny;
    if (cb >= 0 && cb + 64 <= fp.s.Nx) walk_strip<T, LV, FORCE, false, true>(fp, d, cb, keep0, keep1, t.y0, t.y1);
    else walk_strip<T, LV, FORCE, true, true>(fp, d, cb, keep0, keep1, t.y0, t.y1);
}

// One thread per special node (launch::multi_swap).
template <typename T>
__global__ void k_multi_swap(const int2 *__restrict__ nodes, int n, const uint16_t *__restrict__ flags, int pitch,
                             long long plane, const T *cur, T *other, T *odd, T *even2, int enter) {
    const int q = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (q >= n) return;
    const long long o = (long long)nodes[q].y * pitch + (nodes[q].x & ~kSpecialSolid);
    const bool solid = (flags[o] & NF_SOLID) != 0;
#pragma unroll
    for (int k = 0; k < 9; k++) {
        const long long at = k * plane + o;
        if (enter) {
            odd[at] = other[at];
            if (solid) {
                other[at] = cur[at];
                if (even2) even2[at] = cur[at];
            }
        } else {
            other[at] = odd[at];
        }
    }
}

namespace launch {

template <typename T, int LV>
static cudaError_t multi_load_tl(bool plain, bool force) {
    cudaFuncAttributes a;
    if (plain) return force ? cudaFuncGetAttributes(&a, k_multi_plain<T, LV, true>) : cudaFuncGetAttributes(&a, k_multi_plain<T, LV, false>);
    return force ? cudaFuncGetAttributes(&a, k_multi_geo<T, LV, true>) : cudaFuncGetAttributes(&a, k_multi_geo<T, LV, false>);
}

cudaError_t multi_load(int store, int levels, bool plain, bool force) {
    if (store == STORE_F32) return levels == 2 ? multi_load_tl<float, 2>(plain, force) : multi_load_tl<float, 4>(plain, force);
    return levels == 2 ? multi_load_tl<__half, 2>(plain, force) : multi_load_tl<__half, 4>(plain, force);
}

template <typename T, int LV>
static cudaError_t multi_geo_tl(const FastStepParams &p, const uint32_t *deep, int warps_wanted, cudaStream_t s) {
    const int width = 64 - 2 * multi_halo(LV);
    const int strips = (p.s.Nx + width - 1) / width;
    const int chunks = std::max(1, std::min(p.s.Ny / 4, warps_wanted / strips));
    const int height = (p.s.Ny + chunks - 1) / chunks;
    const long long warps = (long long)strips * ((p.s.Ny + height - 1) / height);
    const unsigned blocks = (unsigned)((warps + kMultiThreads / 32 - 1) / (kMultiThreads / 32));
    if (p.s.has_force) k_multi_geo<T, LV, true><<<blocks, kMultiThreads, 0, s>>>(p, deep, strips, height);
    else k_multi_geo<T, LV, false><<<blocks, kMultiThreads, 0, s>>>(p, deep, strips, height);
    return cudaGetLastError();
}

cudaError_t multi_geo(const FastStepParams &p, int store, int levels, const uint32_t *deep, int warps, cudaStream_t s) {
    if (store == STORE_F32) {
        if (levels == 2) return multi_geo_tl<float, 2>(p, deep, warps, s);
        if (levels == 4) return multi_geo_tl<float, 4>(p, deep, warps, s);
    } else {
        if (levels == 2) return multi_geo_tl<__half, 2>(p, deep, warps, s);
        if (levels == 4) return multi_geo_tl<__half, 4>(p, deep, warps, s);
    }
    return cudaErrorInvalidValue;
}

template <typename T, int LV>
static cudaError_t multi_batch_tl(const FastStepParams *sp, int nsp, int sel, const MultiTask *tasks, int ntasks,
                                  const uint32_t *deep, bool force, cudaStream_t s) {
    const unsigned blocks = (unsigned)((ntasks + kMultiThreads / 32 - 1) / (kMultiThreads / 32));
    if (force) k_multi_batch<T, LV, true><<<blocks, kMultiThreads, 0, s>>>(sp, nsp, sel, tasks, ntasks, deep);
    else k_multi_batch<T, LV, false><<<blocks, kMultiThreads, 0, s>>>(sp, nsp, sel, tasks, ntasks, deep);
    return cudaGetLastError();
}

cudaError_t multi_batch(const FastStepParams *sp, int nsp, int sel, const MultiTask *tasks, int ntasks,
                        const uint32_t *deep, int store, int levels, bool force, cudaStream_t s) {
    if (store == STORE_F32) {
        if (levels == 2) return multi_batch_tl<float, 2>(sp, nsp, sel, tasks, ntasks, deep, force, s);
        if (levels == 4) return multi_batch_tl<float, 4>(sp, nsp, sel, tasks, ntasks, deep, force, s);
    } else {
        if (levels == 2) return multi_batch_tl<__half, 2>(sp, nsp, sel, tasks, ntasks, deep, force, s);
        if (levels == 4) return multi_batch_tl<__half, 4>(sp, nsp, sel, tasks, ntasks, deep, force, s);
    }
    return cudaErrorInvalidValue;
}

cudaError_t multi_swap(const int2 *nodes, int n, const uint16_t *flags, int pitch, long long plane, int store,
                       const void *cur, void *other, void *odd, void *even2, bool enter, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const unsigned g = (unsigned)((n + 127) / 128);
    if (store == STORE_F32)
        k_multi_swap<float><<<g, 128, 0, s>>>(nodes, n, flags, pitch, plane, (const float *)cur, (float *)other,
                                              (float *)odd, (float *)even2, enter ? 1 : 0);
    else
        k_multi_swap<__half><<<g, 128, 0, s>>>(nodes, n, flags, pitch, plane, (const __half *)cur, (__half *)other,
                                               (__half *)odd, (__half *)even2, enter ? 1 : 0);
    return cudaGetLastError();
}

template <typename T, int LV>
static cudaError_t multi_plain_tl(const FastStepParams &p, int warps_wanted, cudaStream_t s) {
    const int width = 64 - 2 * multi_halo(LV);
    const int strips = (p.s.Nx + width - 1) / width;
    const int chunks = std::max(1, std::min(p.s.Ny / 4, warps_wanted / strips));
    const int height = (p.s.Ny + chunks - 1) / chunks;
    const long long warps = (long long)strips * ((p.s.Ny + height - 1) / height);
    const unsigned blocks = (unsigned)((warps + kMultiThreads / 32 - 1) / (kMultiThreads / 32));
    if (p.s.has_force) k_multi_plain<T, LV, true><<<blocks, kMultiThreads, 0, s>>>(p, strips, height);
    else k_multi_plain<T, LV, false><<<blocks, kMultiThreads, 0, s>>>(p, strips, height);
    return cudaGetLastError();
}

cudaError_t multi_plain(const FastStepParams &p, int store, int levels, int warps, cudaStream_t s) {
    if (store == STORE_F32) {
        switch (levels) {
        case 2: return multi_plain_tl<float, 2>(p, warps, s);
        case 4: return multi_plain_tl<float, 4>(p, warps, s);
        }
    } else {
        switch (levels) {
        case 2: return multi_plain_tl<__half, 2>(p, warps, s);
        case 4: return multi_plain_tl<__half, 4>(p, warps, s);
        }
    }
    return cudaErrorInvalidValue;
}

}  // namespace launch
}  // namespace lbm
