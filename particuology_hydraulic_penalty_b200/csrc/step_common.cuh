// Storage traits and population-access helpers shared by the step kernels.
#pragma once

#include "collide.cuh"
#include "internal.cuh"

namespace psc {

template <int STORE>
struct StoreTraits;
template <>
struct StoreTraits<PSC_STORE_F64_EXACT> {
    using T = double;
    using R = double;
    using O = double;
    static constexpr bool exact = true;
    static constexpr bool scaled = false;
};
template <>
struct StoreTraits<PSC_STORE_F64> {
    using T = double;
    using R = double;
    using O = double;
    static constexpr bool exact = false;
    static constexpr bool scaled = false;
};
template <>
struct StoreTraits<PSC_STORE_F32> {
    using T = float;
    using R = float;
    using O = float;
    static constexpr bool exact = false;
    static constexpr bool scaled = false;
};
template <>
struct StoreTraits<PSC_STORE_F16> {
    using T = __half;
    using R = float;
    using O = float;
    static constexpr bool exact = false;
    static constexpr bool scaled = true;
};
template <>
struct StoreTraits<PSC_STORE_BF16> {
    using T = __nv_bfloat16;
    using R = float;
    using O = float;
    static constexpr bool exact = false;
    static constexpr bool scaled = true;
};

// Population loads are ordinary (coherent) ones: a chained kernel (launch_chained) is resident while the kernel
// ahead of it still writes them, and read-only (.nc) loads are defined only for data that nobody writes
// while the kernel lives.  asm volatile keeps them behind chain_wait.  FP32 pulls ask L2 for the whole 256-byte line
// pair: a warp's neighbours on the same SM read the rest of it (24 windows 845 -> 831 us a step, 160^3 103.5 -> 102.2).
__device__ __forceinline__ double ld_pop(const double* p) {
    double v;
    asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float ld_pop(const float* p) {
    float v;
    asm volatile("ld.global.L2::256B.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float ld_pop(const __half* p) {
    __half_raw v;
    asm volatile("ld.global.u16 %0, [%1];" : "=h"(v.x) : "l"(p));
    return __half2float(v);
}
__device__ __forceinline__ float ld_pop(const __nv_bfloat16* p) {
    __nv_bfloat16_raw v;
    asm volatile("ld.global.u16 %0, [%1];" : "=h"(v.x) : "l"(p));
    return __bfloat162float(v);
}

// The same of two consecutive populations (p aligned to both).
__device__ __forceinline__ void ld_pair(const float* p, float& a, float& b) {
    asm volatile("ld.global.L2::256B.v2.f32 {%0, %1}, [%2];" : "=f"(a), "=f"(b) : "l"(p));
}
__device__ __forceinline__ void ld_pair(const double* p, double& a, double& b) {
    asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(a), "=d"(b) : "l"(p));
}
__device__ __forceinline__ void ld_pair(const __half* p, float& a, float& b) {
    __half2_raw r;
    asm volatile("ld.global.v2.u16 {%0, %1}, [%2];" : "=h"(r.x), "=h"(r.y) : "l"(p));
    const float2 v = __half22float2(r);
    a = v.x;
    b = v.y;
}
__device__ __forceinline__ void ld_pair(const __nv_bfloat16* p, float& a, float& b) {
    __nv_bfloat162_raw r;
    asm volatile("ld.global.v2.u16 {%0, %1}, [%2];" : "=h"(r.x), "=h"(r.y) : "l"(p));
    const float2 v = __bfloat1622float2(r);
    a = v.x;
    b = v.y;
}

template <typename R>
__device__ __forceinline__ R fast_rcp(R x);
template <>
__device__ __forceinline__ float fast_rcp<float>(float x) {
    return __frcp_rn(x);
}
template <>
__device__ __forceinline__ double fast_rcp<double>(double x) {
    return __drcp_rn(x);
}

// plain (shared-memory) reads of a stored population
__device__ __forceinline__ double ld_smem_pop(const double* p) { return *p; }
__device__ __forceinline__ float ld_smem_pop(const float* p) { return *p; }
__device__ __forceinline__ float ld_smem_pop(const __half* p) { return __half2float(*p); }
__device__ __forceinline__ float ld_smem_pop(const __nv_bfloat16* p) { return __bfloat162float(*p); }

__device__ __forceinline__ void st_pop(double* p, double v) { *p = v; }
__device__ __forceinline__ void st_pop(float* p, float v) { *p = v; }
// 16-bit stores stream (evict-first): measured +7 % for FP16 storage.
__device__ __forceinline__ void st_pop(__half* p, float v) { __stcs(p, __float2half_rn(v)); }
__device__ __forceinline__ void st_pop(__nv_bfloat16* p, float v) { __stcs(p, __float2bfloat16_rn(v)); }

// Offset (in cells) from x to x - c_i for direction i, given the wrapped
// neighbour offsets of this cell.
struct NbrOffsets {
    int32_t xm, xp, ym, yp, zm, zp;  // to ix-1, ix+1, iy-1, iy+1, iz-1, iz+1
};

// Offsets to the six face neighbours, periodic; with open_x the x faces
// point at the cell's own plane instead of wrapping (zero-gradient outflow at
// x = nx - 1; at x = 0 the inlet replaces the pulled values afterwards).
__device__ __forceinline__ NbrOffsets nbr_offsets(uint32_t ix, uint32_t iy, uint32_t iz, int nx, int ny, int nz,
                                                  bool open_x = false) {
    NbrOffsets o;
    const int32_t nyz = ny * nz;
    o.xm = ix == 0 ? (open_x ? 0 : (nx - 1) * nyz) : -nyz;
    o.xp = ix == (uint32_t)(nx - 1) ? (open_x ? 0 : -(nx - 1) * nyz) : nyz;
    o.ym = iy == 0 ? (ny - 1) * nz : -nz;
    o.yp = iy == (uint32_t)(ny - 1) ? -(ny - 1) * nz : nz;
    o.zm = iz == 0 ? nz - 1 : -1;
    o.zp = iz == (uint32_t)(nz - 1) ? -(nz - 1) : 1;
    return o;
}

template <int I>
__device__ __forceinline__ int32_t pull_offset(const NbrOffsets& o) {
    // source of direction I at x is x - c_I
    return (cxv(I) == 1 ? o.xm : (cxv(I) == -1 ? o.xp : 0)) + (cyv(I) == 1 ? o.ym : (cyv(I) == -1 ? o.yp : 0)) +
           (czv(I) == 1 ? o.zm : (czv(I) == -1 ? o.zp : 0));
}

// The constants of the exact arithmetic, by the block: each warp makes a part.
__device__ __forceinline__ void make_exact_win_block(ExactWin& w, double tau, double fx, double fy, double fz) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == 1 && lane == 0) exact_win_force(w, tau, fx, fy, fz);
    if (warp == 2 && lane == 0) exact_win_tau(w, tau);
    if (warp == 3 && lane == 0) exact_win_guo(w, tau);
    if (warp == 4 && lane == 0) exact_win_pairs(w, fx, fy, fz);
}

__device__ __forceinline__ int find_window(const psc_window* wins, const int64_t* s_begin, int nwin, int64_t t) {
    int lo = 0, hi = nwin - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        const int64_t b = s_begin ? s_begin[mid] : wins[mid].tile_begin;
        if (b <= t) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Warp sums of v, written as this warp's row of a tile's partials:
// rows[warp][k] for k < NV (lane k stores value k).  No block barrier.
template <int NV>
__device__ __forceinline__ void warp_reduce_store(double (&v)[NV], double* rows) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double* out = rows + (size_t)warp * NV;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        double x = v[k];
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) x += __shfl_xor_sync(0xffffffffu, x, s);
        if (lane == k) out[k] = x;
    }
}

// The CTA of a persistent grid of `grid` CTAs over `total` tiles (CTA b owns
// [total * b / grid, total * (b + 1) / grid)) that owns tile t.
__device__ __forceinline__ int64_t cta_of_tile(int64_t t, int64_t total, int64_t grid) {
    return ((t + 1) * grid - 1) / total;
}

// End of this CTA's run of tiles inside one window: each warp writes the sums
// of its threads' accumulators as row (b - b_first) * PSC_PARTIAL_ROWS + warp
// of the window's partials (after the header row), and the window's first
// CTA writes the row count into the header.  Resets the accumulators.
template <int NV>
__device__ __forceinline__ void flush_segment(double (&red)[NV], double* partials, int64_t tile_begin,
                                              int64_t tile_count, int64_t total, int64_t grid) {
    const int64_t bf = cta_of_tile(tile_begin, total, grid);
    const int64_t bl = cta_of_tile(tile_begin + tile_count - 1, total, grid);
    const int64_t row = ((int64_t)blockIdx.x - bf) * PSC_PARTIAL_ROWS;
    warp_reduce_store<NV>(red, partials + (1 + row) * NV);
    if ((int64_t)blockIdx.x == bf && threadIdx.x == 0) partials[0] = (double)((bl - bf + 1) * PSC_PARTIAL_ROWS);
#pragma unroll
    for (int k = 0; k < NV; ++k) red[k] = 0.0;
}

// The next window at or after wi that holds tile t (a CTA's tiles ascend).
__device__ __forceinline__ int advance_window(const psc_window* wins, int nwin, int wi, int64_t t) {
    while (wi + 1 < nwin && t >= wins[wi].tile_begin + wins[wi].tile_count) ++wi;
    return wi;
}

// How the tiles of a launch fall to its CTAs: CTA c has the share [start(c), start(c + 1)) of the
// tiles, groups of 2^lg consecutive CTAs pool their shares, and the CTAs of a group take the group's
// tiles in turn.
//
// In turn, a group's CTAs read and write each population plane in one moving front (DRAM pages stay
// open: 200^3 FP32 step 213 -> 197 us with one group; exact 160^3 with sums 292 -> 270 us); with a run
// of its own, a CTA enters fewer windows.  So one window is one group, and a batch gets groups in which
// a CTA takes 32 to 64 tiles per window on average (24 windows, FP32: 871 -> 835 us a step; one group
// for windows of 24^3 to 40^3 took 31 us instead of 19.5).
struct TilePlan {
    uint32_t q, r;  // total tiles = q * grid + r: the first r CTAs have q + 1
    int32_t lg;
};
// (a launch has fewer than 2^31 tiles: as many of 256 cells would hold more than any GPU's memory)
inline TilePlan tile_plan(int64_t total, int nwin, int grid) {
    TilePlan p = {(uint32_t)(total / grid), (uint32_t)(total % grid), 0};
    if (nwin <= 1) {
        p.lg = 30;  // one group
        return p;
    }
    const int64_t size = total / ((int64_t)nwin * 32);
    while (p.lg < 30 && ((int64_t)2 << p.lg) <= size) ++p.lg;
    return p;
}

struct TileWalk {
    uint32_t begin, end;  // the group's tiles
    uint32_t c0, size;    // its first CTA, its CTAs
    // this CTA's first tile; its next ones are `size` further on
    __device__ __forceinline__ uint32_t first() const { return begin + (blockIdx.x - c0); }
};
__device__ __forceinline__ uint32_t tile_start(const TilePlan& p, uint32_t c) { return p.q * c + min(c, p.r); }
__device__ __forceinline__ TileWalk group_walk(const TilePlan& p, uint32_t c) {  // the group of CTA c
    TileWalk w;
    w.c0 = (c >> p.lg) << p.lg;
    const uint32_t c1 = min(w.c0 + (1u << p.lg), gridDim.x);
    w.size = c1 - w.c0;
    w.begin = tile_start(p, w.c0);
    w.end = tile_start(p, c1);
    return w;
}
__device__ __forceinline__ TileWalk tile_walk(const TilePlan& p) { return group_walk(p, blockIdx.x); }
__device__ __forceinline__ TileWalk walk_of_tile(const TilePlan& p, uint32_t t) {
    const uint32_t wide = p.r * (p.q + 1);
    return group_walk(p, t < wide ? t / (p.q + 1) : p.r + (t - wide) / p.q);
}

// End of this CTA's tiles inside the window [tb, te), the first of them t_in: each warp writes the sums
// of its threads as one row of the window's partials (after the header row), the rows of a group's CTAs
// in the order in which they enter the window, group after group; the owner of the window's first tile
// writes the row count into the header.
template <int NV>
__device__ __forceinline__ void flush_walk(double (&red)[NV], double* partials, uint32_t tb, uint32_t te, uint32_t t_in,
                                           const TileWalk& w, const TilePlan& p) {
    uint32_t row = t_in - max(tb, w.begin);
    if (tb < w.begin) {  // the window began in an earlier group: that group's rows and those between
        const TileWalk a = walk_of_tile(p, tb);
        row += min(a.size, a.end - tb) + (w.c0 - (a.c0 + a.size));
    }
    warp_reduce_store<NV>(red, partials + (1 + (int64_t)row * PSC_PARTIAL_ROWS) * NV);
    if (row == 0 && threadIdx.x == 0) {
        uint32_t rows = min(w.size, min(te, w.end) - tb);
        if (te > w.end) {
            const TileWalk b = walk_of_tile(p, te - 1);
            rows += (b.c0 - (w.c0 + w.size)) + min(b.size, te - b.begin);
        }
        partials[0] = (double)((int64_t)rows * PSC_PARTIAL_ROWS);
    }
}

}  // namespace psc
