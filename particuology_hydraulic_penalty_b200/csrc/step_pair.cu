// Pair kernel for the deviation storage modes: the step of k_step_fast
// (pull-stream + PSC-IMB collide, src/lbm_dem/psc3d.py:208-246) with each
// thread owning two consecutive z cells (c, c + 1), c even.
//
// With nz even a pair never crosses a z row, so the nine directions with
// c_z = 0 pull both cells with one aligned 2-element load, and all nineteen
// populations (and the IMB / moment fields) are written with 2-element
// stores; the ten z-shifted directions pull two scalars.  Measured on the
// bare access pattern (19 planes read + 19 written, 33 M cells): 2-element
// accesses at two CTAs per SM move 6.5 TB/s against 5.1-5.9 TB/s for scalar
// ones.  The per-cell arithmetic is the one-cell kernel's: fast_cell() for each
// cell, or for 16-bit storage fast_cell_pair(), which takes both at once in
// packed FP32 and rounds alike, so both kernels produce identical populations.
#include <type_traits>

#include "fast_cell.cuh"
#include "internal.cuh"

namespace psc {

// Set (once) when a launch met a window it cannot run: 0x201 odd nz,
// 0x202 tiles not planned by psc_plan_pair_tiles.  Such windows are skipped.
__device__ int g_pair_status = 0;

constexpr int PAIR_CELLS = 2;

__device__ __forceinline__ void st_pair(float* p, float a, float b) {
    *reinterpret_cast<float2*>(p) = make_float2(a, b);
}
__device__ __forceinline__ void st_pair(double* p, double a, double b) {
    *reinterpret_cast<double2*>(p) = make_double2(a, b);
}
// 16-bit pairs stream (evict-first) like the one-cell stores; the same round-to-nearest conversion
__device__ __forceinline__ void st_pair(__half* p, float a, float b) {
    __stcs(reinterpret_cast<__half2*>(p), __floats2half2_rn(a, b));
}
__device__ __forceinline__ void st_pair(__nv_bfloat16* p, float a, float b) {
    __stcs(reinterpret_cast<__nv_bfloat162*>(p), __floats2bfloat162_rn(a, b));
}

// Resident CTAs the register allocation aims for: two cells per thread need
// about twice the registers of the one-cell kernel.
template <int STORE, bool MOVING, bool RED>
struct PairOccupancy {
    static constexpr int value = (STORE == PSC_STORE_F64) ? 1 : 2;
};

template <int STORE, bool MOVING, bool RED>
__global__ void __launch_bounds__(STEP_THREADS, (PairOccupancy<STORE, MOVING, RED>::value))
    k_step_pair(const psc_window* __restrict__ wins, int nwin, unsigned flags, const __grid_constant__ TilePlan plan) {
    using TR = StoreTraits<STORE>;
    using T = typename TR::T;
    using R = typename TR::R;
    using O = typename TR::O;
    // Both cells in packed FP32 where the arithmetic weighs: 16-bit storage (FP16 160^3 90 -> 82 us plain and
    // 107 -> 99 with IMB and sums, 78 and 96 in a chain of steps; 311 and 394 instructions per cell).  FP32
    // storage is bound by HBM, and there the packed form was slower (114 against 108 us, although at 261
    // instructions per cell instead of 378, 351 now: its shorter bursts of arithmetic leave reads and writes less
    // spread).  FP64 has no packed form.
    constexpr bool PACKED = sizeof(T) == 2;
    using V = std::conditional_t<PACKED, F2, R>;
    __shared__ FastWin<T, R, O, V> sw;
    static_assert(STEP_THREADS / 32 == PSC_PARTIAL_ROWS, "one partial row per warp");
    const bool do_collide = flags & PSC_STEP_COLLIDE;
    const bool do_imb = do_collide && (flags & PSC_STEP_IMB);
    const bool do_mom = flags & PSC_STEP_MOMENTS;
    constexpr bool do_red = RED;
    const TileWalk walk = tile_walk(plan);
    uint32_t win_end = 0, t_in = 0;  // the window's end, the CTA's first tile in it
    int wi = -1, prev = -1;
    constexpr bool SHARED = RED && PACKED;  // (107 -> 104 us with the sums in registers, 99 in shared memory)
    __shared__ double s_red[SHARED ? PSC_NRED : 1][STEP_THREADS];
    CellSums<SHARED> red;  // this thread's sums over the CTA's cells of the current window
    red.s = s_red;
    if (RED) red.clear();
    const auto flush = [&]() {
        double v[PSC_NRED];
#pragma unroll
        for (int q = 0; q < PSC_NRED; ++q) v[q] = red.at(q);
        flush_walk<PSC_NRED>(v, sw.partials, (uint32_t)sw.tile_begin, (uint32_t)sw.tile_end, t_in, walk, plan);
        red.clear();
    };
    bool have = false;
    bool skip = false;  // block-uniform: the window in sw cannot run here
    // this thread's first cell (ix, iy, iz) in the current tile: divided out when the CTA enters a
    // window, then advanced to the CTA's next tile (walk.size tiles on) by a carry-add
    bool fresh = true;
    uint32_t ix = 0, iy = 0, iz = 0;
    for (uint32_t t = walk.first(); t < walk.end; t += walk.size) {
        if (t >= win_end) {  // block-uniform: entering a new window
            if (do_red && have) flush();
            have = false;
            __syncthreads();
            wi = wi < 0 ? find_window(wins, nullptr, nwin, t) : advance_window(wins, nwin, wi, t);
            load_fast_win(sw, wins[wi], MOVING, (int32_t)walk.size, prev >= 0 ? wins + prev : nullptr);
            if (prev < 0) chain_wait();
            prev = wi;
            __syncthreads();
            win_end = (uint32_t)sw.tile_end;
            t_in = t;
            skip = (sw.nz & 1u) != 0 || sw.tile_cells != PAIR_CELLS * (int32_t)blockDim.x;
            fresh = true;
            if (skip && threadIdx.x == 0) atomicCAS(&g_pair_status, 0, (sw.nz & 1u) ? 0x201 : 0x202);
        }
        if (sw.inactive || skip) continue;  // block-uniform
        have = true;
        const uint32_t N = sw.N, nx = sw.nx, ny = sw.ny, nz = sw.nz;
        const uint32_t c0 = (uint32_t)((t - sw.tile_begin) * sw.tile_cells) + PAIR_CELLS * threadIdx.x;
        if (fresh) {
            iz = c0 % nz;
            const uint32_t rr = c0 / nz;
            iy = rr % ny;
            ix = rr / ny;
            fresh = false;
        } else {  // this CTA's next tile: += its step, single carries (each step component < its extent)
            iz += sw.tstep_z;
            const uint32_t cz = iz >= nz;
            iz -= cz ? nz : 0u;
            iy += sw.tstep_y + cz;
            const uint32_t cy = iy >= ny;
            iy -= cy ? ny : 0u;
            ix += sw.tstep_x + cy;
        }
        if (c0 >= N) continue;  // N is even: c0 + 1 < N as well (the window's last tile)
        const bool open_x = sw.open_x;
        const bool inlet = open_x && ix == 0;
        const int32_t nyz = (int32_t)(ny * nz);
        const int32_t xm = ix == 0 ? (open_x ? 0 : (int32_t)(nx - 1) * nyz) : -nyz;
        const int32_t xp = ix == nx - 1 ? (open_x ? 0 : -(int32_t)(nx - 1) * nyz) : nyz;
        const int32_t ym = iy == 0 ? (int32_t)(ny - 1) * (int32_t)nz : -(int32_t)nz;
        const int32_t yp = iy == ny - 1 ? -(int32_t)(ny - 1) * (int32_t)nz : (int32_t)nz;
        // z sources: c0 pulls z - 1 (wraps at iz = 0) and z + 1 (iz + 1 <= nz - 1); c1 pulls z (= iz) and
        // z + 2 (wraps when iz + 1 == nz - 1)
        const int32_t zm0 = iz == 0 ? (int32_t)nz - 1 : -1;
        const int32_t zp1 = iz + 2 == nz ? -(int32_t)(nz - 1) : 1;
        const T* src = sw.src;
        V g[PACKED ? 1 : 2][Q], mom[PACKED ? 1 : 2][4], imb[PACKED ? 1 : 2][3];
        uint32_t plane = 0;
#pragma unroll
        for (int i = 0; i < Q; ++i) {
            const int32_t oxy = (cxv(i) == 1 ? xm : (cxv(i) == -1 ? xp : 0)) + (cyv(i) == 1 ? ym : (cyv(i) == -1 ? yp : 0));
            const T* p = src + (int64_t)(int32_t)(plane + c0 + (uint32_t)oxy);
            R a, b;
            if (czv(i) == 0) {
                ld_pair(p, a, b);  // c0 even, oxy a multiple of nz (even): aligned
            } else if (czv(i) == 1) {
                a = ld_pop(p + zm0);
                b = ld_pop(p);
            } else {
                a = ld_pop(p + 1);
                b = ld_pop(p + 1 + zp1);
            }
            if constexpr (PACKED) {
                g[0][i] = f2(a, b);
            } else {
                g[0][i] = a;
                g[1][i] = b;
            }
            plane += N;
        }
        if constexpr (PACKED) {
            fast_cell_pair<TR, MOVING, RED>(sw, g[0], c0, N, inlet, do_collide, do_imb, mom[0], imb[0], red, do_mom);
        } else {
            fast_cell<TR, MOVING, RED>(sw, g[0], c0, N, inlet, do_collide, do_imb, mom[0], imb[0], red, do_mom);
            fast_cell<TR, MOVING, RED>(sw, g[1], c0 + 1, N, inlet, do_collide, do_imb, mom[1], imb[1], red, do_mom);
        }
        // the two cells' values of one V (packed) or of the two scalars
        const auto both = [](const auto& v, int k, R& x, R& y) {
            if constexpr (PACKED) {
                f2_get(v[0][k], x, y);
            } else {
                x = v[0][k];
                y = v[1][k];
            }
        };
        if (do_collide) {
            T* dst = sw.dst + c0;
            uint32_t pl = 0;
#pragma unroll
            for (int i = 0; i < Q; ++i) {
                if constexpr (PACKED && TR::scaled) g[0][i] = vmul(g[0][i], f2(sw.scale, sw.scale));
                R x, y;
                both(g, i, x, y);
                st_pair(dst + pl, x, y);
                pl += N;
            }
            if (do_imb) {
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    R x, y;
                    both(imb, k, x, y);
                    st_pair(sw.imb + (size_t)k * N + c0, (O)x, (O)y);
                }
            }
        }
        if (do_mom) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                R x, y;
                both(mom, k, x, y);
                if (k == 0) st_pair(sw.mom + c0, (O)(R(1) + x), (O)(R(1) + y));
                else st_pair(sw.mom + (size_t)k * N + c0, (O)x, (O)y);
            }
        }
    }
    if (do_red && have) flush();
}

template <int STORE, bool MOVING, bool RED>
static cudaError_t launch_pair_t(const psc_window* d_windows, int nwin, int64_t total_tiles, unsigned flags,
                                 int grid_ctas, cudaStream_t stream) {
    if (grid_ctas <= 0) {
        static int per_sm[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        int dev = 0;
        cudaGetDevice(&dev);
        int& occ = per_sm[dev & 7];
        if (occ == 0) {
            cudaError_t e =
                cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_step_pair<STORE, MOVING, RED>, STEP_THREADS, 0);
            if (e != cudaSuccess) return e;
            if (occ <= 0) occ = 1;
        }
        const int64_t g = (int64_t)sm_count() * occ;
        grid_ctas = (int)(total_tiles < g ? total_tiles : g);
    }
    if ((int64_t)grid_ctas > total_tiles) grid_ctas = (int)total_tiles;  // every CTA owns >= 1 tile
    if (grid_ctas <= 0) return cudaSuccess;
    return launch_chained(k_step_pair<STORE, MOVING, RED>, grid_ctas, STEP_THREADS, 0, stream, flags & PSC_STEP_CHAINED,
                          d_windows, nwin, flags, tile_plan(total_tiles, nwin, grid_ctas));
}

template <int STORE>
static cudaError_t launch_pair_s(const psc_window* d, int nwin, int64_t tiles, unsigned flags, bool moving, int grid,
                                 cudaStream_t s) {
    const bool red = (flags & PSC_STEP_REDUCE) != 0;
    if (moving) return red ? launch_pair_t<STORE, true, true>(d, nwin, tiles, flags, grid, s)
                           : launch_pair_t<STORE, true, false>(d, nwin, tiles, flags, grid, s);
    return red ? launch_pair_t<STORE, false, true>(d, nwin, tiles, flags, grid, s)
               : launch_pair_t<STORE, false, false>(d, nwin, tiles, flags, grid, s);
}

cudaError_t launch_step_pair(int store, const psc_window* d_windows, int nwin, int64_t total_tiles, unsigned flags,
                             bool moving, int grid_ctas, cudaStream_t stream) {
    switch (store) {
        case PSC_STORE_F64: return launch_pair_s<PSC_STORE_F64>(d_windows, nwin, total_tiles, flags, moving, grid_ctas, stream);
        case PSC_STORE_F32: return launch_pair_s<PSC_STORE_F32>(d_windows, nwin, total_tiles, flags, moving, grid_ctas, stream);
        case PSC_STORE_F16: return launch_pair_s<PSC_STORE_F16>(d_windows, nwin, total_tiles, flags, moving, grid_ctas, stream);
        case PSC_STORE_BF16: return launch_pair_s<PSC_STORE_BF16>(d_windows, nwin, total_tiles, flags, moving, grid_ctas, stream);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t read_pair_status(int* out, bool clear) {
    cudaError_t e = cudaMemcpyFromSymbol(out, g_pair_status, sizeof(int));
    if (e != cudaSuccess || !clear) return e;
    const int zero = 0;
    return cudaMemcpyToSymbol(g_pair_status, &zero, sizeof(int));
}

}  // namespace psc
