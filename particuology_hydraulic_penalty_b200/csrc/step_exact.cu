// Exact FP64 step (PSC_STORE_F64_EXACT): pull-stream + PSC-IMB collide over a list
// of lattice windows, every rounding in the reference's order
// (src/lbm_dem/psc3d.py:208-246):
//   pull      f_i(x) = f*_i(x - c_i)   (periodic; equivalent to the
//             reference's push np.roll(f*_i, c_i) at :239-242)
//   moments   rho, u of the pulled (post-stream) state           (:211-214)
//   collide   Noble-Torczynski PSC + Guo forcing                  (:215-232)
//   write     f*_i(x) to the other buffer, optional IMB momentum   (:234-236)
//   reduce    FP64 partial sums (flux, porosity, IMB, NaN count)
//
// Each persistent CTA takes its share of the 256-cell tiles (TilePlan); a thread owns
// one cell of a tile, so every population plane is read and written with
// consecutive addresses and crosses HBM once per step.  The window's constants
// sit in shared memory, built when the CTA enters the window.
#include "collide.cuh"
#include "internal.cuh"
#include "step_common.cuh"

namespace psc {

struct ExactShared {
    const double* src;
    double* dst;
    const double* solid;
    const double* us;
    double* imb;
    double* mom;
    double* partials;
    int64_t tile_begin, tile_end;
    uint32_t nx, ny, nz, N;
    uint32_t tstep_x, tstep_y, tstep_z;  // a CTA's next tile (tile_cells * stride cells on) as (x, y, z) digits
    int32_t tile_cells;
    int32_t moving, inactive, open_x;
    ExactWin c;
    double corr[Q];  // open_x: bounce-back inlet term 2 w_i rho_in (c_i . u_in) / cs^2
};

// stride: tiles from one of the CTA's tiles to its next.
__device__ void load_exact_win(ExactShared& s, const psc_window& W, bool moving_launch, int32_t stride) {
    if (threadIdx.x == 0) {
        s.src = reinterpret_cast<const double*>(W.f_src);
        s.dst = reinterpret_cast<double*>(W.f_dst);
        s.solid = W.solid;
        s.us = reinterpret_cast<const double*>(W.us);
        s.imb = reinterpret_cast<double*>(W.imb);
        s.mom = reinterpret_cast<double*>(W.moments);
        s.partials = W.partials;
        s.tile_begin = W.tile_begin;
        s.tile_end = W.tile_begin + W.tile_count;
        s.nx = W.nx;
        s.ny = W.ny;
        s.nz = W.nz;
        s.N = (uint32_t)W.nx * W.ny * W.nz;
        const uint64_t tc = (uint64_t)W.tile_cells * stride;
        const uint32_t tq = tc < s.N ? (uint32_t)tc / (uint32_t)W.nz : 0u;  // (a longer step leaves the window)
        s.tstep_z = tc < s.N ? (uint32_t)tc % (uint32_t)W.nz : 0u;
        s.tstep_y = tq % (uint32_t)W.ny;
        s.tstep_x = tq / (uint32_t)W.ny;
        s.tile_cells = W.tile_cells;
        s.moving = (moving_launch && (W.flags & PSC_WIN_MOVING) && W.us != nullptr) ? 1 : 0;
        s.inactive = (W.flags & PSC_WIN_INACTIVE) ? 1 : 0;
        s.open_x = (W.flags & PSC_WIN_OPEN_X) ? 1 : 0;
    }
    make_exact_win_block(s.c, W.tau, W.force[0], W.force[1], W.force[2]);
    if ((W.flags & PSC_WIN_OPEN_X) && threadIdx.x < Q)
        s.corr[threadIdx.x] =
            inlet_correction_exact(threadIdx.x, W.inlet_rho, W.inlet_u[0], W.inlet_u[1], W.inlet_u[2]);
}

// Coordinates of one cell, and the offsets (in cells) of its pull sources.
struct ExactAt {
    uint32_t ix, iy, iz;
};

__device__ __forceinline__ ExactAt exact_decode(const ExactShared& s, uint32_t cell) {
    ExactAt c;
    c.iz = cell % s.nz;
    const uint32_t r = cell / s.nz;
    c.iy = r % s.ny;
    c.ix = r / s.ny;
    return c;
}

// One tile on: += the tile step, single carries (each step component < its extent).
__device__ __forceinline__ void exact_advance(const ExactShared& s, ExactAt& c) {
    c.iz += s.tstep_z;
    const uint32_t cz = c.iz >= s.nz;
    c.iz -= cz ? s.nz : 0u;
    c.iy += s.tstep_y + cz;
    const uint32_t cy = c.iy >= s.ny;
    c.iy -= cy ? s.ny : 0u;
    c.ix += s.tstep_x + cy;
}

__device__ __forceinline__ void exact_pull(const ExactShared& s, uint32_t cell, const ExactAt& c, double (&f)[Q]) {
    const NbrOffsets o = nbr_offsets(c.ix, c.iy, c.iz, (int)s.nx, (int)s.ny, (int)s.nz, s.open_x);
    const double* src = s.src + cell;
    const uint32_t N = s.N;
#pragma unroll
    for (int i = 0; i < Q; ++i) {
        const int32_t off = (cxv(i) == 1 ? o.xm : (cxv(i) == -1 ? o.xp : 0)) +
                            (cyv(i) == 1 ? o.ym : (cyv(i) == -1 ? o.yp : 0)) +
                            (czv(i) == 1 ? o.zm : (czv(i) == -1 ? o.zp : 0));
        f[i] = ld_pop(src + (int64_t)off);
        src += N;
    }
}

// Velocity inlet: the entering populations are the node's own opp(i) bounced back + the momentum term.
__device__ __forceinline__ void exact_inlet(const ExactShared& s, uint32_t cell, double (&f)[Q]) {
#pragma unroll
    for (int i = 0; i < Q; ++i)
        if (enters_x0(i)) f[i] = xadd(ld_pop(s.src + (size_t)opp(i) * s.N + cell), s.corr[i]);
}

// A cell whose operands left the range of the branch-free forms: pulled again and taken
// through the general ones.
struct ExactCell {
    double f[Q], mom[4], imb[3];
};

__device__ __noinline__ void exact_cell_general(const ExactShared& s, uint32_t cell, bool do_collide, ExactCell& r) {
    double f[Q];
    const ExactAt c = exact_decode(s, cell);
    exact_pull(s, cell, c, f);
    if (s.open_x && c.ix == 0) exact_inlet(s, cell, f);
    const ExactMoments mo = moments_exact(f, s.c.hfx, s.c.hfy, s.c.hfz);
    double imb[3] = {0.0, 0.0, 0.0};
    if (do_collide) {
        double us[3] = {0.0, 0.0, 0.0};
        if (s.moving)
            for (int k = 0; k < 3; ++k) us[k] = s.us[(size_t)k * s.N + cell];
        collide_exact(f, mo, s.solid[cell], s.moving != 0, us[0], us[1], us[2], s.c.tau, s.c.fx, s.c.fy, s.c.fz,
                      s.c.hfx, s.c.hfy, s.c.hfz, imb);
    }
    for (int i = 0; i < Q; ++i) r.f[i] = f[i];
    for (int k = 0; k < 3; ++k) r.imb[k] = imb[k];
    r.mom[0] = mo.rho;
    r.mom[1] = mo.ux;
    r.mom[2] = mo.uy;
    r.mom[3] = mo.uz;
}

// Two CTAs per SM (128 registers; three at 80 registers spill).  Bounds, on a 160^3 window: HBM
// (312 B/cell, 196 us at the measured copy rate) and the FP64 pipe (one warp instruction every other
// cycle and SM quarter, about 575 per cell: 130 us).  Measured with branch-free divisions, one window
// set-up per CTA and window, and range tests in integer instructions, in a chain of steps: 231 us
// plain, 271 with IMB and sums (553 and 608 with a branch per division and a window look-up per tile);
// 96^3: 54 and 62 (126 and 137); 24^3: 3.9 and 5.1 (8.9 and 9.8).  Staging the next tile's populations in shared memory by
// cp.async took another 1 to 4 %, at one more kernel per variant: not used.
template <bool MOVING, bool RED>
__global__ void __launch_bounds__(STEP_THREADS, 2)
    k_step_exact(const psc_window* wins, int nwin, unsigned flags, const __grid_constant__ TilePlan plan) {
    __shared__ ExactShared sw;
    __shared__ double s_red[RED ? PSC_NRED : 1][STEP_THREADS];  // running sums per thread (in registers they would spill)
    static_assert(STEP_THREADS / 32 == PSC_PARTIAL_ROWS, "one partial row per warp");
    if (!(flags & PSC_STEP_CHAINED)) chain_wait();  // (the table may be what it waits for)
    const bool do_collide = flags & PSC_STEP_COLLIDE;
    const bool do_imb = do_collide && (flags & PSC_STEP_IMB);
    const bool do_mom = flags & PSC_STEP_MOMENTS;
    const TileWalk walk = tile_walk(plan);
    uint32_t win_end = 0, t_in = 0;  // the window's end, the CTA's first tile in it
    int wi = -1;
    bool have = false;  // block-uniform: s_red holds cells of the window in sw
    ExactAt at = {0, 0, 0};
    auto flush = [&]() {
        double red[PSC_NRED];
#pragma unroll
        for (int q = 0; q < PSC_NRED; ++q) red[q] = s_red[RED ? q : 0][threadIdx.x];
        flush_walk<PSC_NRED>(red, sw.partials, (uint32_t)sw.tile_begin, (uint32_t)sw.tile_end, t_in, walk, plan);
    };
    for (uint32_t t = walk.first(); t < walk.end; t += walk.size) {
        if (t >= win_end) {  // block-uniform: entering a new window
            if (RED && have) flush();
            have = false;
            __syncthreads();
            const bool first = wi < 0;
            wi = first ? find_window(wins, nullptr, nwin, t) : advance_window(wins, nwin, wi, t);
            load_exact_win(sw, wins[wi], MOVING, (int32_t)walk.size);
            if (first && (flags & PSC_STEP_CHAINED)) chain_wait();
            if (RED) {
#pragma unroll
                for (int q = 0; q < (RED ? PSC_NRED : 1); ++q) s_red[q][threadIdx.x] = 0.0;
            }
            __syncthreads();
            win_end = (uint32_t)sw.tile_end;
            t_in = t;
            at = exact_decode(sw, (uint32_t)((t - sw.tile_begin) * sw.tile_cells) + threadIdx.x);
        }
        if (sw.inactive) continue;  // block-uniform
        have = true;
        const uint32_t N = sw.N;
        const uint32_t cell = (uint32_t)((t - sw.tile_begin) * sw.tile_cells) + threadIdx.x;
        if (cell >= N) continue;  // the window's last tile
        double f[Q], imb[3] = {0.0, 0.0, 0.0};
        exact_pull(sw, cell, at, f);
        const double solid = sw.solid[cell];
        if (sw.open_x && at.ix == 0) exact_inlet(sw, cell, f);
        exact_advance(sw, at);
        ExactMomentsS mo = moments_exact_s(f, sw.c.hfx, sw.c.hfy, sw.c.hfz);
        bool out = mo.out | (sw.c.out != 0);  // (the moments divide m + F / 2)
        if (do_collide) {
            bool moves = false;
            double usx = 0.0, usy = 0.0, usz = 0.0;
            if (MOVING && sw.moving) {
                usx = sw.us[cell];
                usy = sw.us[(size_t)N + cell];
                usz = sw.us[2 * (size_t)N + cell];
                // a cell at rest has feq_s = w rho, whichever form computes it
                moves = __any_sync(__activemask(), usx != 0.0 || usy != 0.0 || usz != 0.0);
            }
            if (MOVING && moves)
                out = sw.c.axis >= 0 ? collide_exact_s<MOVING, true, true>(f, mo, solid, usx, usy, usz, sw.c, imb)
                                     : collide_exact_s<MOVING, true, false>(f, mo, solid, usx, usy, usz, sw.c, imb);
            else
                out = sw.c.axis >= 0 ? collide_exact_s<false, true, true>(f, mo, solid, 0.0, 0.0, 0.0, sw.c, imb)
                                     : collide_exact_s<false, true, false>(f, mo, solid, 0.0, 0.0, 0.0, sw.c, imb);
        }
        if (out) {
            ExactCell r;
            exact_cell_general(sw, cell, do_collide, r);
#pragma unroll
            for (int i = 0; i < Q; ++i) f[i] = r.f[i];
#pragma unroll
            for (int k = 0; k < 3; ++k) imb[k] = r.imb[k];
            mo.rho = r.mom[0];
            mo.ux = r.mom[1];
            mo.uy = r.mom[2];
            mo.uz = r.mom[3];
        }
        if (do_collide) {
            double* dst = sw.dst;
            uint32_t plane = cell;
#pragma unroll
            for (int i = 0; i < Q; ++i) {
                st_pop(dst + plane, f[i]);
                plane += N;
            }
            if (do_imb) {
                sw.imb[cell] = imb[0];
                sw.imb[(size_t)N + cell] = imb[1];
                sw.imb[2 * (size_t)N + cell] = imb[2];
            }
        }
        if (do_mom) {
            sw.mom[cell] = mo.rho;
            sw.mom[(size_t)N + cell] = mo.ux;
            sw.mom[2 * (size_t)N + cell] = mo.uy;
            sw.mom[3 * (size_t)N + cell] = mo.uz;
        }
        if (RED) {
            const double fl = 1.0 - solid;
            auto add = [&](int q, double v) { s_red[RED ? q : 0][threadIdx.x] += v; };
            auto add_fluid = [&](int q, double v) {
                double& a = s_red[RED ? q : 0][threadIdx.x];
                a = xfma(fl, v, a);
            };
            add(PSC_RED_RHO, mo.rho);
            add(PSC_RED_UX, mo.ux);
            add(PSC_RED_UY, mo.uy);
            add(PSC_RED_UZ, mo.uz);
            add_fluid(PSC_RED_FLUID_UX, mo.ux);
            add_fluid(PSC_RED_FLUID_UY, mo.uy);
            add_fluid(PSC_RED_FLUID_UZ, mo.uz);
            add(PSC_RED_FLUID, fl);
            if (do_collide) {
                add(PSC_RED_IMBX, imb[0]);
                add(PSC_RED_IMBY, imb[1]);
                add(PSC_RED_IMBZ, imb[2]);
            }
            if (!(isfinite(mo.rho) && isfinite(mo.ux) && isfinite(mo.uy) && isfinite(mo.uz)))
                add(PSC_RED_NONFINITE, 1.0);
            add(PSC_RED_SOLID, solid);
        }
    }
    if (RED && have) flush();
}

template <bool MOVING, bool RED>
static cudaError_t launch_exact_t(const psc_window* d_windows, int nwin, int64_t total_tiles, unsigned flags,
                                  int grid_ctas, cudaStream_t stream) {
    if (grid_ctas <= 0) {
        static int per_sm[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        int dev = 0;
        cudaGetDevice(&dev);
        int& occ = per_sm[dev & 7];
        if (occ == 0) {
            cudaError_t e =
                cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_step_exact<MOVING, RED>, STEP_THREADS, 0);
            if (e != cudaSuccess) return e;
            if (occ <= 0) occ = 1;
        }
        const int64_t g = (int64_t)sm_count() * occ;
        grid_ctas = (int)(total_tiles < g ? total_tiles : g);
    }
    if ((int64_t)grid_ctas > total_tiles) grid_ctas = (int)total_tiles;  // every CTA owns >= 1 tile
    if (grid_ctas <= 0) return cudaSuccess;
    return launch_chained(k_step_exact<MOVING, RED>, grid_ctas, STEP_THREADS, 0, stream, true, d_windows,
                          nwin, flags, tile_plan(total_tiles, nwin, grid_ctas));
}

cudaError_t launch_step_exact(const psc_window* d_windows, int nwin, int64_t total_tiles, unsigned flags, bool moving,
                              int grid_ctas, cudaStream_t stream) {
    const bool red = (flags & PSC_STEP_REDUCE) != 0;
    if (moving) return red ? launch_exact_t<true, true>(d_windows, nwin, total_tiles, flags, grid_ctas, stream)
                           : launch_exact_t<true, false>(d_windows, nwin, total_tiles, flags, grid_ctas, stream);
    return red ? launch_exact_t<false, true>(d_windows, nwin, total_tiles, flags, grid_ctas, stream)
               : launch_exact_t<false, false>(d_windows, nwin, total_tiles, flags, grid_ctas, stream);
}

}  // namespace psc
