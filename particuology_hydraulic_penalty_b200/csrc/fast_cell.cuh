// Per-window set-up and per-cell work shared by the deviation-storage
// kernels (k_step_fast: one cell per thread at a time; k_step_pair: two
// consecutive z cells per thread with paired loads and stores), so both run
// the same arithmetic on every cell.
#pragma once

#include "step_common.cuh"

namespace psc {

template <typename T, typename R, typename O, typename V = R>  // V: what collide_v works on
struct FastWin {
    const T* src;
    T* dst;
    const uint8_t* level;
    const double* solid;
    const O* us;
    O* imb;
    O* mom;
    double* partials;
    int64_t tile_begin;
    int64_t tile_end;
    uint32_t nx, ny, nz, N;
    uint32_t step_x, step_y, step_z;     // blockDim cells as a mixed-radix (x, y, z) increment
    uint32_t tstep_x, tstep_y, tstep_z;  // a CTA's next tile (tile_cells * stride cells on) likewise
    int32_t tile_cells;
    int32_t moving;
    int32_t inactive;
    int32_t trt;
    int32_t open_x;  // PSC_WIN_OPEN_X
    R scale, inv_scale, inv_tau;
    WinConst<V> c;
    R corr[Q];       // open_x: bounce-back inlet term 2 w_i rho_in (c_i . u_in) / cs^2
    R Blut[256];
    R kblut[256];
    R alut[256];  // clipped solid fraction per level
    R tau;
};

// What the level tables and the collision constants depend on.
struct FastKey {
    double tau, tau_minus, f[3];
    int32_t S, level;
    __device__ __forceinline__ bool operator==(const FastKey& o) const {
        return tau == o.tau && tau_minus == o.tau_minus && f[0] == o.f[0] && f[1] == o.f[1] && f[2] == o.f[2] &&
               S == o.S && level == o.level;
    }
};
__device__ __forceinline__ FastKey fast_key(const psc_window& W) {
    return {W.tau, W.tau_minus, {W.force[0], W.force[1], W.force[2]}, W.subsamples, W.level != nullptr ? 1 : 0};
}

// stride: tiles from one of the CTA's tiles to its next.  prev: the window loaded before, or null.  The windows of a batch mostly share their relaxation time
// and force: their tables and constants stay.
template <typename T, typename R, typename O, typename V>
__device__ void load_fast_win(FastWin<T, R, O, V>& s, const psc_window& W, bool moving_launch, int32_t stride,
                              const psc_window* prev) {
    const bool same = prev && fast_key(*prev) == fast_key(W);
    // one warp fills the scalar part, all threads the level tables
    if (threadIdx.x == 0) {
        s.src = reinterpret_cast<const T*>(W.f_src);
        s.dst = reinterpret_cast<T*>(W.f_dst);
        s.level = W.level;
        s.solid = W.solid;
        s.us = reinterpret_cast<const O*>(W.us);
        s.imb = reinterpret_cast<O*>(W.imb);
        s.mom = reinterpret_cast<O*>(W.moments);
        s.partials = W.partials;
        s.tile_begin = W.tile_begin;
        s.tile_end = W.tile_begin + W.tile_count;
        s.nx = W.nx;
        s.ny = W.ny;
        s.nz = W.nz;
        s.N = (uint32_t)W.nx * W.ny * W.nz;
        const uint32_t q = blockDim.x / (uint32_t)W.nz;
        s.step_z = blockDim.x % (uint32_t)W.nz;
        s.step_y = q % (uint32_t)W.ny;
        s.step_x = q / (uint32_t)W.ny;
        const uint64_t tc = W.tile_cells > 0 ? (uint64_t)W.tile_cells * stride : 0u;
        const uint32_t tq = tc < s.N ? (uint32_t)tc / (uint32_t)W.nz : 0u;  // (a longer step leaves the window)
        s.tstep_z = tc < s.N ? (uint32_t)tc % (uint32_t)W.nz : 0u;
        s.tstep_y = tq % (uint32_t)W.ny;
        s.tstep_x = tq / (uint32_t)W.ny;
        s.tile_cells = W.tile_cells;
        s.moving = (moving_launch && (W.flags & PSC_WIN_MOVING) && W.us != nullptr) ? 1 : 0;
        s.inactive = (W.flags & PSC_WIN_INACTIVE) ? 1 : 0;
        s.scale = (R)W.store_scale;
        s.inv_scale = (R)(1.0 / W.store_scale);
        s.tau = (R)W.tau;
        s.inv_tau = (R)(1.0 / W.tau);
        s.trt = W.tau_minus > 0.0 ? 1 : 0;
        s.open_x = (W.flags & PSC_WIN_OPEN_X) ? 1 : 0;
    }
    if (threadIdx.x == 32 && !same) make_win_const(s.c, W.tau, W.force[0], W.force[1], W.force[2], W.tau_minus);
    if ((W.flags & PSC_WIN_OPEN_X) && threadIdx.x < Q) {
        const int i = threadIdx.x;
        s.corr[i] = (R)inlet_correction_exact(i, W.inlet_rho, W.inlet_u[0], W.inlet_u[1], W.inlet_u[2]);
    }
    const int S = W.subsamples;
    const int S3 = S * S * S;
    if (W.level && !same) {
        for (int l = threadIdx.x; l <= S3 && l < 256; l += blockDim.x) {
            const double al = (double)l / (double)S3;
            const double B = al / (al + W.tau * (1.0 - al) + 1.0e-14);
            s.Blut[l] = (R)B;
            s.kblut[l] = (R)((1.0 - B) / W.tau);
            s.alut[l] = (R)al;
        }
    }
}

// 1 / rho, correctly rounded.
__device__ __forceinline__ float rcp_v(float x) { return fast_rcp<float>(x); }
__device__ __forceinline__ double rcp_v(double x) { return fast_rcp<double>(x); }
__device__ __forceinline__ F2 rcp_v(F2 x) {
    float a, b;
    f2_get(x, a, b);
    return f2(fast_rcp<float>(a), fast_rcp<float>(b));
}

// Solid weight B, (1 - B) / tau and the clipped solid fraction of cell c.
template <typename T, typename R, typename O, typename V>
__device__ __forceinline__ void cell_solid(const FastWin<T, R, O, V>& sw, uint32_t c, R& B, R& kb, R& al) {
    if (sw.level) {
        const uint8_t lv = sw.level[c];
        B = sw.Blut[lv];
        kb = sw.kblut[lv];
        al = sw.alut[lv];
    } else {
        al = (R)sw.solid[c];
        B = al * fast_rcp<R>(al + sw.tau * (R(1) - al) + R(1.0e-14));
        kb = (R(1) - B) * sw.inv_tau;
    }
}

// Velocity inlet at x = 0: the entering populations are the node's own opp(i) bounced back
// + 2 w_i rho_in (c_i . u_in) / cs^2, in deviation units.
template <typename TR, typename V>
__device__ __forceinline__ void cell_inlet(const FastWin<typename TR::T, typename TR::R, typename TR::O, V>& sw,
                                           typename TR::R (&g)[Q], uint32_t c, uint32_t N) {
    using R = typename TR::R;
#pragma unroll
    for (int i = 0; i < Q; ++i) {
        if (!enters_x0(i)) continue;
        R back = ld_pop(sw.src + (size_t)opp(i) * N + c);
        if (TR::scaled) back *= sw.inv_scale;
        g[i] = back + sw.corr[i];
    }
}

// This thread's running sums: in registers, or a column of shared memory where the registers buy
// another resident CTA or would spill.
template <bool SHARED>
struct CellSums {
    double (*s)[STEP_THREADS];
    double r[SHARED ? 1 : PSC_NRED];
    __device__ __forceinline__ double& at(int k) { return SHARED ? s[k][threadIdx.x] : r[SHARED ? 0 : k]; }
    __device__ __forceinline__ void add(int k, double v) { at(k) += v; }
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int k = 0; k < PSC_NRED; ++k) at(k) = 0.0;
    }
};

// This cell's share of the reductions.
template <typename S, typename R>
__device__ __forceinline__ void cell_sums(S& red, R al, const R* mom, const R* imb) {
    const double solid = (double)al;
    const double fl = 1.0 - solid;
    const double rho_d = 1.0 + (double)mom[0];
    const double ux = (double)mom[1], uy = (double)mom[2], uz = (double)mom[3];
    red.add(PSC_RED_RHO, rho_d);
    red.add(PSC_RED_UX, ux);
    red.add(PSC_RED_UY, uy);
    red.add(PSC_RED_UZ, uz);
    red.add(PSC_RED_FLUID_UX, fl * ux);
    red.add(PSC_RED_FLUID_UY, fl * uy);
    red.add(PSC_RED_FLUID_UZ, fl * uz);
    red.add(PSC_RED_FLUID, fl);
    red.add(PSC_RED_IMBX, (double)imb[0]);
    red.add(PSC_RED_IMBY, (double)imb[1]);
    red.add(PSC_RED_IMBZ, (double)imb[2]);
    red.add(PSC_RED_NONFINITE, (isfinite(rho_d) && isfinite(ux) && isfinite(uy) && isfinite(uz)) ? 0.0 : 1.0);
    red.add(PSC_RED_SOLID, solid);
}

// The collision of deviations g (one cell, or two in packed FP32), or the moments only: the variant
// follows the window (TRT, moving) and what the launch asks for.
template <bool MOVING, bool RED, typename FW, typename V>
__device__ __forceinline__ void cell_collide(const FW& sw, V (&g)[Q], V B, V kb, V usx, V usy, V usz, bool do_collide,
                                             bool do_imb, V (&mom)[4], V (&imb)[3], bool do_mom) {
    const V drho = sum_populations(g);
    const V irho = rcp_v(vadd(lift<V>(1.0), drho));
    imb[0] = imb[1] = imb[2] = lift<V>(0.0);
    const bool want_mom = do_mom || RED;
    const bool moving = MOVING && sw.moving;
    if (do_collide) {
        if (sw.trt) {
            if (moving) collide_v<V, MOVING, true, true>(g, sw.c, drho, irho, B, kb, usx, usy, usz, mom, imb, want_mom);
            else collide_v<V, false, true, true>(g, sw.c, drho, irho, B, kb, usx, usy, usz, mom, imb, want_mom);
        } else if (do_imb || RED) {
            if (moving) collide_v<V, MOVING, true, false>(g, sw.c, drho, irho, B, kb, usx, usy, usz, mom, imb, want_mom);
            else collide_v<V, false, true, false>(g, sw.c, drho, irho, B, kb, usx, usy, usz, mom, imb, want_mom);
        } else {
            if (moving) collide_v<V, MOVING, false, false>(g, sw.c, drho, irho, B, kb, usx, usy, usz, mom, imb, want_mom);
            else collide_v<V, false, false, false>(g, sw.c, drho, irho, B, kb, usx, usy, usz, mom, imb, want_mom);
        }
    } else {
        V mx, my, mz;
        momentum(g, mx, my, mz);
        moments_v(sw.c, drho, irho, mx, my, mz, mom);
    }
}

// The per-cell work after the pulls (psc3d.py:211-246): inlet fix-up at an
// open x = 0, solid weight from the level tables, collision (or the moments
// only), and this thread's reduction sums.  g holds the pulled populations in
// stored units on entry and the post-collision deviations on exit; mom and
// imb receive the cell's moments (rho - 1, u) and IMB momentum.  The caller
// stores g, imb and mom.
// RED: PSC_STEP_REDUCE as a compile-time switch, so launches without
// reductions carry no loop-carried FP64 accumulators.
template <typename TR, bool MOVING, bool RED, typename S>
__device__ __forceinline__ void fast_cell(const FastWin<typename TR::T, typename TR::R, typename TR::O>& sw,
                                          typename TR::R (&g)[Q], uint32_t c, uint32_t N, bool inlet, bool do_collide,
                                          bool do_imb, typename TR::R (&mom)[4], typename TR::R (&imb)[3],
                                          S& red, bool do_mom = true) {
    using R = typename TR::R;
    if (TR::scaled) {
#pragma unroll
        for (int i = 0; i < Q; ++i) g[i] *= sw.inv_scale;
    }
    if (inlet) cell_inlet<TR>(sw, g, c, N);
    R B, kb, al;
    cell_solid(sw, c, B, kb, al);
    R usx = R(0), usy = R(0), usz = R(0);
    if (MOVING && sw.moving) {
        usx = (R)sw.us[c];
        usy = (R)sw.us[(size_t)N + c];
        usz = (R)sw.us[2 * (size_t)N + c];
    }
    cell_collide<MOVING, RED>(sw, g, B, kb, usx, usy, usz, do_collide, do_imb, mom, imb, do_mom);
    if (RED) cell_sums(red, al, mom, imb);
}

// Two consecutive cells c, c + 1 (c even) in packed FP32: fast_cell on both at once, in half its
// arithmetic instructions.
template <typename TR, bool MOVING, bool RED, typename S>
__device__ __forceinline__ void fast_cell_pair(const FastWin<typename TR::T, float, float, F2>& sw, F2 (&g)[Q],
                                               uint32_t c, uint32_t N, bool inlet, bool do_collide, bool do_imb,
                                               F2 (&mom)[4], F2 (&imb)[3], S& red, bool do_mom) {
    if (TR::scaled) {
        const F2 s = f2(sw.inv_scale, sw.inv_scale);
#pragma unroll
        for (int i = 0; i < Q; ++i) g[i] = vmul(g[i], s);
    }
    if (inlet) {
        float a[Q], b[Q];
#pragma unroll
        for (int i = 0; i < Q; ++i) f2_get(g[i], a[i], b[i]);
        cell_inlet<TR>(sw, a, c, N);
        cell_inlet<TR>(sw, b, c + 1, N);
#pragma unroll
        for (int i = 0; i < Q; ++i) g[i] = f2(a[i], b[i]);
    }
    float B0, B1, k0, k1, al0, al1;
    cell_solid(sw, c, B0, k0, al0);
    cell_solid(sw, c + 1, B1, k1, al1);
    F2 us[3] = {f2(0.0f, 0.0f), f2(0.0f, 0.0f), f2(0.0f, 0.0f)};
    if (MOVING && sw.moving) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float* p = sw.us + (size_t)k * N + c;
            us[k] = f2(p[0], p[1]);
        }
    }
    cell_collide<MOVING, RED>(sw, g, f2(B0, B1), f2(k0, k1), us[0], us[1], us[2], do_collide, do_imb, mom, imb, do_mom);
    if (RED) {
        float m0[4], m1[4], i0[3], i1[3];
#pragma unroll
        for (int k = 0; k < 4; ++k) f2_get(mom[k], m0[k], m1[k]);
#pragma unroll
        for (int k = 0; k < 3; ++k) f2_get(imb[k], i0[k], i1[k]);
        cell_sums(red, al0, m0, i0);
        cell_sums(red, al1, m1, i1);
    }
}

}  // namespace psc
