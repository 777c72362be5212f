// Per-node PSC-IMB collision: moments, Noble-Torczynski solid weighting, Guo
// forcing and the node IMB momentum.  Host+device so that the exact variant
// can be unit-tested on a CPU against the NumPy oracle.
//
// Two formulations of the same step (src/lbm_dem/psc3d.py:211-236):
//  * exact   -- absolute FP64 populations, every rounding in the reference's
//               order (NumPy evaluates one IEEE operation per ufunc call),
//               no FMA: bit-identical to the reference.
//  * fast<R> -- populations stored as deviations g_i = f_i - w_i (rho0 = 1),
//               arithmetic in R (double or float) with FMAs and reciprocal
//               multiplies.  The rest-weight offsets cancel in every
//               difference the step takes, so small deviations keep full
//               relative precision.
//
// Reference quirks reproduced by both (they are the method as published):
//  * moment velocity u = (m + F/2) / rho, and the collision uses a second
//    shift u_eff = u + F/(2 rho) = (m + F) / rho          (psc3d.py:214, 219)
//  * Guo forcing added at every node, not weighted by 1 - B  (psc3d.py:230-232)
//  * B = alpha / (alpha + tau (1 - alpha) + 1e-14)          (psc3d.py:229)
#pragma once

#include "d3q19.cuh"

namespace psc {

// ===========================================================================
// exact FP64
// ===========================================================================
struct ExactMoments {
    double rho, ux, uy, uz;
    Divisor by_rho;  // rho with its reciprocal
};

// x / c_s^2 and x / c_s^4, correctly rounded (Markstein's correction, d3q19.cuh)
PSC_HD double div_cs2(double x) { return xdiv_r(x, CS2, RCS2); }
PSC_HD double div_cs2sq(double x) { return xdiv_r(x, CS2SQ, RCS2SQ); }

// rho and u = (m + F/2)/rho of absolute populations f, psc3d.py:211-214.
PSC_HD ExactMoments moments_exact(const double* f, double hfx, double hfy, double hfz) {
    ExactMoments m;
    double rho = f[0];
#pragma unroll
    for (int i = 1; i < Q; ++i) rho = xadd(rho, f[i]);
    m.rho = rho;
    m.by_rho = make_divisor(rho);
    m.ux = xdiv_d(xadd(seq_moment_exact<0>(f), hfx), m.by_rho);
    m.uy = xdiv_d(xadd(seq_moment_exact<1>(f), hfy), m.by_rho);
    m.uz = xdiv_d(xadd(seq_moment_exact<2>(f), hfz), m.by_rho);
    return m;
}

PSC_HD double cm(int c, double x) { return c == 0 ? 0.0 : (c > 0 ? x : -x); }

// Velocity inlet by moving-wall bounce-back (Ladd 1994): the population i
// entering x = 0 from outside is the node's post-collision population opp(i)
// plus 2 w_i rho_in (c_i . u_in) / cs^2, which injects rho_in u_in per unit
// face area.  This is that term, in the operation order of the oracle.
PSC_HD double inlet_correction_exact(int i, double r, double x, double y, double z) {
    const double cu = xadd(xadd(cm(cxv(i), x), cm(cyv(i), y)), cm(czv(i), z));
    return div_cs2(xmul(xmul(2.0, xmul(wgt(i), r)), cu));
}

// The directions entering x = 0 from outside (c_x = +1).
PSC_HD constexpr bool enters_x0(int i) { return i == 1 || i == 7 || i == 9 || i == 11 || i == 13; }

// Collide f in place.  solid: clipped solid fraction.  moving: use (usx, usy,
// usz), else the solid velocity is zero.  imb receives sum_i c_i B Omega_s,i in
// the reference's sequential order (psc3d.py:234-236).
PSC_HD void collide_exact(double* f, const ExactMoments& mo, double solid, bool moving, double usx, double usy,
                          double usz, double tau, double fx, double fy, double fz, double hfx, double hfy,
                          double hfz, double* imb) {
    const double rho = mo.rho;
    const Divisor by_tau = make_divisor(tau);
    // u_eff = u + 0.5 F / rho   (psc3d.py:217-219)
    const double uex = xadd(mo.ux, xdiv_d(hfx, mo.by_rho));
    const double uey = xadd(mo.uy, xdiv_d(hfy, mo.by_rho));
    const double uez = xadd(mo.uz, xdiv_d(hfz, mo.by_rho));
    // equilibrium pieces shared by all directions (psc3d.py:98, :102)
    const double uu = xadd(xadd(xmul(uex, uex), xmul(uey, uey)), xmul(uez, uez));
    const double ct = div_cs2(xmul(0.5, uu));
    double uus = 0.0, cts = 0.0;
    if (moving) {
        uus = xadd(xadd(xmul(usx, usx), xmul(usy, usy)), xmul(usz, usz));
        cts = div_cs2(xmul(0.5, uus));
    }
    // B (psc3d.py:228-229)
    const double al = solid < 0.0 ? 0.0 : (solid > 1.0 ? 1.0 : solid);
    const double B = xdiv(al, xadd(xadd(al, xmul(tau, xsub(1.0, al))), 1.0e-14));
    const double omB = xsub(1.0, B);
    // Guo prefactor and u.F (psc3d.py:108-109)
    const double pref = xsub(1.0, xdiv_d(0.5, by_tau));
    const double uf = xadd(xadd(xmul(uex, fx), xmul(uey, fy)), xmul(uez, fz));

    double ix = 0.0, iy = 0.0, iz = 0.0;  // imb accumulators, index order from +0

    // rest population: cu = 0, cf = 0
    {
        const double wr = xmul(W0, rho);
        const double feqf = xmul(wr, xsub(1.0, ct));
        const double feqs = moving ? xmul(wr, xsub(1.0, cts)) : wr;
        const double f0 = f[0];
        const double os = xsub(feqs, feqf);  // (f0 - f0) + feqs - feqf
        const double obgk = -xdiv_d(xsub(f0, feqf), by_tau);
        const double coll = xadd(xmul(omB, obgk), xmul(B, os));
        const double g = xmul(xmul(pref, W0), div_cs2(-uf));
        f[0] = xadd(f0, xadd(coll, g));
    }
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        const int i = 2 * k + 1, j = i + 1;  // c_j = -c_i
        const double w = wgt(i);
        const double wr = xmul(w, rho);
        // feq with u_eff: cu_j = -cu_i exactly, so q_j = -q_i and b_j = b_i
        const double cu = xadd(xadd(cm(cxv(i), uex), cm(cyv(i), uey)), cm(czv(i), uez));
        const double q = div_cs2(cu);
        const double b = div_cs2sq(xmul(xmul(0.5, cu), cu));
        const double feqf_i = xmul(wr, xsub(xadd(xadd(1.0, q), b), ct));
        const double feqf_j = xmul(wr, xsub(xadd(xadd(1.0, -q), b), ct));
        double feqs_i = wr, feqs_j = wr;  // u_s = 0: feq = w rho exactly
        if (moving) {
            const double cus = xadd(xadd(cm(cxv(i), usx), cm(cyv(i), usy)), cm(czv(i), usz));
            const double qs = div_cs2(cus);
            const double bs = div_cs2sq(xmul(xmul(0.5, cus), cus));
            feqs_i = xmul(wr, xsub(xadd(xadd(1.0, qs), bs), cts));
            feqs_j = xmul(wr, xsub(xadd(xadd(1.0, -qs), bs), cts));
        }
        const double fi = f[i], fj = f[j];
        // Omega_s = f_opp - f + feq_s - feq_f[opp]   (psc3d.py:223-226)
        const double os_i = xsub(xadd(xsub(fj, fi), feqs_i), feqf_j);
        const double os_j = xsub(xadd(xsub(fi, fj), feqs_j), feqf_i);
        // Omega_bgk = -(f - feq_f) / tau   (psc3d.py:221)
        const double ob_i = -xdiv_d(xsub(fi, feqf_i), by_tau);
        const double ob_j = -xdiv_d(xsub(fj, feqf_j), by_tau);
        const double coll_i = xadd(xmul(omB, ob_i), xmul(B, os_i));
        const double coll_j = xadd(xmul(omB, ob_j), xmul(B, os_j));
        // Guo: pref W ((cf - uf)/cs2 + cu cf / cs2^2), cf_j = -cf_i   (psc3d.py:110-113)
        const double cf = xadd(xadd(cm(cxv(i), fx), cm(cyv(i), fy)), cm(czv(i), fz));
        const double pw = xmul(pref, w);
        const double t2 = div_cs2sq(xmul(cu, cf));
        const double g_i = xmul(pw, xadd(div_cs2(xsub(cf, uf)), t2));
        const double g_j = xmul(pw, xadd(div_cs2(xsub(-cf, uf)), t2));
        f[i] = xadd(fi, xadd(coll_i, g_i));
        f[j] = xadd(fj, xadd(coll_j, g_j));
        // node IMB momentum, sequential in index order (i then j)
        const double bo_i = xmul(B, os_i), bo_j = xmul(B, os_j);
        ix = cxv(i) > 0 ? xadd(ix, bo_i) : (cxv(i) < 0 ? xsub(ix, bo_i) : ix);
        ix = cxv(j) > 0 ? xadd(ix, bo_j) : (cxv(j) < 0 ? xsub(ix, bo_j) : ix);
        iy = cyv(i) > 0 ? xadd(iy, bo_i) : (cyv(i) < 0 ? xsub(iy, bo_i) : iy);
        iy = cyv(j) > 0 ? xadd(iy, bo_j) : (cyv(j) < 0 ? xsub(iy, bo_j) : iy);
        iz = czv(i) > 0 ? xadd(iz, bo_i) : (czv(i) < 0 ? xsub(iz, bo_i) : iz);
        iz = czv(j) > 0 ? xadd(iz, bo_j) : (czv(j) < 0 ? xsub(iz, bo_j) : iz);
    }
    imb[0] = ix;
    imb[1] = iy;
    imb[2] = iz;
}

// ---------------------------------------------------------------------------
// The same arithmetic without branches (the step kernels' path)
// ---------------------------------------------------------------------------
// moments_exact and collide_exact rounding for rounding, with the divisions of
// d3q19.cuh's branch-free forms and the window's constants made once.  Each
// function returns whether an operand left the range of those forms; the
// caller then takes the cell through moments_exact / collide_exact.
//
// The range is tested on the roots of a cell's arithmetic, in integer instructions (the FP64 pipe is
// what bounds the exact kernels): every population in [2^-15, 2), rho in [2^-8, 2^8), tau in
// [2^-8, 2^8], the components of F and of the solid velocity and the solid fraction zero or in
// [2^-200, 2^200).  All other
// operands follow.  A sum or difference of doubles is a multiple of the smaller one's ulp, so
// m + F/2 is zero or >= 2^-253, u + F/(2 rho) zero or >= 2^-313, c.u zero or >= 2^-365 and its
// square >= 2^-730, u.F and c.F - u.F zero or >= 2^-565, (c.u)(c.F) >= 2^-617, feq zero or >= 2^-796
// and f - feq zero or >= 2^-848; nothing exceeds 2^500.  Each form needs zero or 2^-900 .. 2^900.
//
// FP64 operations of a static cell with IMB momentum and F along an axis: about 575 (1360 with
// xdiv_r's five operations and two comparisons per division, and a branch each).
constexpr int kExactRootRange = 200;

struct ExactWin {
    double tau, rtau, rtau_lo;       // 1/tau = rtau + rtau_lo
    double fx, fy, fz, hfx, hfy, hfz;
    double pw[3];                    // (1 - 0.5 / tau) w for the rest, axis and diagonal weights
    double cf[9];                    // c_k . F of the nine direction pairs
    int axis;                        // the axis of a body force along one axis, else -1
    int out;                         // tau or F outside the branch-free forms' range
};

// The parts of ExactWin, independent of one another (a CTA's warps make one each).
PSC_HD void exact_win_force(ExactWin& w, double tau, double fx, double fy, double fz) {
    w.tau = tau;
    w.fx = fx;
    w.fy = fy;
    w.fz = fz;
    w.hfx = xmul(0.5, fx);
    w.hfy = xmul(0.5, fy);
    w.hfz = xmul(0.5, fz);
    w.out = !div_r_divisor_ok(tau) || out_of_range<kExactRootRange>(fx) || out_of_range<kExactRootRange>(fy) ||
            out_of_range<kExactRootRange>(fz);
    w.axis = fx == 0.0 && fy == 0.0 ? 2 : (fx == 0.0 && fz == 0.0 ? 1 : (fy == 0.0 && fz == 0.0 ? 0 : -1));
}
PSC_HD void exact_win_tau(ExactWin& w, double tau) {
    w.rtau = xdiv(1.0, tau);
    w.rtau_lo = xmul(xfma(-w.rtau, tau, 1.0), w.rtau);
}
PSC_HD void exact_win_guo(ExactWin& w, double tau) {
    const double pref = xsub(1.0, xdiv(0.5, tau));
    w.pw[0] = xmul(pref, W0);
    w.pw[1] = xmul(pref, W1);
    w.pw[2] = xmul(pref, W2);
}
PSC_HD void exact_win_pairs(ExactWin& w, double fx, double fy, double fz) {
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        const int i = 2 * k + 1;
        w.cf[k] = xadd(xadd(cm(cxv(i), fx), cm(cyv(i), fy)), cm(czv(i), fz));
    }
}
PSC_HD void make_exact_win(ExactWin& w, double tau, double fx, double fy, double fz) {
    exact_win_force(w, tau, fx, fy, fz);
    exact_win_tau(w, tau);
    exact_win_guo(w, tau);
    exact_win_pairs(w, fx, fy, fz);
}

// What a cell's Guo terms share.  (c_k . F - u . F) / c_s^2 depends on c_k . F alone, which takes three
// values where F lies along one axis: they are divided once per cell (d0, dp, dm) and selected per pair.
struct ExactGuo {
    double uf, d0, dp, dm;
};

// u + F / (2 rho), u . F and the shared Guo terms; AXIS: F lies along the axis w.axis.
template <bool AXIS>
PSC_HD ExactGuo exact_guo_s(const ExactWin& w, double rho, double rrho, double half, double& ux, double& uy, double& uz) {
    ExactGuo g;
    if (AXIS) {
        const int a = w.axis;
        const double F = a == 0 ? w.fx : (a == 1 ? w.fy : w.fz);
        if (half != 0.0) {
            const double h = xdiv_r_s(xmul(half, F), rho, rrho);
            ux = xadd(ux, a == 0 ? h : 0.0);
            uy = xadd(uy, a == 1 ? h : 0.0);
            uz = xadd(uz, a == 2 ? h : 0.0);
        }
        g.uf = xmul(a == 0 ? ux : (a == 1 ? uy : uz), F);
        g.d0 = div_cs2_s(-g.uf);
        g.dp = div_cs2_s(xsub(F, g.uf));
        g.dm = div_cs2_s(xsub(-F, g.uf));
    } else {
        if (half != 0.0) {
            ux = xadd(ux, xdiv_r_s(w.hfx, rho, rrho));
            uy = xadd(uy, xdiv_r_s(w.hfy, rho, rrho));
            uz = xadd(uz, xdiv_r_s(w.hfz, rho, rrho));
        }
        g.uf = xadd(xadd(xmul(ux, w.fx), xmul(uy, w.fy)), xmul(uz, w.fz));
        g.d0 = div_cs2_s(-g.uf);
        g.dp = g.dm = 0.0;
    }
    return g;
}

// (c . F - u . F) / c_s^2 for the direction c = (CX, CY, CZ) and F along `axis`.
template <int C>
PSC_HD double exact_by_sign(const ExactGuo& g) {
    return C == 0 ? g.d0 : (C > 0 ? g.dp : g.dm);
}
template <int CX, int CY, int CZ>
PSC_HD double exact_by_axis(int axis, const ExactGuo& g) {
    if constexpr (CX == CY) return axis == 2 ? exact_by_sign<CZ>(g) : exact_by_sign<CX>(g);
    else if constexpr (CX == CZ) return axis == 1 ? exact_by_sign<CY>(g) : exact_by_sign<CX>(g);
    else if constexpr (CY == CZ) return axis == 0 ? exact_by_sign<CX>(g) : exact_by_sign<CY>(g);
    else return axis == 0 ? exact_by_sign<CX>(g) : (axis == 1 ? exact_by_sign<CY>(g) : exact_by_sign<CZ>(g));
}

// The Guo terms of a pair, pref w ((c . F - u . F) / c_s^2 + (c . u)(c . F) / c_s^4).
template <bool AXIS, int K>
PSC_HD void exact_guo_pair_s(const ExactWin& w, const ExactGuo& g, double pw, double cu, double& g_i, double& g_j) {
    const double cf = w.cf[K];
    const double t2 = div_cs2sq_s(xmul(cu, cf));
    if (AXIS) {
        g_i = xmul(pw, xadd(exact_by_axis<cxv(2 * K + 1), cyv(2 * K + 1), czv(2 * K + 1)>(w.axis, g), t2));
        g_j = xmul(pw, xadd(exact_by_axis<cxv(2 * K + 2), cyv(2 * K + 2), czv(2 * K + 2)>(w.axis, g), t2));
    } else {
        g_i = xmul(pw, xadd(div_cs2_s(xsub(cf, g.uf)), t2));
        g_j = xmul(pw, xadd(div_cs2_s(xsub(-cf, g.uf)), t2));
    }
}

// c_i . v without the additions of a zero component (they change no value).
template <int I>
PSC_HD double cdot_s(double x, double y, double z) {
    constexpr int a = cxv(I), b = cyv(I), c = czv(I);
    if constexpr (a != 0 && b != 0) return xadd(a > 0 ? x : -x, b > 0 ? y : -y);
    else if constexpr (a != 0 && c != 0) return xadd(a > 0 ? x : -x, c > 0 ? z : -z);
    else if constexpr (b != 0 && c != 0) return xadd(b > 0 ? y : -y, c > 0 ? z : -z);
    else if constexpr (a != 0) return a > 0 ? x : -x;
    else if constexpr (b != 0) return b > 0 ? y : -y;
    else return c > 0 ? z : -z;
}

// acc + c v for the component c of direction I along AXIS (the first term starts the sum).
template <int AXIS, int I>
PSC_HD void moment_add_s(double& acc, bool& first, double v) {
    constexpr int c = cv(AXIS, I);
    if constexpr (c != 0) {
        acc = first ? (c > 0 ? v : -v) : (c > 0 ? xadd(acc, v) : xsub(acc, v));
        first = false;
    }
}
template <int AXIS, int I = 0>
PSC_HD void seq_moment_s(const double* f, double& acc, bool& first) {
    if constexpr (I < Q) {
        moment_add_s<AXIS, I>(acc, first, f[I]);
        seq_moment_s<AXIS, I + 1>(f, acc, first);
    }
}

struct ExactMomentsS {
    double rho, ux, uy, uz, rrho;
    bool out;
};

// .out: the populations or rho left the range; F / 2 is ExactWin.out's to test.
PSC_HD ExactMomentsS moments_exact_s(const double* f, double hfx, double hfy, double hfz) {
    ExactMomentsS m;
    double rho = f[0];
#pragma unroll
    for (int i = 1; i < Q; ++i) rho = xadd(rho, f[i]);
    double mx = 0.0, my = 0.0, mz = 0.0;
    bool a = true, b = true, c = true;
    seq_moment_s<0>(f, mx, a);
    seq_moment_s<1>(f, my, b);
    seq_moment_s<2>(f, mz, c);
    mx = xadd(mx, hfx);
    my = xadd(my, hfy);
    mz = xadd(mz, hfz);
    uint32_t h = hi_word(f[0]) ^ 0x3f000000u;  // 2^-15 <= f < 2: the sign and seven exponent bits are 0x3f
#pragma unroll
    for (int i = 1; i < Q; ++i) h |= hi_word(f[i]) ^ 0x3f000000u;
    m.out = (h >= 0x01000000u) | (hi_word(rho) - (1015u << 20) >= (16u << 20));  // 2^-8 <= rho < 2^8
    m.rho = rho;
    m.rrho = xrcp(rho);
    m.ux = xdiv_r_s(mx, rho, m.rrho);
    m.uy = xdiv_r_s(my, rho, m.rrho);
    m.uz = xdiv_r_s(mz, rho, m.rrho);
    return m;
}

template <int K, bool MOVING, bool IMB, bool AXIS>
PSC_HD void exact_pair_s(double* f, const ExactWin& w, double wr, double pw, double ct, const ExactGuo& guo, double B,
                         double omB, double uex, double uey, double uez, double usx, double usy, double usz,
                         double cts, double& ix, double& iy, double& iz) {
    constexpr int i = 2 * K + 1, j = i + 1;
    const double cu = cdot_s<i>(uex, uey, uez);
    const double q = div_cs2_s(cu);
    const double b = half_div_cs2sq_s(xmul(cu, cu));
    const double feqf_i = xmul(wr, xsub(xadd(xadd(1.0, q), b), ct));
    const double feqf_j = xmul(wr, xsub(xadd(xsub(1.0, q), b), ct));
    double feqs_i = wr, feqs_j = wr;
    if (MOVING) {
        const double cus = cdot_s<i>(usx, usy, usz);
        const double qs = div_cs2_s(cus);
        const double bs = half_div_cs2sq_s(xmul(cus, cus));
        feqs_i = xmul(wr, xsub(xadd(xadd(1.0, qs), bs), cts));
        feqs_j = xmul(wr, xsub(xadd(xsub(1.0, qs), bs), cts));
    }
    const double fi = f[i], fj = f[j];
    const double dji = xsub(fj, fi);
    const double os_i = xsub(xadd(dji, feqs_i), feqf_j);
    const double os_j = xsub(xadd(-dji, feqs_j), feqf_i);
    const double di = xsub(fi, feqf_i), dj = xsub(fj, feqf_j);
    const double bo_i = xmul(B, os_i), bo_j = xmul(B, os_j);
    const double coll_i = xsub(bo_i, xmul(omB, xdiv_s(di, w.tau, w.rtau, w.rtau_lo)));
    const double coll_j = xsub(bo_j, xmul(omB, xdiv_s(dj, w.tau, w.rtau, w.rtau_lo)));
    double g_i, g_j;
    exact_guo_pair_s<AXIS, K>(w, guo, pw, cu, g_i, g_j);
    f[i] = xadd(fi, xadd(coll_i, g_i));
    f[j] = xadd(fj, xadd(coll_j, g_j));
    if (IMB) {
        if constexpr (cxv(i) != 0) ix = cxv(i) > 0 ? xsub(xadd(ix, bo_i), bo_j) : xadd(xsub(ix, bo_i), bo_j);
        if constexpr (cyv(i) != 0) iy = cyv(i) > 0 ? xsub(xadd(iy, bo_i), bo_j) : xadd(xsub(iy, bo_i), bo_j);
        if constexpr (czv(i) != 0) iz = czv(i) > 0 ? xsub(xadd(iz, bo_i), bo_j) : xadd(xsub(iz, bo_i), bo_j);
    }
}

// collide_exact in the branch-free forms; true where an operand left their range (f is then undefined).
template <bool MOVING, bool IMB, bool AXIS>
PSC_HD bool collide_exact_s(double* f, const ExactMomentsS& mo, double solid, double usx, double usy, double usz,
                            const ExactWin& w, double* imb) {
    const double rho = mo.rho;
    double uex = mo.ux, uey = mo.uy, uez = mo.uz;
    const ExactGuo guo = exact_guo_s<AXIS>(w, rho, mo.rrho, 0.5, uex, uey, uez);
    bool out = mo.out | (w.out != 0);
    const double ct = half_div_cs2_s(xadd(xadd(xmul(uex, uex), xmul(uey, uey)), xmul(uez, uez)));
    double cts = 0.0;
    if (MOVING) {
        out |= out_of_range<kExactRootRange>(usx) | out_of_range<kExactRootRange>(usy) |
               out_of_range<kExactRootRange>(usz);
        cts = half_div_cs2_s(xadd(xadd(xmul(usx, usx), xmul(usy, usy)), xmul(usz, usz)));
    }
    const double al = solid < 0.0 ? 0.0 : (solid > 1.0 ? 1.0 : solid);
    out |= out_of_range<kExactRootRange>(al);
    const double den = xadd(xadd(al, xmul(w.tau, xsub(1.0, al))), 1.0e-14);  // between 1 and tau
    const double B = xdiv_r_s(al, den, xrcp(den));
    const double omB = xsub(1.0, B);
    double ix = 0.0, iy = 0.0, iz = 0.0;
    {  // rest population
        const double wr = xmul(W0, rho);
        const double feqf = xmul(wr, xsub(1.0, ct));
        const double feqs = MOVING ? xmul(wr, xsub(1.0, cts)) : wr;
        const double d = xsub(f[0], feqf);
        const double coll = xsub(xmul(B, xsub(feqs, feqf)), xmul(omB, xdiv_s(d, w.tau, w.rtau, w.rtau_lo)));
        f[0] = xadd(f[0], xadd(coll, xmul(w.pw[0], guo.d0)));
    }
    const double wr1 = xmul(W1, rho), wr2 = xmul(W2, rho);
    const double pw1 = w.pw[1], pw2 = w.pw[2];
#define PSC_EXACT_PAIR(K)                                                                                          \
    exact_pair_s<K, MOVING, IMB, AXIS>(f, w, K < 3 ? wr1 : wr2, K < 3 ? pw1 : pw2, ct, guo, B, omB, uex, uey, uez,  \
                                       usx, usy, usz, cts, ix, iy, iz)
    PSC_EXACT_PAIR(0);
    PSC_EXACT_PAIR(1);
    PSC_EXACT_PAIR(2);
    PSC_EXACT_PAIR(3);
    PSC_EXACT_PAIR(4);
    PSC_EXACT_PAIR(5);
    PSC_EXACT_PAIR(6);
    PSC_EXACT_PAIR(7);
    PSC_EXACT_PAIR(8);
#undef PSC_EXACT_PAIR
    if (IMB) {
        imb[0] = ix;
        imb[1] = iy;
        imb[2] = iz;
    }
    return out;
}

// ===========================================================================
// fast deviation form, arithmetic type R
// ===========================================================================
template <typename R>
struct FastMoments {
    R drho, rho, mx, my, mz;
};

template <typename R>
PSC_HD FastMoments<R> moments_fast(const R* g) {
    FastMoments<R> m;
    m.drho = (((g[0] + g[1]) + (g[2] + g[3])) + ((g[4] + g[5]) + (g[6] + g[7]))) +
             (((g[8] + g[9]) + (g[10] + g[11])) + ((g[12] + g[13]) + (g[14] + g[15]))) + ((g[16] + g[17]) + g[18]);
    m.rho = R(1) + m.drho;
    m.mx = ((g[1] - g[2]) + (g[7] - g[8])) + ((g[9] - g[10]) + (g[11] - g[12])) + (g[13] - g[14]);
    m.my = ((g[3] - g[4]) + (g[7] - g[8])) + ((g[10] - g[9]) + (g[15] - g[16])) + (g[17] - g[18]);
    m.mz = ((g[5] - g[6]) + (g[11] - g[12])) + ((g[14] - g[13]) + (g[15] - g[16])) + (g[18] - g[17]);
    return m;
}

template <typename R>
struct FastParams {
    R inv_tau, pref, fx, fy, fz;
};

// c * x for a lattice component c in {-1, 0, 1} (folded once loops unroll).
template <typename R>
PSC_HD R csel(int c, R x) {
    return c == 0 ? R(0) : (c > 0 ? x : -x);
}

// Collide deviations g in place; irho = 1 / rho; B solid weight.  The plain form,
// term by term: no kernel runs it, the host tests hold it and the regrouped form
// below, which the kernels run, to the same oracle.  imb gets
// sum_i c_i B Omega_s,i.  Returns nothing else: the caller owns the moments.
template <typename R, bool MOVING, bool IMB>
PSC_HD void collide_fast(R* g, const FastMoments<R>& mo, R irho, R B, R usx, R usy, R usz,
                         const FastParams<R>& p, R* imb) {
    const R rho = mo.rho, drho = mo.drho;
    const R uex = (mo.mx + p.fx) * irho;
    const R uey = (mo.my + p.fy) * irho;
    const R uez = (mo.mz + p.fz) * irho;
    const R uu = uex * uex + uey * uey + uez * uez;
    const R uf = uex * p.fx + uey * p.fy + uez * p.fz;
    const R omB = R(1) - B;
    const R kb = omB * p.inv_tau;  // (1 - B) / tau
    R uus = R(0);
    if (MOVING) uus = usx * usx + usy * usy + usz * usz;
    const R r15 = R(1.5) * rho;
    R ax = R(0), ay = R(0), az = R(0);
    {
        const R geq = R(W0) * (drho - r15 * uu);
        const R os = R(W0) * r15 * (uu - uus);
        const R G = R(-3) * p.pref * R(W0) * uf;
        g[0] = g[0] - kb * (g[0] - geq) + B * os + G;
    }
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        const int i = 2 * k + 1, j = i + 1;
        const R w = R(wgt(i));
        const R cu = csel(cxv(i), uex) + csel(cyv(i), uey) + csel(czv(i), uez);
        const R cF = csel(cxv(i), p.fx) + csel(cyv(i), p.fy) + csel(czv(i), p.fz);
        const R sym = w * (drho + rho * (R(4.5) * cu * cu - R(1.5) * uu));
        const R asym = R(3) * w * rho * cu;
        R ssym, sasym;
        if (MOVING) {
            const R cus = csel(cxv(i), usx) + csel(cyv(i), usy) + csel(czv(i), usz);
            ssym = w * (drho + rho * (R(4.5) * cus * cus - R(1.5) * uus));
            sasym = R(3) * w * rho * cus;
        } else {
            ssym = w * drho;
            sasym = R(0);
        }
        const R gi = g[i], gj = g[j];
        const R d = gj - gi;
        const R e = ssym - sym;
        const R h = sasym + asym;
        const R os_i = d + e + h;
        const R os_j = e - d - h;
        const R pw = p.pref * w;
        const R t9 = R(9) * cu * cF;
        const R G_i = pw * (R(3) * (cF - uf) + t9);
        const R G_j = pw * (R(3) * (-cF - uf) + t9);
        g[i] = gi - kb * (gi - (sym + asym)) + B * os_i + G_i;
        g[j] = gj - kb * (gj - (sym - asym)) + B * os_j + G_j;
        if (IMB) {
            const R dm = B * (os_i - os_j);  // c_i B os_i + c_j B os_j = c_i B (os_i - os_j)
            ax += csel(cxv(i), dm);
            ay += csel(cyv(i), dm);
            az += csel(czv(i), dm);
        }
    }
    if (IMB) {
        imb[0] = ax;
        imb[1] = ay;
        imb[2] = az;
    }
}

}  // namespace psc

namespace psc {

// ===========================================================================
// fast deviation form with per-window constants hoisted (throughput kernels)
// ===========================================================================
// Everything that depends only on the window (tau, F) is computed once per
// window: (1 - B)/tau comes from a per-level table, the Guo terms are split
// into per-direction constants A_k = 3 pref w_k (c_k . F) and
// K_k = 9 pref w_k (c_k . F) so that G_i = K_k cu - 3 pref w uF +- A_k.
//
// V is what one evaluation works on: one cell in float or double, or two cells
// at once in packed FP32 (F2).  Every product that feeds a sum is an explicit
// fused multiply-add, so a packed cell and a scalar cell round alike.
PSC_HD float vadd(float a, float b) { return a + b; }
PSC_HD double vadd(double a, double b) { return a + b; }
PSC_HD float vsub(float a, float b) { return a - b; }
PSC_HD double vsub(double a, double b) { return a - b; }
#if defined(__CUDA_ARCH__)
PSC_HD float vmul(float a, float b) { return __fmul_rn(a, b); }
PSC_HD double vmul(double a, double b) { return __dmul_rn(a, b); }
PSC_HD float vfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
PSC_HD double vfma(double a, double b, double c) { return __fma_rn(a, b, c); }
#else
PSC_HD float vmul(float a, float b) { return a * b; }
PSC_HD double vmul(double a, double b) { return a * b; }
PSC_HD float vfma(float a, float b, float c) { return std::fma(a, b, c); }
PSC_HD double vfma(double a, double b, double c) { return std::fma(a, b, c); }
#endif

// Two floats in one 64-bit register pair: the sm_100 instructions on both halves at once (a host
// build computes the halves one after the other).
struct F2 {
    unsigned long long v;
};
PSC_HD F2 f2(float a, float b) {
    F2 r;
#if defined(__CUDA_ARCH__)
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
#else
    const float h[2] = {a, b};
    std::memcpy(&r.v, h, sizeof(r.v));
#endif
    return r;
}
PSC_HD void f2_get(F2 x, float& a, float& b) {
#if defined(__CUDA_ARCH__)
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x.v));
#else
    float h[2];
    std::memcpy(h, &x.v, sizeof(x.v));
    a = h[0];
    b = h[1];
#endif
}
#if defined(__CUDA_ARCH__)
#define PSC_F2_OP2(NAME)                                                                        \
    PSC_HD F2 v##NAME(F2 a, F2 b) {                                                             \
        F2 r;                                                                                   \
        asm(#NAME ".rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));                    \
        return r;                                                                               \
    }
#else
#define PSC_F2_OP2(NAME)                                                                        \
    PSC_HD F2 v##NAME(F2 a, F2 b) {                                                             \
        float a0, a1, b0, b1;                                                                   \
        f2_get(a, a0, a1);                                                                      \
        f2_get(b, b0, b1);                                                                      \
        return f2(v##NAME(a0, b0), v##NAME(a1, b1));                                            \
    }
#endif
PSC_F2_OP2(add)
PSC_F2_OP2(sub)
PSC_F2_OP2(mul)
#undef PSC_F2_OP2
PSC_HD F2 vfma(F2 a, F2 b, F2 c) {
    F2 r;
#if defined(__CUDA_ARCH__)
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
#else
    float a0, a1, b0, b1, c0, c1;
    f2_get(a, a0, a1);
    f2_get(b, b0, b1);
    f2_get(c, c0, c1);
    r = f2(vfma(a0, b0, c0), vfma(a1, b1, c1));
#endif
    return r;
}

template <typename V>
struct Lift {
    PSC_HD static V of(double x) { return (V)x; }
};
template <>
struct Lift<F2> {
    PSC_HD static F2 of(double x) { return f2((float)x, (float)x); }
};
template <typename V>
PSC_HD V lift(double x) {
    return Lift<V>::of(x);
}

template <typename V>
struct WinConst {
    V inv_tau;
    V trt_ratio;  // omega- / omega+ (1 for BGK)
    V fx, fy, fz;
    V hfx, hfy, hfz;  // F / 2
    V npw3[3];        // -3 pref w for the rest, axis and diagonal weights
    V A[9];           // 3 pref w_k (c_k . F) for the nine direction pairs
    V K[9];           // 9 pref w_k (c_k . F)
};

// tau_minus > 0 selects two-relaxation-time collision (symmetric parts relax
// with 1/tau, antisymmetric with 1/tau_minus; Guo's antisymmetric term takes
// the prefactor 1 - 1/(2 tau_minus)).  tau_minus = tau is BGK.
template <typename V>
PSC_HD void make_win_const(WinConst<V>& c, double tau, double fx, double fy, double fz, double tau_minus = 0.0) {
    const double pref = 1.0 - 0.5 / tau;
    const double tm = tau_minus > 0.0 ? tau_minus : tau;
    const double pref_m = 1.0 - 0.5 / tm;
    c.inv_tau = lift<V>(1.0 / tau);
    c.trt_ratio = lift<V>(tau / tm);
    c.fx = lift<V>(fx);
    c.fy = lift<V>(fy);
    c.fz = lift<V>(fz);
    c.hfx = lift<V>(0.5 * fx);
    c.hfy = lift<V>(0.5 * fy);
    c.hfz = lift<V>(0.5 * fz);
    c.npw3[0] = lift<V>(-3.0 * pref * W0);
    c.npw3[1] = lift<V>(-3.0 * pref * W1);
    c.npw3[2] = lift<V>(-3.0 * pref * W2);
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        const int i = 2 * k + 1;
        const double w = wgt(i);
        const double cf = cxv(i) * fx + cyv(i) * fy + czv(i) * fz;
        c.A[k] = lift<V>(3.0 * pref_m * w * cf);
        c.K[k] = lift<V>(9.0 * pref * w * cf);
    }
}

// c_i . v for the first direction i of pair K (its first non-zero component is +1).
template <int K, typename V>
PSC_HD V cdot_v(V x, V y, V z) {
    constexpr int i = 2 * K + 1, a = cxv(i), b = cyv(i), c = czv(i);
    if constexpr (a != 0 && b != 0) return b > 0 ? vadd(x, y) : vsub(x, y);
    else if constexpr (a != 0 && c != 0) return c > 0 ? vadd(x, z) : vsub(x, z);
    else if constexpr (b != 0 && c != 0) return c > 0 ? vadd(y, z) : vsub(y, z);
    else return a != 0 ? x : (b != 0 ? y : z);
}

template <typename V>
PSC_HD V sum_populations(const V* g) {
    return vadd(vadd(vadd(vadd(vadd(g[0], g[1]), vadd(g[2], g[3])), vadd(vadd(g[4], g[5]), vadd(g[6], g[7]))),
                     vadd(vadd(vadd(g[8], g[9]), vadd(g[10], g[11])), vadd(vadd(g[12], g[13]), vadd(g[14], g[15])))),
                vadd(vadd(g[16], g[17]), g[18]));
}
template <typename V>
PSC_HD void momentum(const V* g, V& mx, V& my, V& mz) {
    mx = vadd(vadd(vadd(vsub(g[1], g[2]), vsub(g[7], g[8])), vadd(vsub(g[9], g[10]), vsub(g[11], g[12]))),
              vsub(g[13], g[14]));
    my = vadd(vadd(vadd(vsub(g[3], g[4]), vsub(g[7], g[8])), vadd(vsub(g[10], g[9]), vsub(g[15], g[16]))),
              vsub(g[17], g[18]));
    mz = vadd(vadd(vadd(vsub(g[5], g[6]), vsub(g[11], g[12])), vadd(vsub(g[14], g[13]), vsub(g[15], g[16]))),
              vsub(g[18], g[17]));
}
// The moments handed on: rho - 1 and u = (m + F/2) / rho of the incoming state.
template <typename V>
PSC_HD void moments_v(const WinConst<V>& c, V drho, V irho, V mx, V my, V mz, V* mom) {
    mom[0] = drho;
    mom[1] = vmul(vadd(mx, c.hfx), irho);
    mom[2] = vmul(vadd(my, c.hfy), irho);
    mom[3] = vmul(vadd(mz, c.hfz), irho);
}

// What the nine pairs of a cell share (see collide_v).
template <typename V>
struct PairTerms {
    V uex, uey, uez, usx, usy, usz, uus15;
    V omB, bB, B, B2;
    V wr[2], q[2], b[2], t[2], a[2];  // axis and diagonal weights
};

template <int K, bool MOVING, bool IMB, typename V>
PSC_HD void collide_pair_v(V* g, const WinConst<V>& c, const PairTerms<V>& p, V* imb) {
    constexpr int i = 2 * K + 1, j = i + 1, d = i < 7 ? 0 : 1;
    const V cu = cdot_v<K>(p.uex, p.uey, p.uez);
    V S = vfma(cu, vfma(p.q[d], cu, c.K[K]), p.b[d]);
    V T = vfma(p.t[d], cu, c.A[K]);
    const V gi = g[i], gj = g[j];
    V h = vsub(gj, gi);  // + h: (os_i - os_j) / 2
    if (IMB) h = vfma(p.a[d], cu, h);
    if (MOVING) {
        const V cus = cdot_v<K>(p.usx, p.usy, p.usz);
        S = vfma(p.B, vmul(p.wr[d], vsub(vmul(lift<V>(4.5), vmul(cus, cus)), p.uus15)), S);
        const V hs = vmul(p.a[d], cus);
        T = vfma(p.B, hs, T);
        if (IMB) h = vadd(h, hs);
    }
    g[i] = vfma(p.omB, gi, vfma(p.bB, gj, vadd(S, T)));
    g[j] = vfma(p.omB, gj, vfma(p.bB, gi, vsub(S, T)));
    if (IMB) {
        const V dm = vmul(p.B2, h);
        if constexpr (cxv(i) != 0) imb[0] = K == 0 ? dm : vadd(imb[0], dm);
        if constexpr (cyv(i) != 0) imb[1] = K == 1 ? dm : (cyv(i) > 0 ? vadd(imb[1], dm) : vsub(imb[1], dm));
        if constexpr (czv(i) != 0) imb[2] = K == 2 ? dm : (czv(i) > 0 ? vadd(imb[2], dm) : vsub(imb[2], dm));
    }
}

// Collide deviations g in place.  drho = rho - 1 and irho = 1 / rho of the
// incoming state, B solid weight, kb = (1 - B) / tau.  mom receives rho - 1
// and the moment velocity u = (m + F/2)/rho of the incoming state when
// want_mom; imb the node IMB momentum when IMB.
//
// The collision regrouped per population pair.  With geq = w drho + wrq +- asym, the solid
// terms os_i = (g_j - g_i) + e + h, os_j = (g_i - g_j) + e - h (e = -wrq + e_s,
// h = asym + h_s, e_s and h_s from the solid velocity), Guo's G = K cu - 3 pref w uF +- A,
// and the fluid part relaxing the pair's symmetric half with kb and its antisymmetric half
// with kbm (= kb for BGK; TRT: kb omega-/omega+):
//   g_i' = a g_i + b g_j + S + T,   g_j' = a g_j + b g_i + S - T,
//   a = 1 - (kb + kbm)/2 - B,  b = B + (kbm - kb)/2   (BGK: 1 - kb - B and B),
//   S = K cu + (kb - B) wrq + (kb w drho - 3 pref w uF) + B e_s,
//   T = 3 (kbm + B) w rho cu + B h_s + A,
// and the pair's IMB momentum B (os_i - os_j) = 2 B ((g_j - g_i) + h).  With
// wrq = w rho (4.5 cu^2 - 1.5 u^2), S without e_s is the quadratic cu (q cu + K) + b,
// q = 4.5 (kb - B) w rho, b = kb w drho - 3 pref w uF - (kb - B) w rho 1.5 u^2: two FMAs per
// pair.  The per-weight factors are computed once per cell.
template <typename V, bool MOVING, bool IMB, bool TRT>
PSC_HD void collide_v(V* g, const WinConst<V>& c, V drho, V irho, V B, V kb, V usx, V usy, V usz, V* mom, V* imb,
                      bool want_mom) {
    const V one = lift<V>(1.0), half = lift<V>(0.5);
    const V rho = vadd(one, drho);
    V mx, my, mz;
    momentum(g, mx, my, mz);
    if (want_mom) moments_v(c, drho, irho, mx, my, mz, mom);  // (plain steps store no moments)
    PairTerms<V> p;
    p.uex = vmul(vadd(mx, c.fx), irho);
    p.uey = vmul(vadd(my, c.fy), irho);
    p.uez = vmul(vadd(mz, c.fz), irho);
    const V uu15 = vmul(lift<V>(1.5), vfma(p.uez, p.uez, vfma(p.uey, p.uey, vmul(p.uex, p.uex))));
    const V uF = vfma(p.uez, c.fz, vfma(p.uey, c.fy, vmul(p.uex, c.fx)));
    const V omk = vsub(one, kb);
    const V rq = vmul(rho, uu15);
    V e0 = rq;  // rho (1.5 u^2 - 1.5 us^2)
    if (MOVING) {
        p.usx = usx;
        p.usy = usy;
        p.usz = usz;
        p.uus15 = vmul(lift<V>(1.5), vfma(usz, usz, vfma(usy, usy, vmul(usx, usx))));
        e0 = vmul(rho, vsub(uu15, p.uus15));
    }
    {
        const V geq = vmul(lift<V>(W0), vsub(drho, rq));
        const V os = vmul(lift<V>(W0), e0);
        g[0] = vfma(omk, g[0], vfma(kb, geq, vfma(B, os, vmul(c.npw3[0], uF))));
    }
    const V kbm = TRT ? vmul(kb, c.trt_ratio) : kb;
    p.B = B;
    p.omB = TRT ? vsub(vsub(one, vmul(half, vadd(kb, kbm))), B) : vsub(omk, B);
    p.bB = TRT ? vfma(half, vsub(kbm, kb), B) : B;
    p.B2 = vadd(B, B);
    const V kmB = vsub(kb, B), kbd = vmul(kb, drho), kp3 = vmul(lift<V>(3.0), vadd(kbm, B));
#pragma unroll
    for (int d = 0; d < 2; ++d) {
        const V w = lift<V>(d == 0 ? W1 : W2);
        const V wr = vmul(w, rho), m = vmul(kmB, wr);
        p.wr[d] = wr;
        p.q[d] = vmul(lift<V>(4.5), m);
        p.b[d] = vsub(vfma(w, kbd, vmul(c.npw3[1 + d], uF)), vmul(m, uu15));
        p.t[d] = vmul(kp3, wr);
        p.a[d] = vmul(lift<V>(3.0), wr);
    }
    collide_pair_v<0, MOVING, IMB>(g, c, p, imb);
    collide_pair_v<1, MOVING, IMB>(g, c, p, imb);
    collide_pair_v<2, MOVING, IMB>(g, c, p, imb);
    collide_pair_v<3, MOVING, IMB>(g, c, p, imb);
    collide_pair_v<4, MOVING, IMB>(g, c, p, imb);
    collide_pair_v<5, MOVING, IMB>(g, c, p, imb);
    collide_pair_v<6, MOVING, IMB>(g, c, p, imb);
    collide_pair_v<7, MOVING, IMB>(g, c, p, imb);
    collide_pair_v<8, MOVING, IMB>(g, c, p, imb);
}

// collide_v with the density taken from g; irho_hint: 1 / rho where the caller has it, else 0.
template <typename R, bool MOVING, bool IMB, bool TRT = false>
PSC_HD void collide_fast2(R* g, const WinConst<R>& c, R B, R kb, R usx, R usy, R usz, R irho_hint, R* mom,
                          R* imb, bool want_mom = true) {
    const R drho = sum_populations(g);
    const R irho = irho_hint > R(0) ? irho_hint : R(1) / (R(1) + drho);
    collide_v<R, MOVING, IMB, TRT>(g, c, drho, irho, B, kb, usx, usy, usz, mom, imb, want_mom);
}

}  // namespace psc

namespace psc {

// ===========================================================================
// voxel bounce-back D3Q19 (scripts/run_3d_window_lbm.py:95-146), exact FP64
// ===========================================================================
// At a solid node the reference overwrites populations in index order,
// f[i] = f[OPP[i]] for i = 0..18 (:117-119); because f[2k+1] is overwritten
// before f[2k+2] reads it, both members of each pair end up holding the old
// f[2k+2].  Reproduced as written.
PSC_HD void bounce_solid_as_reference(double* f) {
#pragma unroll
    for (int k = 0; k < 9; ++k) f[2 * k + 1] = f[2 * k + 2];
}

// BGK + Guo with the single half-force shift of run_3d_window_lbm.py:106-114:
// u = (m + F/2)/rho, u = 0 at solid nodes, f <- f - (f - feq)/tau + guo(u).
PSC_HD void collide_bb_exact(double* f, bool solid, double tau, double fx, double fy, double fz, double* mom) {
    const double hfx = xmul(0.5, fx), hfy = xmul(0.5, fy), hfz = xmul(0.5, fz);
    ExactMoments mo = moments_exact(f, hfx, hfy, hfz);
    if (solid) {
        mo.ux = 0.0;
        mo.uy = 0.0;
        mo.uz = 0.0;
    }
    mom[0] = mo.rho;
    mom[1] = mo.ux;
    mom[2] = mo.uy;
    mom[3] = mo.uz;
    const double rho = mo.rho, ux = mo.ux, uy = mo.uy, uz = mo.uz;
    const Divisor by_tau = make_divisor(tau);
    const double uu = xadd(xadd(xmul(ux, ux), xmul(uy, uy)), xmul(uz, uz));
    const double ct = div_cs2(xmul(0.5, uu));
    const double pref = xsub(1.0, xdiv_d(0.5, by_tau));
    const double uf = xadd(xadd(xmul(ux, fx), xmul(uy, fy)), xmul(uz, fz));
    {
        const double feq = xmul(xmul(W0, rho), xsub(1.0, ct));
        const double g = xmul(xmul(pref, W0), div_cs2(-uf));
        f[0] = xadd(xsub(f[0], xdiv_d(xsub(f[0], feq), by_tau)), g);
    }
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        const int i = 2 * k + 1, j = i + 1;
        const double w = wgt(i);
        const double wr = xmul(w, rho);
        const double cu = xadd(xadd(cm(cxv(i), ux), cm(cyv(i), uy)), cm(czv(i), uz));
        const double q = div_cs2(cu);
        const double b = div_cs2sq(xmul(xmul(0.5, cu), cu));
        const double feq_i = xmul(wr, xsub(xadd(xadd(1.0, q), b), ct));
        const double feq_j = xmul(wr, xsub(xadd(xadd(1.0, -q), b), ct));
        const double cf = xadd(xadd(cm(cxv(i), fx), cm(cyv(i), fy)), cm(czv(i), fz));
        const double pw = xmul(pref, w);
        const double t2 = div_cs2sq(xmul(cu, cf));
        const double g_i = xmul(pw, xadd(div_cs2(xsub(cf, uf)), t2));
        const double g_j = xmul(pw, xadd(div_cs2(xsub(-cf, uf)), t2));
        f[i] = xadd(xsub(f[i], xdiv_d(xsub(f[i], feq_i), by_tau)), g_i);
        f[j] = xadd(xsub(f[j], xdiv_d(xsub(f[j], feq_j), by_tau)), g_j);
    }
}

// collide_bb_exact in the branch-free forms (moments_exact_s, ExactWin); true where an operand left
// their range (f is then undefined).
template <int K, bool AXIS>
PSC_HD void bb_pair_s(double* f, const ExactWin& w, double wr, double pw, double ct, const ExactGuo& guo, double ux, double uy,
                      double uz) {
    constexpr int i = 2 * K + 1, j = i + 1;
    const double cu = cdot_s<i>(ux, uy, uz);
    const double q = div_cs2_s(cu);
    const double b = half_div_cs2sq_s(xmul(cu, cu));
    const double di = xsub(f[i], xmul(wr, xsub(xadd(xadd(1.0, q), b), ct)));
    const double dj = xsub(f[j], xmul(wr, xsub(xadd(xsub(1.0, q), b), ct)));
    double g_i, g_j;
    exact_guo_pair_s<AXIS, K>(w, guo, pw, cu, g_i, g_j);
    f[i] = xadd(xsub(f[i], xdiv_s(di, w.tau, w.rtau, w.rtau_lo)), g_i);
    f[j] = xadd(xsub(f[j], xdiv_s(dj, w.tau, w.rtau, w.rtau_lo)), g_j);
}

template <bool AXIS>
PSC_HD bool collide_bb_exact_s(double* f, const ExactMomentsS& mo, bool solid, const ExactWin& w) {
    double ux = solid ? 0.0 : mo.ux, uy = solid ? 0.0 : mo.uy, uz = solid ? 0.0 : mo.uz;
    const ExactGuo guo = exact_guo_s<AXIS>(w, mo.rho, mo.rrho, 0.0, ux, uy, uz);
    const double ct = half_div_cs2_s(xadd(xadd(xmul(ux, ux), xmul(uy, uy)), xmul(uz, uz)));
    {
        const double d = xsub(f[0], xmul(xmul(W0, mo.rho), xsub(1.0, ct)));
        f[0] = xadd(xsub(f[0], xdiv_s(d, w.tau, w.rtau, w.rtau_lo)), xmul(w.pw[0], guo.d0));
    }
    const double wr1 = xmul(W1, mo.rho), wr2 = xmul(W2, mo.rho);
    bb_pair_s<0, AXIS>(f, w, wr1, w.pw[1], ct, guo, ux, uy, uz);
    bb_pair_s<1, AXIS>(f, w, wr1, w.pw[1], ct, guo, ux, uy, uz);
    bb_pair_s<2, AXIS>(f, w, wr1, w.pw[1], ct, guo, ux, uy, uz);
    bb_pair_s<3, AXIS>(f, w, wr2, w.pw[2], ct, guo, ux, uy, uz);
    bb_pair_s<4, AXIS>(f, w, wr2, w.pw[2], ct, guo, ux, uy, uz);
    bb_pair_s<5, AXIS>(f, w, wr2, w.pw[2], ct, guo, ux, uy, uz);
    bb_pair_s<6, AXIS>(f, w, wr2, w.pw[2], ct, guo, ux, uy, uz);
    bb_pair_s<7, AXIS>(f, w, wr2, w.pw[2], ct, guo, ux, uy, uz);
    bb_pair_s<8, AXIS>(f, w, wr2, w.pw[2], ct, guo, ux, uy, uz);
    return mo.out | (w.out != 0);
}

}  // namespace psc
