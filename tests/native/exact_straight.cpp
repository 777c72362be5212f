// Host build of the branch-free forms of the exact arithmetic (csrc/d3q19.cuh, csrc/collide.cuh)
// for tests/test_exact_straight_host.py: g++ -O2 -ffp-contract=off.
#include <cstdint>
#include <cstring>

#include "collide.cuh"

namespace {
uint64_t bits(double v) {
    uint64_t b;
    std::memcpy(&b, &v, sizeof(b));
    return b;
}
uint64_t next(uint64_t& s) {
    uint64_t z = (s += 0x9e3779b97f4a7c15ull);
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}
// form 0: x / c_s^2, 1: x / c_s^4, 2: (x / 2) / c_s^2, 3: (x / 2) / c_s^4, 4: x / y, 5: x / y from 1/y alone
double form(int k, double x, double y) {
    using namespace psc;
    switch (k) {
        case 0: return div_cs2_s(x);
        case 1: return div_cs2sq_s(x);
        case 2: return half_div_cs2_s(x);
        case 3: return half_div_cs2sq_s(x);
        case 4: {
            const double r = 1.0 / y;
            return xdiv_s(x, y, r, xmul(xfma(-r, y, 1.0), r));
        }
        default: return xdiv_r_s(x, y, 1.0 / y);
    }
}
double ieee(int k, double x, double y) {
    using namespace psc;
    switch (k) {
        case 0: return x / CS2;
        case 1: return x / CS2SQ;
        case 2: return 0.5 * x / CS2;
        case 3: return 0.5 * x / CS2SQ;
        default: return x / y;
    }
}
}  // namespace

extern "C" {

long long straight_list(int k, double y, const double* xs, long long n) {
    long long bad = 0;
    for (long long i = 0; i < n; ++i) bad += bits(form(k, xs[i], y)) != bits(ieee(k, xs[i], y));
    return bad;
}

long long straight_random(int k, double y, long long n, uint64_t seed, int emin, int emax) {
    long long bad = 0;
    uint64_t s = seed;
    for (long long i = 0; i < n; ++i) {
        const uint64_t r = next(s);
        const uint64_t e = (uint64_t)(emin + 1023 + (int64_t)(next(s) % (uint64_t)(emax - emin + 1)));
        const uint64_t b = (r & 0x800fffffffffffffull) | (e << 52);
        double x;
        std::memcpy(&x, &b, sizeof(x));
        bad += bits(form(k, x, y)) != bits(ieee(k, x, y));
    }
    return bad;
}

int range_test(double x) { return psc::out_of_range<psc::kExactRootRange>(x) ? 1 : 0; }

// Cells through the branch-free and the general forms; out[c] is the former's range flag.
void straight_cells(const double* f_in, const double* solid, const double* us, int moving, double tau, double fx,
                    double fy, double fz, int ncell, double* f_s, double* imb_s, double* mom_s, int* out, double* f_g,
                    double* imb_g, double* mom_g) {
    using namespace psc;
    ExactWin w;
    make_exact_win(w, tau, fx, fy, fz);
    for (int c = 0; c < ncell; ++c) {
        double f[Q], g[Q], a[3], b[3];
        for (int i = 0; i < Q; ++i) f[i] = g[i] = f_in[(size_t)i * ncell + c];
        const double u[3] = {moving ? us[c] : 0.0, moving ? us[ncell + c] : 0.0, moving ? us[2 * ncell + c] : 0.0};
        const ExactMomentsS ms = moments_exact_s(f, w.hfx, w.hfy, w.hfz);
        if (w.axis >= 0)
            out[c] = moving ? collide_exact_s<true, true, true>(f, ms, solid[c], u[0], u[1], u[2], w, a)
                            : collide_exact_s<false, true, true>(f, ms, solid[c], 0.0, 0.0, 0.0, w, a);
        else
            out[c] = moving ? collide_exact_s<true, true, false>(f, ms, solid[c], u[0], u[1], u[2], w, a)
                            : collide_exact_s<false, true, false>(f, ms, solid[c], 0.0, 0.0, 0.0, w, a);
        const ExactMoments mg = moments_exact(g, w.hfx, w.hfy, w.hfz);
        collide_exact(g, mg, solid[c], moving != 0, u[0], u[1], u[2], tau, fx, fy, fz, w.hfx, w.hfy, w.hfz, b);
        for (int i = 0; i < Q; ++i) {
            f_s[(size_t)i * ncell + c] = f[i];
            f_g[(size_t)i * ncell + c] = g[i];
        }
        for (int k = 0; k < 3; ++k) {
            imb_s[(size_t)k * ncell + c] = a[k];
            imb_g[(size_t)k * ncell + c] = b[k];
        }
        const double m[4] = {ms.rho, ms.ux, ms.uy, ms.uz}, n[4] = {mg.rho, mg.ux, mg.uy, mg.uz};
        for (int k = 0; k < 4; ++k) {
            mom_s[(size_t)k * ncell + c] = m[k];
            mom_g[(size_t)k * ncell + c] = n[k];
        }
    }
}

}  // extern "C"
