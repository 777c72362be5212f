// The kernels' collision of deviations (csrc/collide.cuh, collide_v) on the host: FP32 cells one by one and two
// at once in the packed form, for tests/test_collide_packed_host.py (g++ -O2 -ffp-contract=off).
#include <cstddef>

#include "collide.cuh"

using namespace psc;

template <typename V, bool MOVING, bool TRT>
static void one(V* g, const WinConst<V>& c, V irho, V B, V kb, const V* us, V* mom, V* imb) {
    imb[0] = imb[1] = imb[2] = lift<V>(0.0);
    collide_v<V, MOVING, true, TRT>(g, c, sum_populations(g), irho, B, kb, us[0], us[1], us[2], mom, imb, true);
}

template <typename V>
static void any(bool moving, bool trt, V* g, const WinConst<V>& c, V irho, V B, V kb, const V* us, V* mom, V* imb) {
    if (moving) trt ? one<V, true, true>(g, c, irho, B, kb, us, mom, imb) : one<V, true, false>(g, c, irho, B, kb, us, mom, imb);
    else trt ? one<V, false, true>(g, c, irho, B, kb, us, mom, imb) : one<V, false, false>(g, c, irho, B, kb, us, mom, imb);
}

// n cells (even), arrays [k][n]; packed: cells 2j and 2j + 1 together.  out: 19 populations, 4 moments, 3 IMB rows.
extern "C" void packed_cells(int packed, int moving, double tau, double tau_minus, double fx, double fy, double fz, int n,
                             const float* g_in, const float* solid, const float* us_in, float* out) {
    const bool trt = tau_minus > 0.0;
    WinConst<float> c;
    WinConst<F2> c2;
    make_win_const(c, tau, fx, fy, fz, tau_minus);
    make_win_const(c2, tau, fx, fy, fz, tau_minus);
    for (int j = 0; j < n; j += 2) {
        float g[2][Q], us[2][3], B[2], kb[2], irho[2], mom[2][4], imb[2][3];
        for (int s = 0; s < 2; ++s) {
            for (int i = 0; i < Q; ++i) g[s][i] = g_in[(size_t)i * n + j + s];
            for (int k = 0; k < 3; ++k) us[s][k] = us_in[(size_t)k * n + j + s];
            const double al = solid[j + s], b = al / (al + tau * (1.0 - al) + 1.0e-14);
            B[s] = (float)b;
            kb[s] = (float)((1.0 - b) / tau);
            irho[s] = 1.0f / (1.0f + sum_populations(g[s]));
        }
        if (packed) {
            F2 G[Q], U[3], M[4], I[3];
            for (int i = 0; i < Q; ++i) G[i] = f2(g[0][i], g[1][i]);
            for (int k = 0; k < 3; ++k) U[k] = f2(us[0][k], us[1][k]);
            any<F2>(moving, trt, G, c2, f2(irho[0], irho[1]), f2(B[0], B[1]), f2(kb[0], kb[1]), U, M, I);
            for (int i = 0; i < Q; ++i) f2_get(G[i], g[0][i], g[1][i]);
            for (int k = 0; k < 4; ++k) f2_get(M[k], mom[0][k], mom[1][k]);
            for (int k = 0; k < 3; ++k) f2_get(I[k], imb[0][k], imb[1][k]);
        } else {
            for (int s = 0; s < 2; ++s) any<float>(moving, trt, g[s], c, irho[s], B[s], kb[s], us[s], mom[s], imb[s]);
        }
        for (int s = 0; s < 2; ++s) {
            for (int i = 0; i < Q; ++i) out[(size_t)i * n + j + s] = g[s][i];
            for (int k = 0; k < 4; ++k) out[(size_t)(Q + k) * n + j + s] = mom[s][k];
            for (int k = 0; k < 3; ++k) out[(size_t)(Q + 4 + k) * n + j + s] = imb[s][k];
        }
    }
}
