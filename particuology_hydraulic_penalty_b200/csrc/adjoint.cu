// Discrete adjoint of the Darcy permeability with respect to the particles'
// centres and radii (no counterpart in the reference; it differentiates the
// reference's step, src/lbm_dem/psc3d.py:208-246, and the caller-side K of
// scripts/run_psc_permeability_resolution.py:144-150).
//
// Forward model: static particles, deviation storage (F64 or F32), smooth
// solid fraction (psc_geometry.smooth_eps > 0), pull streaming with stored
// post-collision states S_t, f_t = pull(S_t), S_{t+1} = C(f_t; B).
// K = kappa * sum_x (1 - solid) u.dir of pull(S_T), u = (m + F/2) / rho.
//
// Reverse pass, one launch per step (t = T-1 .. 0):
//   mu(x)            = J_C(f_t(x))^T lambda_{t+1}(x)      (local 19x19, by hand)
//   lambda_t(x - c_i) = mu_i(x)                          (pull^T = push; one
//                                                         store per element)
//   dK/dB(x)        += lambda_{t+1}(x) . dC/dB(f_t(x))
// Each reverse step reads S_t (pulled) and lambda_{t+1}, writes lambda_t and
// updates one FP64 accumulator per cell: ~1.6x the bytes of a forward step.
#include <cooperative_groups.h>

#include "collide.cuh"
#include "internal.cuh"
#include "smooth.cuh"
#include "step_common.cuh"

namespace psc {

namespace {

template <typename R>
struct Pull19 {
    R v[Q];
};

__device__ __forceinline__ void decode(uint32_t cell, int nx, int ny, int nz, uint32_t& ix, uint32_t& iy,
                                       uint32_t& iz) {
    iz = cell % (uint32_t)nz;
    const uint32_t r = cell / (uint32_t)nz;
    iy = r % (uint32_t)ny;
    ix = r / (uint32_t)ny;
}

// offset from x to x - c_i (periodic)
template <int I>
__device__ __forceinline__ int32_t src_off(int32_t xm, int32_t xp, int32_t ym, int32_t yp, int32_t zm, int32_t zp) {
    return (cxv(I) == 1 ? xm : (cxv(I) == -1 ? xp : 0)) + (cyv(I) == 1 ? ym : (cyv(I) == -1 ? yp : 0)) +
           (czv(I) == 1 ? zm : (czv(I) == -1 ? zp : 0));
}

template <int I = 0>
__device__ __forceinline__ void offsets(int32_t* off, int32_t xm, int32_t xp, int32_t ym, int32_t yp, int32_t zm,
                                        int32_t zp) {
    if constexpr (I < Q) {
        off[I] = src_off<I>(xm, xp, ym, yp, zm, zp);
        offsets<I + 1>(off, xm, xp, ym, yp, zm, zp);
    }
}

__device__ __forceinline__ void coord_offsets(uint32_t ix, uint32_t iy, uint32_t iz, int nx, int ny, int nz,
                                              int32_t* off) {
    const int32_t nyz = ny * nz;
    const int32_t xm = ix == 0 ? (nx - 1) * nyz : -nyz;
    const int32_t xp = ix == (uint32_t)(nx - 1) ? -(nx - 1) * nyz : nyz;
    const int32_t ym = iy == 0 ? (ny - 1) * nz : -nz;
    const int32_t yp = iy == (uint32_t)(ny - 1) ? -(ny - 1) * nz : nz;
    const int32_t zm = iz == 0 ? nz - 1 : -1;
    const int32_t zp = iz == (uint32_t)(nz - 1) ? -(nz - 1) : 1;
    offsets(off, xm, xp, ym, yp, zm, zp);
}

__device__ __forceinline__ void cell_offsets(uint32_t cell, int nx, int ny, int nz, int32_t* off) {
    uint32_t ix, iy, iz;
    decode(cell, nx, ny, nz, ix, iy, iz);
    coord_offsets(ix, iy, iz, nx, ny, nz, off);
}

// Cell coordinates of a grid-stride loop: decoded once, then advanced by the
// stride's own (x, y, z) digits with carries (no division per cell).
struct StrideWalk {
    uint32_t ix, iy, iz, sx, sy, sz, ny, nz;
    __device__ __forceinline__ StrideWalk(uint32_t cell, uint32_t stride, int nx, int ny_, int nz_) {
        ny = (uint32_t)ny_;
        nz = (uint32_t)nz_;
        decode(cell, nx, ny_, nz_, ix, iy, iz);
        sz = stride % nz;
        const uint32_t q = stride / nz;
        sy = q % ny;
        sx = q / ny;
    }
    __device__ __forceinline__ void next() {
        iz += sz;
        const uint32_t cz = iz >= nz;
        iz -= cz ? nz : 0u;
        iy += sy + cz;
        const uint32_t cy = iy >= ny;
        iy -= cy ? ny : 0u;
        ix += sx + cy;
    }
};

}  // namespace

// lambda_T(x - c_i) = dK/df_i(x) = kappa (1 - solid) (c_i.dir - u.dir) / rho ; dK/dsolid = -kappa u.dir
template <typename R>
__global__ void k_adjoint_seed(psc_adjoint_args a) {
    const uint32_t N = (uint32_t)a.nx * a.ny * a.nz;
    const R* S = reinterpret_cast<const R*>(a.state);
    R* lam = reinterpret_cast<R*>(a.lam_out);
    const R dx = (R)a.dir[0], dy = (R)a.dir[1], dz = (R)a.dir[2];
    const R fx = (R)a.force[0], fy = (R)a.force[1], fz = (R)a.force[2];
    for (uint32_t cell = blockIdx.x * blockDim.x + threadIdx.x; cell < N; cell += gridDim.x * blockDim.x) {
        int32_t off[Q];
        cell_offsets(cell, a.nx, a.ny, a.nz, off);
        R g[Q];
#pragma unroll
        for (int i = 0; i < Q; ++i) g[i] = S[(size_t)i * N + (size_t)((int64_t)cell + off[i])];
        const FastMoments<R> mo = moments_fast(g);
        const R irho = R(1) / mo.rho;
        const R uF = ((mo.mx + R(0.5) * fx) * dx + (mo.my + R(0.5) * fy) * dy + (mo.mz + R(0.5) * fz) * dz) * irho;
        const double solid = a.solid[cell];
        const R w = (R)(a.kappa * (1.0 - solid));
#pragma unroll
        for (int i = 0; i < Q; ++i) {
            const R cd = (R)cxv(i) * dx + (R)cyv(i) * dy + (R)czv(i) * dz;
            lam[(size_t)i * N + (size_t)((int64_t)cell + off[i])] = w * (cd - uF) * irho;
        }
        a.dKdsolid[cell] = -a.kappa * (double)uF;
        a.dKdB[cell] = 0.0;
    }
}

// J_C(f)^T lambda of one cell (or two in packed FP32), by hand.  g: the pulled deviations; lam: lambda_{t+1}
// on entry, mu on exit; returns dC/dB . lambda.  Per direction pair with L = l_i + l_j, D = l_i - l_j:
//   the sensitivities to feq_i +- feq_j are P = (kb - B) L and M = (kb + B) D, so with
//   x = 4.5 cu P and y = 3 M
//     d/d(rho - 1) += w cu (x + y)          (and kb sum w L - 1.5 u^2 (kb - B) sum w L once)
//     d/du         += c (w rho (2 x + y) + 9 pref w (c . F) L)
//   (and u by - sum w L (3 rho (kb - B) u + 3 pref F) once), and
//     dC/dB . lambda += L ((gs/2 - sym)/tau - w rho q) + D ((gd/2 - asym)/tau - gd + asym),
//   gs = g_i + g_j, gd = g_i - g_j, feq = sym +- asym, sym = w (drho + rho q), q = 4.5 cu^2 - 1.5 u^2;
//   mu_i = (1 - kb - B) l_i + B l_j + d/d(rho - 1) + c . d/dm.
template <typename V>
struct AdjointConst {
    V inv_tau, fx, fy, fz, pref3;  // pref3 = 3 pref
    V K9[9];                       // 9 pref w_k (c_k . F)
};

template <typename V>
__device__ __forceinline__ void make_adjoint_const(AdjointConst<V>& c, const psc_adjoint_args& a) {
    const double pref = 1.0 - 0.5 / a.tau;
    c.inv_tau = lift<V>(1.0 / a.tau);
    c.fx = lift<V>(a.force[0]);
    c.fy = lift<V>(a.force[1]);
    c.fz = lift<V>(a.force[2]);
    c.pref3 = lift<V>(3.0 * pref);
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        const int i = 2 * k + 1;
        c.K9[k] = lift<V>(9.0 * pref * wgt(i) * (cxv(i) * a.force[0] + cyv(i) * a.force[1] + czv(i) * a.force[2]));
    }
}

template <typename V>
struct AdjointTerms {
    V ux, uy, uz, uu15, rho, drho, kmB, kpB3;  // kb - B, 3 (kb + B)
    V Vx, Vy, Vz, E, dB, Lw;
};

template <int K, typename V>
__device__ __forceinline__ void adjoint_pair(const V* g, const V* lam, const AdjointConst<V>& c, AdjointTerms<V>& p) {
    constexpr int i = 2 * K + 1, j = i + 1;
    const V w = lift<V>(wgt(i)), wr = vmul(w, p.rho);
    const V L = vadd(lam[i], lam[j]), D = vsub(lam[i], lam[j]);
    const V cu = cdot_v<K>(p.ux, p.uy, p.uz), c45 = vmul(lift<V>(4.5), cu);
    const V x = vmul(c45, vmul(p.kmB, L)), y = vmul(p.kpB3, D);
    p.E = vfma(vmul(w, cu), vadd(x, y), p.E);
    const V vc = vfma(wr, vfma(lift<V>(2.0), x, y), vmul(c.K9[K], L));
    if constexpr (cxv(i) != 0) p.Vx = K == 0 ? vc : vadd(p.Vx, vc);
    if constexpr (cyv(i) != 0) p.Vy = K == 1 ? vc : (cyv(i) > 0 ? vadd(p.Vy, vc) : vsub(p.Vy, vc));
    if constexpr (czv(i) != 0) p.Vz = K == 2 ? vc : (czv(i) > 0 ? vadd(p.Vz, vc) : vsub(p.Vz, vc));
    p.Lw = vfma(w, L, p.Lw);
    const V rq = vmul(p.rho, vsub(vmul(c45, cu), p.uu15));
    const V sym = vmul(w, vadd(p.drho, rq)), asym = vmul(lift<V>(3.0), vmul(wr, cu));
    const V half = lift<V>(0.5), gd = vsub(g[i], g[j]);
    const V es = vsub(vmul(half, vadd(g[i], g[j])), sym), ea = vsub(vmul(half, gd), asym);
    p.dB = vfma(L, vsub(vmul(es, c.inv_tau), vmul(w, rq)), p.dB);
    p.dB = vfma(D, vadd(vmul(ea, c.inv_tau), vsub(asym, gd)), p.dB);
}

template <int K, typename V>
__device__ __forceinline__ void adjoint_mu(V* lam, V direct, V B, V rb, V mx, V my, V mz) {
    constexpr int i = 2 * K + 1, j = i + 1;
    const V cm = cdot_v<K>(mx, my, mz), li = lam[i], lj = lam[j];
    lam[i] = vfma(direct, li, vfma(B, lj, vadd(rb, cm)));
    lam[j] = vfma(direct, lj, vfma(B, li, vsub(rb, cm)));
}

template <typename V>
__device__ __forceinline__ V adjoint_cell(const V* g, V* lam, V B, V irho, V drho, const AdjointConst<V>& c) {
    const V one = lift<V>(1.0);
    AdjointTerms<V> p;
    p.drho = drho;
    p.rho = vadd(one, drho);
    V mx, my, mz;
    momentum(g, mx, my, mz);
    p.ux = vmul(vadd(mx, c.fx), irho);
    p.uy = vmul(vadd(my, c.fy), irho);
    p.uz = vmul(vadd(mz, c.fz), irho);
    p.uu15 = vmul(lift<V>(1.5), vfma(p.uz, p.uz, vfma(p.uy, p.uy, vmul(p.ux, p.ux))));
    const V kb = vmul(vsub(one, B), c.inv_tau);
    p.kmB = vsub(kb, B);
    p.kpB3 = vmul(lift<V>(3.0), vadd(kb, B));
    // rest population: cu = 0
    const V w0 = lift<V>(W0), l0 = lam[0];
    const V rq0 = vmul(p.rho, p.uu15), geq0 = vmul(w0, vsub(drho, rq0));
    p.dB = vmul(l0, vfma(vsub(g[0], geq0), c.inv_tau, vmul(w0, rq0)));
    p.E = lift<V>(0.0);
    p.Lw = vmul(w0, l0);
    adjoint_pair<0>(g, lam, c, p);
    adjoint_pair<1>(g, lam, c, p);
    adjoint_pair<2>(g, lam, c, p);
    adjoint_pair<3>(g, lam, c, p);
    adjoint_pair<4>(g, lam, c, p);
    adjoint_pair<5>(g, lam, c, p);
    adjoint_pair<6>(g, lam, c, p);
    adjoint_pair<7>(g, lam, c, p);
    adjoint_pair<8>(g, lam, c, p);
    const V PL = vmul(p.kmB, p.Lw);  // sum of w P
    const V s1 = vmul(vmul(lift<V>(3.0), p.rho), PL), s2 = vmul(c.pref3, p.Lw);
    const V ubx = vsub(vsub(p.Vx, vmul(s1, p.ux)), vmul(s2, c.fx));
    const V uby = vsub(vsub(p.Vy, vmul(s1, p.uy)), vmul(s2, c.fy));
    const V ubz = vsub(vsub(p.Vz, vmul(s1, p.uz)), vmul(s2, c.fz));
    V rb = vadd(vsub(vmul(kb, p.Lw), vmul(p.uu15, PL)), p.E);
    rb = vsub(rb, vmul(vfma(ubz, p.uz, vfma(uby, p.uy, vmul(ubx, p.ux))), irho));
    const V mbx = vmul(ubx, irho), mby = vmul(uby, irho), mbz = vmul(ubz, irho);
    const V direct = vsub(vsub(one, kb), B);
    lam[0] = vfma(vsub(one, kb), l0, rb);
    adjoint_mu<0>(lam, direct, B, rb, mbx, mby, mbz);
    adjoint_mu<1>(lam, direct, B, rb, mbx, mby, mbz);
    adjoint_mu<2>(lam, direct, B, rb, mbx, mby, mbz);
    adjoint_mu<3>(lam, direct, B, rb, mbx, mby, mbz);
    adjoint_mu<4>(lam, direct, B, rb, mbx, mby, mbz);
    adjoint_mu<5>(lam, direct, B, rb, mbx, mby, mbz);
    adjoint_mu<6>(lam, direct, B, rb, mbx, mby, mbz);
    adjoint_mu<7>(lam, direct, B, rb, mbx, mby, mbz);
    adjoint_mu<8>(lam, direct, B, rb, mbx, mby, mbz);
    return p.dB;
}

template <typename R>
__device__ __forceinline__ R adjoint_B(double solid, R tau) {
    const R al = (R)solid;
    return al / (al + tau * (R(1) - al) + R(1.0e-14));
}

// One cell per thread.
template <typename R>
__global__ void __launch_bounds__(256) k_adjoint_step(const __grid_constant__ psc_adjoint_args a) {
    __shared__ AdjointConst<R> c;
    if (threadIdx.x == 0) make_adjoint_const(c, a);
    chain_wait();
    __syncthreads();
    const uint32_t N = (uint32_t)a.nx * a.ny * a.nz;
    const R* S = reinterpret_cast<const R*>(a.state);
    const R* lin = reinterpret_cast<const R*>(a.lam_in);
    R* lout = reinterpret_cast<R*>(a.lam_out);
    const uint32_t stride = gridDim.x * blockDim.x;
    StrideWalk at(blockIdx.x * blockDim.x + threadIdx.x, stride, a.nx, a.ny, a.nz);
    for (uint32_t cell = blockIdx.x * blockDim.x + threadIdx.x; cell < N; cell += stride, at.next()) {
        int32_t off[Q];
        coord_offsets(at.ix, at.iy, at.iz, a.nx, a.ny, a.nz, off);
        R g[Q], lam[Q];
#pragma unroll
        for (int i = 0; i < Q; ++i) {
            g[i] = ld_pop(S + (size_t)i * N + (size_t)((int64_t)cell + off[i]));
            lam[i] = ld_pop(lin + (size_t)i * N + cell);
        }
        const R drho = sum_populations(g);
        const R dB = adjoint_cell<R>(g, lam, adjoint_B<R>(a.solid[cell], (R)a.tau), fast_rcp<R>(R(1) + drho), drho, c);
#pragma unroll
        for (int i = 0; i < Q; ++i) lout[(size_t)i * N + (size_t)((int64_t)cell + off[i])] = lam[i];
        a.dKdB[cell] += (double)dB;
    }
}

// Two consecutive z cells per thread in packed FP32 (nz even, pointers aligned): the accesses of
// k_step_pair, half the arithmetic instructions.  Bound by HBM: 252 B per cell, 34 us on 96^3.  Twelve
// warps per SM at 168 registers: 96^3 48.5 -> 39.1 us, 64^3 14.1 -> 9.7 us (sixteen warps at 128 registers
// spill: 49 us; eight at 255: 46 us; one cell per thread: 45 us).
constexpr int ADJ_THREADS = 128, ADJ_CTAS = 3;
__global__ void __launch_bounds__(ADJ_THREADS, ADJ_CTAS) k_adjoint_pair(const __grid_constant__ psc_adjoint_args a) {
    __shared__ AdjointConst<F2> c;
    if (threadIdx.x == 0) make_adjoint_const(c, a);
    chain_wait();
    __syncthreads();
    const uint32_t N = (uint32_t)a.nx * a.ny * a.nz, nz = (uint32_t)a.nz;
    const float* S = reinterpret_cast<const float*>(a.state);
    const float* lin = reinterpret_cast<const float*>(a.lam_in);
    float* lout = reinterpret_cast<float*>(a.lam_out);
    const float tau = (float)a.tau;
    const uint32_t stride = 2 * gridDim.x * blockDim.x;
    uint32_t c0 = 2 * (blockIdx.x * blockDim.x + threadIdx.x);
    StrideWalk at(c0, stride, a.nx, a.ny, a.nz);
    for (; c0 < N; c0 += stride, at.next()) {
        const int32_t nyz = a.ny * a.nz;
        const int32_t xm = at.ix == 0 ? (a.nx - 1) * nyz : -nyz, xp = at.ix + 1 == (uint32_t)a.nx ? -(a.nx - 1) * nyz : nyz;
        const int32_t ym = at.iy == 0 ? (a.ny - 1) * a.nz : -a.nz;
        const int32_t yp = at.iy + 1 == (uint32_t)a.ny ? -(a.ny - 1) * a.nz : a.nz;
        const int32_t zm0 = at.iz == 0 ? (int32_t)nz - 1 : -1;           // c0's z - 1
        const int32_t zp1 = at.iz + 2 == nz ? 2 - (int32_t)nz : 2;       // c0 + 1's z + 1, from c0
        F2 g[Q], lam[Q];
#pragma unroll
        for (int i = 0; i < Q; ++i) {
            const int32_t oxy = (cxv(i) == 1 ? xm : (cxv(i) == -1 ? xp : 0)) + (cyv(i) == 1 ? ym : (cyv(i) == -1 ? yp : 0));
            const float* p = S + (size_t)i * N + (size_t)((int64_t)c0 + oxy);
            if (czv(i) == 0) {
                float x, y;
                ld_pair(p, x, y);
                g[i] = f2(x, y);
            } else if (czv(i) == 1) {
                g[i] = f2(ld_pop(p + zm0), ld_pop(p));
            } else {
                g[i] = f2(ld_pop(p + 1), ld_pop(p + zp1));
            }
            float l0, l1;
            ld_pair(lin + (size_t)i * N + c0, l0, l1);
            lam[i] = f2(l0, l1);
        }
        const double2 solid = *reinterpret_cast<const double2*>(a.solid + c0);
        const F2 drho = sum_populations(g);
        float d0, d1;
        f2_get(drho, d0, d1);
        const F2 dB = adjoint_cell<F2>(g, lam, f2(adjoint_B<float>(solid.x, tau), adjoint_B<float>(solid.y, tau)),
                                       f2(fast_rcp<float>(1.0f + d0), fast_rcp<float>(1.0f + d1)), drho, c);
#pragma unroll
        for (int i = 0; i < Q; ++i) {
            const int32_t oxy = (cxv(i) == 1 ? xm : (cxv(i) == -1 ? xp : 0)) + (cyv(i) == 1 ? ym : (cyv(i) == -1 ? yp : 0));
            float* p = lout + (size_t)i * N + (size_t)((int64_t)c0 + oxy);
            float x, y;
            f2_get(lam[i], x, y);
            if (czv(i) == 0) {
                *reinterpret_cast<float2*>(p) = make_float2(x, y);
            } else if (czv(i) == 1) {
                p[zm0] = x;
                p[0] = y;
            } else {
                p[1] = x;
                p[zp1] = y;
            }
        }
        float b0, b1;
        f2_get(dB, b0, b1);
        double2 acc = *reinterpret_cast<double2*>(a.dKdB + c0);
        acc.x += (double)b0;
        acc.y += (double)b1;
        *reinterpret_cast<double2*>(a.dKdB + c0) = acc;
    }
}

// Per-cell dK/d(alpha_sum) = (dK/dB dB/dalpha + dK/dsolid) [0 < alpha_sum < 1], then
// per-particle sums over bbox entries of dK/dalpha_sum * d alpha_p / d(x, y, z, r).
constexpr int GRAD_THREADS = 128;
constexpr int GRAD_CTAS = 8;

// One cluster per chunk: an entry near a sphere's surface costs S^3 FP64 exponentials, one away from it none,
// and the chunks differ as much.  64 spheres, S = 4: 33^3 194 -> 80 us and 96^3 478 -> 391 us against a block
// per chunk (clusters of 256-thread CTAs: 497 us; a tanh for every sample of every entry: 1215 us).  Bound by
// the exponentials.  The CTAs' sums are added in order.
template <int S>
__global__ void __cluster_dims__(GRAD_CTAS, 1, 1) __launch_bounds__(GRAD_THREADS)
    k_adjoint_geom_chunks(const __grid_constant__ psc_geometry g, const __grid_constant__ psc_adjoint_args a, double* part) {
    namespace cg = cooperative_groups;
    __shared__ double s[GRAD_THREADS / 32][4];
    __shared__ double s_cta[4];
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t rank = cluster.block_rank();
    const int64_t C = g.totals[1];
    const double Sd = (double)g.subsamples, inv_eps = 1.0 / g.smooth_eps, tau = a.tau;
    const double inv_s3 = 1.0 / (Sd * Sd * Sd);
    for (int64_t chunk = blockIdx.x / GRAD_CTAS; chunk < C; chunk += gridDim.x / GRAD_CTAS) {
        // owner particle of this chunk (largest p with chunk_off[p] <= chunk)
        int lo = 0, hi = g.nparticles - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (g.chunk_off[mid] <= chunk) lo = mid;
            else hi = mid - 1;
        }
        const int p = lo;
        const int64_t e0 = g.ent_off[p] + (chunk - g.chunk_off[p]) * g.chunk_entries;
        const int64_t e1 = min(e0 + (int64_t)g.chunk_entries, g.ent_off[p + 1]);
        const double* q = g.particles + (size_t)p * 10;
        const int32_t* bb = g.bbox + (size_t)p * 6;
        const int64_t eyz = (int64_t)bb[4] * bb[5];
        double acc[4] = {0.0, 0.0, 0.0, 0.0};
        for (int64_t e = e0 + rank * GRAD_THREADS + threadIdx.x; e < e1; e += GRAD_CTAS * GRAD_THREADS) {
            const int64_t local = e - g.ent_off[p];
            const int32_t ia = (int32_t)(local / eyz);
            const int64_t rem = local - (int64_t)ia * eyz;
            const int32_t ib = (int32_t)(rem / bb[5]);
            const int32_t ic = (int32_t)(rem - (int64_t)ib * bb[5]);
            const int32_t ix = bb[0] + ia, iy = bb[1] + ib, iz = bb[2] + ic;
            const uint32_t cell = ((uint32_t)ix * g.ny + iy) * g.nz + iz;
            const double as = g.alpha_sum[cell];
            if (!(as > 0.0 && as < 1.0)) continue;  // clip: zero derivative outside (0, 1)
            const double D = as + tau * (1.0 - as) + 1.0e-14;
            const double gcell = a.dKdB[cell] * (tau + 1.0e-14) / (D * D) + a.dKdsolid[cell];
            double gx, gy, gz, gr;
            smooth_gradient<S>(ix, iy, iz, q[0], q[1], q[2], q[3], g.subsamples, inv_eps, gx, gy, gz, gr);
            const double f = gcell * inv_s3;
            acc[0] += f * gx;
            acc[1] += f * gy;
            acc[2] += f * gz;
            acc[3] += f * gr;
        }
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            double x = acc[k];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
            if (lane == 0) s[warp][k] = x;
        }
        __syncthreads();
        if (threadIdx.x < 4) {
            double t = 0.0;
            for (int w = 0; w < nw; ++w) t += s[w][threadIdx.x];
            s_cta[threadIdx.x] = t;
        }
        cluster.sync();
        if (rank == 0 && threadIdx.x < 4) {
            double t = 0.0;
            for (int r = 0; r < GRAD_CTAS; ++r) t += cluster.map_shared_rank(s_cta, r)[threadIdx.x];
            part[chunk * 4 + threadIdx.x] = t;
        }
        cluster.sync();  // s and s_cta stay in place until they are read
    }
}

__global__ void k_adjoint_geom_final(psc_geometry g, const double* part, double* grad) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < g.nparticles; p += gridDim.x * blockDim.x) {
        double t[4] = {0.0, 0.0, 0.0, 0.0};
        for (int64_t c = g.chunk_off[p]; c < g.chunk_off[p + 1]; ++c)
            for (int k = 0; k < 4; ++k) t[k] += part[c * 4 + k];
        for (int k = 0; k < 4; ++k) grad[(size_t)p * 4 + k] = t[k];
    }
}

static unsigned cap_grid(int64_t work, int threads, int per_sm) {
    int64_t g = (work + threads - 1) / threads;
    const int64_t cap = (int64_t)sm_count() * per_sm;
    if (g > cap) g = cap;
    if (g < 1) g = 1;
    return (unsigned)g;
}

cudaError_t launch_adjoint_seed(const psc_adjoint_args& a, cudaStream_t stream) {
    const int64_t N = (int64_t)a.nx * a.ny * a.nz;
    if (a.store == PSC_STORE_F64) k_adjoint_seed<double><<<cap_grid(N, 256, 8), 256, 0, stream>>>(a);
    else k_adjoint_seed<float><<<cap_grid(N, 256, 8), 256, 0, stream>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_adjoint_step(const psc_adjoint_args& a, cudaStream_t stream) {
    const int64_t N = (int64_t)a.nx * a.ny * a.nz;
    const auto aligned = [](const void* p, uintptr_t n) { return reinterpret_cast<uintptr_t>(p) % n == 0; };
    if (a.store == PSC_STORE_F64)
        return launch_chained(k_adjoint_step<double>, cap_grid(N, 256, 8), 256, 0, stream, true, a);
    else if (a.nz % 2 == 0 && aligned(a.state, 8) && aligned(a.lam_in, 8) && aligned(a.lam_out, 8) &&
             aligned(a.solid, 16) && aligned(a.dKdB, 16))
        return launch_chained(k_adjoint_pair, cap_grid(N / 2, ADJ_THREADS, ADJ_CTAS), ADJ_THREADS, 0, stream, true,
                              a);  // (the resident CTAs)
    else
        return launch_chained(k_adjoint_step<float>, cap_grid(N, 256, 8), 256, 0, stream, true, a);
}

cudaError_t launch_adjoint_geometry_grad(const psc_geometry& g, const psc_adjoint_args& a, double* part,
                                         double* grad, cudaStream_t stream) {
    if (g.nparticles <= 0) return cudaSuccess;
    if (g.capacity_chunks > 0) {
        const int64_t cap = (int64_t)sm_count() * 16;
        const unsigned grid = GRAD_CTAS * (unsigned)(g.capacity_chunks < cap ? g.capacity_chunks : cap);
        PSC_BY_SUBSAMPLES(g.subsamples, k_adjoint_geom_chunks, <<<grid, GRAD_THREADS, 0, stream>>>(g, a, part));
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    k_adjoint_geom_final<<<cap_grid(g.nparticles, 256, 4), 256, 0, stream>>>(g, part, grad);
    return cudaGetLastError();
}

}  // namespace psc
