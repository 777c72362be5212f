// Voxel bounce-back D3Q19 window LBM (the reference's second, simpler
// solver: scripts/run_3d_window_lbm.py, voxelize :73-92, run_lbm :95-146).
//
// Binary solid from sphere centres (cell-centre inside test), then per step,
// fused in one pull pass over post-collision populations:
//   pull f(x) = fpost(x - c)          (the reference's np.roll push, :115-116)
//   solid x: in-place pair overwrite   (:117-119, reproduced as written)
//   moments, u = 0 at solid nodes      (:104-110)
//   BGK + Guo, single half-force shift (:113-114)
// Exact FP64 arithmetic in the reference's operation order.
#include "collide.cuh"
#include "internal.cuh"
#include "step_common.cuh"

namespace psc {

// One block per sphere: cells of its clamped box whose centre lies inside.
__global__ void k_vox_spheres(const double* __restrict__ pts, int M, double lox, double loy, double loz, double dxx,
                              double dxy, double dxz, double radius, int nx, int ny, int nz, uint8_t* solid) {
    const int m = blockIdx.x;
    if (m >= M) return;
    const double x = pts[3 * m], y = pts[3 * m + 1], z = pts[3 * m + 2];
    // box clamp [max(0, floor((c - r - lo)/dx)), min(n - 1, ceil((c + r - lo)/dx))]
    const int ix0 = max(0, (int)floor(xdiv(xsub(xsub(x, radius), lox), dxx)));
    const int ix1 = min(nx - 1, (int)ceil(xdiv(xsub(xadd(x, radius), lox), dxx)));
    const int iy0 = max(0, (int)floor(xdiv(xsub(xsub(y, radius), loy), dxy)));
    const int iy1 = min(ny - 1, (int)ceil(xdiv(xsub(xadd(y, radius), loy), dxy)));
    const int iz0 = max(0, (int)floor(xdiv(xsub(xsub(z, radius), loz), dxz)));
    const int iz1 = min(nz - 1, (int)ceil(xdiv(xsub(xadd(z, radius), loz), dxz)));
    if (ix1 < ix0 || iy1 < iy0 || iz1 < iz0) return;
    const int ex = ix1 - ix0 + 1, ey = iy1 - iy0 + 1, ez = iz1 - iz0 + 1;
    const double rr = xmul(radius, radius);
    for (int e = threadIdx.x; e < ex * ey * ez; e += blockDim.x) {
        const int a = e / (ey * ez), rem = e - a * ey * ez, b = rem / ez, c = rem - b * ez;
        const int ix = ix0 + a, iy = iy0 + b, iz = iz0 + c;
        // cell centre lo + (i + 0.5) dx (:77), distance test (:91)
        const double cx = xadd(lox, xmul((double)ix + 0.5, dxx));
        const double cy = xadd(loy, xmul((double)iy + 0.5, dxy));
        const double cz = xadd(loz, xmul((double)iz + 0.5, dxz));
        const double ddx = xsub(cx, x), ddy = xsub(cy, y), ddz = xsub(cz, z);
        if (xadd(xadd(xmul(ddx, ddx), xmul(ddy, ddy)), xmul(ddz, ddz)) <= rr)
            solid[((size_t)ix * ny + iy) * nz + iz] = 1;
    }
}

struct BbArgs {
    const double* src;
    double* dst;
    const uint8_t* solid;
    double* mom;
    int32_t nx, ny, nz;
    double tau, fx, fy, fz;
    unsigned flags;
};

__device__ __forceinline__ void bb_pull(const double* src, uint32_t N, uint32_t cell, const NbrOffsets& o,
                                        double (&f)[Q]) {
    const double* p = src + cell;  // 64-bit: a window may hold up to 2^31 cells per plane
#pragma unroll
    for (int i = 0; i < Q; ++i) {
        const int32_t off = (cxv(i) == 1 ? o.xm : (cxv(i) == -1 ? o.xp : 0)) +
                            (cyv(i) == 1 ? o.ym : (cyv(i) == -1 ? o.yp : 0)) +
                            (czv(i) == 1 ? o.zm : (czv(i) == -1 ? o.zp : 0));
        f[i] = ld_pop(p + (int64_t)off);
        p += N;
    }
}

// A cell whose operands left the range of the branch-free forms: pulled again, general forms.
struct BbCell {
    double f[Q], mom[4];
};

__device__ __noinline__ void bb_cell_general(const BbArgs& a, uint32_t N, uint32_t cell, NbrOffsets o, bool solid,
                                             BbCell& r) {
    double f[Q], m[4];
    bb_pull(a.src, N, cell, o, f);
    if (solid) bounce_solid_as_reference(f);
    if (a.flags & PSC_STEP_COLLIDE) {
        collide_bb_exact(f, solid, a.tau, a.fx, a.fy, a.fz, m);
    } else {
        const ExactMoments mo = moments_exact(f, xmul(0.5, a.fx), xmul(0.5, a.fy), xmul(0.5, a.fz));
        m[0] = mo.rho;
        m[1] = solid ? 0.0 : mo.ux;
        m[2] = solid ? 0.0 : mo.uy;
        m[3] = solid ? 0.0 : mo.uz;
    }
    for (int i = 0; i < Q; ++i) r.f[i] = f[i];
    for (int k = 0; k < 4; ++k) r.mom[k] = m[k];
}

// One cell per thread of a grid-stride loop, two CTAs per SM (128 registers): bound by the FP64 pipe
// like k_step_exact, whose branch-free forms it shares (64^3: 32.5 us a step with a branch per division,
// 15.0 without, in a chain of steps).
__global__ void __launch_bounds__(256, 2) k_bb_step(const __grid_constant__ BbArgs a) {
    __shared__ ExactWin w;
    make_exact_win_block(w, a.tau, a.fx, a.fy, a.fz);
    chain_wait();
    __syncthreads();
    const uint32_t N = (uint32_t)a.nx * a.ny * a.nz;
    const bool do_collide = a.flags & PSC_STEP_COLLIDE;
    const bool do_mom = a.flags & PSC_STEP_MOMENTS;
    const uint32_t ny = (uint32_t)a.ny, nz = (uint32_t)a.nz;
    const uint32_t stride = gridDim.x * blockDim.x;
    uint32_t cell = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t iz = cell % nz, r = cell / nz, iy = r % ny, ix = r / ny;
    const uint32_t step_z = stride % nz, q = stride / nz, step_y = q % ny, step_x = q / ny;
    for (; cell < N; cell += stride) {
        const NbrOffsets o = nbr_offsets(ix, iy, iz, a.nx, a.ny, a.nz);
        double f[Q];
        bb_pull(a.src, N, cell, o, f);
        const bool s = a.solid[cell] != 0;
        if (s) bounce_solid_as_reference(f);
        const ExactMomentsS mo = moments_exact_s(f, w.hfx, w.hfy, w.hfz);
        double m[4] = {mo.rho, s ? 0.0 : mo.ux, s ? 0.0 : mo.uy, s ? 0.0 : mo.uz};
        bool out = mo.out | (w.out != 0);  // (the moments divide m + F / 2)
        if (do_collide) out = w.axis >= 0 ? collide_bb_exact_s<true>(f, mo, s, w) : collide_bb_exact_s<false>(f, mo, s, w);
        if (out) {
            BbCell g;
            bb_cell_general(a, N, cell, o, s, g);
#pragma unroll
            for (int i = 0; i < Q; ++i) f[i] = g.f[i];
#pragma unroll
            for (int k = 0; k < 4; ++k) m[k] = g.mom[k];
        }
        if (do_collide) {
            double* p = a.dst + cell;
#pragma unroll
            for (int i = 0; i < Q; ++i) {
                *p = f[i];
                p += N;
            }
        }
        if (do_mom) {
#pragma unroll
            for (int k = 0; k < 4; ++k) a.mom[(size_t)k * N + cell] = m[k];
        }
        // the stride's own (x, y, z) digits with carries
        iz += step_z;
        const uint32_t cz = iz >= nz;
        iz -= cz ? nz : 0u;
        iy += step_y + cz;
        const uint32_t cy = iy >= ny;
        iy -= cy ? ny : 0u;
        ix += step_x + cy;
    }
}

cudaError_t launch_vox_spheres(const double* pts, int M, const double* lo, const double* dx, double radius, int nx,
                               int ny, int nz, uint8_t* solid, cudaStream_t s) {
    if (M <= 0) return cudaSuccess;
    k_vox_spheres<<<M, 256, 0, s>>>(pts, M, lo[0], lo[1], lo[2], dx[0], dx[1], dx[2], radius, nx, ny, nz, solid);
    return cudaGetLastError();
}

cudaError_t launch_bb_step(const double* src, double* dst, const uint8_t* solid, int nx, int ny, int nz, double tau,
                           double fx, double fy, double fz, unsigned flags, double* mom, cudaStream_t s) {
    const int64_t N = (int64_t)nx * ny * nz;
    int64_t g = (N + 255) / 256;
    const int64_t cap = (int64_t)sm_count() * 2;  // resident CTAs
    if (g > cap) g = cap;
    const BbArgs a = {src, dst, solid, mom, nx, ny, nz, tau, fx, fy, fz, flags};
    return launch_chained(k_bb_step, (unsigned)g, 256, 0, s, true, a);
}

}  // namespace psc

namespace psc {

// Element-wise equilibrium (src/lbm_dem/psc3d.py:97-103) and Guo forcing
// (:106-114) in the reference's operation order, for the module-level helpers.
__global__ void k_equilibrium(const double* rho, const double* ux, const double* uy, const double* uz, double* out,
                              int64_t n) {
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < n; c += (int64_t)gridDim.x * blockDim.x) {
        const double r = rho[c], x = ux[c], y = uy[c], z = uz[c];
        const double uu = xadd(xadd(xmul(x, x), xmul(y, y)), xmul(z, z));
        const double ct = xdiv(xmul(0.5, uu), CS2);
#pragma unroll
        for (int i = 0; i < Q; ++i) {
            const double cu = xadd(xadd(cm(cxv(i), x), cm(cyv(i), y)), cm(czv(i), z));
            const double a = xadd(1.0, xdiv(cu, CS2));
            const double b = xdiv(xmul(xmul(0.5, cu), cu), CS2SQ);
            out[(size_t)i * n + c] = xmul(xmul(wgt(i), r), xsub(xadd(a, b), ct));
        }
    }
}

__global__ void k_guo(double fx, double fy, double fz, const double* ux, const double* uy, const double* uz,
                      double tau, double* out, int64_t n) {
    const double pref = xsub(1.0, xdiv(0.5, tau));
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < n; c += (int64_t)gridDim.x * blockDim.x) {
        const double x = ux[c], y = uy[c], z = uz[c];
        const double uf = xadd(xadd(xmul(x, fx), xmul(y, fy)), xmul(z, fz));
#pragma unroll
        for (int i = 0; i < Q; ++i) {
            const double cu = xadd(xadd(cm(cxv(i), x), cm(cyv(i), y)), cm(czv(i), z));
            const double cf = xadd(xadd(cm(cxv(i), fx), cm(cyv(i), fy)), cm(czv(i), fz));
            out[(size_t)i * n + c] =
                xmul(xmul(pref, wgt(i)), xadd(xdiv(xsub(cf, uf), CS2), xdiv(xmul(cu, cf), CS2SQ)));
        }
    }
}

cudaError_t launch_equilibrium(const double* rho, const double* ux, const double* uy, const double* uz, double* out,
                               int64_t n, cudaStream_t s) {
    int64_t g = (n + 255) / 256;
    const int64_t cap = (int64_t)sm_count() * 8;
    if (g > cap) g = cap;
    if (g < 1) g = 1;
    k_equilibrium<<<(unsigned)g, 256, 0, s>>>(rho, ux, uy, uz, out, n);
    return cudaGetLastError();
}

cudaError_t launch_guo(double fx, double fy, double fz, const double* ux, const double* uy, const double* uz,
                       double tau, double* out, int64_t n, cudaStream_t s) {
    int64_t g = (n + 255) / 256;
    const int64_t cap = (int64_t)sm_count() * 8;
    if (g > cap) g = cap;
    if (g < 1) g = 1;
    k_guo<<<(unsigned)g, 256, 0, s>>>(fx, fy, fz, ux, uy, uz, tau, out, n);
    return cudaGetLastError();
}

}  // namespace psc
