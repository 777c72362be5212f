// Sums of the step kernels' partial rows, and the conversions between stored
// populations and the reference's post-stream f (src/lbm_dem/psc3d.py:239-242).
#include <cooperative_groups.h>

#include "collide.cuh"
#include "internal.cuh"
#include "step_common.cuh"

namespace psc {

// Window sums of the partial rows (header row: element 0 = row count; the
// rows follow it) by one cluster of REDUCE_CTAS CTAs per window, in a fixed
// order: thread (c, g, k) of CTA c adds column k of the rows c * 32 + g,
// + 32 * REDUCE_CTAS, ...; a warp per column adds the CTA's 32 groups by a
// shuffle tree; the cluster's first CTA adds the CTAs' sums in order through
// distributed shared memory.  A reporting call waits for these sums, so what
// counts is latency: a window of 296 CTAs leaves 2368 rows, nine independent
// loads per thread.  One launch of 3 us instead of two of 3.5 us.
constexpr int REDUCE_CTAS = 8;
constexpr int REDUCE_GROUPS = 32;
constexpr int REDUCE_THREADS = REDUCE_GROUPS * PSC_NRED;  // a warp per column

// Row count from the header, clamped to the window's capacity.
__device__ __forceinline__ int64_t partial_rows(const psc_window& W) {
    const double h = W.partials[0];
    const int64_t cap = W.tile_count * PSC_PARTIAL_ROWS;
    if (!(h > 0.0)) return 0;
    const int64_t r = (int64_t)h;
    return r < cap ? r : cap;
}

// The residual |mean_k - mean_{k-1}| / |mean_k| of step k = cc.step; step 1 has no previous value
// (residual inf, as the reference's first iteration).  On convergence the step's rows are kept and the
// window is marked inactive in both descriptor tables, so the launches already enqueued do nothing.
__device__ void converge_check(const ConvergeCheck& cc, const double* post) {
    double* cs = cc.state;
    if (cs[2] != 0.0) return;
    const double now = post[PSC_RED_UZ] / cc.cells;
    double resid = __longlong_as_double(0x7ff0000000000000ll);  // +inf
    if (cc.step > 1) {
        const double a = fabs(now);
        resid = fabs(now - cc.pre[PSC_RED_UZ] / cc.cells) / (a < 1.0e-30 ? 1.0e-30 : a);
    }
    cs[0] = now;
    cs[1] = (double)cc.step;
    cs[4] = resid;
    const bool done = cc.step >= cc.min_steps && resid < cc.tol;
    if (done || cc.last) {
        for (int k = 0; k < PSC_NRED; ++k) {
            cs[kConvState + k] = cc.pre[k];
            // the sums of the state after the step: an IMB momentum among them is the next step's
            cs[kConvState + PSC_NRED + k] = k >= PSC_RED_IMBX && k <= PSC_RED_IMBZ ? 0.0 : post[k];
        }
    }
    if (done) {
        cs[2] = 1.0;
        cs[3] = (double)cc.step;
        cc.tab[0]->flags |= PSC_WIN_INACTIVE;
        cc.tab[1]->flags |= PSC_WIN_INACTIVE;
    }
}

template <bool CONV>
__global__ void __cluster_dims__(REDUCE_CTAS, 1, 1) __launch_bounds__(REDUCE_THREADS)
    k_reduce_windows(const psc_window* wins, double* out, double* out2, const __grid_constant__ ConvergeCheck cc) {
    namespace cg = cooperative_groups;
    chain_wait();
    __shared__ double s_g[REDUCE_GROUPS * PSC_NRED];
    __shared__ double s_cta[PSC_NRED];
    cg::cluster_group cluster = cg::this_cluster();
    const int c = (int)cluster.block_rank(), t = threadIdx.x;
    const int w = blockIdx.x / REDUCE_CTAS;
    const psc_window& W = wins[w];
    const int64_t rows = partial_rows(W);
    const double* body = W.partials + PSC_NRED;
    double acc = 0.0;
    const int g = t / PSC_NRED, k = t - g * PSC_NRED;
    int64_t r = c * REDUCE_GROUPS + g;
    constexpr int kStride = REDUCE_GROUPS * REDUCE_CTAS, kAhead = 8;
    for (; r + (kAhead - 1) * kStride < rows; r += kAhead * kStride) {
        double v[kAhead];
#pragma unroll
        for (int j = 0; j < kAhead; ++j) v[j] = body[(r + j * kStride) * PSC_NRED + k];
#pragma unroll
        for (int j = 0; j < kAhead; ++j) acc += v[j];
    }
    double v[kAhead];
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
        const int64_t q = r + j * kStride;
        v[j] = q < rows ? body[q * PSC_NRED + k] : 0.0;
    }
#pragma unroll
    for (int j = 0; j < kAhead; ++j) acc += v[j];
    s_g[t] = acc;
    __syncthreads();
    const int lane = t & 31, col = t >> 5;
    double x = s_g[lane * PSC_NRED + col];
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) x += __shfl_xor_sync(0xffffffffu, x, s);
    if (lane == 0) s_cta[col] = x;
    cluster.sync();
    if (c == 0 && t < PSC_NRED) {
        double sum = 0.0;
#pragma unroll
        for (int j = 0; j < REDUCE_CTAS; ++j) sum += cluster.map_shared_rank(s_cta, j)[t];
        out[(size_t)w * PSC_NRED + t] = sum;
        if (out2) out2[(size_t)w * PSC_NRED + t] = sum;
        if (CONV) s_g[t] = sum;
    }
    cluster.sync();  // the CTAs' sums stay in place until they are read
    if (CONV && c == 0 && t < 32) {
        __syncwarp();
        if (t == 0) converge_check(cc, s_g);
    }
}

template <int STORE>
__global__ void k_init_eq(void* f, int64_t ncells) {
    using T = typename StoreTraits<STORE>::T;
    T* p = reinterpret_cast<T*>(f);
    const int64_t total = ncells * Q;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
        const int i = (int)(e / ncells);
        // equilibrium(rho=1, u=0) = w_i exactly (psc3d.py:136-140); deviation 0
        if constexpr (StoreTraits<STORE>::exact) st_pop(p + e, wgt(i));
        else st_pop(p + e, 0.0f);
    }
}

__device__ __forceinline__ double to_double(double v) { return v; }
__device__ __forceinline__ double to_double(float v) { return (double)v; }
__device__ __forceinline__ double to_double(__half v) { return (double)__half2float(v); }
__device__ __forceinline__ double to_double(__nv_bfloat16 v) { return (double)__bfloat162float(v); }

template <typename T>
__device__ __forceinline__ double to_abs(T v, int i, bool exact, bool scaled, double inv_scale) {
    double d = to_double(v);
    if (exact) return d;
    if (scaled) d *= inv_scale;
    return d + wgt(i);
}

// dst_i(x) = src_i(x - c_i) in absolute FP64 (the reference's post-stream f);
// with open_x the x faces follow PSC_WIN_OPEN_X (bounce-back velocity inlet
// at x = 0, zero-gradient outflow at x = nx - 1).
template <int STORE>
__global__ void k_stream_push(const void* src, double* dst, int nx, int ny, int nz, double scale, bool open_x,
                              double in_rho, double in_ux, double in_uy, double in_uz) {
    using TR = StoreTraits<STORE>;
    using T = typename TR::T;
    const uint32_t N = (uint32_t)nx * ny * nz;
    const T* s = reinterpret_cast<const T*>(src);
    for (uint32_t cell = blockIdx.x * blockDim.x + threadIdx.x; cell < N; cell += gridDim.x * blockDim.x) {
        const uint32_t iz = cell % nz, rr = cell / nz, iy = rr % ny, ix = rr / ny;
        const NbrOffsets nb = nbr_offsets(ix, iy, iz, nx, ny, nz, open_x);
        int32_t off[Q];
        off[0] = 0;
        off[1] = pull_offset<1>(nb); off[2] = pull_offset<2>(nb); off[3] = pull_offset<3>(nb);
        off[4] = pull_offset<4>(nb); off[5] = pull_offset<5>(nb); off[6] = pull_offset<6>(nb);
        off[7] = pull_offset<7>(nb); off[8] = pull_offset<8>(nb); off[9] = pull_offset<9>(nb);
        off[10] = pull_offset<10>(nb); off[11] = pull_offset<11>(nb); off[12] = pull_offset<12>(nb);
        off[13] = pull_offset<13>(nb); off[14] = pull_offset<14>(nb); off[15] = pull_offset<15>(nb);
        off[16] = pull_offset<16>(nb); off[17] = pull_offset<17>(nb); off[18] = pull_offset<18>(nb);
#pragma unroll
        for (int i = 0; i < Q; ++i) {
            const T v = s[(size_t)i * N + (size_t)((int64_t)cell + off[i])];
            double a = to_abs(v, i, TR::exact, TR::scaled, 1.0 / scale);
            if (open_x && ix == 0 && enters_x0(i)) {  // inlet: bounce-back of opp(i) at the node + momentum term
                const double back = to_abs(s[(size_t)opp(i) * N + cell], opp(i), TR::exact, TR::scaled, 1.0 / scale);
                a = xadd(back, inlet_correction_exact(i, in_rho, in_ux, in_uy, in_uz));
            }
            dst[(size_t)i * N + cell] = a;
        }
    }
}

// dst_i(y) = store(src_i(y + c_i)): inverse of k_stream_push.
template <int STORE>
__global__ void k_stream_pull_store(const double* src, void* dst, int nx, int ny, int nz, double scale) {
    using TR = StoreTraits<STORE>;
    using T = typename TR::T;
    const uint32_t N = (uint32_t)nx * ny * nz;
    T* d = reinterpret_cast<T*>(dst);
    for (uint32_t cell = blockIdx.x * blockDim.x + threadIdx.x; cell < N; cell += gridDim.x * blockDim.x) {
        const uint32_t iz = cell % nz, rr = cell / nz, iy = rr % ny, ix = rr / ny;
        const NbrOffsets nb = nbr_offsets(ix, iy, iz, nx, ny, nz);
        // y + c_i is the pull source of direction opp(i)
        int32_t off[Q];
        off[0] = 0;
        off[1] = pull_offset<2>(nb); off[2] = pull_offset<1>(nb); off[3] = pull_offset<4>(nb);
        off[4] = pull_offset<3>(nb); off[5] = pull_offset<6>(nb); off[6] = pull_offset<5>(nb);
        off[7] = pull_offset<8>(nb); off[8] = pull_offset<7>(nb); off[9] = pull_offset<10>(nb);
        off[10] = pull_offset<9>(nb); off[11] = pull_offset<12>(nb); off[12] = pull_offset<11>(nb);
        off[13] = pull_offset<14>(nb); off[14] = pull_offset<13>(nb); off[15] = pull_offset<16>(nb);
        off[16] = pull_offset<15>(nb); off[17] = pull_offset<18>(nb); off[18] = pull_offset<17>(nb);
#pragma unroll
        for (int i = 0; i < Q; ++i) {
            double v = src[(size_t)i * N + (size_t)((int64_t)cell + off[i])];
            if (!TR::exact) {
                v -= wgt(i);
                if (TR::scaled) v *= scale;
            }
            if constexpr (sizeof(T) == 8) d[(size_t)i * N + cell] = (T)v;
            else if constexpr (sizeof(T) == 4) d[(size_t)i * N + cell] = (T)v;
            else st_pop(d + (size_t)i * N + cell, (float)v);
        }
    }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
cudaError_t launch_reduce_windows(const psc_window* d_windows, int nwin, double* out, cudaStream_t stream,
                                  double* out2) {
    return launch_chained(k_reduce_windows<false>, nwin * REDUCE_CTAS, REDUCE_THREADS, 0, stream, true, d_windows, out, out2,
                          ConvergeCheck{});
}

cudaError_t launch_reduce_converge(const psc_window* d_window, double* out, const ConvergeCheck& cc,
                                   cudaStream_t stream) {
    return launch_chained(k_reduce_windows<true>, REDUCE_CTAS, REDUCE_THREADS, 0, stream, true, d_window, out,
                          static_cast<double*>(nullptr), cc);
}

static int grid_for(int64_t work, int threads) {
    int64_t g = (work + threads - 1) / threads;
    const int64_t cap = (int64_t)sm_count() * 16;
    if (g > cap) g = cap;
    if (g < 1) g = 1;
    return (int)g;
}

cudaError_t launch_init_equilibrium(int store, double scale, void* f, int64_t ncells, cudaStream_t stream) {
    (void)scale;
    const int g = grid_for(ncells * Q, 256);
    switch (store) {
        case PSC_STORE_F64_EXACT: k_init_eq<PSC_STORE_F64_EXACT><<<g, 256, 0, stream>>>(f, ncells); break;
        case PSC_STORE_F64: k_init_eq<PSC_STORE_F64><<<g, 256, 0, stream>>>(f, ncells); break;
        case PSC_STORE_F32: k_init_eq<PSC_STORE_F32><<<g, 256, 0, stream>>>(f, ncells); break;
        case PSC_STORE_F16: k_init_eq<PSC_STORE_F16><<<g, 256, 0, stream>>>(f, ncells); break;
        case PSC_STORE_BF16: k_init_eq<PSC_STORE_BF16><<<g, 256, 0, stream>>>(f, ncells); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_stream_push(int store, double scale, const void* src, double* dst, int nx, int ny, int nz,
                               cudaStream_t stream, bool open_x, const double* inlet) {
    const int g = grid_for((int64_t)nx * ny * nz, 256);
    const double r = open_x ? inlet[0] : 1.0, ux = open_x ? inlet[1] : 0.0, uy = open_x ? inlet[2] : 0.0,
                 uz = open_x ? inlet[3] : 0.0;
#define PSC_PUSH_CASE(S) \
    case S: k_stream_push<S><<<g, 256, 0, stream>>>(src, dst, nx, ny, nz, scale, open_x, r, ux, uy, uz); break;
    switch (store) {
        PSC_PUSH_CASE(PSC_STORE_F64_EXACT)
        PSC_PUSH_CASE(PSC_STORE_F64)
        PSC_PUSH_CASE(PSC_STORE_F32)
        PSC_PUSH_CASE(PSC_STORE_F16)
        PSC_PUSH_CASE(PSC_STORE_BF16)
        default: return cudaErrorInvalidValue;
    }
#undef PSC_PUSH_CASE
    return cudaGetLastError();
}

// Open-x inverse at the inlet plane: the populations that only the inlet's
// bounce-back reads (c_x = -1 at x = 0) are set so that the pulled value of
// the entering direction i = opp(j) is f_i(0): stored_j = f_i - term_i (to
// rounding in the exact mode).
template <int STORE>
__global__ void k_open_x_unpull(const double* src, void* dst, int nx, int ny, int nz, double scale, double in_rho,
                                double in_ux, double in_uy, double in_uz) {
    using TR = StoreTraits<STORE>;
    using T = typename TR::T;
    const uint32_t N = (uint32_t)nx * ny * nz;
    const uint32_t plane = (uint32_t)ny * nz;  // the cells of x = 0
    T* d = reinterpret_cast<T*>(dst);
    for (uint32_t cell = blockIdx.x * blockDim.x + threadIdx.x; cell < plane; cell += gridDim.x * blockDim.x) {
#pragma unroll
        for (int i = 0; i < Q; ++i) {
            if (!enters_x0(i)) continue;
            const int j = opp(i);
            double v = xsub(src[(size_t)i * N + cell], inlet_correction_exact(i, in_rho, in_ux, in_uy, in_uz));
            if (!TR::exact) {
                v -= wgt(j);
                if (TR::scaled) v *= scale;
            }
            if constexpr (sizeof(T) == 8) d[(size_t)j * N + cell] = (T)v;
            else if constexpr (sizeof(T) == 4) d[(size_t)j * N + cell] = (T)v;
            else st_pop(d + (size_t)j * N + cell, (float)v);
        }
    }
}

cudaError_t launch_stream_pull_store(int store, double scale, const double* src, void* dst, int nx, int ny, int nz,
                                     cudaStream_t stream, bool open_x, const double* inlet) {
    const int g = grid_for((int64_t)nx * ny * nz, 256);
    switch (store) {
        case PSC_STORE_F64_EXACT: k_stream_pull_store<PSC_STORE_F64_EXACT><<<g, 256, 0, stream>>>(src, dst, nx, ny, nz, scale); break;
        case PSC_STORE_F64: k_stream_pull_store<PSC_STORE_F64><<<g, 256, 0, stream>>>(src, dst, nx, ny, nz, scale); break;
        case PSC_STORE_F32: k_stream_pull_store<PSC_STORE_F32><<<g, 256, 0, stream>>>(src, dst, nx, ny, nz, scale); break;
        case PSC_STORE_F16: k_stream_pull_store<PSC_STORE_F16><<<g, 256, 0, stream>>>(src, dst, nx, ny, nz, scale); break;
        case PSC_STORE_BF16: k_stream_pull_store<PSC_STORE_BF16><<<g, 256, 0, stream>>>(src, dst, nx, ny, nz, scale); break;
        default: return cudaErrorInvalidValue;
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess || !open_x) return e;
    const int gp = grid_for((int64_t)ny * nz, 256);
    const double r = inlet[0], ux = inlet[1], uy = inlet[2], uz = inlet[3];
#define PSC_UNPULL_CASE(S) \
    case S: k_open_x_unpull<S><<<gp, 256, 0, stream>>>(src, dst, nx, ny, nz, scale, r, ux, uy, uz); break;
    switch (store) {
        PSC_UNPULL_CASE(PSC_STORE_F64_EXACT)
        PSC_UNPULL_CASE(PSC_STORE_F64)
        PSC_UNPULL_CASE(PSC_STORE_F32)
        PSC_UNPULL_CASE(PSC_STORE_F16)
        PSC_UNPULL_CASE(PSC_STORE_BF16)
        default: return cudaErrorInvalidValue;
    }
#undef PSC_UNPULL_CASE
    return cudaGetLastError();
}

}  // namespace psc
