// The handle layer's result transfers (csrc/solver.cu) on the host, over stand-ins of the CUDA calls that they make
// (device memory is host memory): page-locked allocations can be made to fail, copies are counted.
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "solver.cu"

namespace {
bool g_no_pinned = false;       // page-locked allocations fail
cudaError_t g_last = cudaSuccess;
long long g_copied = 0;         // bytes copied off the device
long long g_pinned = 0;         // page-locked bytes asked for
int g_waits = 0;                // stream synchronisations
int g_handle;
}  // namespace

extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) { *p = std::malloc(n); return cudaSuccess; }
cudaError_t cudaFree(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) {
    g_pinned += (long long)n;
    if (g_no_pinned) return g_last = cudaErrorMemoryAllocation;
    *p = std::malloc(n);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = g_last; g_last = cudaSuccess; return e; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    std::memcpy(d, s, n);
    g_copied += (long long)n;
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { ++g_waits; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = reinterpret_cast<cudaEvent_t>(&g_handle); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
}

namespace psc {
int fail(int code, const std::string&) { return code; }
int cuda_fail(cudaError_t, const char*) { return PSC_E_CUDA; }
uint64_t error_seq() { return 0; }
const std::string& last_error_string() { static std::string s; return s; }
cudaError_t launch_copy_rows(const RowCopy* r, int count, double* dst, cudaStream_t) {
    for (int k = 0; k < count; ++k) {
        std::memcpy(dst + r[k].at, r[k].src, (size_t)r[k].n * 8);
        g_copied += r[k].n * 8;
    }
    return cudaSuccess;
}
}  // namespace psc

// 0 where every value arrived and no error is left behind, else 1.
static int fields() {
    int bad = 0;
    for (int64_t n : {1, 7, 65536, 65537, 600001}) {
        std::vector<float> f((size_t)n);
        std::vector<double> d((size_t)n), out((size_t)n + 1);
        for (int64_t i = 0; i < n; ++i) d[(size_t)i] = f[(size_t)i] = (float)(1.0 + 0.37 * (double)i);
        for (bool f64 : {false, true}) {
            HArray<int64_t> ring;
            std::fill(out.begin(), out.end(), -1.0);
            bad |= values_to_host(f64 ? (const void*)d.data() : (const void*)f.data(), f64, n, out.data(), nullptr, ring,
                                  "x") != PSC_OK;
            bad |= std::memcmp(out.data(), d.data(), (size_t)n * 8) != 0 || out[(size_t)n] != -1.0 || g_last != cudaSuccess;
        }
    }
    return bad;
}

// One float field of n values.
static int field(int64_t n) {
    std::vector<float> f((size_t)n, 0.25f);
    std::vector<double> out((size_t)n, -1.0);
    HArray<int64_t> ring;
    int bad = values_to_host(f.data(), false, n, out.data(), nullptr, ring, "x") != PSC_OK;
    for (double v : out) bad |= v != 0.25;
    return bad;
}

static void make_batch(psc_batch& b, int nwin, int P) {
    for (int k = 0; k < nwin; ++k) {
        b.w.emplace_back(new Window);
        Window& w = *b.w.back();
        w.P = P;
        w.loads_ready = true;
        w.forces.ensure(3 * P, true, nullptr);
        w.torques.ensure(3 * P, true, nullptr);
        for (int i = 0; i < 3 * P; ++i) {
            w.forces.p[i] = 1000.0 * k + i;
            w.torques.p[i] = -1000.0 * k - i;
        }
    }
}

static int read(psc_batch& b, int k) {
    const size_t n = 3 * (size_t)b.w[(size_t)k]->P;
    std::vector<double> f(n, -1.0), t(n, -1.0);
    if (psc_batch_get_loads(&b, k, f.data(), t.data()) != PSC_OK) return 1;
    return std::memcmp(f.data(), b.w[(size_t)k]->forces.p, n * 8) != 0 ||
           std::memcmp(t.data(), b.w[(size_t)k]->torques.p, n * 8) != 0 || g_last != cudaSuccess;
}

// results_host fields NO_PINNED | results_host field NO_PINNED VALUES | results_host loads NO_PINNED NWIN P (WINDOW | step)...
int main(int argc, char** argv) {
    g_no_pinned = std::atoi(argv[2]) != 0;
    int bad = 0;
    if (!std::strcmp(argv[1], "fields")) {
        bad = fields();
    } else if (!std::strcmp(argv[1], "field")) {
        bad = field(std::atoll(argv[3]));
    } else {
        psc_batch b;
        make_batch(b, std::atoi(argv[3]), std::atoi(argv[4]));
        for (int k = 5; k < argc; ++k) {
            if (!std::strcmp(argv[k], "step")) {  // what a reporting step leaves; counted from here
                b.loads_at.clear();
                b.loads_take = 1;
                b.loads_last = -1;
                g_copied = g_pinned = g_waits = 0;
            } else {
                bad |= read(b, std::atoi(argv[k]));
            }
        }
    }
    std::printf("%d %lld %lld %d\n", bad, g_copied, g_pinned, g_waits);
    return 0;
}
