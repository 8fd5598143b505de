// ps_gpu_power_spectrum_noalloc: the power spectrum P(k) of a device-resident
// field without any device allocation.
//
// Who needs it: host programs whose GPU memory is owned by another allocator
// and may not be taken by a library behind its back - a framework's caching
// pool that has reserved the device's memory for itself, or a real-time or
// embedded host with a fixed, pre-planned memory budget - where a cudaMalloc
// of the library's own would fail or break that budget.  Everything the
// computation needs beyond the caller's input field and output arrays lives
// in one file-scope device array of fixed size, which the CUDA runtime
// reserves when it loads the library's device code.
//
// Limits and sharing:
//   * grids up to PS_NOALLOC_MAX_N^3 (64^3), at most PS_NOALLOC_MAX_SHELLS
//     shells per call; larger requests are rejected with PS_ERR_ARG;
//   * every GPU that loads the library holds the array (8 MiB) until exit;
//   * all calls on a device share the array and leave their data in it; calls
//     that overlap on the GPU (different streams, or host threads without
//     ordering between them) race on it - serialise them;
//   * the call copies its small tables from host memory, reads its results
//     back and synchronises `stream` before it returns;
//   * the first call on each device looks up the array's device address
//     (cudaGetSymbolAddress) with that device current; make that first call
//     before any stream capture begins.
#include <algorithm>
#include <cmath>
#include <exception>
#include <mutex>
#include <vector>

#include "ps_launch.cuh"
#include "ps_pair2.cuh"

namespace ps {
PS_EXTERN_L3(float)
}  // namespace ps

using namespace ps;

#define PS_NOALLOC_MAX_N 64
#define PS_NOALLOC_MAX_SHELLS 256
#define PS_NOALLOC_SCRATCH_BYTES (8u << 20)

// The scratch memory of ps_gpu_power_spectrum_noalloc.  In host code this name
// is only a host-side stand-in: its device address comes from
// cudaGetSymbolAddress (noalloc_scratch_ptr below).
static __device__ __align__(256) unsigned char g_noalloc_scratch[PS_NOALLOC_SCRATCH_BYTES];

namespace {

constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mu;
unsigned char* g_noalloc_ptr[kMaxDevices] = {nullptr};

// Device address of g_noalloc_scratch on the current device (set up once per device).
int noalloc_scratch_ptr(int dev, unsigned char** out)
{
    if (dev < 0 || dev >= kMaxDevices) return report_error(PS_ERR_ARG, "device ordinal out of range");
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (!g_noalloc_ptr[dev]) {
        void* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p) return launch_fail(e != cudaSuccess ? e : cudaErrorInvalidSymbol,
                                                       "cudaGetSymbolAddress(g_noalloc_scratch)");
        g_noalloc_ptr[dev] = (unsigned char*)p;
    }
    *out = g_noalloc_ptr[dev];
    return PS_OK;
}

size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

// B = coef * sumD / (N^3 * count), Npoly = count: the batched method's
// normalisation.
__global__ void k_noalloc_finalize(int ns, double coef, double n3, const double* __restrict__ sums,
                                   double* __restrict__ out)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= ns) return;
    const double cnt = sums[ns + s];
    out[2 * s] = __ddiv_rn(__dmul_rn(coef, sums[s]), __dmul_rn(cnt, n3));
    out[2 * s + 1] = cnt;
}

template <int N>
int run_noalloc(cudaStream_t st, unsigned char* base, double L, const float* field, int phase, int ns,
                const double* k, double bw, double* P, double* Npoly)
{
    using V32 = float2;
    constexpr int W32 = PencilGeom<float, N>::W;
    constexpr int S32 = (N / 2 + 1 + W32 - 1) / W32 * W32;
    // host values of what the call copies in, one block: the twiddle tables (the
    // context's expressions, made once per size) and the sorted shells
    struct Head {
        V32 tw[N], twp[N], twr[N / 2];
        P2Chunk chunks[(PS_NOALLOC_MAX_SHELLS + kP2Shells - 1) / kP2Shells];
        P2Range iv[PS_NOALLOC_MAX_SHELLS];
        int idx[PS_NOALLOC_MAX_SHELLS];
    };
    static thread_local Head h;
    static thread_local bool tables = false;
    if (!tables) {
        const long double two_pi = 6.283185307179586476925286766559005768L;
        for (int m = 0; m < N; m++) {
            const long double a = two_pi * (long double)m / (long double)N;
            h.tw[m] = V32{(float)cosl(a), (float)(-sinl(a))};
        }
        L3<float, N>::host_tables(h.twp, h.twr);
        tables = true;
    }
    std::vector<P2Range> iv(ns);
    std::vector<int> order(ns);
    std::vector<P2Range> by_cfg(ns);
    for (int s = 0; s < ns; s++) {
        const Shell sh = host_shell(SHELL_DEFAULT, k[s], 0.0, 0.0, bw, L, N);
        by_cfg[s] = P2Range{sh.r2lo, sh.r2hi};
        order[s] = s;
    }
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return by_cfg[x].lo < by_cfg[y].lo; });
    for (int s = 0; s < ns; s++) {
        h.iv[s] = iv[s] = by_cfg[order[s]];
        h.idx[s] = order[s];
    }
    const std::vector<P2Chunk> chunks = pair2_chunks(iv, N, 148 * 4);
    std::copy(chunks.begin(), chunks.end(), h.chunks);
    const int nch = (int)chunks.size(), blocks = chunks.back().block0 + chunks.back().nblocks;

    size_t off = 0;
    auto carve = [&](size_t bytes) {
        unsigned char* p = base + off;
        off += align256(bytes);
        return p;
    };
    V32* spec32 = (V32*)carve(sizeof(V32) * (size_t)N * N * S32);
    Head* d = (Head*)carve(sizeof(Head));
    double* cparts = (double*)carve(sizeof(double) * (size_t)ns * kP2CountParts);
    double* partials = (double*)carve(sizeof(double) * (size_t)blocks * kP2Shells);
    double* sums = (double*)carve(sizeof(double) * 2 * PS_NOALLOC_MAX_SHELLS);
    double* out = (double*)carve(sizeof(double) * 2 * PS_NOALLOC_MAX_SHELLS);
    if (off > PS_NOALLOC_SCRATCH_BYTES) return report_error(PS_ERR_ARG, "no-alloc scratch too small");
    PS_LCK(cudaMemcpyAsync(d, &h, sizeof(Head), cudaMemcpyHostToDevice, st));
    const Tables<float> tb32{d->twp, d->twr, d->tw};

    // forward transform of the field (get_FT_field + optional phase normalisation)
    PS_LTRY((L3<float, N>::fwd_z(st, SRC_F32, field, nullptr, spec32, S32, N / 2 + 1, tb32)));
    PS_LTRY((L3<float, N>::pass_y(st, spec32, S32, false, tb32)));
    FwdXItem<float> it{};
    it.data = spec32;
    it.stride = it.ncols = S32;
    it.hvalid = N / 2 + 1;
    PS_LTRY((L3<float, N>::fwd_x(st, &it, 1, S32, phase == 1 ? SPEC_STORE_PHASE : SPEC_STORE, spec32, S32,
                                 nullptr, 0, tb32, nullptr)));
    // all shells in one sweep over the spectrum (Parseval): sums of |dk|^2 in
    // FP64 and exact counts; per-shell inverse transforms (six passes and two
    // reductions each) took 1.45 ms for 32 shells at 64^3
    const double n3 = (double)N * (double)N * (double)N;
    k_pair2_sweep<float><<<blocks, kP2Threads, 0, st>>>(N, spec32, S32, d->chunks, nch, d->iv, partials);
    k_pair2_counts<<<dim3(ns, kP2CountParts), 256, 0, st>>>(N, d->iv, cparts);
    k_pair2_finish<<<nch, 256, 0, st>>>(d->chunks, partials, d->idx, n3, sums, cparts, sums + ns);
    k_noalloc_finalize<<<(ns + 127) / 128, 128, 0, st>>>(ns, host_norm_coef(L, N, 2), n3, sums, out);
    PS_LCK(cudaGetLastError());
    static thread_local double hout[2 * PS_NOALLOC_MAX_SHELLS];
    PS_LCK(cudaMemcpyAsync(hout, out, sizeof(double) * 2 * ns, cudaMemcpyDeviceToHost, st));
    PS_LCK(cudaStreamSynchronize(st));
    for (int s = 0; s < ns; s++) {
        P[s] = hout[2 * s];
        Npoly[s] = hout[2 * s + 1];
    }
    return PS_OK;
}

}  // namespace

extern "C" int ps_gpu_power_spectrum_noalloc(int nbins, double boxsize, const float* field_dev,
                                             int use_only_phase, int nshell, const double* k,
                                             double kbinwidth, double* P, double* Npoly, void* stream)
{
    if (!field_dev || !k || !P || !Npoly) return report_error(PS_ERR_ARG, "NULL argument");
    if (nbins != 16 && nbins != 32 && nbins != 64)
        return report_error(PS_ERR_ARG, "ps_gpu_power_spectrum_noalloc: grid size must be 16, 32 or 64 "
                                        "(the fixed scratch holds at most 64^3)");
    if (nshell < 1 || nshell > PS_NOALLOC_MAX_SHELLS)
        return report_error(PS_ERR_ARG, "ps_gpu_power_spectrum_noalloc: 1..256 shells per call");
    if (!(boxsize > 0.0) || !std::isfinite(boxsize))
        return report_error(PS_ERR_ARG, "box size must be positive and finite");
    if (!(kbinwidth > 0.0) || !std::isfinite(kbinwidth))
        return report_error(PS_ERR_ARG, "kbinwidth must be positive and finite");
    if (use_only_phase != 0 && use_only_phase != 1) return report_error(PS_ERR_ARG, "use_only_phase must be 0 or 1");
    int dev = 0;
    PS_LCK(cudaGetDevice(&dev));
    unsigned char* base = nullptr;
    PS_LTRY(noalloc_scratch_ptr(dev, &base));
    cudaStream_t st = (cudaStream_t)stream;
    try {
        switch (nbins) {
        case 16: return run_noalloc<16>(st, base, boxsize, field_dev, use_only_phase, nshell, k, kbinwidth, P, Npoly);
        case 32: return run_noalloc<32>(st, base, boxsize, field_dev, use_only_phase, nshell, k, kbinwidth, P, Npoly);
        default: return run_noalloc<64>(st, base, boxsize, field_dev, use_only_phase, nshell, k, kbinwidth, P, Npoly);
        }
    } catch (const std::exception&) {  // the host's small tables
        return report_error(PS_ERR_OOM, "host memory");
    }
}
