// Launch wrappers of the pass kernels for one (precision, N), instantiated
// explicitly in the ps_inst_*.cu units (their bodies: ps_launch_impl.cuh, which
// only those include) so the heavy unrolled kernels compile once, in parallel.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "../../include/ps_gpu.h"
#include "ps_kernels.cuh"

namespace ps {

int launch_fail(cudaError_t e, const char* what);
// Records a message for ps_gpu_last_error() and returns code.
int report_error(int code, const char* msg);
// Shell descriptor as the context builds it (filter.c expressions, host side).
Shell host_shell(int kind, double k, double kmin, double kmax, double binwidth, double L, int N);
// pow(V, n-1) * pow(N, -3n) with V = L^3 (polyspectrum.c:155).
double host_norm_coef(double L, int N, int n);

#define PS_LTRY(x)                \
    do {                          \
        int rc_ = (x);            \
        if (rc_ != 0) return rc_; \
    } while (0)
#define PS_LCK(x)                                        \
    do {                                                 \
        cudaError_t e_ = (x);                            \
        if (e_ != cudaSuccess) return launch_fail(e_, #x); \
    } while (0)

// A kernel reads its transform's table without a test: a launch without one is refused here.
#define PS_NEED_TABLE(p) \
    if (!(p)) return launch_fail(cudaErrorInvalidValue, "twiddle table " #p " of this transform is missing")

template <typename K> int set_smem(K kernel, size_t bytes)
{
    if (bytes > 48 * 1024)
        PS_LCK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    return PS_OK;
}

// Grid of a persistent kernel: as many CTAs as fit on the device at once.
template <typename K> int persistent_grid(K kernel, int threads, size_t smem, int work_items, int* grid)
{
    int dev = 0, sms = 0, per_sm = 0;
    PS_LCK(cudaGetDevice(&dev));
    PS_LCK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    PS_LCK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem));
    if (per_sm < 1) per_sm = 1;
    *grid = std::min(work_items, per_sm * sms);
    return PS_OK;
}

template <class I> inline Items<I> pack(const I* items, int n)
{
    Items<I> b;
    for (int q = 0; q < kItems; q++) b.at[q] = items[q < n ? q : 0];
    return b;
}

// Twiddle tables of one precision: twp = Stockham table of the pencil
// transforms (length N), twr = of the row transforms (length N/2), twpp =
// W_N^k for the r2c / c2r pre- and post-processing (k < N).  twp_alt is not optional
// where the Y pass's default geometry is not the pencils' (host_alt_table says so).
template <typename T> struct Tables {
    const V2<T>* twp;
    const V2<T>* twr;
    const V2<T>* twpp;
    const V2<T>* twp_alt = nullptr;  // Stockham table of the alternative pencil geometry or the Y pass's own, if any
    const V2<T>* twr_alt = nullptr;  // row table of pair kernel variant 2 (PairVariants::ALT_RX), if any
};

template <typename T, int N> struct L3 {
    using V = V2<T>;
    using PG = PencilGeom<T, N>;
    using RG = RowGeom<T, N>;
    static_assert(N == 16 || N == 1024 || PG::W == PencilWidth<T>::value, "tiles of one 128-byte segment");
    static constexpr int ALT = PencilAlt<T, N>::value;
    // the Y pass's alternative geometry (0: none, or its default already is that one)
    static constexpr int Y_ALT = YGeom<T, N, 0>::LONG ? 0 : ALT;
    static constexpr int DOT_ALT = PencilAlt<T, N>::dot_default;
    // host copy of the alternative pencil table, or of the Y pass's where it has a
    // geometry of its own (false: neither)
    static bool host_alt_table(V* twp_alt);
    static constexpr int PAIR_RX2 = PairVariants<T, N>::ALT_RX;
    // host copy of the row table of pair kernel variant 2 (false: no such variant)
    static bool host_pair_alt_table(V* twr_alt);
    // the pair kernel variants this length has (PairVariants): bit v set = variant v runs
    static int pair_variants();
    // host copies of the tables for this N
    static void host_tables(V* twp, V* twr);
    // quad: the xy-quadrant layout of data even in x and y ([i <= N/2][j <= N/2][h])
    // nsrc: grid size of the source spectrum src (0: N; a larger field grid
    // when this N-grid holds a band-limited sub-grid transform)
    // skip_dead: tiles of all-zero pencils (|my| above the shell's band) are
    // left unwritten; the following pass_y must then be given that band
    static int inv_x(cudaStream_t st, const V* src, int ss, V* dst, int ds, int mode, const Shell* sh,
                     int hvalid, const Tables<T>& tb, int quad = 0, int nsrc = 0, int skip_dead = 0, int band = N)
    {
        const XItem<T> it{dst, ds, hvalid, sh, band, 0};
        return inv_x_b(st, src, ss, &it, 1, ds, mode, tb, quad, nsrc, skip_dead);
    }
    // The batched forms take nitems <= kItems descriptions (copied into the launch);
    // ds, ncols, hva, hvb: the widest of the batch.
    static int inv_x_b(cudaStream_t st, const V* src, int ss, const XItem<T>* items, int nitems,
                       int ds, int mode, const Tables<T>& tb, int quad, int nsrc, int skip_dead);
    // jband < N/2: input rows with |my| > jband are zero and are not read
    // ncols (0: stride): only columns h < ncols, a multiple of the pencil width
    // jout < N/2: output rows with |my| > jout are not stored
    // alt: the alternative geometry (PencilAlt) when this length has one
    static int pass_y(cudaStream_t st, V* data, int stride, bool inv, const Tables<T>& tb, int quad = 0,
                      int jband = N, int ncols = 0, int jout = N, int alt = 0, int r2 = 0)
    {
        const int nc = ncols > 0 ? ncols : stride;
        const YItem<T> it{data, stride, nc, jband, jout, r2};
        return pass_y_b(st, &it, 1, nc, inv, tb, quad, alt);
    }
    static int pass_y_b(cudaStream_t st, const YItem<T>* items, int nitems, int ncols, bool inv,
                        const Tables<T>& tb, int quad, int alt);
    static int inv_z(cudaStream_t st, const V* src, int ss, int hvalid, T* out, const T* aux, int epi,
                     int power, double* partials, const Tables<T>& tb, int* nblocks, double scale = 1.0);
    // stage: 1 copies the input rows to shared memory first (k_fwd_z STAGED),
    // 0 loads them straight into registers, -1 picks staging when it applies
    // (16-byte aligned inputs of 4- or 8-byte values, tile fits shared memory)
    // nrows (0: all N^2): rows processed, from the row the pointers start at
    // (a multiple of the row tile RG::WZ)
    // status (non-NULL): stage by bulk copies (cp.async.bulk, one per input
    // array and tile) whose bounded wait sets *status to 1 if it expires
    static int fwd_z(cudaStream_t st, int kind, const void* a, const void* b, V* dst, int ds, int hout,
                     const Tables<T>& tb, int stage = -1, size_t nrows = 0, int* status = nullptr, int tx_extra = 0);
    // variant: the autotuned pair kernel variant (PairVariants; 0 the default,
    // and the default wherever the length lacks the one asked for)
    static int pair_z(cudaStream_t st, const V* a, int sa, int hva, const V* b, int sb, int hvb, V* dst,
                      int ds, int hout, const Tables<T>& tb, int quad = 0, int variant = 0)
    {
        const PairItem<T> it{a, b, dst, sa, hva, sb, hvb, ds, hout};
        return pair_z_b(st, &it, 1, b ? 2 : 1, hva, hvb, tb, quad,
                        variant);
    }
    // hva, hvb: the widest legs of the batch; ninputs: 2 when any item has two
    static int pair_z_b(cudaStream_t st, const PairItem<T>* items, int nitems, int ninputs,
                        int hva, int hvb, const Tables<T>& tb, int quad, int variant);
    template <int RX, bool KEEP, bool REAL, bool TWO>
    static int pair_z_v(cudaStream_t st, const PairItem<T>* items, int nitems, int ninputs,
                        int hva, int hvb, const V* twr, const V* twpp, int quad);
    // Grid sums of products (k_prod_z) of nitems lists of factors, the widest row of
    // hv columns; real: quad rows.  Partials per item: *nblocks (at most prod_blocks()).
    static int prod_z(cudaStream_t st, const ProdItem<T>* items, int nitems, int hv, bool real, int abs_terms,
                      const Tables<T>& tb, int* nblocks);
    static constexpr int prod_blocks(bool real)
    {
        return ((real ? (N / 2 + 1) * (N / 2 + 1) : N * N) + RG::WZ - 1) / RG::WZ;
    }
    // The forward X pass, storing (epi SPEC_STORE, SPEC_STORE_PHASE, SPEC_MASK_ADD)
    // or summing per shell; ndk: grid size of the field spectrum dk (0: N).
    // Returns the blocks per item of the widest spectrum in *nblocks.
    static int fwd_x(cudaStream_t st, const FwdXItem<T>* items, int nitems, int ncols, int epi,
                     V* out, int ostride, const V* dk, int dks, const Tables<T>& tb, int* nblocks, int quad = 0,
                     int ndk = 0, T* mod_out = nullptr, int jband = N, int alt = 0);
};

// Grid sizes.  Powers of two 16..1024, the 3 2^k / 5 2^k sizes of the
// alias-free sub-grids of pair groups (192, 320, 384), and further grid sizes
// 2^a 3^b 5^c a context may run on (48, 60, 96, 300, 600), instantiated in three
// translation units per precision.
#define PS_INSTANTIATE_L3_A(T)        \
    template struct L3<T, 16>;        \
    template struct L3<T, 32>;        \
    template struct L3<T, 64>;        \
    template struct L3<T, 128>;       \
    template struct L3<T, 192>;       \
    template struct L3<T, 256>;
#define PS_INSTANTIATE_L3_B(T)        \
    template struct L3<T, 320>;       \
    template struct L3<T, 384>;
#define PS_INSTANTIATE_L3_C(T)        \
    template struct L3<T, 512>;       \
    template struct L3<T, 1024>;

#define PS_INSTANTIATE_L3_MIXED(T)    \
    template struct L3<T, 48>;        \
    template struct L3<T, 60>;        \
    template struct L3<T, 96>;        \
    template struct L3<T, 300>;       \
    template struct L3<T, 600>;

#define PS_EXTERN_L3(T)                  \
    extern template struct L3<T, 16>;    \
    extern template struct L3<T, 32>;    \
    extern template struct L3<T, 48>;    \
    extern template struct L3<T, 60>;    \
    extern template struct L3<T, 64>;    \
    extern template struct L3<T, 96>;    \
    extern template struct L3<T, 128>;   \
    extern template struct L3<T, 192>;   \
    extern template struct L3<T, 256>;   \
    extern template struct L3<T, 300>;   \
    extern template struct L3<T, 320>;   \
    extern template struct L3<T, 384>;   \
    extern template struct L3<T, 512>;   \
    extern template struct L3<T, 600>;   \
    extern template struct L3<T, 1024>;

}  // namespace ps
