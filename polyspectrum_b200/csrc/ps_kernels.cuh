// 3D r2c / c2r pass kernels with fused loaders and epilogues.
//
// Layouts (row-major, i = axis 0, j = axis 1, l = axis 2 as in the reference's
// [i][j][l], filter.c:59):
//   real grid     x[(i*N + j)*N + l]
//   half spectrum X[(i*N + j)*S + h], h in [0, S), S >= band, S % W == 0;
//                 only h <= N/2 is spectrum, columns above hold don't-care data
//
// Inverse 3D transform (c2r, unnormalised like FFTW_BACKWARD, fft.c:52):
//   inv_x  : along i for every (j,h) pencil; loads through a shell filter
//   pass_y : along j for every (i,h) pencil, in place
//   inv_z  : c2r along l for every (i,j) row; epilogue stores / multiplies /
//            reduces the real field
//   pair_z : c2r of two rows, product, r2c of the product (pair groups)
// Forward 3D transform (r2c, unnormalised like FFTW_FORWARD, fft.c:32):
//   fwd_z  : r2c along l, loader composes the input field
//   pass_y : along j
//   fwd_x  : along i; epilogue stores the spectrum (optionally phase only) or
//            folds it into per-shell dot products
//
// Unit shells (polygon counts) are even in every axis, so their transforms are
// real and even too and are kept on the xy-quadrant i, j <= N/2 as real numbers
// ("quad" below, FP64): a row of the quadrant spectrum holds columns 2p and
// 2p + 1 as the two lanes of complex element p, and one complex transform along x
// or y of the pair is the transform of both columns, each staying in its lane.
//
// Every kernel stages the twiddle table W_N^m (m < N) in shared memory first;
// row kernels synchronise per row (warp or named barrier), pencil kernels per
// CTA (a pencil's threads span several warps).
#pragma once

#include <type_traits>

#include "ps_common.cuh"
#include "ps_fft.cuh"

namespace ps {

constexpr int MAX_DOT_SHELLS = 16;

// Pencils per CTA in the strided passes: one 128-byte segment of a row.
template <typename T> struct PencilWidth { static constexpr int value = 128 / (int)sizeof(V2<T>); };

// Threads per pencil (strided-axis) transform: N / (register-plan radix),
// with radix 16 for FP32 at N = 512 so a CTA of 16 pencils is 512 threads;
// split lengths take the larger factor, rounded up so that a CTA is whole warps.
template <typename T, int N> struct PencilThreads {
    static constexpr int split(int v) { return v * PencilWidth<T>::value % 32 ? split(v + 1) : v; }
    static constexpr int value = LenKind<N>::SPLIT ? split(SplitPlan<N>::RB)
                               : N / ((sizeof(T) == 4 && N == 512) ? 16 : DefaultRadix<N>::value);
};
// RX > 0 takes the register plan with RX elements per thread (pass variants).
// MAXT: most threads of a CTA (the tile is then narrower than a 128-byte segment).
template <typename T, int N, int RX = 0, int MAXT = 512> struct PencilGeom {
    static constexpr bool SPLIT = LenKind<N>::SPLIT && RX == 0;
    static constexpr int TPF = RX > 0 ? N / RX : PencilThreads<T, N>::value;
    using SG = SplitGeom<SPLIT ? N : 600, TPF>;
    // slots of a thread going in and coming out, and what they hold: position
    // ip(t, e) where il(t, e), op and ol likewise (register plans: t + TPF e, all live)
    static constexpr int RI = SPLIT ? SG::RI : N / TPF, RO = SPLIT ? SG::RO : N / TPF;
    static constexpr int R = RI > RO ? RI : RO;
    __device__ static constexpr int ip(int t, int e) { return SPLIT ? SG::ip(t, e) : t + TPF * e; }
    __device__ static constexpr bool il(int t, int e) { return !SPLIT || SG::il(t, e); }
    __device__ static constexpr int op(int t, int e) { return SPLIT ? SG::op(t, e) : t + TPF * e; }
    __device__ static constexpr bool ol(int t, int e) { return !SPLIT || SG::ol(t, e); }
    // one 128-byte segment per row, whole warps per CTA, at most MAXT threads
    // (512: an epilogue keeps 16 FP64 accumulators in registers)
    static constexpr int W0 = PencilWidth<T>::value * TPF >= 32 ? PencilWidth<T>::value : 32 / TPF;
    static constexpr int W = W0 * TPF > MAXT ? MAXT / TPF : W0;
    static constexpr int THREADS = TPF * W;
    static constexpr size_t TW_BYTES = (size_t)N * sizeof(V2<T>);  // Stockham table (N-1 used)
    static constexpr size_t SMEM = TW_BYTES + (size_t)N * W * sizeof(V2<T>);
    // FP32 dot passes also stage the tile's field-spectrum pencils ([N][W],
    // interleaved like the exchange buffer) when that fits in shared memory
    static constexpr size_t DK_BYTES = (size_t)N * W * sizeof(V2<T>);
    static constexpr bool DK_SMEM = sizeof(T) == 4 && SMEM + DK_BYTES <= 227 * 1024;
    static constexpr size_t SMEM_DOT = SMEM + (DK_SMEM ? DK_BYTES : 0);
};

// Geometries of single passes at 512 and 1024 points in FP32.  The storing X pass, whose rows
// lie 4 MB apart, takes whole 128-byte segments and one CTA of 1024 threads per SM
// (2.43 against 2.92 ms for the 1024^3 field with 64-byte segments and two CTAs of
// 512), the Y pass 32 elements per thread in two passes (1.91 against 2.11 ms; at 512
// points 0.146 against 0.156 ms).
template <typename T, int N, int RX> struct StoreXGeom {
    static constexpr bool WIDE = sizeof(T) == 4 && N == 1024 && RX == 0;
    using type = PencilGeom<T, N, RX, WIDE ? 1024 : 512>;
};
template <typename T, int N, int RX> struct YGeom {
    static constexpr bool LONG = sizeof(T) == 4 && (N == 512 || N == 1024) && RX == 0;
    using type = PencilGeom<T, N, LONG ? 32 : RX, LONG && N == 1024 ? 256 : 512>;
};

// The alternative pencil geometry of the FP32 Y and dot passes for the larger
// lengths: twice the elements per thread, half the threads per pencil, one radix
// pass fewer; for a split length its register plan, which needs fewer registers (0:
// none).  Chosen per length by the plan autotuner against the default; the 512-point Y
// pass has this geometry anyway (YGeom).
template <typename T, int N> struct PencilAlt {
    static constexpr int odd = LenKind<N>::odd_of(N);
    static constexpr int value = !(sizeof(T) == 4 && N >= 128 && N <= 512 && odd <= 5) ? 0
                               : LenKind<N>::SPLIT ? DefaultRadix<N>::value : 2 * PencilGeom<T, N>::R;
    // the dot pass without a timed choice: 0.136 against 0.155 ms at 384 points (the
    // split plan's 24 elements and 16 sums per thread spill at two CTAs per SM), the
    // split plan below
    static constexpr int dot_default = N == 384 && value > 0 ? 1 : 0;
};

// Elements per thread of the row (contiguous-axis) transforms of length NH:
// at most 32 threads per row (warp-synchronous) except FP64 rows of 512,
// which use radix 8 and 64 threads (two transforms must fit in registers).
template <typename T, int NH> struct RowRadix {
    static constexpr bool POW2 = (NH & (NH - 1)) == 0;
    // rows of 160 (320-point grids): radix 10 keeps two row transforms in
    // registers (radix 20 needed over 220 registers per thread)
    static constexpr int value = NH == 160 ? 10 : !POW2 ? DefaultRadix<NH>::value
                               : NH <= 16 ? NH : ((sizeof(T) == 4 && NH == 512) ? 16 : 8);
};
// RX > 0 overrides the elements per thread of a register-plan row length
// (the pair kernel's variants).
template <typename T, int N, int RX = 0> struct RowGeom {
    static constexpr int NH = N / 2;
    static constexpr bool SPLIT = LenKind<NH>::SPLIT && RX == 0;
    // split rows (30, 96, 150, 160, 192, 300): a power of two of threads, so that rows pack warps
    static constexpr int TPF = SPLIT ? (NH == 30 || NH == 96 ? 8 : NH <= 192 || sizeof(T) == 4 ? 16 : 32)
                                     : NH / (RX > 0 ? RX : RowRadix<T, NH>::value);
    using SG = SplitGeom<SPLIT ? NH : 300, TPF>;
    // slots of a thread on the spectrum side (kp, kl: column k) and on the real side
    // (tp, tl: pair n of the row); register plans: t + TPF e on both, all live
    static constexpr int RK = SPLIT ? SG::RI : NH / TPF, RT = SPLIT ? SG::RO : NH / TPF;
    static constexpr int R = RK > RT ? RK : RT;
    __device__ static constexpr int kp(int t, int e) { return SPLIT ? SG::ip(t, e) : t + TPF * e; }
    __device__ static constexpr bool kl(int t, int e) { return !SPLIT || SG::il(t, e); }
    __device__ static constexpr int tp(int t, int e) { return SPLIT ? SG::op(t, e) : t + TPF * e; }
    __device__ static constexpr bool tl(int t, int e) { return !SPLIT || SG::ol(t, e); }
    static constexpr int EPC = 16 / (int)sizeof(V2<T>);  // complex elements per 16-byte copy
    // Rows shorter than a 128-byte block of threads share a warp: their buffers are
    // set apart by SKEW elements modulo a block, so that the rows of a warp fall on
    // different banks (rows of 4 threads at 96 points: two of three shared-memory
    // accesses were conflicts; pair kernel of a batch there 0.031 -> 0.015 ms).
    static constexpr int BLOCK = 128 / (int)sizeof(V2<T>);
    static constexpr int SKEW = TPF < BLOCK ? (TPF < EPC ? EPC : TPF) : 0;
    // rows per CTA (tile): up to 256 threads and 32 rows, and as many as fit
    // in 227 KB of shared memory with two double-buffered full-length inputs
    // (FP64: 128 threads, whose smaller tiles leave less of an SM unused)
    static constexpr int WZ0 = ((sizeof(T) == 8 ? 128 : 256) / TPF) < 32 ? ((sizeof(T) == 8 ? 128 : 256) / TPF) : 32;
    // exchange buffer of a row: its padded passes, rounded up to the skew
    static constexpr int ROWBUF0 = (SmemRow<V2<T>>::template size<NH, R, SPLIT>() + EPC - 1) / EPC * EPC;
    static constexpr int ROWBUF = SKEW ? ROWBUF0 + (SKEW + BLOCK - ROWBUF0 % BLOCK) % BLOCK : ROWBUF0;
    // input stage pitch (elements) for rows of hv valid entries
    __host__ __device__ static constexpr int pitch(int hv)
    {
        const int p = (hv + EPC - 1) / EPC * EPC;
        return SKEW ? p + (SKEW + BLOCK - p % BLOCK) % BLOCK : p;
    }
    static constexpr size_t ROW_BYTES = (size_t)(ROWBUF + 4 * pitch(NH + 1)) * sizeof(V2<T>);
    static constexpr int WZ_FIT = (int)((227 * 1024 - (size_t)(2 * NH + 2) * sizeof(V2<T>)) / ROW_BYTES);
    __host__ __device__ static constexpr int pow2_floor(int v) { return v >= 2 ? 2 * pow2_floor(v / 2) : 1; }
    // and a divisor of the N^2 rows, so whole tiles cover the grid
    __host__ __device__ static constexpr int pow2_dividing(int v, int cap) { return cap > 1 && v % cap ? pow2_dividing(v, cap / 2) : cap; }
    static constexpr int WZ = pow2_dividing(N * N, pow2_floor(WZ0 < WZ_FIT ? WZ0 : WZ_FIT));
    static constexpr int THREADS = TPF * WZ;
    // shared memory: row Stockham table [NH], pre/post twiddles W_N^k, k <= NH
    // [NH+2], per-row exchange buffers [WZ][NH], then the input stages
    static constexpr size_t TWR_OFF = 0;
    static constexpr size_t TWPP_OFF = TWR_OFF + (size_t)NH * sizeof(V2<T>);
    static constexpr size_t ROWBUF_OFF = TWPP_OFF + (size_t)(NH + 2) * sizeof(V2<T>);
    static constexpr size_t STAGE_OFF = ROWBUF_OFF + (size_t)WZ * ROWBUF * sizeof(V2<T>);
    // dynamic shared memory of a kernel with `ninputs` double-buffered inputs
    __host__ __device__ static constexpr size_t smem(int ninputs, int hva, int hvb)
    {
        return STAGE_OFF + (size_t)2 * WZ * (pitch(hva) + (ninputs > 1 ? pitch(hvb) : 0)) * sizeof(V2<T>);
    }
    static_assert(TPF <= 32 || WZ <= 15, "one named barrier per row");
    static_assert(THREADS % 32 == 0, "whole warps per CTA");
    static_assert(smem(2, NH + 1, NH + 1) <= 227 * 1024, "row tile exceeds shared memory");
};

// Copy a twiddle table into shared memory (whole CTA).
template <typename V>
__device__ __forceinline__ V* stage_table(unsigned char* smem, const V* __restrict__ src, int n)
{
    V* dst = reinterpret_cast<V*>(smem);
    for (int q = threadIdx.x; q < n; q += blockDim.x) dst[q] = src[q];
    return dst;
}

// cp.async (16-byte, L2-only) copies global -> shared, grouped; the waits are
// the hardware's own (no polling loop in this code).
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem)
{
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_prev() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// One level of a warp's recursive-halving sum of per-lane arrays: v[0..2H)
// -> v[0..H) holding, for lanes with (lane & O), the upper half plus the
// partner lane's upper half, else the lower halves.
template <int N2, int O> __device__ __forceinline__ void halve_sums(double* v, int lane)
{
    constexpr int H = N2 / 2;
    const bool up = (lane & O) != 0;
#pragma unroll
    for (int k = 0; k < H; k++) {
        const double keep = up ? v[k + H] : v[k];
        const double send = up ? v[k] : v[k + H];
        v[k] = keep + __shfl_xor_sync(0xffffffffu, send, O);
    }
}

// Stage WZ consecutive spectrum rows (first hv entries, rounded up to a
// 16-byte multiple, which stays inside the row stride ss) into `stage`
// (pitch P) with the whole CTA.
template <typename V, int WZ, int THREADS>
__device__ __forceinline__ void stage_rows(V* stage, int P, const V* __restrict__ src, size_t row0, int ss, int hv,
                                           int nrows = 0x7fffffff)
{
    constexpr int EPC = 16 / (int)sizeof(V);
    const int chunks = (hv + EPC - 1) / EPC;
    for (int c = threadIdx.x; c < WZ * chunks; c += THREADS) {
        const int w = c / chunks, q = c - w * chunks;
        if (row0 + w < (size_t)nrows) cp_async16(stage + w * P + q * EPC, src + (row0 + w) * ss + q * EPC);
    }
}

// ------------------------------------------------------------------ reductions
// Deterministic block sum: fixed shuffle tree, then warp partials in order.
template <int THREADS> __device__ __forceinline__ double block_sum(double v, double* red)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    constexpr int NW = (THREADS + 31) / 32;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) red[wid] = v;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x == 0) {
#pragma unroll 1
        for (int q = 0; q < NW; q++) s += red[q];
    }
    return s;
}

// ------------------------------------------------------------------ batches
// The passes of a pair group run on spectra of one transform size but of
// different bands.  A launch works on up to kItems of them, blockIdx.y picking
// its description: a sweep of small groups (64 equilateral triangles on 16- to
// 128-point grids, say) is a few launches instead of a dozen per triangle.
// blockIdx.x covers the largest spectrum of the batch; blocks past a smaller one
// return at once.  The descriptions are kernel arguments, so their fields are
// uniform constants: read from device memory they took 10 to 20 registers per
// thread, which cost the 512-point Y pass half its CTAs (0.138 -> 0.207 ms).
constexpr int kItems = 32;
template <class I> struct Items {
    I at[kItems];
};
template <class I> __device__ __forceinline__ const I& item_at(const Items<I>& b) { return b.at[blockIdx.y]; }
template <class I> __device__ __forceinline__ const I& item_at(const I& one) { return one; }
template <typename T> struct XItem {  // inverse X
    V2<T>* dst;
    int ds;              // row stride, a multiple of the pencil width
    int hvalid;
    const Shell* shell;  // NULL for plain loads
    int band;            // plain loads: components above it are zero and not read
    int r2;              // > 0: no mode with |m|^2 > r2 (skip_dead leaves those tiles unwritten)
};
template <typename T> struct YItem {  // Y pass
    V2<T>* data;
    int stride, ncols;  // columns h < ncols, a multiple of the pencil width
    int jband, jout;
    int r2;             // > 0: as XItem's, of the input rows (inverse) or of the rows to store (forward)
};
template <typename T> struct PairItem {  // pair kernel
    const V2<T>* A;
    const V2<T>* B;  // NULL: the square of A
    V2<T>* dst;
    int sa, hva, sb, hvb, ds, hout;
};
template <typename T> struct FwdXItem {  // forward X
    V2<T>* data;
    int stride, hvalid;
    int ncols;                  // columns h < ncols, a multiple of the pencil width
    int nshell;
    const Shell* shells;
    const unsigned short* lut;  // r2 -> shell bitmask (interval shells; NULL: the shells themselves)
    int lut_size;
    const unsigned short* vol;  // |m| components <= vol_band -> shell bitmask (other shells; NULL: evaluated here)
    int vol_band;
    int interval;               // the shells are at most two r2 intervals, compared directly
    int r2max;                  // no shell holds a mode with |m|^2 > r2max
    double weight;
    double* partials;           // [nshell][blocks]
};

// The pencils (my, h) that can hold a mode of a spectrum with |m|^2 <= r2 are those
// with my^2 + h^2 <= r2: a disc, which a shell's X and Y passes leave out a fifth of
// the band's square for.  Decided per 16 columns (per tile at most), so that passes of
// different tile widths agree: the first real column of the 16 that element h is in.
__device__ __forceinline__ int cut_column(int h, int quad) { return (h & ~15) * (quad ? 2 : 1); }
constexpr int kCutFrom = 192;  // points: below, the kernels have no such test (the items' r2 is 0)

// ------------------------------------------------------------------ inverse X
enum InvLoad : int { LOAD_PLAIN = 0, LOAD_MASKED = 1, LOAD_UNIT = 2 };  // LOAD_UNIT: quad only

template <typename T, int N>
__global__ void __launch_bounds__(PencilGeom<T, N>::THREADS)
    k_inv_x(const V2<T>* __restrict__ src, int src_stride, int nsrc, const __grid_constant__ Items<XItem<T>> items,
            int mode, int quad_arg, int skip_dead, const V2<T>* __restrict__ tw_g)
{
    using G = PencilGeom<T, N>;
    using V = V2<T>;
    const int quad = quad_arg;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const XItem<T>& it = items.at[blockIdx.y];
    V* __restrict__ dst = it.dst;
    const int dst_stride = it.ds, hvalid = it.hvalid;
    const Shell* __restrict__ shell_p = it.shell;
    const int tiles_per_row = dst_stride / G::W;
    if ((int)blockIdx.x >= (quad ? N / 2 + 1 : N) * tiles_per_row) return;
    // skip_dead: a filtered tile whose |my| exceeds the shell's band, or that lies
    // outside the disc of its r2, holds only zeros and is not written (the inverse Y
    // pass then treats those rows as zero, its jband and r2)
    static_assert(N == 16 || 16 % G::W == 0, "cut_column");
    if (skip_dead) {
        const int my = lattice_freq((int)(blockIdx.x / tiles_per_row), N);
        if (abs(my) > (mode == LOAD_PLAIN ? it.band : shell_p->band)) return;
        if constexpr (N >= kCutFrom) {
            const int hc = cut_column((int)(blockIdx.x % tiles_per_row) * G::W, quad);
            if (it.r2 > 0 && my * my + hc * hc > it.r2) return;
        }
    }
    const V* tw = stage_table<V>(smem_raw, tw_g, N);
    __syncthreads();
    SmemInterleaved<V, G::W> sm{reinterpret_cast<V*>(smem_raw + G::TW_BYTES), (int)(threadIdx.x % G::W)};
    const int w = threadIdx.x % G::W, t = threadIdx.x / G::W;
    // quad: pencils j <= N/2 only, outputs i <= N/2 only, stored [i][j][h] with
    // N/2+1 rows per plane; column element h holds the unit filter's columns 2h
    // and 2h + 1.
    // nsrc: grid size of the source spectrum ([nsrc][nsrc][src_stride]); a mode
    // m of this N-grid is read at index m mod nsrc there (nsrc >= N, and the
    // shell's band is below N/2, so every selected mode has one home in both).
    const int nj = quad ? N / 2 + 1 : N;
    const int j = blockIdx.x / tiles_per_row;
    const int h = (blockIdx.x % tiles_per_row) * G::W + w;
    const int my = lattice_freq(j, N);
    const int mz = h == N / 2 ? -(N / 2) : h;
    const bool col_ok = h < hvalid && h <= N / 2;
    const size_t js = (size_t)(my < 0 ? my + nsrc : my);
    Shell sh;
    if (mode != LOAD_PLAIN) sh = *shell_p;
    else sh.band = it.band;
    const bool pencil_live =
        !quad && col_ok && abs(my) <= sh.band && abs(mz) <= sh.band;
    // filter bits of this thread's R modes, one predicate instance (loop not unrolled)
    unsigned bits = 0u;
    if (pencil_live) {
        if (mode == LOAD_PLAIN) {
#pragma unroll
            for (int e = 0; e < G::RI; e++)
                if (G::il(t, e) && abs(lattice_freq(G::ip(t, e), N)) <= sh.band) bits |= 1u << e;
        } else {
#pragma unroll 1
            for (int e = 0; e < G::RI; e++) {
                if (!G::il(t, e)) continue;
                const int mx = lattice_freq(G::ip(t, e), N);
                if (abs(mx) <= sh.band && shell_bit(sh, mx, my, mz)) bits |= 1u << e;
            }
        }
    }
    V a[G::R];
    if constexpr (sizeof(T) == 8) {
        if (quad) {
#pragma unroll
            for (int e = 0; e < G::RI; e++) a[e] = czero<V>();
            for (int lane = 0; lane < 2; lane++) {
                const int hz = 2 * h + lane, mzq = hz == N / 2 ? -(N / 2) : hz;
                if (hz > N / 2 || hz >= hvalid || abs(my) > sh.band || abs(mzq) > sh.band) continue;
                unsigned in = 0u;
#pragma unroll 1
                for (int e = 0; e < G::RI; e++) {
                    if (!G::il(t, e)) continue;
                    const int mx = lattice_freq(G::ip(t, e), N);
                    if (abs(mx) <= sh.band && shell_bit(sh, mx, my, mzq)) in |= 1u << e;
                }
#pragma unroll
                for (int e = 0; e < G::RI; e++)
                    if ((in >> e) & 1u) (lane ? a[e].y : a[e].x) = (T)1;
            }
        }
    }
#pragma unroll
    for (int e = 0; e < G::RI; e++) {
        if (sizeof(T) == 8 && quad) break;
        const int mx = lattice_freq(G::ip(t, e), N);
        V v = czero<V>();
        if ((bits >> e) & 1u) {
            v = src[((size_t)(mx < 0 ? mx + nsrc : mx) * nsrc + js) * src_stride + h];
        }
        a[e] = v;
    }
    fft_geom<G, V, N, true>(a, t, sm, tw, BlockSync{});
#pragma unroll
    for (int e = 0; e < G::RO; e++) {
        const int i = G::op(t, e);
        if (G::ol(t, e) && (!quad || i <= N / 2)) dst[((size_t)i * nj + j) * dst_stride + h] = a[e];
    }
}

// ------------------------------------------------------------------ Y pass
template <typename T, int N, bool INV, int RX = 0>
__global__ void __launch_bounds__(YGeom<T, N, RX>::type::THREADS)
    k_pass_y(const __grid_constant__ Items<YItem<T>> items, int quad_arg, const V2<T>* __restrict__ tw_g)
{
    using G = typename YGeom<T, N, RX>::type;
    using V = V2<T>;
    const int quad = quad_arg;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const YItem<T>& it = items.at[blockIdx.y];
    V* __restrict__ data = it.data;
    const int stride = it.stride, ncols = it.ncols;
    const int jband = it.jband, jout = it.jout;
    if ((int)blockIdx.x >= (quad ? N / 2 + 1 : N) * (ncols / G::W)) return;
    const int w = threadIdx.x % G::W, t = threadIdx.x / G::W;
    const int tiles_per_plane = ncols / G::W;  // columns h < ncols of rows of stride `stride`
    static_assert(N == 16 || 16 % G::W == 0, "cut_column");
    int cut = 0x7fffffff;  // rows my^2 > cut: zero, or not to be stored
    if constexpr (N >= kCutFrom) {
        const int hc = cut_column((int)(blockIdx.x % tiles_per_plane) * G::W, quad);
        if (it.r2 > 0) cut = it.r2 - hc * hc;
        if (!INV && cut < 0) return;
    }
    const auto inside = [&](int my, int band) {
        return (band >= N / 2 || abs(my) <= band) && (N < kCutFrom || my * my <= cut);
    };
    // quad: planes i <= N/2, rows j <= N/2 stored, row N-j read as row j
    // (data even in y)
    const int nj = quad ? N / 2 + 1 : N;
    const int i = blockIdx.x / tiles_per_plane;
    const int h = (blockIdx.x % tiles_per_plane) * G::W + w;
    V* base = data + (size_t)i * nj * stride + h;
    // jband < N/2: rows with |my| > jband are zero and not read (the inverse X
    // pass of a band-limited shell leaves them unwritten)
    V a[G::R];
#pragma unroll
    for (int e = 0; e < G::RI; e++) {
        const int j = G::ip(t, e);
        const int jr = quad && j > N / 2 ? N - j : j;
        const bool in = INV ? inside(lattice_freq(j, N), jband) : jband >= N / 2 || abs(lattice_freq(j, N)) <= jband;
        a[e] = G::il(t, e) && in ? base[(size_t)jr * stride] : czero<V>();
    }
    const V* tw = stage_table<V>(smem_raw, tw_g, N);
    __syncthreads();
    SmemInterleaved<V, G::W> sm{reinterpret_cast<V*>(smem_raw + G::TW_BYTES), w};
    fft_geom<G, V, N, INV>(a, t, sm, tw, BlockSync{});
#pragma unroll
    for (int e = 0; e < G::RO; e++) {
        const int j = G::op(t, e);
        // jout < N/2: rows with |my| > jout are read by no later pass and not stored
        const bool in = INV ? jout >= N / 2 || abs(lattice_freq(j, N)) <= jout : inside(lattice_freq(j, N), jout);
        if (G::ol(t, e) && (!quad || j <= N / 2) && in)
            base[(size_t)j * stride] = a[e];
    }
}

// ------------------------------------------------------------------ row helpers
// A CTA works on tiles of WZ consecutive (i,j) rows; row w of a tile is done
// by threads [w*TPF, (w+1)*TPF), which synchronise among themselves only.
template <typename T, int N, int RX = 0> struct RowCtx {
    using G = RowGeom<T, N, RX>;
    using V = V2<T>;
    int w, t;
    V* rowbuf;       // this row's exchange buffer [ROWBUF >= NH]
    const V* twr;    // Stockham table of the NH-point transform
    const V* twpp;   // W_N^k, k <= NH (r2c / c2r pre- and post-processing)
    RowSync<G::TPF> sync;
    // stage both tables (caller issues the __syncthreads that publishes them)
    __device__ __forceinline__ RowCtx(unsigned char* smem, const V* __restrict__ twr_g,
                                      const V* __restrict__ twpp_g)
    {
        twr = stage_table<V>(smem + G::TWR_OFF, twr_g, G::NH);
        twpp = stage_table<V>(smem + G::TWPP_OFF, twpp_g, G::NH + 1);
        w = threadIdx.x / G::TPF;
        t = threadIdx.x % G::TPF;
        rowbuf = reinterpret_cast<V*>(smem + G::ROWBUF_OFF) + w * G::ROWBUF;
        sync.bar = 1 + w;
        if constexpr (G::TPF >= 32) {
            sync.mask = 0xffffffffu;
        } else {
            const int base = (threadIdx.x & 31) / G::TPF * G::TPF;
            sync.mask = ((1u << G::TPF) - 1u) << base;
        }
    }
};

// c2r of one spectrum row held in shared memory (entries h < hv, zero above)
// into registers, canonical layout: a[e] = (x[2n], x[2n+1]), n = t + TPF*e.
template <typename T, int N, int RX = 0>
__device__ __forceinline__ void c2r_row(const V2<T>* zr, int hv, RowCtx<T, N, RX>& rc,
                                        V2<T> (&a)[RowGeom<T, N, RX>::R])
{
    using G = RowGeom<T, N, RX>;
    using V = V2<T>;
    constexpr int NH = G::NH;
#pragma unroll
    for (int e = 0; e < G::RK; e++) {
        const int k = G::kp(rc.t, e);
        if (!G::kl(rc.t, e)) {
            a[e] = czero<V>();
            continue;
        }
        const V zk = k < hv ? zr[k] : czero<V>();
        const V zm = (NH - k) < hv ? cconj(zr[NH - k]) : czero<V>();
        const V A = cadd(zk, zm);
        const V B = cmul(csub(zk, zm), cconj(rc.twpp[k]));  // exp(+2 pi i k / N)
        a[e] = V{A.x - B.y, A.y + B.x};
    }
    rc.sync();  // the exchange buffer may be the row just read
    SmemRow<V> sm{rc.rowbuf};
    fft_geom<G, V, NH, true>(a, rc.t, sm, rc.twr, rc.sync);
    rc.sync();
}

// The same of a real spectrum row (quad layout: the transform of an even row).
template <typename T, int N, int RX = 0>
__device__ __forceinline__ void c2r_row_real(const T* zr, int hv, RowCtx<T, N, RX>& rc,
                                             V2<T> (&a)[RowGeom<T, N, RX>::R])
{
    using G = RowGeom<T, N, RX>;
    using V = V2<T>;
    constexpr int NH = G::NH;
#pragma unroll
    for (int e = 0; e < G::RK; e++) {
        const int k = G::kp(rc.t, e);
        if (!G::kl(rc.t, e)) {
            a[e] = czero<V>();
            continue;
        }
        const T zk = k < hv ? zr[k] : (T)0, zm = (NH - k) < hv ? zr[NH - k] : (T)0;
        const T A = zk + zm, D = zk - zm;
        const V w = rc.twpp[k];  // B = D conj(w)
        a[e] = V{A + D * w.y, D * w.x};
    }
    rc.sync();  // the exchange buffer may be the row just read
    SmemRow<V> sm{rc.rowbuf};
    fft_geom<G, V, NH, true>(a, rc.t, sm, rc.twr, rc.sync);
    rc.sync();
}

// r2c of a real row held in registers (canonical pairs), writing h < hout (REAL:
// the real parts only, for even rows).
template <typename T, int N, int RX = 0, bool REAL = false>
__device__ __forceinline__ void r2c_row(V2<T> (&a)[RowGeom<T, N, RX>::R], RowCtx<T, N, RX>& rc,
                                        std::conditional_t<REAL, T, V2<T>>* __restrict__ xo, int hout)
{
    using G = RowGeom<T, N, RX>;
    using V = V2<T>;
    constexpr int NH = G::NH;
    SmemRow<V> sm{rc.rowbuf};
    fft_geom<G, V, NH, false, true>(a, rc.t, sm, rc.twr, rc.sync);
    rc.sync();
#pragma unroll
    for (int e = 0; e < G::RK; e++)
        if (G::kl(rc.t, e)) sm.st(G::kp(rc.t, e), a[e]);
    rc.sync();
    const T half = (T)0.5;
    // column k from elements k and NH - k; column NH (element 0 twice) by thread 0
#pragma unroll
    for (int e = 0; e <= (NH + G::TPF - 1) / G::TPF; e++) {
        const int k = e * G::TPF >= NH ? NH : rc.t + e * G::TPF;
        if ((e * G::TPF >= NH && rc.t != 0) || (e * G::TPF < NH && k >= NH) || k >= hout) continue;
        const V yk = sm.ld(k == NH ? 0 : k);
        const V ym = cconj(sm.ld(k == 0 ? 0 : NH - k));
        const V E = V{(yk.x + ym.x) * half, (yk.y + ym.y) * half};
        const V D = csub(yk, ym);
        const V O = V{D.y * half, -D.x * half};  // D / (2i)
        const V X = cadd(E, cmul(rc.twpp[k], O));
        if constexpr (REAL) xo[k] = X.x;
        else xo[k] = X;
    }
    // the partner lane of an odd last column: the complex passes mix lanes that are not real and even
    if (REAL && (hout & 1) && rc.t == 0) reinterpret_cast<T*>(xo)[hout] = (T)0;
    rc.sync();
}

// ------------------------------------------------------------------ inverse Z (c2r)
enum RealEpi : int {
    EPI_STORE = 0,      // out = x^p
    EPI_MUL_STORE = 1,  // out = x^p * aux   (aux may alias out)
    EPI_MUL_REDUCE = 2, // sum x^p * aux
    EPI_REDUCE = 3,     // sum x^p
    EPI_MUL_REDUCE_ABS = 4,  // sum |x^p * aux|  (condition numbers)
    EPI_REDUCE_ABS = 5,      // sum |x^p|
    EPI_SCALE = 6            // out = scale * x, the product in FP64
};

template <typename T> __device__ __forceinline__ T ipow(T x, int p)
{
    T r = x;
    for (int q = 1; q < p; q++) r *= x;
    return r;
}

// Persistent: CTA b handles tiles b, b + gridDim.x, ...; the next tile's rows
// are copied into the other stage buffer while the current one is computed.
template <typename T, int N>
__global__ void __launch_bounds__(RowGeom<T, N>::THREADS)
    k_inv_z(const V2<T>* __restrict__ src, int src_stride, int hvalid, T* out, const T* aux,
            int epi, int power, double scale, double* __restrict__ partials, const V2<T>* __restrict__ twr_g,
            const V2<T>* __restrict__ twpp_g)
{
    using G = RowGeom<T, N>;
    using V = V2<T>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double red[(G::THREADS + 31) / 32];
    RowCtx<T, N> rc(smem_raw, twr_g, twpp_g);
    const int P = G::pitch(hvalid);
    V* stage = reinterpret_cast<V*>(smem_raw + G::STAGE_OFF);
    const int ntiles = N * N / G::WZ;
    int tile = blockIdx.x;
    if (tile < ntiles) stage_rows<V, G::WZ, G::THREADS>(stage, P, src, (size_t)tile * G::WZ, src_stride, hvalid);
    cp_async_commit();
    double acc = 0.0;
    for (int st = 0; tile < ntiles; tile += gridDim.x, st ^= 1) {
        const int next = tile + gridDim.x;
        if (next < ntiles)
            stage_rows<V, G::WZ, G::THREADS>(stage + (st ^ 1) * G::WZ * P, P, src, (size_t)next * G::WZ,
                                             src_stride, hvalid);
        cp_async_commit();
        cp_async_wait_prev();
        __syncthreads();
        const size_t row = (size_t)tile * G::WZ + rc.w;
        V a[G::R];
        c2r_row<T, N>(stage + st * G::WZ * P + rc.w * P, hvalid, rc, a);
        T* orow = out ? out + row * N : nullptr;
        const T* arow = aux ? aux + row * N : nullptr;
#pragma unroll
        for (int e = 0; e < G::RT; e++) {
            if (!G::tl(rc.t, e)) continue;
            const int n2 = 2 * (G::tp(rc.t, e));
            T x0 = ipow(a[e].x, power), x1 = ipow(a[e].y, power);
            if (epi == EPI_STORE) {
                *reinterpret_cast<V*>(orow + n2) = V{x0, x1};
            } else if (epi == EPI_SCALE) {
                *reinterpret_cast<V*>(orow + n2) = V{(T)(scale * (double)x0), (T)(scale * (double)x1)};
            } else if (epi == EPI_MUL_STORE) {
                const V q = *reinterpret_cast<const V*>(arow + n2);
                *reinterpret_cast<V*>(orow + n2) = V{x0 * q.x, x1 * q.y};
            } else if (epi == EPI_MUL_REDUCE) {
                const V q = *reinterpret_cast<const V*>(arow + n2);
                acc += (double)x0 * (double)q.x + (double)x1 * (double)q.y;
            } else if (epi == EPI_MUL_REDUCE_ABS) {
                const V q = *reinterpret_cast<const V*>(arow + n2);
                acc += fabs((double)x0 * (double)q.x) + fabs((double)x1 * (double)q.y);
            } else if (epi == EPI_REDUCE_ABS) {
                acc += fabs((double)x0) + fabs((double)x1);
            } else {
                acc += (double)x0 + (double)x1;
            }
        }
        __syncthreads();  // stage st is refilled two tiles later
    }
    if (epi >= EPI_MUL_REDUCE && epi != EPI_SCALE) {
        const double s = block_sum<G::THREADS>(acc, red);
        if (threadIdx.x == 0) partials[blockIdx.x] = s;
    }
}

// ------------------------------------------------------------------ forward Z (r2c)
enum RealSrcKind : int {
    SRC_F32 = 0,       // a
    SRC_F64 = 1,       // a
    SRC_XHI_F32 = 2,   // (double)a * (1 - (double)b), input_field.c:33
    SRC_XHI_F64 = 3,
    SRC_T = 4          // array of the transform's own type
};

template <typename T>
__device__ __forceinline__ T load_real(int kind, const void* a, const void* b, size_t idx)
{
    switch (kind) {
    case SRC_F32:
        return (T)((const float*)a)[idx];
    case SRC_F64:
        return (T)((const double*)a)[idx];
    case SRC_XHI_F32: {
        const double d = (double)((const float*)a)[idx], x = (double)((const float*)b)[idx];
        return (T)__dmul_rn(d, __dsub_rn(1.0, x));
    }
    case SRC_XHI_F64: {
        const double d = ((const double*)a)[idx], x = ((const double*)b)[idx];
        return (T)__dmul_rn(d, __dsub_rn(1.0, x));
    }
    default:
        return ((const T*)a)[idx];
    }
}

// Real values 2n and 2n+1 of a row (ra, and rb for XHI_DENS), composed as
// load_real does, with one vector load per array.
template <typename T>
__device__ __forceinline__ V2<T> load_pair(int kind, const unsigned char* ra, const unsigned char* rb, int n)
{
    switch (kind) {
    case SRC_F32: {
        const float2 v = reinterpret_cast<const float2*>(ra)[n];
        return V2<T>{(T)v.x, (T)v.y};
    }
    case SRC_F64: {
        const double2 v = reinterpret_cast<const double2*>(ra)[n];
        return V2<T>{(T)v.x, (T)v.y};
    }
    case SRC_XHI_F32: {
        const float2 d = reinterpret_cast<const float2*>(ra)[n], x = reinterpret_cast<const float2*>(rb)[n];
        return V2<T>{(T)__dmul_rn((double)d.x, __dsub_rn(1.0, (double)x.x)),
                     (T)__dmul_rn((double)d.y, __dsub_rn(1.0, (double)x.y))};
    }
    default: {  // SRC_XHI_F64
        const double2 d = reinterpret_cast<const double2*>(ra)[n], x = reinterpret_cast<const double2*>(rb)[n];
        return V2<T>{(T)__dmul_rn(d.x, __dsub_rn(1.0, x.x)), (T)__dmul_rn(d.y, __dsub_rn(1.0, x.y))};
    }
    }
}

// One tile of WZ consecutive rows per CTA.  Two ways to bring the rows in:
//  * STAGED: the tile's input bytes (contiguous: WZ rows of N values per input
//    array) are copied to shared memory by cp.async (16-byte, L2-only) and the
//    loader reads its value pairs from there, so no register holds a load in
//    flight; the exchange buffers of the rows then take the stage's place, and FP32
//    rows of 512 run five 256-thread CTAs per SM.  Needs 16-byte aligned inputs of 4- or 8-byte values.
//    With BULK the tile arrives by one bulk copy per input array
//    (cp.async.bulk through the TMA engine, completion counted on an mbarrier)
//    instead of one 16-byte cp.async per thread and chunk.  The wait on the
//    mbarrier is bounded (kBulkWaitNs of the global timer): past the limit the
//    kernel sets *status to 1, waits once more (bounded) for the copies and
//    returns without writing.  tx_extra > 0 (fault injection in tests) makes
//    the barrier expect more bytes than the copies bring, so the wait runs out.
//  * direct: all loads issued up front into registers (`vec`: one vector load
//    per value pair); FP32 rows of 512 are held to 32 registers so that eight
//    CTAs (every warp slot of the SM) keep their loads in flight.
constexpr unsigned long long kBulkWaitNs = 200000000ull;  // 0.2 s before a bulk copy counts as lost

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ bool mbar_try_wait_parity(unsigned bar, unsigned parity)
{
    unsigned done;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(done)
                 : "r"(bar), "r"(parity)
                 : "memory");
    return done != 0u;
}

template <typename T, int N, bool STAGED, bool BULK = false>
__global__ void __launch_bounds__(RowGeom<T, N>::THREADS,
                                  (sizeof(T) == 4 && N == 512) ? (STAGED ? 5 : 8) : 1)
    k_fwd_z(int kind, const void* __restrict__ a_src, const void* __restrict__ b_src,
            V2<T>* __restrict__ dst, int dst_stride, int hout, int vec, const V2<T>* __restrict__ twr_g,
            const V2<T>* __restrict__ twpp_g, int* __restrict__ status = nullptr, int tx_extra = 0)
{
    using G = RowGeom<T, N>;
    using V = V2<T>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int w0 = threadIdx.x / G::TPF, t0 = threadIdx.x % G::TPF;
    const size_t row = (size_t)blockIdx.x * G::WZ + w0;
    V a[G::R];
    if constexpr (STAGED) {
        const int eb = (kind == SRC_F32 || kind == SRC_XHI_F32) ? 4 : 8;
        const size_t tile_bytes = (size_t)G::WZ * N * eb;
        unsigned char* sa = smem_raw + G::ROWBUF_OFF;  // the exchange buffers take its place later
        unsigned char* sb = sa + tile_bytes;
        const unsigned char* ga = reinterpret_cast<const unsigned char*>(a_src) + (size_t)blockIdx.x * tile_bytes;
        const unsigned char* gb =
            b_src ? reinterpret_cast<const unsigned char*>(b_src) + (size_t)blockIdx.x * tile_bytes : nullptr;
        __shared__ __align__(8) unsigned long long bar;  // BULK: completion of the tile's copies
        const unsigned bar_s = (unsigned)__cvta_generic_to_shared(&bar);
        if constexpr (BULK) {
            if (threadIdx.x == 0) {
                asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar_s) : "memory");
                asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            }
            __syncthreads();
            if (threadIdx.x == 0) {
                const unsigned bytes = (unsigned)tile_bytes, total = bytes * (gb ? 2u : 1u) + (unsigned)tx_extra;
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar_s), "r"(total)
                             : "memory");
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                             ::"r"((unsigned)__cvta_generic_to_shared(sa)), "l"(ga), "r"(bytes), "r"(bar_s)
                             : "memory");
                if (gb)
                    asm volatile(
                        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                        ::"r"((unsigned)__cvta_generic_to_shared(sb)), "l"(gb), "r"(bytes), "r"(bar_s)
                        : "memory");
            }
        } else {
            for (size_t c = threadIdx.x; c < tile_bytes / 16; c += G::THREADS) {
                cp_async16(sa + 16 * c, ga + 16 * c);
                if (gb) cp_async16(sb + 16 * c, gb + 16 * c);
            }
            cp_async_commit();
        }
        RowCtx<T, N> rc(smem_raw, twr_g, twpp_g);  // tables staged while the copies fly
        if constexpr (BULK) {
            bool arrived = mbar_try_wait_parity(bar_s, 0u);
            for (const unsigned long long t0 = global_ns(); !arrived && global_ns() - t0 < kBulkWaitNs;)
                arrived = mbar_try_wait_parity(bar_s, 0u);
            if (!__syncthreads_and(arrived)) {  // the copy never completed: report, wait once more, leave
                if (threadIdx.x == 0 && status) atomicExch(status, 1);
                for (const unsigned long long t0 = global_ns(); !arrived && global_ns() - t0 < kBulkWaitNs;)
                    arrived = mbar_try_wait_parity(bar_s, 0u);
                return;
            }
        } else {
            cp_async_wait_all();
        }
        __syncthreads();
        const unsigned char* ra = sa + (size_t)w0 * N * eb;
        const unsigned char* rb = gb ? sb + (size_t)w0 * N * eb : nullptr;
#pragma unroll
        for (int e = 0; e < G::RT; e++)
            a[e] = G::tl(t0, e) ? load_pair<T>(kind, ra, rb, G::tp(t0, e)) : czero<V>();
        __syncthreads();  // every row is in registers
        r2c_row<T, N>(a, rc, dst + row * dst_stride, hout);
    } else {
        if (kind == SRC_T) {
            const V* xr = reinterpret_cast<const V*>((const T*)a_src + row * N);
#pragma unroll
            for (int e = 0; e < G::RT; e++) a[e] = G::tl(t0, e) ? xr[G::tp(t0, e)] : czero<V>();
        } else if (vec) {
            // both values of a pair in one 8- or 16-byte load per array
            const int eb = (kind == SRC_F32 || kind == SRC_XHI_F32) ? 4 : 8;
            const unsigned char* ra = reinterpret_cast<const unsigned char*>(a_src) + row * N * eb;
            const unsigned char* rb = b_src ? reinterpret_cast<const unsigned char*>(b_src) + row * N * eb : nullptr;
#pragma unroll
            for (int e = 0; e < G::RT; e++)
                a[e] = G::tl(t0, e) ? load_pair<T>(kind, ra, rb, G::tp(t0, e)) : czero<V>();
        } else {
#pragma unroll
            for (int e = 0; e < G::RT; e++) {
                const size_t n2 = row * N + 2 * (G::tp(t0, e));
                a[e] = G::tl(t0, e)
                           ? V{load_real<T>(kind, a_src, b_src, n2), load_real<T>(kind, a_src, b_src, n2 + 1)}
                           : czero<V>();
            }
        }
        RowCtx<T, N> rc(smem_raw, twr_g, twpp_g);
        __syncthreads();
        r2c_row<T, N>(a, rc, dst + row * dst_stride, hout);
    }
}

// ------------------------------------------------------------------ pair Z
// One (i,j) row of the product of two band-limited inverse transforms,
// transformed forward again: c2r(A) * c2r(B) -> r2c, all along l, so the real
// product D_a*D_b (or D_a^2 when B is NULL) never leaves the SM.  Output rows
// keep h < hout.  Persistent and double-buffered like k_inv_z.
//   RX   : elements per thread of the row transforms (0: RowRadix's choice)
//   KEEP : c2r(A)'s values wait in shared memory (each thread its own slots,
//          no synchronisation) while c2r(B) runs, so one row transform is
//          live in registers at a time instead of two
template <typename T, int N, int RX, bool KEEP> struct PairGeom {
    using G = RowGeom<T, N, RX>;
    // dynamic shared memory: the row kernels' layout, then the keep buffers
    __host__ __device__ static constexpr size_t smem(int ninputs, int hva, int hvb, bool alias = false)
    {
        const int pa = G::pitch(hva);
        return (alias ? G::ROWBUF_OFF + (size_t)2 * G::WZ * ((pa > G::ROWBUF ? pa : G::ROWBUF) + (ninputs > 1 ? G::pitch(hvb) : 0)) * sizeof(V2<T>)
                      : G::smem(ninputs, hva, hvb)) +
               (KEEP ? (size_t)G::WZ * G::ROWBUF * sizeof(V2<T>) : 0);
    }
    static constexpr bool FITS = smem(2, N / 2 + 1, N / 2 + 1) <= 227 * 1024;
};

// Pair kernel variants the plan autotuner times per FP32 transform size of
// register-plan rows from 128 to 512 points: 0 the default, 1 KEEP (one row
// transform live in registers), 2 KEEP with twice the default elements per
// thread (one radix pass fewer, half the threads per row).  KEEP_OK /
// ALT_RX (0: none) say which exist for a length.
template <typename T, int N> struct PairVariants {
    static constexpr bool REG = sizeof(T) == 4 && !LenKind<N / 2>::SPLIT && N >= 128 && N <= 512;
    static constexpr int RX2 = 2 * RowGeom<T, N>::R;
    static constexpr bool KEEP_OK = REG && PairGeom<T, N, 0, true>::FITS;
    static constexpr int ALT_RX = REG && (N / 2) % RX2 == 0 && (N / 2) / RX2 >= 4 ? RX2 : 0;
};

//   REAL : rows of the quad layout (real spectra, two columns per element;
//          hva, hvb, hout count columns)
//   TWO  : two legs (else A squared: no second row in registers)
// alias: the exchange buffer of a row is its current stage buffer of A, whose pitch
// is then at least ROWBUF (full-band legs: a third less shared memory per row).
template <typename T, int N, int RX = 0, bool KEEP = false, bool REAL = false, bool TWO = true>
__global__ void __launch_bounds__(RowGeom<T, N, RX>::THREADS, sizeof(T) == 8 ? 0 : !TWO && N <= 512 ? 3 : LenKind<N / 2>::SPLIT ? 2 : 0)
    k_pair_z(const __grid_constant__ Items<PairItem<T>> items, int nrows, int alias,
             const V2<T>* __restrict__ twr_g, const V2<T>* __restrict__ twpp_g)
{
    using G = RowGeom<T, N, RX>;
    using V = V2<T>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const PairItem<T>& it = items.at[blockIdx.y];
    const V* __restrict__ srcA = it.A;
    const V* __restrict__ srcB = it.B;
    V* __restrict__ dst = it.dst;
    const int sa = it.sa, sb = it.sb, ds = it.ds, hout = it.hout;
    RowCtx<T, N, RX> rc(smem_raw, twr_g, twpp_g);
    // elements of a staged row
    const int hva = REAL ? (it.hva + 1) / 2 : it.hva, hvb = REAL ? (it.hvb + 1) / 2 : it.hvb;
    auto c2r = [&](const V* z, int hv, V(&x)[G::R]) {
        if constexpr (REAL) c2r_row_real<T, N, RX>(reinterpret_cast<const T*>(z), hv, rc, x);
        else c2r_row<T, N, RX>(z, hv, rc, x);
    };
    constexpr bool two = TWO;
    const int PA = alias ? max(G::pitch(hva), G::ROWBUF) : G::pitch(hva), PB = two ? G::pitch(hvb) : 0;
    V* stA = reinterpret_cast<V*>(smem_raw + (alias ? G::ROWBUF_OFF : G::STAGE_OFF));
    V* stB = stA + 2 * G::WZ * PA;
    V* keep = stB + 2 * G::WZ * PB + rc.w * G::ROWBUF;  // KEEP: this row's slots
    const int ntiles = (nrows + G::WZ - 1) / G::WZ;
    int tile = blockIdx.x;
    if (tile < ntiles) {
        stage_rows<V, G::WZ, G::THREADS>(stA, PA, srcA, (size_t)tile * G::WZ, sa, hva, nrows);
        if (two) stage_rows<V, G::WZ, G::THREADS>(stB, PB, srcB, (size_t)tile * G::WZ, sb, hvb, nrows);
    }
    cp_async_commit();
    for (int st = 0; tile < ntiles; tile += gridDim.x, st ^= 1) {
        const int next = tile + gridDim.x;
        if (next < ntiles) {
            stage_rows<V, G::WZ, G::THREADS>(stA + (st ^ 1) * G::WZ * PA, PA, srcA, (size_t)next * G::WZ, sa, hva,
                                             nrows);
            if (two)
                stage_rows<V, G::WZ, G::THREADS>(stB + (st ^ 1) * G::WZ * PB, PB, srcB, (size_t)next * G::WZ, sb,
                                                 hvb, nrows);
        }
        cp_async_commit();
        cp_async_wait_prev();
        __syncthreads();
        const size_t row = (size_t)tile * G::WZ + rc.w;
        // A row group past the quadrant's last row idles; every thread reaches the one
        // barrier below (rows of a warp on different barriers is what the hardware's
        // CTA barrier does not allow).  The N^2 rows of a full grid are whole tiles.
        static_assert(REAL || N * N % G::WZ == 0, "whole tiles");
        if (!REAL || row < (size_t)nrows) {
            if (alias) rc.rowbuf = stA + st * G::WZ * PA + rc.w * PA;
            V a[G::R];
            c2r(stA + st * G::WZ * PA + rc.w * PA, it.hva, a);
            if constexpr (two) {
                if constexpr (KEEP) {
#pragma unroll
                    for (int e = 0; e < G::RT; e++)
                        if (G::tl(rc.t, e)) keep[G::tp(rc.t, e)] = a[e];
                    c2r(stB + st * G::WZ * PB + rc.w * PB, it.hvb, a);
#pragma unroll
                    for (int e = 0; e < G::RT; e++) {
                        const V q = G::tl(rc.t, e) ? keep[G::tp(rc.t, e)] : czero<V>();
                        a[e] = V{a[e].x * q.x, a[e].y * q.y};
                    }
                } else {
                    V b[G::R];
                    c2r(stB + st * G::WZ * PB + rc.w * PB, it.hvb, b);
#pragma unroll
                    for (int e = 0; e < G::RT; e++) a[e] = V{a[e].x * b[e].x, a[e].y * b[e].y};
                }
            } else {
#pragma unroll
                for (int e = 0; e < G::RT; e++) a[e] = V{a[e].x * a[e].x, a[e].y * a[e].y};
            }
            // the products sit in canonical layout as (x[2n], x[2n+1]): r2c input as is
            if constexpr (REAL) r2c_row<T, N, RX, true>(a, rc, reinterpret_cast<T*>(dst + row * ds), hout);
            else r2c_row<T, N, RX>(a, rc, dst + row * ds, hout);
        }
        __syncthreads();  // this stage is refilled two tiles later
    }
}

// ------------------------------------------------------------------ products of n fields
// Grid sums of prod_f x_f^p_f over the rows of up to kMaxFactors inverse
// transforms: every row's factors are brought back to real space one after the
// other and multiplied in registers, so no real field is stored or read (three
// legs as separate passes moved 6 N^3 values beside the spectra).  Persistent and
// double-buffered over the (row tile, factor) sequence.  REAL: quad rows, weighted
// by the points each stands for.
constexpr int kMaxFactors = 8;
template <typename T> struct ProdItem {
    const V2<T>* src[kMaxFactors];
    int stride[kMaxFactors];
    short hv[kMaxFactors];     // columns
    short power[kMaxFactors];
    int nf;
    double* partials;          // one per block
};
template <typename T, int N, bool REAL>
__global__ void __launch_bounds__(RowGeom<T, N>::THREADS)
    k_prod_z(const __grid_constant__ Items<ProdItem<T>> items, int P, int alias, int abs_terms, const V2<T>* __restrict__ twr_g,
             const V2<T>* __restrict__ twpp_g)
{
    using G = RowGeom<T, N>;
    using V = V2<T>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double red[(G::THREADS + 31) / 32];
    const ProdItem<T>& it = item_at(items);
    RowCtx<T, N> rc(smem_raw, twr_g, twpp_g);
    V* stage = reinterpret_cast<V*>(smem_raw + (alias ? G::ROWBUF_OFF : G::STAGE_OFF));  // two tiles of pitch P
    constexpr int NQ = N / 2 + 1;
    constexpr int nrows = REAL ? NQ * NQ : N * N, ntiles = (nrows + G::WZ - 1) / G::WZ;
    const int nf = it.nf;
    auto fetch = [&](int tile, int f, int buf) {
        if (tile < ntiles)
            stage_rows<V, G::WZ, G::THREADS>(stage + buf * G::WZ * P, P, it.src[f], (size_t)tile * G::WZ, it.stride[f],
                                             REAL ? (it.hv[f] + 1) / 2 : it.hv[f], nrows);
        cp_async_commit();
    };
    int buf = 0;
    fetch(blockIdx.x, 0, 0);
    double acc = 0.0;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int row = tile * G::WZ + rc.w;
        const bool live = row < nrows;
        V prod[G::R];
        for (int f = 0; f < nf; f++, buf ^= 1) {
            const bool last = f + 1 == nf;
            fetch(last ? tile + gridDim.x : tile, last ? 0 : f + 1, buf ^ 1);
            cp_async_wait_prev();
            __syncthreads();
            if (live) {  // whole row groups
                V a[G::R];
                V* z = stage + buf * G::WZ * P + rc.w * P;
                if (alias) rc.rowbuf = z;  // the row's own stage buffer is its exchange buffer
                if constexpr (REAL) c2r_row_real<T, N>(reinterpret_cast<const T*>(z), it.hv[f], rc, a);
                else c2r_row<T, N>(z, it.hv[f], rc, a);
                const int p = it.power[f];
                if (p == 2) {  // one branch for the row, not a loop per element
#pragma unroll
                    for (int e = 0; e < G::RT; e++) a[e] = V{a[e].x * a[e].x, a[e].y * a[e].y};
                } else if (p == 3) {
#pragma unroll
                    for (int e = 0; e < G::RT; e++) a[e] = V{a[e].x * a[e].x * a[e].x, a[e].y * a[e].y * a[e].y};
                } else if (p > 3 && sizeof(T) == 8) {
#pragma unroll
                    for (int e = 0; e < G::RT; e++) a[e] = V{ipow(a[e].x, p), ipow(a[e].y, p)};
                } else if (p > 3) {
                    // the last factor's power in two halves, whose product the sum takes in
                    // double: the eighth power of 6e4 is above FP32's range
                    const int q = last ? p - p / 2 : p;
#pragma unroll
                    for (int e = 0; e < G::RT; e++) {
                        if (last) {
                            const V h{ipow(a[e].x, p / 2), ipow(a[e].y, p / 2)};
                            prod[e] = f == 0 ? h : V{prod[e].x * h.x, prod[e].y * h.y};
                        }
                        a[e] = V{ipow(a[e].x, q), ipow(a[e].y, q)};
                    }
                }
                const bool alone = f == 0 && (sizeof(T) == 8 || p <= 3);
                double s = 0.0;
#pragma unroll
                for (int e = 0; e < G::RT; e++) {
                    const T x0 = a[e].x, x1 = a[e].y;
                    if (!last) {
                        prod[e] = f == 0 ? V{x0, x1} : V{prod[e].x * x0, prod[e].y * x1};
                    } else if (G::tl(rc.t, e)) {
                        const double y0 = alone ? (double)x0 : (double)prod[e].x * (double)x0;
                        const double y1 = alone ? (double)x1 : (double)prod[e].y * (double)x1;
                        s += abs_terms ? fabs(y0) + fabs(y1) : y0 + y1;
                    }
                }
                if (last) {
                    if constexpr (REAL) {
                        const int i = row / NQ, j = row - i * NQ;
                        s *= (double)((i == 0 || i == N / 2 ? 1 : 2) * (j == 0 || j == N / 2 ? 1 : 2));
                    }
                    acc += s;
                }
            }
            __syncthreads();  // this buffer is refilled by the next fetch but one
        }
    }
    const double total = block_sum<G::THREADS>(acc, red);
    if (threadIdx.x == 0) it.partials[blockIdx.x] = total;
}

// ------------------------------------------------------------------ forward X
enum SpecEpi : int {
    SPEC_STORE = 0,        // out = X
    SPEC_STORE_PHASE = 1,  // out = X / |X|  (utils_fftw.c:78-93)
    SPEC_DOT = 2,          // per shell c: sum_m w(h) F_c(m) Re(dk(m) conj(X(m)))
    SPEC_COUNT = 3,        // per shell c: sum_m w(h) F_c(m) rint(Re X(m) / N^3)
    SPEC_MASK_ADD = 4,     // out += weight * F(m) X(m) where F selects (adjoint); out is of an ndk-grid
    SPEC_DOT_ABS = 5       // as SPEC_DOT with |term| (condition numbers)
};

// KIND: FWD_SUMS for the per-shell sum epilogues (SPEC_DOT, SPEC_COUNT,
// SPEC_DOT_ABS), FWD_STORE for SPEC_STORE and SPEC_STORE_PHASE, FWD_MASK for
// SPEC_MASK_ADD; separate instantiations so that no pass is sized for another's
// registers (with the masked sum in it the storing pass at 512 points spills
// 128 bytes per thread at its two CTAs per SM, without it none).
// r2max (sums only): no shell of the launch holds a mode with |m|^2 > r2max,
// so a tile of pencils whose (my, mz) lie outside that ball is skipped.
// FP32 sums up to 384 points run two CTAs per SM (64 registers, a few bytes
// of spill: the 384-point pass 0.149 against 0.165 ms at one CTA per SM).
// RX > 0 (FP32 dot passes, autotuned): the alternative pencil geometry of
// PencilAlt, twice the elements per thread and one radix pass fewer.
enum FwdKind : int { FWD_STORE = 0, FWD_SUMS = 1, FWD_MASK = 2 };
template <typename T, int N, int KIND, int RX>
using FwdXGeom = std::conditional_t<KIND == FWD_STORE, typename StoreXGeom<T, N, RX>::type, PencilGeom<T, N, RX>>;
template <typename T, int N, int KIND, int RX = 0>
__global__ void __launch_bounds__(FwdXGeom<T, N, KIND, RX>::THREADS,
                                  KIND == FWD_SUMS ? (((sizeof(T) == 4 && N <= 384) || PencilGeom<T, N, RX>::THREADS <= 256) ? 2 : 1)
                                      : (sizeof(T) == 8 || FwdXGeom<T, N, KIND, RX>::THREADS > 512 ? 1 : 2))
    k_fwd_x(const __grid_constant__ std::conditional_t<KIND == FWD_SUMS, Items<FwdXItem<T>>, FwdXItem<T>> items, int epi,
            V2<T>* out, int out_stride, const V2<T>* __restrict__ dk, int dk_stride, int ndk, int quad_arg, const V2<T>* __restrict__ tw_g,
            T* __restrict__ mod_out, int jband)
{
    using G = FwdXGeom<T, N, KIND, RX>;
    using V = V2<T>;
    constexpr bool DOT = KIND == FWD_SUMS;
    const int quad = DOT && sizeof(T) == 8 ? quad_arg : 0;  // FP64 counts only
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const FwdXItem<T>& it = item_at(items);
    V* data = it.data;
    const int stride = it.stride, hvalid = it.hvalid, ncols = it.ncols, r2max = it.r2max;
    // blocks of this item: blockIdx.x < nblk
    const int nblk = (quad ? N / 2 + 1 : N) * (ncols / G::W);
    if ((int)blockIdx.x >= nblk) return;
    const int w = threadIdx.x % G::W, t = threadIdx.x / G::W;
    // pencils of columns h < ncols (rows of stride `stride`); storing passes
    // with jband < N/2 (a band-limited field spectrum) skip the tiles whose
    // |my| exceeds it and write only modes with |mx| <= jband
    const int tiles_per_row = ncols / G::W;
    // quad (counts only): pencils j <= N/2 of data even in x and y stored
    // [i <= N/2][j <= N/2][h]; plane N-i read as plane i; interior j weigh 2;
    // column element h holds columns 2h (real part) and 2h + 1 (imaginary part)
    const int nj = quad ? N / 2 + 1 : N;
    const int j = blockIdx.x / tiles_per_row;
    const int h = (blockIdx.x % tiles_per_row) * G::W + w;
    const bool packed = DOT && sizeof(T) == 8 && quad;
    const int hz = packed ? 2 * h : h;
    const bool col_ok = hz < hvalid && hz <= N / 2;
    const int my = lattice_freq(j, N);
    const int mz = hz == N / 2 ? -(N / 2) : hz;
    if constexpr (!DOT) {
        if (jband < N / 2 && abs(my) > jband) return;  // rows outside the field's band
    }
    const bool use_dk = epi == SPEC_DOT || epi == SPEC_DOT_ABS;
    const size_t jdk = (size_t)(my < 0 ? my + ndk : my);
    V* sdk = reinterpret_cast<V*>(smem_raw + G::SMEM);
    if constexpr (DOT) {
        // the whole tile outside every shell: no transform, zero partials
        const bool live = col_ok && my * my + mz * mz <= r2max;
        if (!__syncthreads_or(live)) {
            if ((int)threadIdx.x < it.nshell) it.partials[(size_t)threadIdx.x * nblk + blockIdx.x] = 0.0;
            return;
        }
        if constexpr (G::DK_SMEM) {
            // field-spectrum pencils of the tile (128 bytes per x row, rows
            // that can hold a shell mode only) copied while the transform runs
            if (use_dk) {
                constexpr int EPC = 16 / (int)sizeof(V), CPR = G::W / EPC;
                const int h0 = (blockIdx.x % tiles_per_row) * G::W;
                const long long rest = (long long)r2max - (long long)my * my - (long long)h0 * h0;
                for (int c = threadIdx.x; c < N * CPR; c += G::THREADS) {
                    const int i = c / CPR, q = c - i * CPR;
                    const int mx = lattice_freq(i, N);
                    if ((long long)mx * mx <= rest)
                        cp_async16(sdk + i * G::W + q * EPC,
                                   dk + ((size_t)(mx < 0 ? mx + ndk : mx) * ndk + jdk) * dk_stride + h0 + q * EPC);
                }
            }
            cp_async_commit();
        }
    }
    V a[G::R];
#pragma unroll
    for (int e = 0; e < G::RI; e++) {
        const int i = G::ip(t, e);
        a[e] = G::il(t, e) ? data[((size_t)(quad && i > N / 2 ? N - i : i) * nj + j) * stride + h] : czero<V>();
    }
    // sums: the shell bits depend on indices only and are found before the
    // transform (16 bits per mode, two modes per register)
    unsigned bits2[(G::RO + 1) / 2];
    [[maybe_unused]] unsigned bits2b[(G::RO + 1) / 2];  // packed: of the odd column
    if constexpr (DOT) {
#pragma unroll
        for (int e = 0; e < (G::RO + 1) / 2; e++) bits2[e] = bits2b[e] = 0u;
        const auto each = [&](auto&& bits_of) {  // bits_of(mx) of every mode of this thread
#pragma unroll
            for (int e = 0; e < G::RO; e++) {
                if (col_ok && G::ol(t, e))
                    bits2[e / 2] |= (bits_of(lattice_freq(G::op(t, e), N)) & 0xffffu) << (16 * (e & 1));
            }
        };
        const int s2 = my * my + mz * mz;
        if (it.interval) {  // one or two r2 intervals
            const int lo0 = it.shells[0].r2lo, hi0 = it.shells[0].r2hi;
            each([&](int mx) { return (unsigned)(mx * mx + s2 >= lo0 && mx * mx + s2 <= hi0); });
            if (it.nshell > 1) {
                const int lo1 = it.shells[1].r2lo, hi1 = it.shells[1].r2hi;
                each([&](int mx) { return mx * mx + s2 >= lo1 && mx * mx + s2 <= hi1 ? 2u : 0u; });
            }
        } else if (it.lut) {
            const unsigned short* __restrict__ lut = it.lut;
            const int lut_size = it.lut_size;
            each([&](int mx) { return mx * mx + s2 < lut_size ? (unsigned)__ldg(lut + mx * mx + s2) : 0u; });
        } else if (it.vol) {
            const int vb = it.vol_band, ay = abs(my);
            const unsigned short* __restrict__ vol = it.vol + (size_t)ay * (vb + 1) + abs(mz);
            const size_t step = (size_t)(vb + 1) * (vb + 1);
            const bool in = ay <= vb && abs(mz) <= vb;
            each([&](int mx) { return in && abs(mx) <= vb ? (unsigned)__ldg(vol + abs(mx) * step) : 0u; });
        } else {
            each([&](int mx) { return shell_bits(it.shells, it.nshell, mx, my, mz); });
        }
        if constexpr (sizeof(T) == 8) {
            if (packed && hz + 1 < hvalid && hz + 1 <= N / 2) {
                const int mzb = hz + 1 == N / 2 ? -(N / 2) : hz + 1;
                const unsigned short* __restrict__ lut = it.lut;
                const int s2b = my * my + mzb * mzb;
#pragma unroll
                for (int e = 0; e < G::RO; e++) {
                    if (!G::ol(t, e)) continue;
                    const int mx = lattice_freq(G::op(t, e), N), r2 = mx * mx + s2b;
                    const int vb = it.vol_band;
                    unsigned bb = 0u;
                    if (lut) bb = r2 < it.lut_size ? (unsigned)__ldg(lut + r2) : 0u;
                    else if (!it.vol) bb = shell_bits(it.shells, it.nshell, mx, my, mzb);
                    else if (abs(mx) <= vb && abs(my) <= vb && abs(mzb) <= vb)
                        bb = __ldg(it.vol + ((size_t)abs(mx) * (vb + 1) + abs(my)) * (vb + 1) + abs(mzb));
                    bits2b[e / 2] |= (bb & 0xffffu) << (16 * (e & 1));
                }
            }
        }
    }
    const V* tw = stage_table<V>(smem_raw, tw_g, N);
    __syncthreads();
    SmemInterleaved<V, G::W> sm{reinterpret_cast<V*>(smem_raw + G::TW_BYTES), w};
    fft_geom<G, V, N, false>(a, t, sm, tw, BlockSync{});
    if constexpr (!DOT) {
        unsigned keep = 0u;
        if constexpr (KIND == FWD_MASK) {
            const Shell sh = it.shells[0];
            if (col_ok) {
#pragma unroll 1
                for (int e = 0; e < G::RO; e++) {
                    if (!G::ol(t, e)) continue;
                    const int mx = lattice_freq(G::op(t, e), N);
                    if (in_band(sh, mx, my, mz) && shell_bit(sh, mx, my, mz)) keep |= 1u << e;
                }
            }
        }
        if (h >= out_stride) return;
#pragma unroll
        for (int e = 0; e < G::RO; e++) {
            const int i = G::op(t, e);
            if (!G::ol(t, e)) continue;
            if (jband < N / 2 && abs(lattice_freq(i, N)) > jband) continue;
            V v = a[e];
            if constexpr (KIND == FWD_MASK) {
                if (!((keep >> e) & 1u)) continue;
                // mode m of this grid sits at m mod ndk of the accumulated spectrum
                const int mx = lattice_freq(i, N);
                V* o = out + ((size_t)(mx < 0 ? mx + ndk : mx) * ndk + jdk) * out_stride + h;
                const V prev = *o;
                *o = V{prev.x + (T)it.weight * v.x, prev.y + (T)it.weight * v.y};
                continue;
            }
            if (epi == SPEC_STORE_PHASE) {
                // mod_out (optional) keeps |X| for the phase-only adjoint
                T m;
                if constexpr (sizeof(T) == 8) {
                    m = hypot(v.x, v.y);
                    v = V{v.x / m, v.y / m};
                } else {
                    // FP32 spectra: one reciprocal square root when |v|^2 is a
                    // normal float, the overflow-safe quotient otherwise (a zero
                    // mode stays 0/0 = NaN, as utils_fftw.c:89 gives)
                    const float m2 = v.x * v.x + v.y * v.y;
                    if (m2 >= 1.17549435e-38f && m2 <= 3.40282347e38f) {
                        const float r = rsqrtf(m2);
                        v = V{v.x * r, v.y * r};
                        m = m2 * r;
                    } else {
                        m = hypotf(v.x, v.y);
                        v = V{v.x / m, v.y / m};
                    }
                }
                if (mod_out) mod_out[((size_t)i * N + j) * out_stride + h] = m;
            }
            out[((size_t)i * N + j) * out_stride + h] = v;
        }
    } else {
        // dk: field spectrum of an ndk-grid ([ndk][ndk][dk_stride], ndk >= N);
        // mode m of this grid sits at index m mod ndk there (shells lie below N/2).
        // Per-shell FP64 sums in registers, then one fixed-order reduction for
        // all shells at once (deterministic): warp xor-trees, per-warp rows in
        // shared memory, one thread per shell sums the rows in warp order.
        if constexpr (G::DK_SMEM) {
            cp_async_wait_all();
            __syncthreads();
        }
        // DOT sums carry `weight` (the (N_field / N)^3 of a sub-grid product spectrum)
        const double wgt =
            (double)(herm_weight(hz, N) * (quad && j != 0 && j != N / 2 ? 2 : 1)) * (use_dk ? it.weight : 1.0);
        const double inv_n3 = 1.0 / ((double)N * (double)N * (double)N);
        // the 16 shells in two halves of 8 (8 FP64 accumulators live at a
        // time; a mode's term is formed once per half it has shells in).
        // Warp sums of a half by recursive halving: at lane offset o each lane
        // keeps half of its shells (the upper half when lane & o) and adds the
        // partner's copy of that half, so after offsets 16, 8, 4 lane l holds
        // shell c(l) = 4 b4 + 2 b3 + b2 of the half (b_k the lane bits), summed
        // over 8 lanes; offsets 2 and 1 complete it.
        static_assert(MAX_DOT_SHELLS == 16, "two halving trees of 8 shells");
        constexpr int NW = G::THREADS / 32;
        __shared__ double wsum[NW][MAX_DOT_SHELLS];
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
        for (int half = 0; half < 2; half++) {
            double acc[8];
#pragma unroll
            for (int c = 0; c < 8; c++) acc[c] = 0.0;
#pragma unroll
            for (int e = 0; e < G::RO; e++) {
                const unsigned b = (bits2[e / 2] >> (16 * (e & 1) + 8 * half)) & 0xffu;
                if (b) {
                    double val;
                    if (use_dk) {
                        V d;
                        if constexpr (G::DK_SMEM) {
                            d = sdk[G::op(t, e) * G::W + w];
                        } else {
                            const int mx = lattice_freq(G::op(t, e), N);
                            d = dk[((size_t)(mx < 0 ? mx + ndk : mx) * ndk + jdk) * dk_stride + h];
                        }
                        val = wgt * ((double)d.x * (double)a[e].x + (double)d.y * (double)a[e].y);
                    } else {
                        val = wgt * rint((double)a[e].x * inv_n3);
                    }
                    if (epi == SPEC_DOT_ABS) val = fabs(val);
#pragma unroll
                    for (int c = 0; c < 8; c++)
                        if ((b >> c) & 1u) acc[c] += val;
                }
            }
            if constexpr (sizeof(T) == 8) {
                if (packed) {
                    const double wgtb = (double)(herm_weight(hz + 1, N) * (j != 0 && j != N / 2 ? 2 : 1));
#pragma unroll
                    for (int e = 0; e < G::RO; e++) {
                        const unsigned b = (bits2b[e / 2] >> (16 * (e & 1) + 8 * half)) & 0xffu;
                        if (b) {
                            const double val = wgtb * rint((double)a[e].y * inv_n3);
#pragma unroll
                            for (int c = 0; c < 8; c++)
                                if ((b >> c) & 1u) acc[c] += val;
                        }
                    }
                }
            }
            halve_sums<8, 16>(acc, lane);
            halve_sums<4, 8>(acc, lane);
            halve_sums<2, 4>(acc, lane);
            acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 2);
            acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 1);
            if ((lane & 3) == 0) wsum[wid][8 * half + ((lane >> 2) & 7)] = acc[0];
        }
        __syncthreads();
        if ((int)threadIdx.x < it.nshell) {
            double sum = 0.0;
#pragma unroll 1
            for (int q = 0; q < NW; q++) sum += wsum[q][threadIdx.x];
            it.partials[(size_t)threadIdx.x * nblk + blockIdx.x] = sum;
        }
    }
}

// Shell bitmask per r2 value (shells of the DEFAULT / RANGE kinds); blockIdx.y
// picks the table.
struct LutItem {
    const Shell* shells;
    unsigned short* lut;
    int ns, size;
};
static __global__ void k_shell_lut(const __grid_constant__ Items<LutItem> items)
{
    const LutItem& it = items.at[blockIdx.y];
    const int r2 = blockIdx.x * blockDim.x + threadIdx.x;
    if (r2 >= it.size) return;
    unsigned bits = 0u;
    for (int c = 0; c < it.ns; c++) bits |= (unsigned)(r2 >= it.shells[c].r2lo && r2 <= it.shells[c].r2hi) << c;
    it.lut[r2] = (unsigned short)bits;
}

// The same for shells that are no r2 intervals (WATKINSON): every predicate is even
// in each axis, so the bitmask of the octant 0 <= x, y, z <= band serves all modes.
// Made once per plan; evaluating 12 shells for every mode in the dot passes took
// 0.085 of the 0.101 ms (FP32) and most of the 0.119 ms (FP64) at 128 points.
static __global__ void __launch_bounds__(256)
    k_shell_volume(const Shell* __restrict__ shells, int ns, int band, unsigned short* __restrict__ vol)
{
    const int side = band + 1;
    const long long total = (long long)side * side * side;
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < total; q += (long long)gridDim.x * blockDim.x) {
        const int z = (int)(q % side), y = (int)(q / side % side), x = (int)(q / side / side);
        vol[q] = (unsigned short)shell_bits(shells, ns, x, y, z);
    }
}

// ------------------------------------------------------------------ adjoint helpers
// Mode q of the cube |components| <= band of an n-grid's half spectrum (stride S):
// its index, or false for +n/2 (the index of -n/2, visited as such).
__device__ __forceinline__ bool cube_index(size_t q, int n, int band, int S, size_t& idx)
{
    const int side = 2 * band + 1, hb = band + 1;
    const int h = (int)(q % hb);
    const int my = (int)(q / hb % side) - band, mx = (int)(q / hb / side) - band;
    if (mx >= n / 2 || my >= n / 2) return false;
    idx = ((size_t)(mx < 0 ? mx + n : mx) * n + (my < 0 ? my + n : my)) * S + h;
    return true;
}
// n = 2: dB/d(delta) needs L_a D_b + L_b D_a = IFFT[F_a FFT[D_b] + F_b FFT[D_a]]
// with FFT[D] = N^3 F dk (the inverse transform is unnormalised), i.e.
// IFFT[2 N^3 F_a F_b dk]; this writes that spectrum on the cube |components| <= band.
template <typename T>
__global__ void k_grad_pair2(int n, const V2<T>* __restrict__ dk, int dks, const Shell* __restrict__ shells,
                             V2<T>* __restrict__ hacc, int S, int band)
{
    const size_t total = (size_t)(2 * band + 1) * (2 * band + 1) * (band + 1);
    for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < total; q += (size_t)gridDim.x * blockDim.x) {
        size_t idx;
        if (!cube_index(q, n, band, S, idx)) continue;
        const int h = (int)(q % (band + 1));
        const int my = (int)(q / (band + 1) % (2 * band + 1)) - band, mx = (int)(q / (band + 1) / (2 * band + 1)) - band;
        const int mz = h == n / 2 ? -(n / 2) : h;
        V2<T> v = czero<V2<T>>();
        if (in_band(shells[0], mx, my, mz) && shell_bit(shells[0], mx, my, mz) && in_band(shells[1], mx, my, mz) &&
            shell_bit(shells[1], mx, my, mz)) {
            const V2<T> d = dk[idx / S * dks + h];
            const T f = (T)(2.0 * (double)n * (double)n * (double)n);
            v = V2<T>{f * d.x, f * d.y};
        }
        hacc[idx] = v;
    }
}

// Phase-only adjoint: the field enters through phi = z/|z| per mode, whose
// differential is (dz - phi Re(conj(phi) dz)) / |z|; its transpose maps the
// accumulated gradient spectrum H to (H - phi Re(conj(phi) H)) / |z| (in
// place, on the cube |components| <= band).  Modes with H = 0 stay 0.
template <typename T>
__global__ void k_phase_adjoint(int n, int band, V2<T>* __restrict__ hacc, int S, const V2<T>* __restrict__ phi,
                                const T* __restrict__ mod)
{
    const size_t total = (size_t)(2 * band + 1) * (2 * band + 1) * (band + 1);
    for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < total; q += (size_t)gridDim.x * blockDim.x) {
        size_t idx;
        if (!cube_index(q, n, band, S, idx)) continue;
        const V2<T> H = hacc[idx];
        if (H.x == (T)0 && H.y == (T)0) continue;
        const V2<T> u = phi[idx];
        const T m = mod[idx];
        const T p = u.x * H.x + u.y * H.y;  // Re(conj(phi) H)
        hacc[idx] = V2<T>{(H.x - u.x * p) / m, (H.y - u.y * p) / m};
    }
}
template <typename T> __global__ void k_zero_cube(int n, int band, V2<T>* __restrict__ hacc, int S)
{
    const size_t total = (size_t)(2 * band + 1) * (2 * band + 1) * (band + 1);
    for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < total; q += (size_t)gridDim.x * blockDim.x) {
        size_t idx;
        if (cube_index(q, n, band, S, idx)) hacc[idx] = czero<V2<T>>();
    }
}

// out[x] = scale * in[x], converted to the output type.
template <typename T, typename O>
__global__ void k_scale_out(const T* __restrict__ in, O* __restrict__ out, size_t count, double scale)
{
    for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < count; q += (size_t)gridDim.x * blockDim.x)
        out[q] = (O)(scale * (double)in[q]);
}

// ------------------------------------------------------------------ n = 2 (Parseval)
// Per configuration c (legs a, b): S_D = N^3 sum_half w(h) F_a F_b |dk|^2 and
// the count sum_half w(h) F_a F_b (exact), over the band cube |m| <= band.
// For shells that are no r^2 intervals (those take k_pair2_sweep): the per-mode
// configuration bitmask comes from the shell pairs legs[2c], legs[2c+1].
// Per-thread FP64 sums, one fixed-order reduction: partials[c] (sums) and
// partials[MAX + c] (counts).
template <typename T>
__global__ void __launch_bounds__(256)
    k_pair2_sums(int n, const V2<T>* __restrict__ dk, int dks, const Shell* __restrict__ legs, int ncfg, int band,
                 double* __restrict__ partials)
{
    double acc[MAX_DOT_SHELLS], cnt[MAX_DOT_SHELLS];
#pragma unroll
    for (int c = 0; c < MAX_DOT_SHELLS; c++) acc[c] = cnt[c] = 0.0;
    const int b = min(band, n / 2);
    const int side = 2 * b + 1;
    const long long total = (long long)side * side * (b + 1);
    const double n3 = (double)n * (double)n * (double)n;
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < total;
         q += (long long)gridDim.x * blockDim.x) {
        const int h = (int)(q % (b + 1));
        const long long r = q / (b + 1);
        const int mx = (int)(r / side) - b, my = (int)(r % side) - b;
        if (mx >= n / 2 || my >= n / 2) continue;  // +N/2 is the index of -N/2, visited as such
        const int mz = h == n / 2 ? -(n / 2) : h;
        unsigned bits = 0u;
        for (int c = 0; c < ncfg; c++) {
            const Shell& sa = legs[2 * c];
            const Shell& sb = legs[2 * c + 1];
            if (in_band(sa, mx, my, mz) && shell_bit(sa, mx, my, mz) && in_band(sb, mx, my, mz) &&
                shell_bit(sb, mx, my, mz))
                bits |= 1u << c;
        }
        if (!bits) continue;
        const int i = mx < 0 ? mx + n : mx, j = my < 0 ? my + n : my;
        const V2<T> d = dk[((size_t)i * n + j) * dks + h];
        const double wgt = (double)herm_weight(h, n);
        const double val = wgt * n3 * ((double)d.x * (double)d.x + (double)d.y * (double)d.y);
#pragma unroll
        for (int c = 0; c < MAX_DOT_SHELLS; c++)
            if ((bits >> c) & 1u) {
                acc[c] += val;
                cnt[c] += wgt;
            }
    }
    __shared__ double wsum[8][2 * MAX_DOT_SHELLS];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int c = 0; c < MAX_DOT_SHELLS; c++) {
        double v = acc[c], u = cnt[c];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            v += __shfl_xor_sync(0xffffffffu, v, o);
            u += __shfl_xor_sync(0xffffffffu, u, o);
        }
        if (lane == c) {
            wsum[wid][c] = v;
            wsum[wid][MAX_DOT_SHELLS + c] = u;
        }
    }
    __syncthreads();
    if (threadIdx.x < 2 * MAX_DOT_SHELLS) {
        double sum = 0.0;
#pragma unroll 1
        for (int q = 0; q < 8; q++) sum += wsum[q][threadIdx.x];
        partials[(size_t)threadIdx.x * gridDim.x + blockIdx.x] = sum;
    }
}

// dst[idx[q]] = src[q]
static __global__ void k_scatter(const double* __restrict__ src, const int* __restrict__ idx, int count,
                                 double* __restrict__ dst)
{
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q < count) dst[idx[q]] = src[q];
}

// ------------------------------------------------------------------ final sums
// out[c] = sum_b partials[c*nblocks + b], fixed order (one CTA per column).
// Column c of the partial sums, summed in a fixed order, lands in
// out[c * out_stride], or in out[idx[c]] (the configuration it belongs to).
static __global__ void k_sum_partials(const double* __restrict__ partials, int nblocks, double* out,
                                      int out_stride, const int* __restrict__ idx)
{
    __shared__ double red[32];
    const double* p = partials + (size_t)blockIdx.x * nblocks;
    double s = 0.0;
    for (int b = threadIdx.x; b < nblocks; b += blockDim.x) s += p[b];
    s = block_sum<1024>(s, red);
    if (threadIdx.x == 0) out[idx ? (size_t)idx[blockIdx.x] : (size_t)blockIdx.x * out_stride] = s;
}

// Column blockIdx.x of item blockIdx.y of a list of partial sums, in a fixed
// order: one launch for all pair groups of a plan.  (Summed by the last block of
// each dot pass instead, the 384-point pass took 0.203 against 0.145 + 0.008 ms:
// every block then waits for a fence and an atomic before it leaves its SM.)
struct SumItem {
    const double* partials;  // [ncol][nblk]
    int nblk, ncol;
    double scale;
    double* out;             // column c lands at out[idx[c]], or out[c] (idx NULL)
    const int* idx;
};
static __global__ void __launch_bounds__(256) k_sum_items(const __grid_constant__ Items<SumItem> items)
{
    const SumItem& it = item_at(items);
    const int c = blockIdx.x;
    if (c >= it.ncol) return;
    __shared__ double red[8];
    const double* p = it.partials + (size_t)c * it.nblk;
    double s = 0.0;
    for (int b = threadIdx.x; b < it.nblk; b += 256) s += p[b];
    s = block_sum<256>(s, red);
    if (threadIdx.x == 0) it.out[it.idx ? it.idx[c] : c] = it.scale * s;
}

// ------------------------------------------------------------------ DERIVED k-range
// min/max of squared corner radii over the DEFAULT-filter modes of a shell
// (construct_kfilter_with_determining_kbinwidth, filter.c:78-114).  The
// reference folds the running min/max through sqrt and back per voxel; for
// binary64 sqrt(fl(s*s)) = s, so that equals sqrt of the global min/max of the
// squared corners whatever the visiting order.  Non-negative doubles order
// like their bit patterns, so the fold is an integer atomicMin/atomicMax.
__device__ __forceinline__ int isqrt_floor(int v)  // floor(sqrt(v)), v >= 0
{
    int r = (int)sqrt((double)v);
    while (r * r > v) r--;
    while ((r + 1) * (r + 1) <= v) r++;
    return r;
}

// DERIVED range of one shell: min/max of the squared corner radii over its
// modes with |mz| <= hmax, folded into minmax_bits[0..1] (bit patterns of
// non-negative doubles order as integers).  The grid's x extent strides the
// shell's modes.
__device__ __forceinline__ void derived_range_body(int n, const Shell& sh, int hmax, unsigned long long* minmax_bits);

static __global__ void k_derived_range(int n, const Shell* __restrict__ shell_p, int hmax,
                                       unsigned long long* minmax_bits)
{
    derived_range_body(n, *shell_p, hmax, minmax_bits);
}

// nd shells in one launch: blockIdx.y selects the shell (hmax = its band, at
// most n/2); blocks past what a shell needs find no mode and fold nothing.
static __global__ void k_derived_ranges(int n, const Shell* __restrict__ shells, unsigned long long* minmax_bits)
{
    const Shell sh = shells[blockIdx.y];
    derived_range_body(n, sh, min(sh.band, n / 2), minmax_bits + 2 * blockIdx.y);
}

__device__ __forceinline__ void derived_range_body(int n, const Shell& sh, int hmax, unsigned long long* minmax_bits)
{
    const int band = min(sh.band, n / 2);
    const int side = 2 * band + 1;
    double min2 = sh.min2_init, max2 = 0.0;
    if (sh.kind == SHELL_DEFAULT || sh.kind == SHELL_RANGE) {
        // interval shells: one thread per (mx, my) column, mz over the exact
        // range r2lo <= mx^2 + my^2 + mz^2 <= r2hi (mz >= 0: the corner radii
        // of (mx, my, -mz) are those of (mx, my, mz))
        for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < side * side; q += gridDim.x * blockDim.x) {
            const int mx = q / side - band, my = q % side - band;
            if (mx >= n / 2 || my >= n / 2 || mx < -(n / 2) || my < -(n / 2)) continue;
            const int s = mx * mx + my * my;
            if (sh.r2hi < 0 || s > sh.r2hi) continue;
            int z0 = 0;
            if (sh.r2lo - s > 0) {
                z0 = isqrt_floor(sh.r2lo - s);
                if (z0 * z0 < sh.r2lo - s) z0++;
            }
            const int z1 = min(isqrt_floor(sh.r2hi - s), hmax);
            for (int hz = z0; hz <= z1; hz++)
                corners_fold(mx, my, hz == n / 2 ? -(n / 2) : hz, sh.half, min2, max2);
        }
    } else {
        const long long total = (long long)side * side * (hmax + 1);
        for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < total;
             q += (long long)gridDim.x * blockDim.x) {
            const int hz = (int)(q % (hmax + 1));
            const long long r = q / (hmax + 1);
            const int mx = (int)(r / side) - band, my = (int)(r % side) - band;
            if (mx >= n / 2 || my >= n / 2 || mx < -(n / 2) || my < -(n / 2)) continue;
            const int mz = hz == n / 2 ? -(n / 2) : hz;
            if (shell_bit(sh, mx, my, mz)) corners_fold(mx, my, mz, sh.half, min2, max2);
        }
    }
    // min2/max2 are non-negative (or the +huge start value)
    unsigned long long lo = __double_as_longlong(min2), hi = __double_as_longlong(max2);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = min(lo, __shfl_down_sync(0xffffffffu, lo, o));
        hi = max(hi, __shfl_down_sync(0xffffffffu, hi, o));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMin(&minmax_bits[0], lo);
        atomicMax(&minmax_bits[1], hi);
    }
}

}  // namespace ps
