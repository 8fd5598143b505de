// In-CTA Stockham FFT of length N with R elements per thread.
//
// A transform of length N is done by TPF = N/R threads.  Thread t holds
// a[e] = x[t + TPF*e] ("canonical layout") on entry and X[t + TPF*e] on exit.
// N is a power of two, or 3 or 5 times one, for the register passes below; the
// other lengths 2^a 3^b 5^c are two passes of unequal radices (SplitPlan).  Passes are
// radix-R (for N = f 2^k, R = f 2^r: radix-2^r passes, one of a smaller power
// of two if needed, then one radix-R pass last); each thread does R/Rp
// butterflies per pass.  Pass p with radix Rp and span Ns (product of the
// previous radices) computes, for butterfly v in [0, N/Rp):
//     b_q = x[v + q*N/Rp] * W_{Ns*Rp}^{q*(v mod Ns)},  b = DFT_Rp(b),
//     y[(v/Ns)*Ns*Rp + (v mod Ns) + q*Ns] = b_q
// (the Stockham auto-sort form), so no bit reversal is ever needed and the
// last pass writes its outputs back into the registers it read, already in
// canonical layout.  Between passes the data goes through shared memory
// through an accessor (interleaved [pos][lane] for pencil passes, or one row
// per transform for the contiguous axis).
#pragma once

#include "ps_common.cuh"

namespace ps {

// cos(2 pi j / 32), j = 0..31: constants of the in-register butterflies.
__device__ __forceinline__ constexpr double cos32(int j)
{
    constexpr double c[8] = {1.0,
                             0.98078528040323044913,
                             0.92387953251128675613,
                             0.83146961230254523708,
                             0.70710678118654752440,
                             0.55557023301960222474,
                             0.38268343236508977173,
                             0.19509032201612826785};
    j &= 31;
    if (j <= 8) return j == 8 ? 0.0 : c[j];
    if (j <= 16) return -cos32(16 - j);
    return cos32(32 - j);
}

// cos(2 pi p / q) for integers p, q > 0, evaluated at compile time: the angle
// is folded into [0, pi/4] by the exact symmetries of cos and sin on the
// rational p/q, then summed as a Taylor series (13 terms; the remainder is
// below 1e-24 there).  For the radix-3 / radix-5 constants, whose angles are
// not multiples of pi/16.
__host__ __device__ constexpr double taylor_cos(double t)
{
    double term = 1.0, sum = 1.0;
    for (int i = 1; i <= 13; i++) {
        term *= -t * t / ((2.0 * i - 1.0) * (2.0 * i));
        sum += term;
    }
    return sum;
}
__host__ __device__ constexpr double taylor_sin(double t)
{
    double term = t, sum = t;
    for (int i = 1; i <= 13; i++) {
        term *= -t * t / ((2.0 * i) * (2.0 * i + 1.0));
        sum += term;
    }
    return sum;
}
__host__ __device__ constexpr double cos_2pi(long long p, long long q)
{
    p %= q;
    if (p < 0) p += q;
    if (2 * p > q) p = q - p;                                  // cos(2pi(1-x)) = cos(2pi x)
    if (4 * p > q) return -cos_2pi(q - 2 * p, 2 * q);          // x > 1/4: -cos(2pi(1/2-x))
    if (8 * p > q) return taylor_sin(6.283185307179586477 * (double)(q - 4 * p) / (double)(4 * q));
    return taylor_cos(6.283185307179586477 * (double)p / (double)q);
}
__host__ __device__ constexpr double sin_2pi(long long p, long long q) { return cos_2pi(q - 4 * p, 4 * q); }

// W_R^k for the forward (e^{-}) or inverse (e^{+}) direction, applied to v.
template <int R, int K, bool INV, typename V> __device__ __forceinline__ V twiddle_const(V v)
{
    if constexpr (K == 0) {
        return v;
    } else if constexpr (4 * K == R) {
        return mul_mi<INV>(v);
    } else if constexpr (32 % R != 0) {
        using T = decltype(v.x);
        constexpr double cd = cos_2pi(K, R), sd = sin_2pi(K, R);
        const T c = (T)cd;
        const T s = INV ? (T)sd : (T)-sd;
        return V{v.x * c - v.y * s, v.x * s + v.y * c};
    } else {
        using T = decltype(v.x);
        constexpr int j = K * (32 / R);
        const T c = (T)cos32(j);
        const T s = INV ? (T)cos32(j - 8) : (T)-cos32(j - 8);  // sin(2 pi j/32) = cos(2 pi (j-8)/32)
        return V{v.x * c - v.y * s, v.x * s + v.y * c};
    }
}

// Decimation-in-frequency DFT of length R in registers, natural order in and
// out: even R splits into two halves, R = 3 and 5 are direct butterflies, 15 and 25
// go through columns of five.
template <int R, bool INV> struct Dft {
    static_assert(R % 2 == 0 || R == 15 || R == 25, "odd DFT lengths other than 3, 5, 15 and 25 are not provided");
    // R = P Q odd: x[Q i + j] -> P-point DFTs over i, twiddles W_R^{j k}, Q-point
    // DFTs over j, output P l + k
    template <int J, int K, typename V> static __device__ __forceinline__ void twist(V* y)
    {
        constexpr int P = R / 5;
        if constexpr (K < P) {
            y[K] = twiddle_const<R, (J * K) % R, INV>(y[K]);
            twist<J, K + 1>(y);
        }
    }
    template <int J, typename V> static __device__ __forceinline__ void columns(const V* a, V (&y)[5][R / 5])
    {
        constexpr int P = R / 5;
        if constexpr (J < 5) {
#pragma unroll
            for (int i = 0; i < P; i++) y[J][i] = a[5 * i + J];
            Dft<P, INV>::run(y[J]);
            twist<J, 0>(y[J]);
            columns<J + 1>(a, y);
        }
    }
    template <typename V> static __device__ __forceinline__ void run(V* a)
    {
        if constexpr (R % 2 != 0) {
            constexpr int P = R / 5;
            V y[5][P];
            columns<0>(a, y);
#pragma unroll
            for (int k = 0; k < P; k++) {
                V z[5];
#pragma unroll
                for (int j = 0; j < 5; j++) z[j] = y[j][k];
                Dft<5, INV>::run(z);
#pragma unroll
                for (int l = 0; l < 5; l++) a[P * l + k] = z[l];
            }
        } else {
            halves(a);
        }
    }
    template <typename V> static __device__ __forceinline__ void halves(V* a)
    {
        constexpr int H = R / 2;
        V b[H], c[H];
        apply<0>(a, b, c);
        Dft<H, INV>::run(b);
        Dft<H, INV>::run(c);
#pragma unroll
        for (int k = 0; k < H; k++) {
            a[2 * k] = b[k];
            a[2 * k + 1] = c[k];
        }
    }
    template <int K, typename V> static __device__ __forceinline__ void apply(const V* a, V* b, V* c)
    {
        if constexpr (K < R / 2) {
            b[K] = cadd(a[K], a[K + R / 2]);
            c[K] = twiddle_const<R, K, INV>(csub(a[K], a[K + R / 2]));
            apply<K + 1>(a, b, c);
        }
    }
};
template <bool INV> struct Dft<1, INV> {
    template <typename V> static __device__ __forceinline__ void run(V*) {}
};
// y_k = sum_n a_n W_3^{nk}: y0 = a0 + s, y1,2 = a0 - s/2 -/+ i sin(2pi/3) d
// (forward), s = a1 + a2, d = a1 - a2; the inverse swaps the +/- i terms.
template <bool INV> struct Dft<3, INV> {
    template <typename V> static __device__ __forceinline__ void run(V* a)
    {
        using T = decltype(a[0].x);
        constexpr T s3 = (T)sin_2pi(1, 3);
        const V s = cadd(a[1], a[2]), d = csub(a[1], a[2]);
        const V t = V{a[0].x - (T)0.5 * s.x, a[0].y - (T)0.5 * s.y};
        const V u = V{-s3 * d.y, s3 * d.x};  // i sin(2pi/3) d
        a[0] = cadd(a[0], s);
        a[1] = INV ? cadd(t, u) : csub(t, u);
        a[2] = INV ? csub(t, u) : cadd(t, u);
    }
};
// Length 5: with t1 = a1 + a4, t2 = a2 + a3, d1 = a1 - a4, d2 = a2 - a3,
// y0 = a0 + t1 + t2, y1,4 = a0 + c1 t1 + c2 t2 -/+ i (s1 d1 + s2 d2),
// y2,3 = a0 + c2 t1 + c1 t2 -/+ i (s2 d1 - s1 d2) (forward signs),
// c_j = cos(2pi j/5), s_j = sin(2pi j/5).
template <bool INV> struct Dft<5, INV> {
    template <typename V> static __device__ __forceinline__ void run(V* a)
    {
        using T = decltype(a[0].x);
        constexpr T c1 = (T)cos_2pi(1, 5), c2 = (T)cos_2pi(2, 5);
        constexpr T s1 = (T)sin_2pi(1, 5), s2 = (T)sin_2pi(2, 5);
        const V t1 = cadd(a[1], a[4]), t2 = cadd(a[2], a[3]);
        const V d1 = csub(a[1], a[4]), d2 = csub(a[2], a[3]);
        const V r1 = V{a[0].x + c1 * t1.x + c2 * t2.x, a[0].y + c1 * t1.y + c2 * t2.y};
        const V r2 = V{a[0].x + c2 * t1.x + c1 * t2.x, a[0].y + c2 * t1.y + c1 * t2.y};
        const V p1 = V{s1 * d1.x + s2 * d2.x, s1 * d1.y + s2 * d2.y};
        const V p2 = V{s2 * d1.x - s1 * d2.x, s2 * d1.y - s1 * d2.y};
        const V i1 = V{-p1.y, p1.x}, i2 = V{-p2.y, p2.x};  // i p
        a[0] = cadd(a[0], cadd(t1, t2));
        a[1] = INV ? cadd(r1, i1) : csub(r1, i1);
        a[4] = INV ? csub(r1, i1) : cadd(r1, i1);
        a[2] = INV ? cadd(r2, i2) : csub(r2, i2);
        a[3] = INV ? csub(r2, i2) : cadd(r2, i2);
    }
};

// Radix plan.  R = f 2^r with f in {1, 3, 5} the odd part of N: passes of
// radix 2^r while possible, then one pass of the power-of-two remainder; for
// f > 1 these cover N / R and one radix-R pass (it carries the odd factor)
// comes last.  Every radix divides R.  With the odd pass last, every pass
// that goes through shared memory has a power-of-two radix and span, which
// the row layout (SmemRow) makes conflict-free.
template <int N, int R> struct RadixPlan {
    __host__ __device__ static constexpr int odd_of(int n) { return n % 2 ? n : odd_of(n / 2); }
    static constexpr int F = odd_of(R);
    static constexpr int R2 = R / F;                  // radix of the power-of-two passes
    static constexpr int TAIL = F > 1 ? 1 : 0;        // the radix-R pass of a mixed length
    static constexpr int N2 = N / (F > 1 ? R : 1);    // what the power-of-two passes cover
    __host__ __device__ static constexpr int count_full(int n) { return n >= R2 ? 1 + count_full(n / R2) : 0; }
    __host__ __device__ static constexpr int rem_of(int n) { return n >= R2 ? rem_of(n / R2) : n; }
    static constexpr int FULL = count_full(N2);
    static constexpr int REM = rem_of(N2);  // 1 if N2 is a power of R2
    static constexpr int NREM = REM > 1 ? 1 : 0;
    static constexpr int P = FULL + NREM + TAIL;
    __host__ __device__ static constexpr int radix(int p)
    {
        return p < FULL ? R2 : (p < FULL + NREM ? REM : R);
    }
    __host__ __device__ static constexpr int span(int p)
    {
        int s = 1;
        for (int q = 0; q < p; q++) s *= radix(q);
        return s;
    }
    // offset of pass p's twiddles in the Stockham table (entries [k][q-1],
    // k < span(p), q in [1, radix(p))); the table has N - 1 entries in all
    __host__ __device__ static constexpr int tw_off(int p)
    {
        int o = 0;
        for (int q = 0; q < p; q++) o += span(q) * (radix(q) - 1);
        return o;
    }
    static_assert(F == 1 || F == 3 || F == 5, "radix must be 2^r, 3*2^r or 5*2^r");
    static_assert(R2 >= 2 || F > 1, "power-of-two radix must be >= 2");
    static_assert(N % R == 0 && odd_of(N) == F, "length must be R times a power of two");
    static_assert(F == 1 || R2 >= 2 || N == R, "mixed lengths need a power-of-two part in R");
};

// Elements per thread used for each register-plan length (3 2^k and 5 2^k:
// the odd factor times 2 or 4, 4 to 32 threads per transform).
template <int N> struct DefaultRadix {
    static constexpr int value = N == 24 ? 6 : N == 40 ? 10 : N == 48 ? 12 : N == 80 ? 20 : N == 96 ? 12
                               : N == 160 ? 20 : N == 192 ? 12 : N == 320 ? 20 : N == 384 ? 12
                               : N <= 16 ? N : (N == 32 || N == 64 || N == 128 || N == 512) ? 8 : 16;
};

// Lengths whose odd part is not 1, 3 or 5, and those with a factor 3 or 5 whose
// register plan needs three or more passes: N = RA RB in two passes, the factors as
// equal as they come (the second at least the first), so that either pass is one
// butterfly per thread and one exchange through shared memory lies between them.
// Thread t does the butterflies v = t, t + TPF, ... of a pass: slot u R + q of its
// array holds element v + q N / R, v = t + TPF u; slots of v >= N / R are idle.  The
// layouts of input (pass A) and output (pass B) therefore differ, see SplitGeom.  A
// sequence of radix-8/4/2, 3 and 5 passes through shared memory (five exchanges at 600
// points) took 0.54 ms for a Y pass of 600^2 x 304 columns.  Against the register plans
// (160: 2 2 2 2 10, 192: 4 4 12, 320: 4 4 20, 384: 4 4 2 12): pair kernel at 320 points
// 0.170 -> 0.135 ms, at 384 points 0.224 -> 0.215 ms, inverse X pass at 384 points 0.048
// -> 0.041 ms, Y passes at 320 points 9% and at 384 points 10 to 14% faster.
template <int N> struct SplitPlan {
    static constexpr int RA = N == 30 ? 5 : N == 60 ? 6 : N == 96 ? 8 : N == 150 || N == 160 ? 10 : N == 192 ? 12
                            : N == 300 ? 15 : N == 320 || N == 384 ? 16 : N == 600 ? 24 : 0;
    static constexpr int RB = RA ? N / RA : 0;
    static constexpr bool value = RA > 0;
};
template <int N, int TPF> struct SplitGeom {
    static constexpr int RA = SplitPlan<N>::RA, RB = SplitPlan<N>::RB;
    static constexpr int BA = (RB + TPF - 1) / TPF, BB = (RA + TPF - 1) / TPF;  // butterflies per thread (N / RA = RB)
    static constexpr int RI = BA * RA, RO = BB * RB;                            // slots in, out
    __device__ static constexpr int ip(int t, int e) { return t + TPF * (e / RA) + (e % RA) * RB; }
    __device__ static constexpr bool il(int t, int e) { return t + TPF * (e / RA) < RB; }
    __device__ static constexpr int op(int t, int e) { return t + TPF * (e / RB) + (e % RB) * RA; }
    __device__ static constexpr bool ol(int t, int e) { return t + TPF * (e / RB) < RA; }
};

template <int L> struct LenKind {
    __host__ __device__ static constexpr int odd_of(int n) { return n % 2 ? n : odd_of(n / 2); }
    static constexpr bool SPLIT = SplitPlan<L>::value;
    static_assert(SPLIT || odd_of(L) == 1 || odd_of(L) == 3 || odd_of(L) == 5, "no plan for this length");
};

// Synchronisation between passes: the whole CTA (pencil kernels, whose
// transforms span several warps), or only the threads of one row (row
// kernels): __syncwarp when a row lives in one warp, else a named barrier per
// row (ids 1..15; id 0 is __syncthreads').
struct BlockSync {
    __device__ __forceinline__ void operator()() const { __syncthreads(); }
};
template <int TPF> struct RowSync {
    int bar;         // named barrier id (TPF > 32)
    unsigned mask;   // this row's lanes (TPF <= 32)
    __device__ __forceinline__ void operator()() const
    {
        if constexpr (TPF <= 32) __syncwarp(mask);
        else asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"(TPF) : "memory");
    }
};

// Stockham passes.  twt is the transform's twiddle table: for pass p, entry
// tw_off(p) + k*(Rp-1) + (q-1) = W_{Ns*Rp}^{q*k} (forward sign), so the lanes
// of a warp (consecutive k) read it with a stride of Rp-1 entries, which maps
// 8 (FP64) or 16 (FP32) consecutive lanes to distinct shared-memory banks.
template <typename V, int N, int R, bool INV, int P_ = 0, class Acc, class Sync>
__device__ __forceinline__ void fft_passes(V (&a)[R], int t, Acc& sm, const V* __restrict__ twt, const Sync& sync)
{
    using Plan = RadixPlan<N, R>;
    if constexpr (P_ < Plan::P) {
        constexpr int Rp = Plan::radix(P_);
        constexpr int Ns = Plan::span(P_);
        constexpr int BPT = R / Rp;
        constexpr int TPF = N / R;
        constexpr bool LAST = (P_ == Plan::P - 1);
#pragma unroll
        for (int u = 0; u < BPT; u++) {
            V b[Rp];
#pragma unroll
            for (int q = 0; q < Rp; q++) b[q] = a[u + q * BPT];
            const int v = t + TPF * u;
            const int k = v % Ns;
            if constexpr (Ns > 1) {
                const V* tp = twt + Plan::tw_off(P_) + k * (Rp - 1);
#pragma unroll
                for (int q = 1; q < Rp; q++) {
                    V w = tp[q - 1];
                    if constexpr (INV) w.y = -w.y;
                    b[q] = cmul(b[q], w);
                }
            }
            Dft<Rp, INV>::run(b);
            if constexpr (LAST) {
#pragma unroll
                for (int q = 0; q < Rp; q++) a[u + q * BPT] = b[q];
            } else {
                const int j = (v / Ns) * Ns * Rp + k;
#pragma unroll
                for (int q = 0; q < Rp; q++) sm.template st<Rp, Ns>(j, q * Ns, b[q]);
            }
        }
        if constexpr (!LAST) {
            sync();
#pragma unroll
            for (int e = 0; e < R; e++) a[e] = sm.template ld<Rp, Ns>(t, TPF * e);
            sync();
            fft_passes<V, N, R, INV, P_ + 1>(a, t, sm, twt, sync);
        }
    }
}

// The two passes of N = RA RB (see SplitPlan).  twt holds W_N^{k q}, k < A, q in
// [1, B), at k (B - 1) + q - 1 for the factors A <= B of SplitPlan; with SWAP the
// passes run as RB RA (RA, RB here being the swapped pair) on the same table.
template <typename V, int N, int RA, int RB, int TPF, bool INV, bool SWAP, int SLOTS, class Acc, class Sync>
__device__ __forceinline__ void split_passes(V (&a)[SLOTS], int t, Acc& sm, const V* __restrict__ twt, const Sync& sync)
{
    constexpr int BA = (RB + TPF - 1) / TPF, BB = (RA + TPF - 1) / TPF;
    static_assert(BA * RA <= SLOTS && BB * RB <= SLOTS && RA * RB == N, "slots");
#pragma unroll
    for (int u = 0; u < BA; u++) {
        const int v = t + TPF * u;
        if (v < RB) {
            Dft<RA, INV>::run(&a[u * RA]);
#pragma unroll
            for (int q = 0; q < RA; q++) sm.template st_split<RA, RB>(v, q, a[u * RA + q]);
        }
    }
    sync();
#pragma unroll
    for (int u = 0; u < BB; u++) {
        const int v = t + TPF * u;
        if (v < RA) {
#pragma unroll
            for (int q = 0; q < RB; q++) a[u * RB + q] = sm.template ld_split<RA, RB>(v, q);
        }
    }
    sync();
#pragma unroll
    for (int u = 0; u < BB; u++) {
        const int v = t + TPF * u;
        if (v < RA) {
#pragma unroll
            for (int q = 1; q < RB; q++) {
                V w;
                if constexpr (!SWAP) {
                    w = twt[v * (RB - 1) + q - 1];
                } else {  // entry (k = q, q = v), 1 for v = 0
                    w = v > 0 ? twt[q * (RA - 1) + v - 1] : V{1, 0};
                }
                if constexpr (INV) w.y = -w.y;
                a[u * RB + q] = cmul(a[u * RB + q], w);
            }
            Dft<RB, INV>::run(&a[u * RB]);
        }
    }
}

// A transform in the geometry G of a kernel (input layout G::ip, output G::op; SWAP:
// the other way round), register passes or split.
template <class G, typename V, int N, bool INV, bool SWAP = false, class Acc, class Sync>
__device__ __forceinline__ void fft_geom(V (&a)[G::R], int t, Acc& sm, const V* __restrict__ twt, const Sync& sync)
{
    if constexpr (!G::SPLIT) {
        fft_passes<V, N, G::R, INV>(a, t, sm, twt, sync);
    } else if constexpr (SWAP) {
        split_passes<V, N, SplitPlan<N>::RB, SplitPlan<N>::RA, G::TPF, INV, true>(a, t, sm, twt, sync);
    } else {
        split_passes<V, N, SplitPlan<N>::RA, SplitPlan<N>::RB, G::TPF, INV, false>(a, t, sm, twt, sync);
    }
}

// Host side: the Stockham table of a pass plan (forward sign), from
// exp(-2 pi i m / M) evaluated in long double.
template <typename V, class Plan> inline void plan_table(V* out)
{
    const long double two_pi = 6.283185307179586476925286766559005768L;
    for (int p = 0; p < Plan::P; p++) {
        const int Rp = Plan::radix(p), Ns = Plan::span(p);
        V* tp = out + Plan::tw_off(p);
        for (int k = 0; k < Ns; k++)
            for (int q = 1; q < Rp; q++) {
                const long double a = two_pi * (long double)(q * k) / (long double)(Ns * Rp);
                tp[k * (Rp - 1) + q - 1].x = (decltype(tp->x))cosl(a);
                tp[k * (Rp - 1) + q - 1].y = (decltype(tp->x))(-sinl(a));
            }
    }
}
// the table of the transform fft_geom runs in geometry G
template <typename V, int N, class G> inline void transform_table(V* out)
{
    if constexpr (!G::SPLIT) {
        plan_table<V, RadixPlan<N, G::R>>(out);
    } else {
        const long double two_pi = 6.283185307179586476925286766559005768L;
        constexpr int RA = SplitPlan<N>::RA, RB = SplitPlan<N>::RB;
        for (int k = 0; k < RA; k++)
            for (int q = 1; q < RB; q++) {
                const long double a = two_pi * (long double)(q * k) / (long double)N;
                out[k * (RB - 1) + q - 1].x = (decltype(out->x))cosl(a);
                out[k * (RB - 1) + q - 1].y = (decltype(out->x))(-sinl(a));
            }
    }
}

// Shared-memory accessor for pencil passes: W transforms interleaved, element
// `pos` of transform `lane` at s[pos*W + lane] (conflict-free when W*sizeof(V)
// = 128 bytes, the tile width of one global row segment).  In the exchange of the
// split passes butterfly v of the first stores its output q, and butterfly v of the
// second loads its input q.
template <typename V, int W> struct SmemInterleaved {
    V* s;
    int lane;
    template <int Rp, int Ns> __device__ __forceinline__ void st(int base, int off, V v) { s[(base + off) * W + lane] = v; }
    template <int Rp, int Ns> __device__ __forceinline__ V ld(int base, int off) const { return s[(base + off) * W + lane]; }
    template <int RA, int RB> __device__ __forceinline__ void st_split(int v, int q, V x) { s[(v * RA + q) * W + lane] = x; }
    template <int RA, int RB> __device__ __forceinline__ V ld_split(int v, int q) const { return s[(v + q * RA) * W + lane]; }
};

// Shared-memory accessor for row passes: one row per transform, padded per exchange
// so that no store of an instruction meets another on a bank and every address is a
// thread's base plus a constant (no arithmetic per element; an XOR swizzle took two
// instructions for each, a fifth of the row kernels').  Blocks are G elements (128
// bytes).
//  * Exchange after a pass of radix Rp and span Ns (powers of two): lane t stores at
//    (t/Ns)*Ns*Rp + t%Ns + q*Ns; block a is moved up by a*PAD elements.  When Ns*Rp <=
//    G the lanes that share an offset lie in Rp consecutive blocks and PAD = Ns moves
//    them apart; else they lie K = Ns*Rp/G blocks apart and PAD = Ns/K = G/Rp does.  From
//    Ns = G on the lanes are consecutive anyway.  The loads that follow (consecutive
//    positions, one block per G lanes) stay conflict-free.
//  * Split passes: output q of butterfly v at q * pitch + v, so both the stores
//    (consecutive v) and the loads (v of the second pass pitch apart, the pitch odd)
//    are conflict-free.
//  * r2c post-processing: consecutive positions both ways, no padding.
template <typename V> struct SmemRow {
    static constexpr int G = 128 / (int)sizeof(V);
    V* s;
    template <int Rp, int Ns> __host__ __device__ static constexpr int pad()
    {
        static_assert((Rp & (Rp - 1)) == 0 && (Ns & (Ns - 1)) == 0, "power-of-two passes go through shared memory");
        return Ns >= G ? 0 : Ns * Rp <= G ? Ns : Rp >= G ? 1 : G / Rp;
    }
    // base: the thread's part of the position, off: the constant part; their offsets
    // within a block never add up to a whole one (a store's base is r < Ns past a
    // multiple of min(Ns Rp, G), its off a multiple of Ns below Ns Rp; a load's base is
    // t and its off a multiple of TPF), so the padded position is the sum of both
    template <int Rp, int Ns> __device__ __forceinline__ static int at(int pos) { return pos + pos / G * pad<Rp, Ns>(); }
    template <int Rp, int Ns> __device__ __forceinline__ void st(int base, int off, V v) { s[at<Rp, Ns>(base) + at<Rp, Ns>(off)] = v; }
    template <int Rp, int Ns> __device__ __forceinline__ V ld(int base, int off) const { return s[at<Rp, Ns>(base) + at<Rp, Ns>(off)]; }
    __host__ __device__ static constexpr int pitch(int rb) { return rb | 1; }
    template <int RA, int RB> __device__ __forceinline__ void st_split(int v, int q, V x) { s[q * pitch(RB) + v] = x; }
    template <int RA, int RB> __device__ __forceinline__ V ld_split(int v, int q) const { return s[v * pitch(RB) + q]; }
    __device__ __forceinline__ void st(int pos, V v) { s[pos] = v; }
    __device__ __forceinline__ V ld(int pos) const { return s[pos]; }
    // elements a row of N takes through the passes of radix R (register plan) or split
    template <int N, int R, int P = 0> __host__ __device__ static constexpr int size_reg()
    {
        using Plan = RadixPlan<N, R>;
        if constexpr (P + 1 >= Plan::P) {
            return N;
        } else {
            constexpr int here = N + (N + G - 1) / G * pad<Plan::radix(P), Plan::span(P)>(), rest = size_reg<N, R, P + 1>();
            return here > rest ? here : rest;
        }
    }
    template <int N, int R, bool SPLIT> __host__ __device__ static constexpr int size()
    {
        if constexpr (SPLIT) {
            constexpr int A = SplitPlan<N>::RA, B = SplitPlan<N>::RB;
            constexpr int x = A * pitch(B), y = B * pitch(A);
            return x > y ? x : y;
        } else {
            return size_reg<N, R>();
        }
    }
};

}  // namespace ps
