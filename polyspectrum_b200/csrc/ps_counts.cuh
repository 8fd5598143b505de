// Exact polygon counts of a pair group by enumeration in integers: the mode
// lists (host) and the histogram kernel.  Shared by the library and the
// stand-alone timing harness.
#pragma once

#include <algorithm>
#include <cmath>
#include <vector>

#include "ps_common.cuh"

namespace ps {

// ------------------------------------------------------------------ exact pair counts
// Polygon counts of a pair group whose shells are all r^2 intervals, by
// enumeration in integers instead of FP64 transforms of unit shells:
//     count(c) = #{(m_a, m_b) in S_a x S_b : |w(m_a + m_b)|^2 in [r2lo_c, r2hi_c]},
// w = componentwise wrap into the grid's lattice frequencies [-N/2, N/2)
// (WRAP: only when a component can reach N/2; aliased triples are counted, as
// the reference's N-grid sums count them).  That is the number of triples
// m_a + m_b + m_c = 0 (mod N) with m_c in S_c (S_c = -S_c).  S_a enters as
// representatives of its orbits under the 48 axis permutations and sign
// flips with their orbit sizes as weights: S_b, the closing shells and |w(.)|^2
// are invariant under them.  The pairs are cut into work items (a chunk of
// THREADS BPT modes of S_b times a slice of rep_slice representatives); each CTA
// of a group takes every nctas-th item into
// its own histogram of |w(m_a + m_b)|^2 - s_lo over nbins bins in shared
// memory (integer atomics: the result does not depend on their order), so
// the clearing and the interval sums are paid once per CTA.  Each CTA then sums each closing shell's
// interval and adds it to counts[c].  Without WRAP the bin is
// |m_a|^2 - s_lo + |m_b|^2 + 2 m_a.m_b: the representatives are staged as
// (2x, 2y, 2z, weight) beside |m_a|^2 - s_lo, the modes keep |m_b|^2 (a large
// negative value for the idle slots past nb), so a pair costs three
// multiply-adds, an add and the range test before its atomic.
// WRAP: with a >= 0 and b >= -n/2 a component q = a + b can pass the upper edge
// only, and (q - n)^2 - q^2 = n (n - 2 q) is at most 0 exactly where q >= n/2, so the
// wrapped norm is the plain one plus min(0, n^2 - 2 n q) per component: one fused
// add-minimum each (compares and selects per component took 27 instructions a pair,
// 0.24 ms for the 2.2e8 wrapping pairs of 64 equilateral triangles at 128^3).
constexpr int kCountBPT = 4;
constexpr int kCountThreads = 1024;  // one CTA per SM: 32 warps to hide the atomics' latency
// Short histograms hold no SM's shared memory, and a list of such groups is cut
// finer: CTAs of 256 threads, six per SM in all, so that no group's last CTA is left
// over.
constexpr int kCountSmallBins = 2048, kCountSmallThreads = 256;
constexpr int kCountRepChunk = 512;  // largest rep_slice
constexpr size_t kCountStageBytes = kCountRepChunk * 2 * sizeof(int4);
constexpr int kCountMaxBins = 44 * 1024;  // 176 KB of uint32 bins beside the staged representatives

// One launch counts for a list of groups: group g has the CTAs cta0 .. cta0 +
// nctas - 1 (about in proportion to its pairs), each with a histogram of its own.
struct CountItem {
    const int4* reps;
    const short4* modes;
    const Shell* closing;
    unsigned long long* counts;
    int nrep, nb, s_lo, nbins, rep_slice, ncl;
    int cta0, nctas;
};
template <bool WRAP, int BPT = kCountBPT, int THREADS = kCountThreads>
__global__ void __launch_bounds__(THREADS, THREADS == kCountSmallThreads ? 6 : 1)
    k_pair_counts(const CountItem* __restrict__ items, int ngroups, int n)
{
    int gi = 0;  // the group of this CTA
    for (int e = ngroups; gi + 1 < e;) {
        const int mid = (gi + e) >> 1;
        if (items[mid].cta0 <= (int)blockIdx.x) gi = mid;
        else e = mid;
    }
    const CountItem it = items[gi];
    const int4* __restrict__ reps = it.reps;
    const short4* __restrict__ modes = it.modes;
    const Shell* __restrict__ closing = it.closing;
    unsigned long long* __restrict__ counts = it.counts;
    const int nrep = it.nrep, nb = it.nb, s_lo = it.s_lo, nbins = it.nbins, ncl = it.ncl;
    int rep_slice = it.rep_slice;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    int4* srep = reinterpret_cast<int4*>(smem_raw);
    int4* sedge = srep + kCountRepChunk;  // -2 n a (WRAP), |a|^2 - s_lo
    unsigned int* hist = reinterpret_cast<unsigned int*>(smem_raw + kCountStageBytes);
    for (int i = threadIdx.x; i < nbins; i += blockDim.x) hist[i] = 0u;
    constexpr int kChunk = THREADS * BPT;
    rep_slice = max(1, min(rep_slice, kCountRepChunk));  // the staging buffer's size
    const int nmc = (nb + kChunk - 1) / kChunk, nrs = (nrep + rep_slice - 1) / rep_slice;
    const int nitems = nmc * nrs;
    for (int item = (int)blockIdx.x - it.cta0; item < nitems; item += it.nctas) {
        const int mc = item % nmc, r0 = (item / nmc) * rep_slice;
        const int cnt = min(rep_slice, nrep - r0);
        int bx[BPT], by[BPT], bz[BPT], bn[BPT];
        int ex[BPT], ey[BPT], ez[BPT];  // n^2 - 2 n b
#pragma unroll
        for (int u = 0; u < BPT; u++) {
            const int idx = mc * kChunk + u * THREADS + (int)threadIdx.x;
            const bool valid = idx < nb;
            const short4 m = valid ? modes[idx] : short4{0, 0, 0, 0};
            bx[u] = m.x;
            by[u] = m.y;
            bz[u] = m.z;
            // idle slots: every bin index of theirs is negative (|.|^2 sums stay below 2^29)
            bn[u] = valid ? m.x * m.x + m.y * m.y + m.z * m.z : -(1 << 30);
            ex[u] = n * (n - 2 * m.x);
            ey[u] = n * (n - 2 * m.y);
            ez[u] = n * (n - 2 * m.z);
        }
        __syncthreads();  // the previous item's representatives are no longer read
        for (int i = threadIdx.x; i < cnt; i += blockDim.x) {
            const int4 a = reps[r0 + i];
            srep[i] = int4{2 * a.x, 2 * a.y, 2 * a.z, a.w};
            sedge[i] = int4{-2 * n * a.x, -2 * n * a.y, -2 * n * a.z, a.x * a.x + a.y * a.y + a.z * a.z - s_lo};
        }
        __syncthreads();
#pragma unroll 2
        for (int r = 0; r < cnt; r++) {
            const int4 a = srep[r];
            const int4 d = sedge[r];
#pragma unroll
            for (int u = 0; u < BPT; u++) {
                int sb = d.w + bn[u] + a.x * bx[u] + a.y * by[u] + a.z * bz[u];
                if constexpr (WRAP)
                    sb += __viaddmin_s32(d.x, ex[u], 0) + __viaddmin_s32(d.y, ey[u], 0) + __viaddmin_s32(d.z, ez[u], 0);
                if ((unsigned)sb < (unsigned)nbins) atomicAdd(&hist[sb], (unsigned)a.w);
            }
        }
    }
    __syncthreads();
    // closing shell c: the bins of its interval (clamped to the histogram)
    const int lane = threadIdx.x & 31;
    for (int c = 0; c < ncl; c++) {
        const Shell sh = closing[c];
        const int lo = max(sh.r2lo - s_lo, 0), hi = min(sh.r2hi - s_lo, nbins - 1);
        unsigned long long v = 0ull;
        for (int i = lo + (int)threadIdx.x; i <= hi; i += blockDim.x) v += hist[i];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0 && v) atomicAdd(&counts[c], v);
    }
}

// The same for groups with one closing shell each (equilateral and single triangles),
// without a histogram: a pair inside the shell's interval adds its weight in a
// register.  The norms are computed in FP32, where every value is an integer or a half
// below 2^23 (WRAP: doubled, below 2^24) and so exact, two modes per packed
// instruction: about four instructions a pair, nine with WRAP, where
// min(0, x) = (x - |x|) / 2 leaves one packed sum and an |x| operand per component.
// (In integers, whose multiply-adds and minima issue at half rate, the 2.4e8 pairs of 64
// equilateral triangles at 128^3 took 0.197 instead of 0.156 ms, with histograms 0.42 ms.)
constexpr int kOneThreads = 256, kOneBPT = 4, kOneRepChunk = 256;
struct __align__(16) OneRep {  // a staged representative, read as two float4
    float2 v[4];
    __device__ __forceinline__ float4 pair(int q) const { return reinterpret_cast<const float4*>(v)[q]; }
};
static_assert(alignof(OneRep) == alignof(float4) && sizeof(OneRep) == 2 * sizeof(float4), "vector reads of shared rows");

__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c)
{
    float2 r;
    asm("{\n\t.reg .b64 pa, pb, pc, pd;\n\tmov.b64 pa, {%2, %3};\n\tmov.b64 pb, {%4, %5};\n\tmov.b64 pc, {%6, %7};\n\t"
        "fma.rn.f32x2 pd, pa, pb, pc;\n\tmov.b64 {%0, %1}, pd;\n\t}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return r;
}

template <bool WRAP>
__global__ void __launch_bounds__(kOneThreads, 4)
    k_pair_counts_one(const CountItem* __restrict__ items, int ngroups, int n)
{
    int gi = 0;  // the group of this CTA
    for (int e = ngroups; gi + 1 < e;) {
        const int mid = (gi + e) >> 1;
        if (items[mid].cta0 <= (int)blockIdx.x) gi = mid;
        else e = mid;
    }
    const CountItem it = items[gi];
    // representatives, each value twice (packed operands): f (a, c), f a = 2 a (WRAP: 4 a),
    // c the constant part; WRAP: -2 n a
    __shared__ OneRep sa[kOneRepChunk], su[WRAP ? kOneRepChunk : 1];
    __shared__ unsigned sw[kOneRepChunk];
    const int lo = it.closing[0].r2lo, hi = it.closing[0].r2hi;
    const float f = WRAP ? 2.f : 1.f, fn = (float)n;
    const float mid = 0.5f * f * ((float)lo + (float)hi);
    const float hw = hi >= lo ? 0.5f * f * ((float)hi - (float)lo) : -1.f;  // no value is within -1
    constexpr int kChunk = kOneThreads * kOneBPT, NP = kOneBPT / 2;
    const int rep_slice = max(1, min(it.rep_slice, kOneRepChunk));
    const int nmc = (it.nb + kChunk - 1) / kChunk, nrs = (it.nrep + rep_slice - 1) / rep_slice;
    unsigned long long inside = 0ull;
    for (int item = (int)blockIdx.x - it.cta0; item < nmc * nrs; item += it.nctas) {
        const int mc = item % nmc, r0 = (item / nmc) * rep_slice;
        const int cnt = min(rep_slice, it.nrep - r0);
        float2 bx[NP], by[NP], bz[NP], bc[NP], ex[NP], ey[NP], ez[NP];
#pragma unroll
        for (int p = 0; p < NP; p++)
#pragma unroll
            for (int l = 0; l < 2; l++) {
                const int idx = mc * kChunk + (2 * p + l) * kOneThreads + (int)threadIdx.x;
                const bool valid = idx < it.nb;
                const short4 m = valid ? it.modes[idx] : short4{0, 0, 0, 0};
                const float x = (float)m.x, y = (float)m.y, z = (float)m.z;
                const float qx = fn * (fn - 2.f * x), qy = fn * (fn - 2.f * y), qz = fn * (fn - 2.f * z);
                float c = f * (x * x + y * y + z * z);
                if (WRAP) c += qx + qy + qz;
                if (!valid) c = 1e30f;  // never inside
                (l ? bx[p].y : bx[p].x) = x;
                (l ? by[p].y : by[p].x) = y;
                (l ? bz[p].y : bz[p].x) = z;
                (l ? bc[p].y : bc[p].x) = c;
                (l ? ex[p].y : ex[p].x) = qx;
                (l ? ey[p].y : ey[p].x) = qy;
                (l ? ez[p].y : ez[p].x) = qz;
            }
        __syncthreads();  // the previous item's representatives are no longer read
        for (int i = threadIdx.x; i < cnt; i += kOneThreads) {
            const int4 a = it.reps[r0 + i];
            const float x = (float)a.x, y = (float)a.y, z = (float)a.z;
            const float ux = -2.f * fn * x, uy = -2.f * fn * y, uz = -2.f * fn * z;
            float c = f * (x * x + y * y + z * z) - mid;
            if (WRAP) c += ux + uy + uz;
            sa[i].v[0] = float2{2.f * f * x, 2.f * f * x};
            sa[i].v[1] = float2{2.f * f * y, 2.f * f * y};
            sa[i].v[2] = float2{2.f * f * z, 2.f * f * z};
            sa[i].v[3] = float2{c, c};
            if constexpr (WRAP) {
                su[i].v[0] = float2{ux, ux};
                su[i].v[1] = float2{uy, uy};
                su[i].v[2] = float2{uz, uz};
            }
            sw[i] = (unsigned)a.w;
        }
        __syncthreads();
        unsigned here = 0u;  // at most rep_slice BPT 48
#pragma unroll 2
        for (int r = 0; r < cnt; r++) {
            const float4 a01 = sa[r].pair(0), a23 = sa[r].pair(1);
            const unsigned w = sw[r];
#pragma unroll
            for (int p = 0; p < NP; p++) {
                float2 v = cadd(float2{a23.z, a23.w}, bc[p]);
                v = fma2(float2{a01.x, a01.y}, bx[p], v);
                v = fma2(float2{a01.z, a01.w}, by[p], v);
                v = fma2(float2{a23.x, a23.y}, bz[p], v);
                if constexpr (WRAP) {
                    const float4 u01 = su[r].pair(0);
                    const float2 tx = cadd(float2{u01.x, u01.y}, ex[p]), ty = cadd(float2{u01.z, u01.w}, ey[p]),
                                 tz = cadd(su[r].v[2], ez[p]);
                    v.x = ((v.x - fabsf(tx.x)) - fabsf(ty.x)) - fabsf(tz.x);
                    v.y = ((v.y - fabsf(tx.y)) - fabsf(ty.y)) - fabsf(tz.y);
                }
                if (fabsf(v.x) <= hw) here += w;
                if (fabsf(v.y) <= hw) here += w;
            }
        }
        inside += here;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) inside += __shfl_xor_sync(0xffffffffu, inside, o);
    if ((threadIdx.x & 31) == 0 && inside) atomicAdd(&it.counts[0], inside);
}

// sumI[idx[c]] = counts[c] (exact integers, below 2^53)
static __global__ void k_counts_out(int n, const unsigned long long* __restrict__ counts, const int* __restrict__ idx,
                             double* __restrict__ sumI)
{
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c < n) sumI[idx[c]] = (double)counts[c];
}

// Mode lists of an exact pair count (k_pair_counts): the modes of S_b, the
// orbit representatives of S_a with their orbit sizes, the histogram range.
struct PairCountLists {
    std::vector<short4> modes;
    std::vector<int4> reps;
    int s_lo = 0, nbins = 0;
    bool wrap = false;
};

// Representatives 0 <= x <= y <= z (N/2 stands for -N/2, which is the same index) of the
// orbits of an interval shell's modes under the 48 axis permutations and sign
// flips, with the orbit sizes: 6, 3 or 1 permutations, two signs per component
// but for 0 and the single index of |N/2|.
inline std::vector<int4> interval_orbits(const Shell& sh, int N)
{
    std::vector<int4> out;
    if (sh.r2hi < 0 || sh.r2lo > sh.r2hi) return out;
    const int b = std::min(sh.band, N / 2);
    const auto signs = [&](int v) { return v == 0 || v == N / 2 ? 1 : 2; };
    for (int x = 0; x <= b && 3 * x * x <= sh.r2hi; x++)
        for (int y = x; y <= b && x * x + 2 * y * y <= sh.r2hi; y++) {
            const int s = x * x + y * y;
            int z = y;
            if (sh.r2lo - s > z * z) {
                z = (int)sqrt((double)(sh.r2lo - s));
                while (z * z < sh.r2lo - s) z++;
                while (z > y && (z - 1) * (z - 1) >= sh.r2lo - s) z--;
            }
            for (; z <= b && s + z * z <= sh.r2hi; z++) {
                const int perms = x == y && y == z ? 1 : x == y || y == z ? 3 : 6;
                out.push_back(int4{x, y, z, perms * signs(x) * signs(y) * signs(z)});
            }
        }
    return out;
}

inline size_t orbit_total(const std::vector<int4>& reps)
{
    size_t n = 0;
    for (const int4& a : reps) n += (size_t)a.w;
    return n;
}

// The modes of a shell from its orbits (lattice frequencies [-N/2, N/2)): one pass over
// the representatives per permutation and signs, so that neighbours in the list are
// neighbours on the shell.  2 to 4 ns a mode on the host; a walk over all (x, y) columns
// with their square roots took 9 to 20 (126 170 modes at radius 100: 0.27 against 1.08 ms).
template <int A, int B, int C>  // component A takes x, B takes y, C takes z
inline void orbit_images(const std::vector<int4>& reps, int N, short4*& out)
{
    constexpr bool xy = B < A, yz = C < B;  // equal components in one order only
    for (int signs = 0; signs < 8; signs++) {
        // no -0, and N/2 as -N/2 only: the value that a sign leaves out
        const int sx = signs & 1 ? -1 : 1, sy = signs & 2 ? -1 : 1, sz = signs & 4 ? -1 : 1;
        const int ox = sx < 0 ? 0 : N / 2, oy = sy < 0 ? 0 : N / 2, oz = sz < 0 ? 0 : N / 2;
        for (const int4& a : reps) {
            if ((a.x == ox) | (a.y == oy) | (a.z == oz) | (xy & (a.x == a.y)) | (yz & (a.y == a.z))) continue;
            const short x = (short)(sx * a.x), y = (short)(sy * a.y), z = (short)(sz * a.z);
            *out++ = short4{A == 0 ? x : B == 0 ? y : z, A == 1 ? x : B == 1 ? y : z, A == 2 ? x : B == 2 ? y : z, 0};
        }
    }
}
inline std::vector<short4> orbit_modes(const std::vector<int4>& reps, int N)
{
    std::vector<short4> modes(orbit_total(reps));
    short4* out = modes.data();
    orbit_images<0, 1, 2>(reps, N, out);
    orbit_images<0, 2, 1>(reps, N, out);
    orbit_images<1, 0, 2>(reps, N, out);
    orbit_images<1, 2, 0>(reps, N, out);
    orbit_images<2, 0, 1>(reps, N, out);
    orbit_images<2, 1, 0>(reps, N, out);
    return modes;
}

// Pairs up to which the counts of a group with one closing shell are enumerated; beyond,
// the FP64 transforms of the unit shells on the group's M-grid are the cheaper.  A group's
// transforms take about 60 us and 7 ps a cell (96 points 65 us, 256 points 180 us, 600
// points 1.57 ms), the enumeration 1 ps a pair where components wrap, 0.37 ps where none
// can, beside the field's part.  Lone triangles at 128 points: 4.9e7 pairs 107 us against
// 94 us by transforms, 5.9e8 pairs 356 against 107; at 320 points 2.8e8 pairs 491 against
// 501, 1.1e9 pairs 849 against 501.  Lists of many small groups, whose transforms are chains
// of launches one after the other, are why the line is not lower at 128 points (64
// equilateral triangles, up to 5.4e7 pairs each: 0.49 ms in all).
inline double one_shell_pairs(int M, bool wrap) { return (60e6 + 7.0 * (double)M * M * M) * (wrap ? 1.0 : 2.67); }
constexpr double kHistPairs = 4e9;  // the same with histograms (several closing shells share them)

// The lists of a group with interval legs a, b on an N-grid whose transforms would run on
// the M-grid, the histogram over the squared radii [c_lo, c_hi] its closing shells may
// hold (one: a single closing shell, no histogram); false when the enumeration does not
// apply (histogram too large for shared memory, or more pairs than the FP64 transforms of
// the shells would cost).  Nothing is listed before that is known, but the orbits: listing
// the modes of thick shells first took longer than all transforms (a one-shot call at 256^3
// for sides of 64 to 77 modes, 13 modes thick: 8.3 ms, now 0.32).
inline bool pair_count_lists(const Shell& sa, const Shell& sb, int N, int M, int c_lo, int c_hi, bool one, PairCountLists* L)
{
    const double est = 4.0 * 3.14159 * (double)std::max(sa.r2hi, 1) * 4.0 * 3.14159 * (double)std::max(sb.r2hi, 1);
    if (std::max(sa.band, sb.band) > 300 || est / 48.0 > 4e10) return false;
    const int bmax_a = std::min(sa.band, N / 2), bmax_b = std::min(sb.band, N / 2);
    L->wrap = bmax_a + bmax_b >= N / 2;
    const double most = one ? one_shell_pairs(M, L->wrap) : kHistPairs;
    const double ra_hi = sqrt((double)std::max(sa.r2hi, 0)), rb_hi = sqrt((double)std::max(sb.r2hi, 0));
    const double ra_lo = sqrt((double)std::max(sa.r2lo, 0)), rb_lo = sqrt((double)std::max(sb.r2lo, 0));
    double smax = (ra_hi + rb_hi) * (ra_hi + rb_hi);
    if (L->wrap) smax = std::min(smax, 3.0 * (N / 2) * (N / 2));
    const double dmin = L->wrap ? 0.0 : std::max({0.0, ra_lo - rb_hi, rb_lo - ra_hi});
    L->s_lo = std::max(0, (int)floor(dmin * dmin) - 1);
    L->s_lo = std::max(L->s_lo, c_lo);
    const long long s_hi = std::max<long long>(L->s_lo, std::min<long long>((long long)ceil(smax) + 1, c_hi));
    if (!one && s_hi - L->s_lo + 1 > kCountMaxBins) return false;
    L->nbins = one ? 0 : (int)(s_hi - L->s_lo + 1);
    const auto volume = [](const Shell& h) {
        return 4.18879 * (pow((double)std::max(h.r2hi, 0), 1.5) - pow((double)std::max(h.r2lo, 0), 1.5));
    };
    // shells inside the grid's cube hold about their volume of modes: far too many are
    // refused before their orbits are listed
    const double inside = (double)(N / 2) * (N / 2);
    if (sa.r2hi < inside && sb.r2hi < inside && volume(sa) * volume(sb) / 48.0 > 1.5 * most) return false;
    // representatives from the smaller shell
    const Shell *pa = &sa, *pb = &sb;
    if (volume(sa) > volume(sb)) std::swap(pa, pb);
    L->reps = interval_orbits(*pa, N);
    const bool same = sa.r2lo == sb.r2lo && sa.r2hi == sb.r2hi && sa.band == sb.band;
    const std::vector<int4> other = same ? std::vector<int4>() : interval_orbits(*pb, N);
    const std::vector<int4>& orbits_b = same ? L->reps : other;
    if ((double)L->reps.size() * (double)orbit_total(orbits_b) > most) return false;
    L->modes = orbit_modes(orbits_b, N);
    return true;
}

}  // namespace ps
