// Power spectra (n = 2) of interval shells by Parseval's identity, every
// configuration of a list in one sweep over the field spectrum.
//
//     S_D(c) = N^3 sum_half w(h) F_c |dk|^2,   count(c) = sum_half w(h) F_c,
//
// F_c the modes with r2lo_c <= |m|^2 <= r2hi_c (the intersection of the two
// legs' intervals).  The configurations, sorted by r2lo, are cut into chunks of
// 16; a chunk visits the modes of its own radius range [lo, hi] only, so the
// sweep reads each mode about once however many shells there are.  Reading the
// whole band cube once per 16 shells instead took 29.9 ms for the 512 shells of
// a 1024^3 grid (about ten reads of the spectrum's ball).
//
// What bounds it: the loads.  A (mx, my) column contributes one or two short
// runs of consecutive h (32 modes on average for 16 unit shells), one warp per
// column; four columns are in flight per warp.  Each lane adds into slots of its
// own in shared memory ([shell][lane], no conflicts, no atomics, so the sums do
// not depend on timing), which keeps the 16 sums out of the registers.
#pragma once

#include <algorithm>
#include <vector>

#include "ps_common.cuh"

namespace ps {

constexpr int kP2Shells = 16;    // shells per chunk
constexpr int kP2Threads = 128;  // four warps: 24 KB of slots per CTA, nine CTAs per SM

struct P2Chunk {
    int lo, hi;      // squared radii the chunk's shells cover
    int band;        // largest |component|
    int lut_ofs;     // its bitmask table: entry r2 - lo
    int cnt;         // shells
    int first;       // first shell, in sorted order
    int block0, nblocks;
};
struct P2Range { int lo, hi; };  // one configuration's r2 interval (sorted order)

// The chunks of a list of intervals (sorted by lo) on an n-grid; total_blocks
// CTAs are shared out by the area of the columns a chunk visits.
inline std::vector<P2Chunk> pair2_chunks(const std::vector<P2Range>& iv, int n, int total_blocks, int* lut_size)
{
    std::vector<P2Chunk> out;
    const long long top = 3ll * (n / 2) * (n / 2);
    double area = 0.0;
    *lut_size = 0;
    for (size_t q0 = 0; q0 < iv.size(); q0 += kP2Shells) {
        P2Chunk ch;
        ch.first = (int)q0;
        ch.cnt = (int)std::min<size_t>(kP2Shells, iv.size() - q0);
        long long lo = top + 1, hi = -1;
        for (int x = 0; x < ch.cnt; x++) {
            const P2Range& r = iv[q0 + x];
            if (r.lo > r.hi || r.hi < 0) continue;  // an empty intersection selects nothing
            lo = std::min<long long>(lo, std::max(r.lo, 0));
            hi = std::max<long long>(hi, std::min<long long>(r.hi, top));
        }
        if (hi < lo) lo = 0, hi = -1;
        ch.lo = (int)lo;
        ch.hi = (int)hi;
        int b = 0;
        while (b < n / 2 && (long long)(b + 1) * (b + 1) <= hi) b++;
        ch.band = b;
        ch.lut_ofs = *lut_size;
        *lut_size += (int)(hi - lo + 1);
        ch.block0 = ch.nblocks = 0;
        area += (double)(2 * b + 1) * (2 * b + 1);
        out.push_back(ch);
    }
    int base = 0;
    for (P2Chunk& ch : out) {
        const int cols = (2 * ch.band + 1) * (2 * ch.band + 1);
        const int most = std::max(1, (cols + 32 * (kP2Threads / 32) - 1) / (32 * (kP2Threads / 32)));
        ch.block0 = base;
        ch.nblocks = std::max(1, std::min(most, (int)(total_blocks * (cols / area))));
        base += ch.nblocks;
    }
    return out;
}

// Bitmask tables of all chunks: bit x of entry r2 - lo = shell first + x selects r2.
static __global__ void k_pair2_lut(const P2Chunk* __restrict__ chunks, const P2Range* __restrict__ iv,
                                   unsigned short* __restrict__ lut)
{
    const P2Chunk ch = chunks[blockIdx.y];
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q <= ch.hi - ch.lo; q += gridDim.x * blockDim.x) {
        const int r2 = ch.lo + q;
        unsigned bits = 0u;
        for (int x = 0; x < ch.cnt; x++) {
            const P2Range r = iv[ch.first + x];
            bits |= (unsigned)(r2 >= r.lo && r2 <= r.hi) << x;
        }
        lut[ch.lut_ofs + q] = (unsigned short)bits;
    }
}

__device__ __forceinline__ int isqrt_i(int v)  // floor(sqrt(v)), v >= 0
{
    int r = (int)sqrtf((float)v);
    while (r * r > v) r--;
    while ((r + 1) * (r + 1) <= v) r++;
    return r;
}

// Block partials: partials[(block0 + b) 32 + x] of chunk block b: x < 16 the
// sums (without N^3), x >= 16 the counts.
template <typename T>
__global__ void __launch_bounds__(kP2Threads)
    k_pair2_sweep(int n, const V2<T>* __restrict__ dk, int dks, const P2Chunk* __restrict__ chunks, int nchunks,
                  const unsigned short* __restrict__ lut, double* __restrict__ partials)
{
    constexpr int NW = kP2Threads / 32, U = 4;
    __shared__ double ssum[NW][kP2Shells][32];
    __shared__ int scnt[NW][kP2Shells][32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int c = 0;  // the chunk this block belongs to
    for (int s = nchunks; c + 1 < s;) {
        const int mid = (c + s) >> 1;
        if (chunks[mid].block0 <= (int)blockIdx.x) c = mid;
        else s = mid;
    }
    const P2Chunk ch = chunks[c];
#pragma unroll
    for (int x = 0; x < kP2Shells; x++) {
        ssum[wid][x][lane] = 0.0;
        scnt[wid][x][lane] = 0;
    }
    auto add = [&](unsigned bits, V2<T> d, int z) {
        const int w = herm_weight(z, n);
        const double v = (double)w * ((double)d.x * (double)d.x + (double)d.y * (double)d.y);
        while (bits) {
            const int x = __ffs(bits) - 1;
            bits &= bits - 1;
            ssum[wid][x][lane] += v;
            scnt[wid][x][lane] += w;
        }
    };
    const int half = n / 2, side = 2 * ch.band + 1, ncol = side * side;
    const int nw = ch.nblocks * NW;
    const unsigned short* tab = lut + ch.lut_ofs;
    for (int g = ((int)blockIdx.x - ch.block0) * NW + wid; g * 32 < ncol; g += nw) {
        // lane l finds the h range of column 32 g + l
        const int q = g * 32 + lane;
        const int mx = q / side - ch.band, my = q % side - ch.band;
        const int s = mx * mx + my * my;
        int z0 = 0, z1 = -1;
        if (q < ncol && mx < half && my < half && s <= ch.hi) {  // +n/2 is the index of -n/2
            if (s < ch.lo) {
                z0 = isqrt_i(ch.lo - s);
                if (z0 * z0 < ch.lo - s) z0++;
            }
            z1 = min(isqrt_i(ch.hi - s), half);
        }
        const int row = (mx < 0 ? mx + n : mx) * n + (my < 0 ? my + n : my);
        unsigned todo = __ballot_sync(0xffffffffu, z0 <= z1);
        while (todo) {
            V2<T> d[U];
            unsigned bits[U];
            int zz[U], ze[U], ss[U];
            const V2<T>* p[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const bool on = todo != 0u;
                const int src = on ? __ffs(todo) - 1 : 0;
                todo &= todo - 1;
                zz[u] = __shfl_sync(0xffffffffu, z0, src) + lane;
                ze[u] = on ? __shfl_sync(0xffffffffu, z1, src) : -1;
                ss[u] = __shfl_sync(0xffffffffu, s, src) - ch.lo;
                p[u] = dk + (size_t)__shfl_sync(0xffffffffu, row, src) * dks;
                bits[u] = 0u;
                if (zz[u] <= ze[u]) {
                    d[u] = p[u][zz[u]];
                    bits[u] = __ldg(tab + (ss[u] + zz[u] * zz[u]));
                }
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                if (bits[u]) add(bits[u], d[u], zz[u]);
                for (int z = zz[u] + 32; z <= ze[u]; z += 32) {
                    const unsigned b = __ldg(tab + (ss[u] + z * z));
                    if (b) add(b, p[u][z], z);
                }
            }
        }
    }
    // fixed-order sums: lanes by a shuffle tree, then the warps in order
    __syncthreads();
    __shared__ double wsum[NW][2 * kP2Shells];
    for (int x = 0; x < ch.cnt; x++) {
        double v = ssum[wid][x][lane], k = (double)scnt[wid][x][lane];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            v += __shfl_xor_sync(0xffffffffu, v, o);
            k += __shfl_xor_sync(0xffffffffu, k, o);
        }
        if (lane == 0) {
            wsum[wid][x] = v;
            wsum[wid][kP2Shells + x] = k;
        }
    }
    __syncthreads();
    const int x = threadIdx.x;
    if (x < 2 * kP2Shells && (x % kP2Shells) < ch.cnt) {
        double v = 0.0;
#pragma unroll
        for (int q = 0; q < NW; q++) v += wsum[q][x];
        partials[(size_t)blockIdx.x * 2 * kP2Shells + x] = v;
    }
}

// Sums of shell `first + x` of every chunk over its blocks, in order: one CTA
// per chunk, eight threads per column; sumD (times n3) and sumI land at idx.
static __global__ void __launch_bounds__(256)
    k_pair2_finish(const P2Chunk* __restrict__ chunks, const double* __restrict__ partials, const int* __restrict__ idx,
                   double n3, double* __restrict__ sumD, double* __restrict__ sumI)
{
    const P2Chunk ch = chunks[blockIdx.x];
    __shared__ double part[8][2 * kP2Shells];
    const int x = threadIdx.x % (2 * kP2Shells), r = threadIdx.x / (2 * kP2Shells);
    double v = 0.0;
    if ((x % kP2Shells) < ch.cnt)
        for (int b = r; b < ch.nblocks; b += 8) v += partials[(size_t)(ch.block0 + b) * 2 * kP2Shells + x];
    part[r][x] = v;
    __syncthreads();
    if (r == 0 && (x % kP2Shells) < ch.cnt) {
        double t = 0.0;
#pragma unroll
        for (int q = 0; q < 8; q++) t += part[q][x];
        const int c = idx[ch.first + x % kP2Shells];
        if (x < kP2Shells) sumD[c] = t * n3;
        else sumI[c] = t;
    }
}

}  // namespace ps
