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
// What bounds it: instruction latency around short runs of loads.  A (mx, my)
// column contributes one run of consecutive h (32 modes on average for 16 unit
// shells), one warp per 32 modes of a column; four such pieces are in flight per
// warp and the path from load to sum has no branch for lists of disjoint
// shells (the shell of an r2 by a four-step search in the chunk's sorted
// bounds; a table indexed by r2 made every lane fetch a sector of its own and
// took 3.4 ms for the 512 shells at 1024^3).  Slot 16 collects the modes of no shell.
// Each lane adds into slots of its own in shared memory ([shell][lane]: no
// conflicts, no atomics, so the sums do not depend on timing), which keeps the 16
// sums out of the registers.  The counts follow from the columns alone and are
// taken on one column in eight (k_pair2_counts).
#pragma once

#include <algorithm>
#include <vector>

#include "ps_common.cuh"

namespace ps {

constexpr int kP2Shells = 16;    // shells per chunk
constexpr int kP2Threads = 128;  // four warps: 17 KB of slots per CTA, twelve CTAs per SM

struct P2Chunk {
    int lo, hi;      // squared radii the chunk's shells cover
    int band;        // largest |component|
    int disjoint;    // no r2 belongs to two of its shells, and none is empty
    int cnt;         // shells
    int first;       // first shell, in sorted order
    int block0, nblocks;
};
struct P2Range { int lo, hi; };  // one configuration's r2 interval (sorted order)

// The chunks of a list of intervals (sorted by lo) on an n-grid; total_blocks
// CTAs are shared out by the area of the columns a chunk visits.
inline std::vector<P2Chunk> pair2_chunks(const std::vector<P2Range>& iv, int n, int total_blocks)
{
    std::vector<P2Chunk> out;
    const long long top = 3ll * (n / 2) * (n / 2);
    double area = 0.0;
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
        ch.disjoint = 1;
        for (int x = 0, last = -1; x < ch.cnt; x++) {
            const P2Range& r = iv[q0 + x];
            if (r.lo > r.hi || r.lo <= last) ch.disjoint = 0;
            last = std::max(last, r.hi);
        }
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

__device__ __forceinline__ int isqrt_i(int v)  // floor(sqrt(v)), v >= 0
{
    int r = (int)sqrtf((float)v);
    while (r * r > v) r--;
    while ((r + 1) * (r + 1) <= v) r++;
    return r;
}

// Block partials: partials[(block0 + b) 16 + x] of chunk block b, without N^3.
template <typename T>
__global__ void __launch_bounds__(kP2Threads, 12)
    k_pair2_sweep(int n, const V2<T>* __restrict__ dk, int dks, const P2Chunk* __restrict__ chunks, int nchunks,
                  const P2Range* __restrict__ iv, double* __restrict__ partials)
{
    constexpr int NW = kP2Threads / 32, U = 4;
    __shared__ double ssum[NW][kP2Shells + 1][32];
    __shared__ int slo[kP2Shells], shi[kP2Shells];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int c = 0;  // the chunk this block belongs to
    for (int s = nchunks; c + 1 < s;) {
        const int mid = (c + s) >> 1;
        if (chunks[mid].block0 <= (int)blockIdx.x) c = mid;
        else s = mid;
    }
    const P2Chunk ch = chunks[c];
#pragma unroll
    for (int x = 0; x <= kP2Shells; x++) ssum[wid][x][lane] = 0.0;
    double* slot = &ssum[wid][0][lane];
    const int half = n / 2, side = 2 * ch.band + 1, ncol = side * side;
    const int nw = ch.nblocks * NW;
    const bool one = ch.disjoint != 0;
    if (threadIdx.x < kP2Shells) {
        const bool have = (int)threadIdx.x < ch.cnt;
        slo[threadIdx.x] = have ? iv[ch.first + threadIdx.x].lo : 0x7fffffff;
        shi[threadIdx.x] = have ? iv[ch.first + threadIdx.x].hi : -1;
    }
    __syncthreads();
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
        int zz = z0 | (z1 << 16);
        unsigned todo = __ballot_sync(0xffffffffu, z0 <= z1);
        while (todo) {
            V2<T> d[U];
            int r2[U];  // -1: no mode
            bool edge[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int src = todo ? __ffs(todo) - 1 : 0;
                const int zp = __shfl_sync(0xffffffffu, zz, src), sc = __shfl_sync(0xffffffffu, s, src);
                const int rw = __shfl_sync(0xffffffffu, row, src);
                const int zb = zp & 0xffff, zl = zp >> 16, z = zb + lane;
                const bool in = todo && z <= zl;
                d[u] = V2<T>{0, 0};
                if (in) d[u] = dk[(size_t)rw * dks + z];
                r2[u] = in ? sc + z * z : -1;
                edge[u] = z == 0 || z == half;
                if (lane == src) zz += 32;            // the rest of a longer run is the next piece
                if (zb + 32 > zl) todo &= todo - 1u;  // (todo = 0 stays 0)
            }
            if (one) {
                int sel[U];  // the last shell whose lo is at most r2
#pragma unroll
                for (int u = 0; u < U; u++) sel[u] = 0;
#pragma unroll
                for (int w = 8; w > 0; w >>= 1)
#pragma unroll
                    for (int u = 0; u < U; u++) sel[u] += slo[sel[u] + w] <= r2[u] ? w : 0;
#pragma unroll
                for (int u = 0; u < U; u++) {
                    // (r2 = -1 lies below every lo and fails the first test)
                    const int x = slo[sel[u]] <= r2[u] && r2[u] <= shi[sel[u]] ? sel[u] : kP2Shells;
                    const double dx = (double)d[u].x, dy = (double)d[u].y;
                    double v = dx * dx + dy * dy;
                    if (!edge[u]) v += v;  // modes 0 < h < n/2 stand for their mirrors too
                    slot[x * 32] += v;
                }
            } else {
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const double dx = (double)d[u].x, dy = (double)d[u].y;
                    double v = dx * dx + dy * dy;
                    if (!edge[u]) v += v;
                    for (int x = 0; x < ch.cnt; x++)
                        if (r2[u] >= 0 && r2[u] >= slo[x] && r2[u] <= shi[x]) slot[x * 32] += v;
                }
            }
        }
    }
    // fixed-order sums: lanes by a shuffle tree, then the warps in order
    __shared__ double wsum[NW][kP2Shells];
    for (int x = 0; x < ch.cnt; x++) {
        double v = slot[x * 32];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) wsum[wid][x] = v;
    }
    __syncthreads();
    const int x = threadIdx.x;
    if (x < ch.cnt) {
        double v = 0.0;
#pragma unroll
        for (int q = 0; q < NW; q++) v += wsum[q][x];
        partials[(size_t)blockIdx.x * kP2Shells + x] = v;
    }
}

// Modes of one list entry on the n-grid, exactly: over the columns x >= y >= 0
// with their multiplicities on the lattice [-n/2, n/2), the number of lattice z
// with r2lo <= s + z^2 <= r2hi.  kP2CountParts CTAs per entry (grid y), their
// parts summed by k_pair2_finish.
constexpr int kP2CountParts = 8;
static __global__ void __launch_bounds__(256)
    k_pair2_counts(int n, const P2Range* __restrict__ iv, double* __restrict__ parts)
{
    const P2Range r = iv[blockIdx.x];
    const int half = n / 2;
    long long cnt = 0;
    if (r.hi >= 0 && r.lo <= r.hi) {
        const int band = min(half, isqrt_i(r.hi));
        for (int x = blockIdx.y; x <= band; x += kP2CountParts)
            for (int y = threadIdx.x; y <= x; y += blockDim.x) {
                const int s = x * x + y * y;
                if (s > r.hi) break;
                const int zh = min(isqrt_i(r.hi - s), half);
                int zl = 0;
                if (s < r.lo) {
                    zl = isqrt_i(r.lo - s);
                    if (zl * zl < r.lo - s) zl++;
                }
                if (zl > zh) continue;
                // |z| in [zl, zh], twice each but for 0 and the single index of |z| = n/2
                const int nz = 2 * (zh - zl + 1) - (zl == 0) - (zh == half);
                const int mult = (x == 0 || x == half ? 1 : 2) * (y == 0 || y == half ? 1 : 2) * (x == y ? 1 : 2);
                cnt += (long long)nz * mult;
            }
    }
    __shared__ long long red[8];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = cnt;
    __syncthreads();
    if (threadIdx.x == 0) {
        long long t = 0;
        for (int w = 0; w < 8; w++) t += red[w];
        parts[blockIdx.x * kP2CountParts + blockIdx.y] = (double)t;
    }
}

// Sums of shell first + x of every chunk over its blocks, in order: one CTA per
// chunk, sixteen threads per column; the sum times n3 and the count land at idx.
static __global__ void __launch_bounds__(256)
    k_pair2_finish(const P2Chunk* __restrict__ chunks, const double* __restrict__ partials, const int* __restrict__ idx,
                   double n3, double* __restrict__ sumD, const double* __restrict__ cparts, double* __restrict__ sumI)
{
    const P2Chunk ch = chunks[blockIdx.x];
    __shared__ double part[16][kP2Shells];
    const int x = threadIdx.x % kP2Shells, r = threadIdx.x / kP2Shells;
    double v = 0.0;
    if (x < ch.cnt)
        for (int b = r; b < ch.nblocks; b += 16) v += partials[(size_t)(ch.block0 + b) * kP2Shells + x];
    part[r][x] = v;
    __syncthreads();
    if (r == 0 && x < ch.cnt) {
        double t = 0.0;
#pragma unroll
        for (int q = 0; q < 16; q++) t += part[q][x];
        const int c = idx[ch.first + x];
        sumD[c] = t * n3;
        double k = 0.0;
        for (int q = 0; q < kP2CountParts; q++) k += cparts[(ch.first + x) * kP2CountParts + q];
        sumI[c] = k;
    }
}

}  // namespace ps
