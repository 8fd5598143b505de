// Bodies of the launch wrappers declared in ps_launch.cuh, for the units that
// instantiate them.
#pragma once

#include "ps_launch.cuh"

namespace ps {

template <typename T, int N>
bool L3<T, N>::host_alt_table(V* twp_alt)
{
    if constexpr (ALT > 0) {
        static_assert(PencilGeom<T, N, ALT>::W == PG::W, "same pencil tile width");
        transform_table<V, N, ALT, PencilGeom<T, N, ALT>::TPF>(twp_alt);
        return true;
    } else {
        (void)twp_alt;
        return false;
    }
}

template <typename T, int N>
bool L3<T, N>::host_pair_alt_table(V* twr_alt)
{
    if constexpr (PAIR_RX2 > 0) {
        using G2 = RowGeom<T, N, PAIR_RX2>;
        transform_table<V, N / 2, G2::R, G2::TPF>(twr_alt);
        return true;
    } else {
        (void)twr_alt;
        return false;
    }
}

template <typename T, int N>
int L3<T, N>::pair_variants()
{
    int m = 1;
    if constexpr (PairVariants<T, N>::KEEP_OK) m |= 2;
    if constexpr (PAIR_RX2 > 0) {
        if constexpr (PairGeom<T, N, PAIR_RX2, true>::FITS) m |= 4;
    }
    return m;
}

template <typename T, int N>
void L3<T, N>::host_tables(V* twp, V* twr)
{
    transform_table<V, N, PG::R, PG::TPF>(twp);
    transform_table<V, N / 2, RG::R, RG::TPF>(twr);
}

template <typename T, int N>
int L3<T, N>::inv_x(cudaStream_t st, const V* src, int ss, V* dst, int ds, int mode, const Shell* sh,
                 int hvalid, const Tables<T>& tb, int quad, int nsrc, int skip_dead)
{
    PS_LTRY(set_smem(k_inv_x<T, N>, PG::SMEM));
    const int nj = quad ? N / 2 + 1 : N;
    k_inv_x<T, N><<<(unsigned)(nj * (ds / PG::W)), PG::THREADS, PG::SMEM, st>>>(
        src, ss, nsrc > 0 ? nsrc : N, dst, ds, mode, sh, hvalid, quad, skip_dead, tb.twp);
    return PS_OK;
}

template <typename T, int N>
int L3<T, N>::pass_y(cudaStream_t st, V* data, int stride, bool inv, const Tables<T>& tb, int quad,
                  int jband, int ncols, int jout, int alt)
{
    const int ni = quad ? N / 2 + 1 : N;
    const int nc = ncols > 0 ? ncols : stride;
    const unsigned blocks = (unsigned)(ni * (nc / PG::W));
    if constexpr (ALT > 0) {
        if (alt && tb.twp_alt) {
            using PA = PencilGeom<T, N, ALT>;
            if (inv) {
                PS_LTRY(set_smem(k_pass_y<T, N, true, ALT>, PA::SMEM));
                k_pass_y<T, N, true, ALT><<<blocks, PA::THREADS, PA::SMEM, st>>>(data, stride, nc, quad, jband, jout,
                                                                                 tb.twp_alt);
            } else {
                PS_LTRY(set_smem(k_pass_y<T, N, false, ALT>, PA::SMEM));
                k_pass_y<T, N, false, ALT><<<blocks, PA::THREADS, PA::SMEM, st>>>(data, stride, nc, quad, jband,
                                                                                  jout, tb.twp_alt);
            }
            return PS_OK;
        }
    }
    if (inv) {
        PS_LTRY(set_smem(k_pass_y<T, N, true>, PG::SMEM));
        k_pass_y<T, N, true><<<blocks, PG::THREADS, PG::SMEM, st>>>(data, stride, nc, quad, jband, jout, tb.twp);
    } else {
        PS_LTRY(set_smem(k_pass_y<T, N, false>, PG::SMEM));
        k_pass_y<T, N, false><<<blocks, PG::THREADS, PG::SMEM, st>>>(data, stride, nc, quad, jband, jout, tb.twp);
    }
    return PS_OK;
}

template <typename T, int N>
int L3<T, N>::inv_z(cudaStream_t st, const V* src, int ss, int hvalid, T* out, const T* aux, int epi,
                 int power, double* partials, const Tables<T>& tb, int* nblocks)
{
    const size_t smem = RG::smem(1, hvalid, 0);
    PS_LTRY(set_smem(k_inv_z<T, N>, RG::smem(1, N / 2 + 1, 0)));
    int grid = 0;
    PS_LTRY(persistent_grid(k_inv_z<T, N>, RG::THREADS, smem, N * N / RG::WZ, &grid));
    k_inv_z<T, N><<<grid, RG::THREADS, smem, st>>>(src, ss, hvalid, out, aux, epi, power, partials,
                                                   tb.twr, tb.twpp);
    if (nblocks) *nblocks = grid;
    return PS_OK;
}

template <typename T, int N>
int L3<T, N>::fwd_z(cudaStream_t st, int kind, const void* a, const void* b, V* dst, int ds, int hout,
                 const Tables<T>& tb, int stage, size_t nrows, int* status, int tx_extra)
{
    const bool two = kind == SRC_XHI_F32 || kind == SRC_XHI_F64;
    const size_t eb = (kind == SRC_F32 || kind == SRC_XHI_F32) ? 4 : 8;
    const uintptr_t addr = (uintptr_t)a | (two ? (uintptr_t)b : 0);
    const size_t smem_staged = RG::STAGE_OFF + (two ? 2 : 1) * (size_t)RG::WZ * N * eb;
    const bool can_stage = kind != SRC_T && addr % 16 == 0 && smem_staged <= 227 * 1024;
    const unsigned blocks = (unsigned)((nrows ? nrows : (size_t)N * N) / RG::WZ);
    if (blocks == 0) return PS_OK;
    if (stage != 0 && can_stage && status) {
        PS_LTRY(set_smem(k_fwd_z<T, N, true, true>, smem_staged));
        k_fwd_z<T, N, true, true><<<blocks, RG::THREADS, smem_staged, st>>>(kind, a, b, dst, ds, hout, 1, tb.twr,
                                                                             tb.twpp, status, tx_extra);
        return PS_OK;
    }
    if (stage != 0 && can_stage) {
        PS_LTRY(set_smem(k_fwd_z<T, N, true>, smem_staged));
        k_fwd_z<T, N, true><<<blocks, RG::THREADS, smem_staged, st>>>(kind, a, b, dst, ds, hout, 1, tb.twr,
                                                                       tb.twpp);
        return PS_OK;
    }
    constexpr size_t smem = RG::STAGE_OFF;
    PS_LTRY(set_smem(k_fwd_z<T, N, false>, smem));
    const uintptr_t need = (kind == SRC_F32 || kind == SRC_XHI_F32) ? 8 : 16;  // float2 / double2
    const int vec = kind != SRC_T && (addr % need) == 0;
    k_fwd_z<T, N, false><<<blocks, RG::THREADS, smem, st>>>(kind, a, b, dst, ds, hout, vec, tb.twr, tb.twpp);
    return PS_OK;
}

template <typename T, int N>
template <int RX, bool KEEP>
int L3<T, N>::pair_z_v(cudaStream_t st, const V* a, int sa, int hva, const V* b, int sb, int hvb, V* dst, int ds,
                    int hout, const V* twr, const V* twpp, int quad)
{
    using G = RowGeom<T, N, RX>;
    using PGm = PairGeom<T, N, RX, KEEP>;
    const size_t smem = PGm::smem(b ? 2 : 1, hva, hvb);
    PS_LTRY(set_smem(k_pair_z<T, N, RX, KEEP>, PGm::smem(2, N / 2 + 1, N / 2 + 1)));
    const int nrows = quad ? (N / 2 + 1) * (N / 2 + 1) : N * N;
    int grid = 0;
    PS_LTRY(persistent_grid(k_pair_z<T, N, RX, KEEP>, G::THREADS, smem, (nrows + G::WZ - 1) / G::WZ, &grid));
    k_pair_z<T, N, RX, KEEP><<<grid, G::THREADS, smem, st>>>(a, sa, hva, b, sb, hvb, dst, ds, hout, nrows, twr,
                                                             twpp);
    return PS_OK;
}

template <typename T, int N>
int L3<T, N>::pair_z(cudaStream_t st, const V* a, int sa, int hva, const V* b, int sb, int hvb, V* dst,
                  int ds, int hout, const Tables<T>& tb, int quad, int variant)
{
    if constexpr (PAIR_RX2 > 0) {
        if constexpr (PairGeom<T, N, PAIR_RX2, true>::FITS) {
            if (variant == 2 && tb.twr_alt && !quad)
                return pair_z_v<PAIR_RX2, true>(st, a, sa, hva, b, sb, hvb, dst, ds, hout, tb.twr_alt, tb.twpp,
                                                quad);
        }
    }
    if constexpr (PairVariants<T, N>::KEEP_OK) {
        if (variant == 1 && !quad)
            return pair_z_v<0, true>(st, a, sa, hva, b, sb, hvb, dst, ds, hout, tb.twr, tb.twpp, quad);
    }
    return pair_z_v<0, false>(st, a, sa, hva, b, sb, hvb, dst, ds, hout, tb.twr, tb.twpp, quad);
}

template <typename T, int N>
int L3<T, N>::fwd_x(cudaStream_t st, V* data, int stride, int hvalid, int epi, V* out, int ostride,
                 const V* dk, int dks, const Shell* shells, int nshell, const unsigned short* lut,
                 int lut_size, double* partials, const Tables<T>& tb, int* nblocks, double weight,
                 int quad, int ndk, int r2max, T* mod_out, int ncols,
                 int jband, int alt)
{
    const int nj = quad ? N / 2 + 1 : N;
    const int nc = ncols > 0 ? ncols : stride;
    const unsigned blocks = (unsigned)(nj * (nc / PG::W));
    const bool dot = epi == SPEC_DOT || epi == SPEC_COUNT || epi == SPEC_DOT_ABS;
    if constexpr (ALT > 0) {  // alt: the dot pass in the alternative geometry (PencilAlt)
        if (dot && alt && tb.twp_alt) {
            using PA = PencilGeom<T, N, ALT>;
            PS_LTRY(set_smem(k_fwd_x<T, N, true, ALT>, PA::SMEM_DOT));
            k_fwd_x<T, N, true, ALT><<<blocks, PA::THREADS, PA::SMEM_DOT, st>>>(
                data, stride, hvalid, epi, out, ostride, dk, dks, ndk > 0 ? ndk : N, shells, nshell, lut, lut_size,
                weight, quad, r2max, partials, tb.twp_alt, mod_out, nc, jband);
            if (nblocks) *nblocks = (int)blocks;
            return PS_OK;
        }
    }
    if (dot) {
        PS_LTRY(set_smem(k_fwd_x<T, N, true>, PG::SMEM_DOT));
        k_fwd_x<T, N, true><<<blocks, PG::THREADS, PG::SMEM_DOT, st>>>(
            data, stride, hvalid, epi, out, ostride, dk, dks, ndk > 0 ? ndk : N, shells, nshell, lut, lut_size,
            weight, quad, r2max, partials, tb.twp, mod_out, nc, jband);
    } else {
        PS_LTRY(set_smem(k_fwd_x<T, N, false>, PG::SMEM));
        k_fwd_x<T, N, false><<<blocks, PG::THREADS, PG::SMEM, st>>>(
            data, stride, hvalid, epi, out, ostride, dk, dks, ndk > 0 ? ndk : N, shells, nshell, lut, lut_size,
            weight, quad, r2max, partials, tb.twp, mod_out, nc, jband);
    }
    if (nblocks) *nblocks = (int)blocks;
    return PS_OK;
}

}  // namespace ps
