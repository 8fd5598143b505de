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
        transform_table<V, N, PencilGeom<T, N, ALT>>(twp_alt);
        return true;
    } else if constexpr (YGeom<T, N, 0>::LONG) {  // the Y pass's own geometry
        transform_table<V, N, typename YGeom<T, N, 0>::type>(twp_alt);
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
        transform_table<V, N / 2, G2>(twr_alt);
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
    transform_table<V, N, PG>(twp);
    transform_table<V, N / 2, RG>(twr);
}

template <typename T, int N>
int L3<T, N>::inv_x_b(cudaStream_t st, const V* src, int ss, const XItem<T>* items, int nitems,
                      int ds, int mode, const Tables<T>& tb, int quad, int nsrc, int skip_dead)
{
    PS_NEED_TABLE(tb.twp);
    PS_LTRY(set_smem(k_inv_x<T, N>, PG::SMEM));
    const int nj = quad ? N / 2 + 1 : N;
    k_inv_x<T, N><<<dim3((unsigned)(nj * (ds / PG::W)), (unsigned)nitems), PG::THREADS, PG::SMEM, st>>>(
        src, ss, nsrc > 0 ? nsrc : N, pack(items, nitems), mode, quad, skip_dead, tb.twp);
    return PS_OK;
}

template <typename T, int N>
int L3<T, N>::pass_y_b(cudaStream_t st, const YItem<T>* items, int nitems, int ncols, bool inv,
                       const Tables<T>& tb, int quad, int alt)
{
    using YG = typename YGeom<T, N, 0>::type;  // (the alternative geometries have the default's tile width)
    const dim3 grid((unsigned)((quad ? N / 2 + 1 : N) * (ncols / YG::W)), (unsigned)nitems);
    auto go = [&](auto kernel, int threads, size_t smem, const V* tw) -> int {
        PS_NEED_TABLE(tw);
        PS_LTRY(set_smem(kernel, smem));
        kernel<<<grid, threads, smem, st>>>(pack(items, nitems), quad, tw);
        return PS_OK;
    };
    if constexpr (Y_ALT > 0) {
        using PA = PencilGeom<T, N, ALT>;
        if (alt && tb.twp_alt)
            return inv ? go(k_pass_y<T, N, true, ALT>, PA::THREADS, PA::SMEM, tb.twp_alt)
                       : go(k_pass_y<T, N, false, ALT>, PA::THREADS, PA::SMEM, tb.twp_alt);
    }
    const V* tw = YGeom<T, N, 0>::LONG ? tb.twp_alt : tb.twp;
    return inv ? go(k_pass_y<T, N, true>, YG::THREADS, YG::SMEM, tw) : go(k_pass_y<T, N, false>, YG::THREADS, YG::SMEM, tw);
}

template <typename T, int N>
int L3<T, N>::inv_z(cudaStream_t st, const V* src, int ss, int hvalid, T* out, const T* aux, int epi,
                 int power, double* partials, const Tables<T>& tb, int* nblocks, double scale)
{
    PS_NEED_TABLE(tb.twr);
    PS_NEED_TABLE(tb.twpp);
    const size_t smem = RG::smem(1, hvalid, 0);
    PS_LTRY(set_smem(k_inv_z<T, N>, RG::smem(1, N / 2 + 1, 0)));
    int grid = 0;
    PS_LTRY(persistent_grid(k_inv_z<T, N>, RG::THREADS, smem, N * N / RG::WZ, &grid));
    k_inv_z<T, N><<<grid, RG::THREADS, smem, st>>>(src, ss, hvalid, out, aux, epi, power, scale, partials,
                                                   tb.twr, tb.twpp);
    if (nblocks) *nblocks = grid;
    return PS_OK;
}

template <typename T, int N>
int L3<T, N>::fwd_z(cudaStream_t st, int kind, const void* a, const void* b, V* dst, int ds, int hout,
                 const Tables<T>& tb, int stage, size_t nrows, int* status, int tx_extra)
{
    PS_NEED_TABLE(tb.twr);
    PS_NEED_TABLE(tb.twpp);
    const bool two = kind == SRC_XHI_F32 || kind == SRC_XHI_F64;
    const size_t eb = (kind == SRC_F32 || kind == SRC_XHI_F32) ? 4 : 8;
    const uintptr_t addr = (uintptr_t)a | (two ? (uintptr_t)b : 0);
    const size_t smem_staged = RG::ROWBUF_OFF + std::max((two ? 2 : 1) * (size_t)RG::WZ * N * eb,
                                                         (size_t)RG::WZ * RG::ROWBUF * sizeof(V));
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
template <int RX, bool KEEP, bool REAL, bool TWO>
int L3<T, N>::pair_z_v(cudaStream_t st, const PairItem<T>* items, int nitems, int ninputs,
                       int hva, int hvb, const V* twr, const V* twpp, int quad)
{
    PS_NEED_TABLE(twr);
    PS_NEED_TABLE(twpp);
    using G = RowGeom<T, N, RX>;
    using PGm = PairGeom<T, N, RX, KEEP>;
    const int ea = REAL ? (hva + 1) / 2 : hva, eb = REAL ? (hvb + 1) / 2 : hvb;
    const bool alias = PGm::smem(ninputs, ea, eb, true) < PGm::smem(ninputs, ea, eb, false);
    const size_t smem = PGm::smem(ninputs, ea, eb, alias);
    PS_LTRY(set_smem(k_pair_z<T, N, RX, KEEP, REAL, TWO>, PGm::smem(2, N / 2 + 1, N / 2 + 1)));
    const int nrows = REAL ? (N / 2 + 1) * (N / 2 + 1) : N * N;
    const int tiles = (nrows + G::WZ - 1) / G::WZ;
    int grid = 0;  // resident CTAs, shared out among the items
    PS_LTRY(persistent_grid(k_pair_z<T, N, RX, KEEP, REAL, TWO>, G::THREADS, smem, tiles * nitems, &grid));
    grid = std::max(1, std::min(tiles, grid / nitems));
    k_pair_z<T, N, RX, KEEP, REAL, TWO><<<dim3((unsigned)grid, (unsigned)nitems), G::THREADS, smem, st>>>(pack(items, nitems), nrows, alias ? 1 : 0, twr, twpp);
    return PS_OK;
}

template <typename T, int N>
int L3<T, N>::pair_z_b(cudaStream_t st, const PairItem<T>* items, int nitems, int ninputs,
                       int hva, int hvb, const Tables<T>& tb, int quad, int variant)
{
    if constexpr (sizeof(T) == 8) {
        if (quad)
            return ninputs > 1 ? pair_z_v<0, false, true, true>(st, items, nitems, ninputs, hva, hvb, tb.twr, tb.twpp, quad)
                               : pair_z_v<0, false, true, false>(st, items, nitems, ninputs, hva, hvb, tb.twr, tb.twpp, quad);
    }
    if (ninputs == 1)  // one leg squared: one row transform in registers anyway
        return pair_z_v<0, false, false, false>(st, items, nitems, 1, hva, 0, tb.twr, tb.twpp, quad);
    if constexpr (PAIR_RX2 > 0) {
        if constexpr (PairGeom<T, N, PAIR_RX2, true>::FITS) {
            if (variant == 2 && tb.twr_alt)
                return pair_z_v<PAIR_RX2, true, false, true>(st, items, nitems, 2, hva, hvb, tb.twr_alt, tb.twpp, quad);
        }
    }
    if constexpr (PairVariants<T, N>::KEEP_OK) {
        if (variant == 1) return pair_z_v<0, true, false, true>(st, items, nitems, 2, hva, hvb, tb.twr, tb.twpp, quad);
    }
    return pair_z_v<0, false, false, true>(st, items, nitems, 2, hva, hvb, tb.twr, tb.twpp, quad);
}

template <typename T, int N>
int L3<T, N>::prod_z(cudaStream_t st, const ProdItem<T>* items, int nitems, int hv, bool real, int abs_terms,
                     const Tables<T>& tb, int* nblocks)
{
    PS_NEED_TABLE(tb.twr);
    PS_NEED_TABLE(tb.twpp);
    const int P0 = RG::pitch(real ? (hv + 1) / 2 : hv);
    const bool alias = 2 * std::max(P0, RG::ROWBUF) < 2 * P0 + RG::ROWBUF;  // rows' exchange buffers in their stages
    const int P = alias ? std::max(P0, RG::ROWBUF) : P0;
    const size_t smem = (alias ? RG::ROWBUF_OFF : RG::STAGE_OFF) + (size_t)2 * RG::WZ * P * sizeof(V);
    auto go = [&](auto kernel) -> int {
        PS_LTRY(set_smem(kernel, RG::smem(1, N / 2 + 1, 0)));
        int grid = 0;  // resident CTAs, shared out among the items
        PS_LTRY(persistent_grid(kernel, RG::THREADS, smem, prod_blocks(real) * nitems, &grid));
        grid = std::max(1, std::min(prod_blocks(real), grid / nitems));
        kernel<<<dim3((unsigned)grid, (unsigned)nitems), RG::THREADS, smem, st>>>(pack(items, nitems), P, alias ? 1 : 0, abs_terms, tb.twr,
                                                                                  tb.twpp);
        *nblocks = grid;
        return PS_OK;
    };
    if constexpr (sizeof(T) == 8) {
        if (real) return go(k_prod_z<T, N, true>);
    }
    return go(k_prod_z<T, N, false>);
}

template <typename T, int N>
int L3<T, N>::fwd_x(cudaStream_t st, const FwdXItem<T>* items, int nitems, int ncols, int epi,
                    V* out, int ostride, const V* dk, int dks, const Tables<T>& tb, int* nblocks, int quad, int ndk,
                    T* mod_out, int jband, int alt)
{
    using SG = typename StoreXGeom<T, N, 0>::type;
    const bool store = epi == SPEC_STORE || epi == SPEC_STORE_PHASE;
    const dim3 grid((unsigned)((quad ? N / 2 + 1 : N) * (ncols / (store ? SG::W : PG::W))), (unsigned)nitems);
    const bool dot = epi == SPEC_DOT || epi == SPEC_COUNT || epi == SPEC_DOT_ABS;
    if (nblocks) *nblocks = (int)grid.x;
    auto go = [&](auto batch, auto kernel, int threads, size_t smem, const V* tw) -> int {
        PS_NEED_TABLE(tw);
        PS_LTRY(set_smem(kernel, smem));
        if constexpr (std::is_same_v<decltype(batch), std::true_type>)
            kernel<<<grid, threads, smem, st>>>(pack(items, nitems), epi, out, ostride, dk, dks, ndk > 0 ? ndk : N, quad,
                                                tw, mod_out, jband);
        else
            kernel<<<grid, threads, smem, st>>>(items[0], epi, out, ostride, dk, dks, ndk > 0 ? ndk : N, quad, tw, mod_out,
                                                jband);
        return PS_OK;
    };
    if constexpr (ALT > 0) {  // alt: the dot pass in the alternative geometry (PencilAlt)
        using PA = PencilGeom<T, N, ALT>;
        if (dot && alt && tb.twp_alt)
            return go(std::true_type{}, k_fwd_x<T, N, FWD_SUMS, ALT>, PA::THREADS, PA::SMEM_DOT, tb.twp_alt);
    }
    if (dot) return go(std::true_type{}, k_fwd_x<T, N, FWD_SUMS>, PG::THREADS, PG::SMEM_DOT, tb.twp);
    return epi == SPEC_MASK_ADD ? go(std::false_type{}, k_fwd_x<T, N, FWD_MASK>, PG::THREADS, PG::SMEM, tb.twp)
                                : go(std::false_type{}, k_fwd_x<T, N, FWD_STORE>, SG::THREADS, SG::SMEM, tb.twp);
}

}  // namespace ps
