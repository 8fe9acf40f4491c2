// Launch wrappers for the mat-vec passes, dispatched on the FFT length of each
// axis.  Included by one translation unit per precision.
#pragma once
#include "engine.cuh"

namespace ifdda {

template <class T, int L, class Pre>
void launch_fwd_x(const MvArgs<T>& a, const Pre& pre, const MvRed& red, int nrhs, bool tab, cudaStream_t st) {
    using TT = MvTiles<T, L>;
    dim3 grid((a.g.ny + TT::TLX - 1) / TT::TLX, a.g.nz, nrhs);
    PassScope ps(PASS_FWD_X, TT::S, st);
    if (tab) {
        ensure_smem(k_fwd_x<T, L, true, TT, Pre>, TT::smem_x);
        launch_pdl(k_fwd_x<T, L, true, TT, Pre>, grid, TT::NTX, TT::smem_x, st, a, pre, red);
    } else {
        ensure_smem(k_fwd_x<T, L, false, TT, Pre>, TT::smem_x);
        launch_pdl(k_fwd_x<T, L, false, TT, Pre>, grid, TT::NTX, TT::smem_x, st, a, pre, red);
    }
}

template <class T, int L, class Epi>
void launch_inv_x(const MvArgs<T>& a, const Epi& epi, const MvRed& red, int nrhs, bool tab, cudaStream_t st) {
    using TT = MvTiles<T, L>;
    dim3 grid((a.g.ny + TT::TLX - 1) / TT::TLX, a.g.nz, nrhs);
    PassScope ps(PASS_INV_X, TT::S, st);
    if (tab) {
        ensure_smem(k_inv_x<T, L, true, Epi, TT>, TT::smem_x);
        launch_pdl(k_inv_x<T, L, true, Epi, TT>, grid, TT::NTX, TT::smem_x, st, a, epi, red);
    } else {
        ensure_smem(k_inv_x<T, L, false, Epi, TT>, TT::smem_x);
        launch_pdl(k_inv_x<T, L, false, Epi, TT>, grid, TT::NTX, TT::smem_x, st, a, epi, red);
    }
}

#define IFDDA_CASE_FWDX(L) \
    case L: launch_fwd_x<T, L, Pre>(a, pre, red, nrhs, tab, st); break;
#define IFDDA_CASE_INVX(L) \
    case L: launch_inv_x<T, L, Epi>(a, epi, red, nrhs, tab, st); break;

// The five passes with a solver's input functor (first x pass) and output
// functor (last x pass); red holds their reduction buffers.
template <class T, class Pre, class Epi>
bool matvec_launch_fused(const MvArgs<T>& a, const Pre& pre, const Epi& epi, const MvRed& red, int nrhs, bool tab,
                         cudaStream_t st) {
    if (!fft_length_supported(a.g.X) || !fft_length_supported(a.g.Y) || !fft_length_supported(a.g.Z)) return false;
    switch (a.g.X) { IFDDA_FFT_LENGTHS(IFDDA_CASE_FWDX) default: return false; }
    IFDDA_CUDA(cudaGetLastError());
    launch_yz<T>(a, nrhs, st);
    switch (a.g.X) { IFDDA_FFT_LENGTHS(IFDDA_CASE_INVX) default: return false; }
    IFDDA_CUDA(cudaGetLastError());
    return true;
}

}  // namespace ifdda
