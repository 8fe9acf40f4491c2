// Launches of the y passes and of zconv, dispatched on the FFT length, and the
// tile chooser that times their shapes.  Included by one translation unit per
// precision (the x passes, instantiated per solver step, have their own).
#pragma once
#include "engine.cuh"

namespace ifdda {

template <class T, int L, int DIR, int V> void launch_pass_y_v(const MvArgs<T>& a, int nrhs, cudaStream_t st) {
    using TT = MvTiles<T, L, V>;
    dim3 grid((a.g.X * TT::S / TT::SE + TT::TLY - 1) / TT::TLY, a.g.nz, 3 * nrhs);
    PassScope ps(DIR > 0 ? PASS_FWD_Y : PASS_INV_Y, TT::S, st);
    ensure_smem(k_pass_y<T, L, DIR, TT>, TT::smem_y);
    launch_pdl(k_pass_y<T, L, DIR, TT>, grid, TT::NTY, TT::smem_y, st, a);
}
template <class T, int L, int DIR> void launch_pass_y(const MvArgs<T>& a, int nrhs, cudaStream_t st) {
    if constexpr (tile_variants(L) > 1) {
        if (a.yvar == 1) return launch_pass_y_v<T, L, DIR, 1>(a, nrhs, st);
    }
    launch_pass_y_v<T, L, DIR, 0>(a, nrhs, st);
}

template <class T, int L, int V> void launch_zconv_v(const MvArgs<T>& a, int nrhs, cudaStream_t st) {
    using TT = MvTiles<T, L, V>;
    dim3 grid(2 * nrhs, (a.g.X * TT::S / TT::SE + TT::TLZ - 1) / TT::TLZ, a.g.ny + 1);
    PassScope ps(PASS_ZCONV, TT::S, st);
    ensure_smem(k_zconv<T, L, TT>, TT::smem_z);
    launch_pdl(k_zconv<T, L, TT>, grid, TT::NTZ, TT::smem_z, st, a);
}
template <class T, int L> void launch_zconv(const MvArgs<T>& a, int nrhs, cudaStream_t st) {
    if constexpr (tile_variants(L) > 1) {
        if (a.zvar == 1) return launch_zconv_v<T, L, 1>(a, nrhs, st);
    }
    launch_zconv_v<T, L, 0>(a, nrhs, st);
}

#define IFDDA_CASE_FWDY(L) \
    case L: launch_pass_y<T, L, +1>(a, nrhs, st); break;
#define IFDDA_CASE_INVY(L) \
    case L: launch_pass_y<T, L, -1>(a, nrhs, st); break;
#define IFDDA_CASE_ZC(L) \
    case L: launch_zconv<T, L>(a, nrhs, st); break;

// passes 2 to 4 of the mat-vec (every length is supported: the caller checked)
template <class T> void launch_yz_impl(const MvArgs<T>& a, int nrhs, cudaStream_t st) {
    switch (a.g.Y) { IFDDA_FFT_LENGTHS(IFDDA_CASE_FWDY) default: break; }
    switch (a.g.Z) { IFDDA_FFT_LENGTHS(IFDDA_CASE_ZC) default: break; }
    switch (a.g.Y) { IFDDA_FFT_LENGTHS(IFDDA_CASE_INVY) default: break; }
}

#define IFDDA_CASE_TY(L) \
    case L: launch_pass_y<T, L, +1>(a, nrhs, st); launch_pass_y<T, L, -1>(a, nrhs, st); break;
#define IFDDA_CASE_TZ(L) \
    case L: launch_zconv<T, L>(a, nrhs, st); break;

// Tile chooser: with G's mat-vec scratch for nrhs right-hand sides (whose
// contents are about to be overwritten by the next mat-vec anyway), time each
// tile variant of the y passes (forward then inverse) and of zconv, best of
// three launches with CUDA events on st, and record the choice for G's grid,
// device and precision (tile_put: every spectrum and batch size on that grid
// then uses it).  Variant 0 is the one to beat by 5%, so that timing noise
// between near-equal shapes does not flip the choice; where a row does not
// half fill its tile (nx up to 8 in the y passes, 4 in zconv, in FP32; half
// that in FP64), variant 1 is (products of 1x64x64 in FP32 13.3 -> 12.6 us,
// 2x64x64 in FP64 15.9 -> 12.7).  Never runs while st is being captured.
template <class T> void tune_tiles_impl(Green& G, int nrhs, cudaStream_t st) {
    const int pk = sizeof(T) == 4 ? 1 : 0;
    TileChoice have;
    if (G.tile_choice<T>(have)) return;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    IFDDA_CUDA(cudaStreamIsCapturing(st, &cs));
    if (cs != cudaStreamCaptureStatusNone) return;
    MvArgs<T> a = mv_args<T>(G, nrhs, nullptr, nullptr, nullptr, 0, ALPHA_NONE, nullptr, 0, nullptr, nullptr);
    TileChoice tc{};
    const int nyv = tile_variants(G.g.Y), nzv = tile_variants(G.g.Z);
    const int columns = G.g.X * (int)sizeof(cplx<T>) / (int)sizeof(typename yz_elem<T>::type);
    tc.yvar = nyv > 1 && columns <= 8 ? 1 : 0;
    tc.zvar = nzv > 1 && G.g.Z < 160 && columns <= 4 ? 1 : 0;
    if (nyv > 1 || nzv > 1) {
        cudaEvent_t e0, e1;
        IFDDA_CUDA(cudaEventCreate(&e0));
        IFDDA_CUDA(cudaEventCreate(&e1));
        auto time_it = [&](auto&& launch) {
            float best = 1e30f;
            for (int r = 0; r < 4; r++) {
                IFDDA_CUDA(cudaEventRecord(e0, st));
                launch();
                IFDDA_CUDA(cudaEventRecord(e1, st));
                IFDDA_CUDA(cudaEventSynchronize(e1));
                float ms = 0;
                IFDDA_CUDA(cudaEventElapsedTime(&ms, e0, e1));
                if (r > 0) best = ms < best ? ms : best;  // the first launch sets up the kernel
            }
            return best;
        };
        for (int v = 0; v < nyv; v++) {
            a.yvar = v;
            tc.y_ms[v] = time_it([&] {
                switch (G.g.Y) { IFDDA_FFT_LENGTHS(IFDDA_CASE_TY) default: break; }
            });
        }
        if (nyv > 1 && tc.y_ms[1 - tc.yvar] < 0.95f * tc.y_ms[tc.yvar]) tc.yvar = 1 - tc.yvar;
        for (int v = 0; v < nzv; v++) {
            a.zvar = v;
            tc.z_ms[v] = time_it([&] {
                switch (G.g.Z) { IFDDA_FFT_LENGTHS(IFDDA_CASE_TZ) default: break; }
            });
        }
        if (nzv > 1 && tc.z_ms[1 - tc.zvar] < 0.95f * tc.z_ms[tc.zvar]) tc.zvar = 1 - tc.zvar;
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
    }
    tile_put(G.device, pk, G.g, tc);
}

}  // namespace ifdda
