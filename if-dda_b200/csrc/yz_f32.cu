// F32-complex y passes, zconv and their tile chooser.
#include "yz_impl.cuh"

namespace ifdda {
template <> void launch_yz<float>(const MvArgs<float>& a, int nrhs, cudaStream_t st) { launch_yz_impl<float>(a, nrhs, st); }
template <> void tune_tiles<float>(Green& G, int nrhs, cudaStream_t st) { tune_tiles_impl<float>(G, nrhs, st); }
}  // namespace ifdda
