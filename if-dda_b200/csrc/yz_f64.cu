// F64-complex y passes, zconv and their tile chooser.
#include "yz_impl.cuh"

namespace ifdda {
template <> void launch_yz<double>(const MvArgs<double>& a, int nrhs, cudaStream_t st) { launch_yz_impl<double>(a, nrhs, st); }
template <> void tune_tiles<double>(Green& G, int nrhs, cudaStream_t st) { tune_tiles_impl<double>(G, nrhs, st); }
}  // namespace ifdda
