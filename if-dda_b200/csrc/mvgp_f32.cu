// F32-complex mat-vecs with GPBiCG's steps in their x passes.
#include "mv_impl.cuh"
#include "gpbicg_fused.cuh"

namespace ifdda {
template bool matvec_launch_fused<float, PreGpP<float>, EpiGpAlpha<float>>(const MvArgs<float>&, const PreGpP<float>&,
                                                                   const EpiGpAlpha<float>&, const MvRed&, int,
                                                                   bool, cudaStream_t);
template bool matvec_launch_fused<float, PreGpYT<float>, EpiGpZeta<float>>(const MvArgs<float>&, const PreGpYT<float>&,
                                                                   const EpiGpZeta<float>&, const MvRed&, int,
                                                                   bool, cudaStream_t);
}  // namespace ifdda
