// F64-complex mat-vecs with GPBiCG's steps in their x passes.
#include "mv_impl.cuh"
#include "gpbicg_fused.cuh"

namespace ifdda {
template bool matvec_launch_fused<double, PreGpP<double>, EpiGpAlpha<double>>(const MvArgs<double>&, const PreGpP<double>&,
                                                                   const EpiGpAlpha<double>&, const MvRed&, int,
                                                                   bool, cudaStream_t);
template bool matvec_launch_fused<double, PreGpYT<double>, EpiGpZeta<double>>(const MvArgs<double>&, const PreGpYT<double>&,
                                                                   const EpiGpZeta<double>&, const MvRed&, int,
                                                                   bool, cudaStream_t);
}  // namespace ifdda
