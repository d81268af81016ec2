// small_m2.cu -- smallsys.cuh for 2 orbitals.
#include "smallsys.cuh"

namespace mctdhb {
template int small_prepare_tmpl<2>();
template int small_waves_tmpl<2>(int (&)[kClusterSizes]);
template int small_launch_tmpl<2>(const SmallSys&, int, int, cudaStream_t);
template int small_batch_tmpl<2>(const BatchSlot*, const int*, const int*, int, int, int,
                                 cudaStream_t);
}  // namespace mctdhb
