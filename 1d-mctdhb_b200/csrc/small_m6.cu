// small_m6.cu -- smallsys.cuh for 6 orbitals.
#include "smallsys.cuh"

namespace mctdhb {
template int small_prepare_tmpl<6>();
template int small_waves_tmpl<6>(int (&)[kClusterSizes]);
template int small_launch_tmpl<6>(const SmallSys&, int, int, cudaStream_t);
template int small_batch_tmpl<6>(const BatchSlot*, const int*, const int*, int, int, int,
                                 cudaStream_t);
}  // namespace mctdhb
