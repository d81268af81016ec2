// small_m3.cu -- smallsys.cuh for 3 orbitals.
#include "smallsys.cuh"

namespace mctdhb {
template int small_prepare_tmpl<3>();
template int small_waves_tmpl<3>(int (&)[kClusterSizes]);
template int small_launch_tmpl<3>(const SmallSys&, int, int, cudaStream_t);
template int small_batch_tmpl<3>(const BatchSlot*, const int*, const int*, int, int, int,
                                 cudaStream_t);
}  // namespace mctdhb
