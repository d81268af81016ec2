// small_m4.cu -- smallsys.cuh for 4 orbitals.
#include "smallsys.cuh"

namespace mctdhb {
template int small_prepare_tmpl<4>();
template int small_waves_tmpl<4>(int (&)[kClusterSizes]);
template int small_launch_tmpl<4>(const SmallSys&, int, int, cudaStream_t);
template int small_batch_tmpl<4>(const BatchSlot*, const int*, const int*, int, int, int,
                                 cudaStream_t);
}  // namespace mctdhb
