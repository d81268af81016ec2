// small_m7.cu -- smallsys.cuh for 7 orbitals.
#include "smallsys.cuh"

namespace mctdhb {
template int small_prepare_tmpl<7>();
template int small_waves_tmpl<7>(int (&)[kClusterSizes]);
template int small_launch_tmpl<7>(const SmallSys&, int, int, cudaStream_t);
template int small_batch_tmpl<7>(const BatchSlot*, const int*, const int*, int, int, int,
                                 cudaStream_t);
}  // namespace mctdhb
