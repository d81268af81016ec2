// small_m5.cu -- smallsys.cuh for 5 orbitals.
#include "smallsys.cuh"

namespace mctdhb {
template int small_prepare_tmpl<5>();
template int small_waves_tmpl<5>(int (&)[kClusterSizes]);
template int small_launch_tmpl<5>(const SmallSys&, int, int, cudaStream_t);
template int small_batch_tmpl<5>(const BatchSlot*, const int*, const int*, int, int, int,
                                 cudaStream_t);
}  // namespace mctdhb
