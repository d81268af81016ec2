// small_m8.cu -- smallsys.cuh for 8 orbitals.
#include "smallsys.cuh"

namespace mctdhb {
template int small_prepare_tmpl<8>();
template int small_waves_tmpl<8>(int (&)[kClusterSizes]);
template int small_launch_tmpl<8>(const SmallSys&, int, int, cudaStream_t);
template int small_batch_tmpl<8>(const BatchSlot*, const int*, const int*, int, int, int,
                                 cudaStream_t);
}  // namespace mctdhb
