// batch_m7.cu -- batched H.C and density kernels for 7 orbitals
#include "batch_tmpl.cuh"
namespace mctdhb {
template int hcp_batch_launch<7>(const BatchSlot*, const BatchTile*, const BatchTile*, const int*,
                                 int, int, int, bool, cudaStream_t);
template int gram_batch_launch<7>(const BatchSlot*, const BatchTile*, const int*, const int*,
                                  const int*, int, cudaStream_t);
template int batch_prepare<7>();
template int batch_prepare_nowait<7>();
}  // namespace mctdhb
