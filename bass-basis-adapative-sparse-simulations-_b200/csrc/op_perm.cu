// op_perm.cu -- the kernels of op.cuh for reorders (the first pass of a 2-qubit gate).
#include "op.cuh"

namespace bass {
template cudaError_t merge_op<K_PERM>(const OpArgs&, cudaStream_t);
template cudaError_t merge_op_seg_t<K_PERM>(const OpArgs*, int, int, int, SegPlan*, cudaStream_t);
template cudaError_t seg_stages_t<K_PERM>(OpArgs*, int, int, int*);
}  // namespace bass
