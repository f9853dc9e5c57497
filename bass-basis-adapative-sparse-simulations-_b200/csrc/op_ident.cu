// op_ident.cu -- the kernels of op.cuh for truncations.
#include "op.cuh"

namespace bass {
template cudaError_t merge_op<K_IDENT>(const OpArgs&, cudaStream_t);
template cudaError_t merge_op_seg_t<K_IDENT>(const OpArgs*, int, int, int, SegPlan*, cudaStream_t);
template cudaError_t seg_stages_t<K_IDENT>(OpArgs*, int, int, int*);
}  // namespace bass
