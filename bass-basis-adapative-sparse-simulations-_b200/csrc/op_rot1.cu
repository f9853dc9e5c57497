// op_rot1.cu -- the kernels of op.cuh for rotation steps.
#include "op.cuh"

namespace bass {
template cudaError_t merge_op<K_ROT1>(const OpArgs&, cudaStream_t);
template cudaError_t merge_op_seg_t<K_ROT1>(const OpArgs*, int, int, int, SegPlan*, cudaStream_t);
template cudaError_t seg_stages_t<K_ROT1>(OpArgs*, int, int, int*);
}  // namespace bass
