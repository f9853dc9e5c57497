// op_gate2.cu -- the kernels of op.cuh for 2-qubit gates (their second pass).
#include "op.cuh"

namespace bass {
template cudaError_t merge_op<K_GATE2>(const OpArgs&, cudaStream_t);
template cudaError_t merge_op_seg_t<K_GATE2>(const OpArgs*, int, int, SegPlan*, cudaStream_t);
template cudaError_t seg_op_grid<K_GATE2, false>(int*);
}  // namespace bass
