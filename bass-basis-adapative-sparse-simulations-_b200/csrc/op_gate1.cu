// op_gate1.cu -- the kernels of op.cuh for 1-qubit gates.
#include "op.cuh"

namespace bass {
template cudaError_t merge_op<K_GATE1>(const OpArgs&, cudaStream_t);
template cudaError_t merge_op_seg_t<K_GATE1>(const OpArgs*, int, int, int, SegPlan*, cudaStream_t);
template cudaError_t seg_stages_t<K_GATE1>(OpArgs*, int, int, int*);
}  // namespace bass
