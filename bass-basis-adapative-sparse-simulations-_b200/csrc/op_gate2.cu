// op_gate2.cu -- the kernels of op.cuh for 2-qubit gates (their second pass).
#include "op.cuh"

namespace bass {
template cudaError_t merge_op<K_GATE2>(const OpArgs&, cudaStream_t);
template cudaError_t merge_op_seg_t<K_GATE2>(const OpArgs*, int, int, int, SegPlan*, cudaStream_t);
template cudaError_t seg_stages_t<K_GATE2>(OpArgs*, int, int, int*);
cudaError_t seg_grid_gate2(int* grid) { return seg_op_grid<K_GATE2, false>(grid); }
}  // namespace bass
