// op.cu -- the op kinds' dispatch (op.cuh; a file per kind instantiates it).
#include "internal.h"

namespace bass {

template <int KIND>
cudaError_t merge_op(const OpArgs& a, cudaStream_t s);
template <int KIND>
cudaError_t merge_op_seg_t(const OpArgs* ops, int nseg, int c64, int staged, SegPlan* plan, cudaStream_t s);
template <int KIND>
cudaError_t seg_stages_t(OpArgs* ops, int nseg, int slots, int* staged);
cudaError_t seg_grid_gate2(int* grid);

cudaError_t run_merge_op(int kind, OpArgs a, const bass_trunc& tr, int finalize_mode, int j, cudaStream_t s) {
  a.k_cond = tr.k_cond;
  a.k_keep = tr.k_keep;
  a.nsets = 1;
  a.fin_mode = finalize_mode;
  a.tr = tr;
  a.j = j;
  a.prof = prof_on() ? 1 : 0;
  switch (kind) {
    case K_GATE1: return merge_op<K_GATE1>(a, s);
    case K_ROT1: return merge_op<K_ROT1>(a, s);
    case K_GATE2: return merge_op<K_GATE2>(a, s);
    case K_PERM: return merge_op<K_PERM>(a, s);
    case K_IDENT: return merge_op<K_IDENT>(a, s);
  }
  return cudaErrorInvalidValue;
}

// ---- segmented ------------------------------------------------------------------
// One state per SM: a launch could take as many as it has resident blocks (four
// times that), but a state's barriers and chains of loads want several.
cudaError_t seg_max_segments(int* out) {
  int g = 0;
  const cudaError_t e = seg_grid_gate2(&g);
  if (e != cudaSuccess) return e;
  *out = g < device().sms ? g : device().sms;
  return cudaSuccess;
}

cudaError_t seg_stages(int kind, OpArgs* ops, int nseg, int slots, int* staged) {
  if (nseg < 1 || nseg > kMaxSeg) return cudaErrorInvalidValue;
  switch (kind) {
    case K_GATE1: return seg_stages_t<K_GATE1>(ops, nseg, slots, staged);
    case K_ROT1: return seg_stages_t<K_ROT1>(ops, nseg, slots, staged);
    case K_GATE2: return seg_stages_t<K_GATE2>(ops, nseg, slots, staged);
    case K_PERM: return seg_stages_t<K_PERM>(ops, nseg, slots, staged);
    case K_IDENT: return seg_stages_t<K_IDENT>(ops, nseg, slots, staged);
  }
  return cudaErrorInvalidValue;
}

cudaError_t run_merge_op_seg(int kind, const OpArgs* ops, int nseg, int c64, int staged, SegPlan* plan,
                             cudaStream_t s) {
  if (nseg < 1 || nseg > kMaxSeg) return cudaErrorInvalidValue;
  switch (kind) {
    case K_GATE1: return merge_op_seg_t<K_GATE1>(ops, nseg, c64, staged, plan, s);
    case K_ROT1: return merge_op_seg_t<K_ROT1>(ops, nseg, c64, staged, plan, s);
    case K_GATE2: return merge_op_seg_t<K_GATE2>(ops, nseg, c64, staged, plan, s);
    case K_PERM: return merge_op_seg_t<K_PERM>(ops, nseg, c64, staged, plan, s);
    case K_IDENT: return merge_op_seg_t<K_IDENT>(ops, nseg, c64, staged, plan, s);
  }
  return cudaErrorInvalidValue;
}

}  // namespace bass
