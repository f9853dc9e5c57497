// merge.cu -- the RDM moment passes and the guarded compaction of diagonal
// 1-qubit gates, on the tiles of tile.cuh:
//
//   k_partition   one warp per tile boundary and qubit;
//   k_tile        loads a tile, merges it into Z order and sums the moments of
//                 its groups (one qubit, or the 4x4 moments of a pair), or
//                 compacts a state whose amplitudes a diagonal gate zeroed;
//   k_rdm_low     the moments of the qubits at low physical bits, in one pass.
#include <math.h>

#include "tile.cuh"

namespace bass {

// ---------------------------------------------------------------------------
// partition
// ---------------------------------------------------------------------------
// The small workspace region (tile counters, histograms, SelState, look-back
// status words: what zero_small clears), zeroed by a group.
__device__ __forceinline__ void zero_op_region(const OpArgs& a, Grp g) {
  unsigned long long* zp = reinterpret_cast<unsigned long long*>(a.ws.counters);
  const long long nw =
      (long long)((reinterpret_cast<const char*>(a.ws.status + a.ws.max_tiles) - reinterpret_cast<const char*>(zp)) / 8);
  for (long long i = (long long)g.bid * blockDim.x + threadIdx.x; i < nw; i += (long long)g.nblk * blockDim.x)
    zp[i] = 0ULL;
}

// zero: also clear the op's small workspace region; nothing here reads it, and
// the kernels after the partition find it zeroed.
__device__ __forceinline__ void partition_body(const OpArgs& a, int kind, int zero, int set, Grp g) {
  if (zero && set == 0) zero_op_region(a, g);
  const bass_state* in = a.in;
  const long long n = in->nnz;
  const int q = (kind == K_RDM) ? set : a.q;
  const int t = in->pos[q];
  if (kind == K_RDM && a.rdm_low && t < kRdmLowBits) return;  // paired by k_rdm_low
  const long long ntiles = merge_tiles(n);
  long long* recs = a.ws.part + (long long)set * (a.ws.max_tiles + 1) * 6;
  const int lane = threadIdx.x & 31;
  const long long warp = ((long long)g.bid * blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = ((long long)g.nblk * blockDim.x) >> 5;
  if (ntiles + 1 > a.ws.max_tiles + 1) {
    if (warp == 0 && lane == 0) set_error(a.ctrl, BASS_ERR_WORKSPACE);
    return;
  }
  for (long long b = warp; b <= ntiles; b += nwarps) {
    long long r[6];
    if (kind == K_GATE2) tile_boundary<1>(in->keys, n, b * kStep, t, true, r);
    else tile_boundary<0>(in->keys, n, b * kStep, t, true, r);
    if (lane == 0) {
      long long* o = recs + b * 6;
      for (int k = 0; k < 6; ++k) o[k] = r[k];
    }
  }
  pdl_trigger();
}

__global__ void k_partition(const __grid_constant__ OpArgs a, int kind, int zero) {
  pdl_wait();
  partition_body(a, kind, zero, blockIdx.y, whole_grid());
}

// ---------------------------------------------------------------------------
// block scan
// ---------------------------------------------------------------------------
__device__ __forceinline__ int block_excl_scan(int v, int* sWarp, int* total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  int x = v;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    int y = __shfl_up_sync(0xffffffffu, x, off);
    if (lane >= off) x += y;
  }
  if (lane == 31) sWarp[w] = x;
  __syncthreads();
  if (w == 0) {
    int s = (lane < nw) ? sWarp[lane] : 0;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      int y = __shfl_up_sync(0xffffffffu, s, off);
      if (lane >= off) s += y;
    }
    if (lane < nw) sWarp[lane] = s;
  }
  __syncthreads();
  int excl = x - v + (w > 0 ? sWarp[w - 1] : 0);
  *total = sWarp[nw - 1];
  __syncthreads();
  return excl;
}

// The selection state into shared memory, one 8-byte word per thread (the
// caller synchronises before reading it).
__device__ __forceinline__ void load_sel(SelState* dst, const SelState* src) {
  constexpr int kWords = (int)(sizeof(SelState) / 8);
  static_assert(sizeof(SelState) % 8 == 0, "selection state words");
  if ((int)threadIdx.x < kWords)
    reinterpret_cast<unsigned long long*>(dst)[threadIdx.x] =
        __ldcg(reinterpret_cast<const unsigned long long*>(src) + threadIdx.x);
}

// ---------------------------------------------------------------------------
// the tile kernel
// ---------------------------------------------------------------------------
// Passes: P_RDM (moments per qubit, or of a qubit pair), P_WRITE (the
// compaction after a diagonal 1-qubit gate, K_IDENT: the entries the drop rule
// keeps, based by a decoupled look-back).
template <int KIND, int PASS, bool C64>
__device__ __forceinline__ void tile_body(const OpArgs& a, Grp g) {
  extern __shared__ __align__(16) unsigned char smem[];
  double2* sA = reinterpret_cast<double2*>(smem);
  uint64_t* sZ = reinterpret_cast<uint64_t*>(sA + kTilePad);
  uint16_t* sIdx = reinterpret_cast<uint16_t*>(sZ + kTilePad);
  // write pass only: per-position offsets and kept masks
  uint16_t* sOff = sIdx + kTilePad;
  uint8_t* sMask = reinterpret_cast<uint8_t*>(sOff + kTilePad);
  __shared__ SelState Sel;
  __shared__ TileSeg T;
  __shared__ long long sItem, sBase;
  __shared__ uint64_t sBar;  // completion of the tile's bulk copies
  __shared__ int sWarp[32];
  __shared__ i128 sRed[4 * (kThreads / 32)];

  const int tid = threadIdx.x;
  if (PASS == P_WRITE) load_sel(&Sel, a.ws.sel);
  if (tid == 0) mbar_init(&sBar, 1);
  __syncthreads();
  if (PASS == P_WRITE && a.guard && Sel.pad == 0) return;

  const bass_state* in = a.in;
  TileSrc S;
  S.keys = in->keys;
  S.amps = reinterpret_cast<const double2*>(in->amps);
  S.n = in->nnz;
  // bulk copies need 16-byte aligned arrays (every allocation of this library
  // is; a caller's arrays at an 8-byte offset take the per-entry copies)
  S.tma = ((reinterpret_cast<uintptr_t>(S.keys) | reinterpret_cast<uintptr_t>(S.amps)) & 15) == 0;
  const double r0 = in->rscale[0], r1 = in->rscale[1];
  const bool wrong_type = (in->amp_type == BASS_AMP_C64) != C64;  // launched for the other amplitude type
  const long long ntiles = (KIND == K_IDENT) ? plain_tiles(S.n) : merge_tiles(S.n);
  const bool bad = ntiles > a.ws.max_tiles || wrong_type;
  if (bad && g.bid == 0 && tid == 0) {
    if (wrong_type) set_error(a.ctrl, BASS_ERR_ARG);
    set_error(a.ctrl, BASS_ERR_WORKSPACE);
  }
  if (bad) return;
  unsigned phase = 0;  // parity of sBar's current phase
  const bool scaled = !(r0 == 1.0 && r1 == 1.0);
  // P_RDM: items are (set, tile); K_RDM sets are qubits, the 4x4 moments of
  // a qubit pair (K_GATE2) split into a.nsets = 4 sets of four values that
  // share one partition
  // P_RDM of K_RDM with rdm_low: the items cover only the sets whose qubit
  // sits at physical bit kRdmLowBits or above (sHigh, the same list in every
  // CTA); k_rdm_low does the others
  __shared__ int8_t sHigh[64];
  __shared__ int sNHigh;
  if (PASS == P_RDM && tid == 0) {
    int nh = 0;
    for (int s2 = 0; s2 < a.nsets && s2 < 64; ++s2)
      if (!(KIND == K_RDM && a.rdm_low && in->pos[a.q + s2] < kRdmLowBits)) sHigh[nh++] = (int8_t)s2;
    sNHigh = nh;
  }
  __syncthreads();
  const long long nitems = (PASS == P_RDM) ? ntiles * sNHigh : ntiles;

  for (;;) {
    if (tid == 0) sItem = (long long)atomicAdd(&reinterpret_cast<unsigned long long*>(a.ws.counters)[a.counter], 1ULL);
    __syncthreads();
    const long long item = sItem;
    if (item >= nitems) break;
    const int set = (PASS == P_RDM) ? (int)sHigh[item / ntiles] : 0;
    const long long tile = (PASS == P_RDM) ? item % ntiles : item;
    const int t = (KIND == K_RDM) ? in->pos[a.q + set] : KIND == K_IDENT ? 0 : in->pos[a.q];
    const int pset = (KIND == K_RDM) ? set : 0;  // the partition records this item reads
    if (tid == 0) {
      if (KIND == K_IDENT) {
        const long long lo = tile * kTile, hi = lo + kTile < S.n ? lo + kTile : S.n;
        const long long rc[6] = {lo, 0, S.n, S.n, lo, 0}, rn[6] = {hi, 0, S.n, S.n, hi, 0};
        tile_segments<C64>(T, rc, rn, S, kTile, sZ, sA, &sBar, a.ctrl);
      } else {
        const long long* rc = a.ws.part + ((long long)pset * (a.ws.max_tiles + 1) + tile) * 6;
        tile_segments<C64>(T, rc, rc + 6, S, kTile, sZ, sA, &sBar, a.ctrl);
      }
      if (a.prof) atomicAdd(reinterpret_cast<unsigned long long*>(&a.ctrl->prof_in[KIND * 5 + PASS]),
                            (unsigned long long)T.off[5]);
    }
    __syncthreads();
    const int E = (int)T.off[5];
    if (!tile_fetch<kPerThread, C64>(T, S, sZ, sA, &sBar, &phase, a.ctrl, wait_limit(a.ctrl))) break;
    if (KIND != K_IDENT) tile_zorder<kPerThread, group_bit(KIND)>(T, sZ, sIdx, sWarp, t);
    const TileView V{sZ, sA, reinterpret_cast<const float2*>(sA), KIND == K_IDENT ? nullptr : sIdx, r0, r1, scaled, C64};

    // ---- evaluate ------------------------------------------------------------
    // Round r gives position r * kThreads + tid to thread tid, so neighbouring
    // threads handle neighbouring groups.
    if (PASS == P_RDM && KIND == K_GATE2) {
      // 4x4 moments of the pair (q1 at bit 1, q2 at bit 0 after the first
      // pass): per group of up to four entries a_i (i = (b_q1 << 1) | b_q2),
      // set 0: |a_0|^2 .. |a_3|^2; set 1: Re/Im a_0 conj(a_1), a_0 conj(a_2);
      // set 2: a_0 conj(a_3), a_1 conj(a_2); set 3: a_1 conj(a_3), a_2 conj(a_3)
      // (bass_simulator.py:200-231, rho[p][q] += a_p conj(a_q)).
      i128 v[4] = {0, 0, 0, 0};
      double dh[4] = {0.0, 0.0, 0.0, 0.0}, dl[4] = {0.0, 0.0, 0.0, 0.0};
      for (int p = tid; p < E; p += kThreads) {
        unsigned w = V.word(p);
        if (!(w & kPlaceStart)) continue;
        const double2 zero = make_double2(0.0, 0.0);
        double2 g0 = zero, g1 = zero, g2 = zero, g3 = zero;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const double2 v2 = V.amp_at((int)(w & kPlaceMask));
          const unsigned i = (w >> kPlaceLocal) & 3u;
          if (i == 0) g0 = v2;
          else if (i == 1) g1 = v2;
          else if (i == 2) g2 = v2;
          else g3 = v2;
          if (!(w & kPlaceNext)) break;
          w = V.word(p + r + 1);
        }
        double m[4];
        if (set == 0) {
          m[0] = prob(g0); m[1] = prob(g1); m[2] = prob(g2); m[3] = prob(g3);
        } else {
          // the set's two pairs (i, j), i < j: a_i conj(a_j)
          const double2 ai = set == 3 ? g1 : g0, aj = set == 1 ? g1 : g3;
          const double2 bi = set == 1 ? g0 : set == 2 ? g1 : g2, bj = set == 3 ? g3 : g2;
          const double2 c0 = cmul(ai, make_double2(aj.x, -aj.y));
          const double2 c1 = cmul(bi, make_double2(bj.x, -bj.y));
          m[0] = c0.x; m[1] = c0.y; m[2] = c1.x; m[3] = c1.y;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) fx_acc96(m[k], dh[k], dl[k], v[k]);
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) v[k] += fx_join96s(dh[k], dl[k]);
      block_sum_i128<4>(v, sRed);
      if (tid == 0) {
        Partial* pt = a.ws.partials + (long long)set * a.ws.max_tiles + tile;
        pt->s[0] = v[0]; pt->s[1] = v[1]; pt->s[2] = v[2]; pt->s[3] = v[3];
      }
    } else if (PASS == P_RDM) {
      // at most kPerThread positions per thread, so at most eight terms per
      // split accumulator (fx_acc96) before they are joined
      i128 v[4] = {0, 0, 0, 0};
      double dh[4] = {0.0, 0.0, 0.0, 0.0}, dl[4] = {0.0, 0.0, 0.0, 0.0};
      for (int p = tid; p < E; p += kThreads) {
        const unsigned w = V.word(p);
        if (!(w & kPlaceStart)) continue;
        const double2 x0 = V.amp_at((int)(w & kPlaceMask));
        if (((w >> kPlaceLocal) & 1u) == 0) {
          fx_acc96(prob(x0), dh[0], dl[0], v[0]);
          if (w & kPlaceNext) {
            const double2 x1 = V.amp(p + 1);
            fx_acc96(prob(x1), dh[1], dl[1], v[1]);
            const double2 c = cmul(x0, make_double2(x1.x, -x1.y));
            fx_acc96(c.x, dh[2], dl[2], v[2]);
            fx_acc96(c.y, dh[3], dl[3], v[3]);
          }
        } else {
          fx_acc96(prob(x0), dh[1], dl[1], v[1]);
        }
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) v[k] += fx_join96s(dh[k], dl[k]);
      block_sum_i128<4>(v, sRed);
      if (tid == 0) {
        Partial* pt = a.ws.partials + (long long)set * a.ws.max_tiles + tile;
        pt->s[0] = v[0]; pt->s[1] = v[1]; pt->s[2] = v[2]; pt->s[3] = v[3];
      }
    } else if (PASS == P_WRITE) {
      double2 ca[1];
      // (a) the entries the drop rule keeps
      for (int p = tid; p < E; p += kThreads) {
        const unsigned mk = group_children_t<KIND>(C64, p, V, a.G, a.drop_zero, ca) & 1u;
        sMask[p] = (uint8_t)mk;
        sOff[p] = (uint16_t)mk;
      }
      __syncthreads();
      // (b) counts -> exclusive offsets in place (position order)
      const int base_e = tid * kPerThread;
      int run = 0;
#pragma unroll
      for (int k = 0; k < kPerThread; ++k)
        if (base_e + k < E) run += sOff[base_e + k];
      int tile_total;
      int ex = block_excl_scan(run, sWarp, &tile_total);
#pragma unroll
      for (int k = 0; k < kPerThread; ++k) {
        const int p = base_e + k;
        if (p < E) {
          const int c = sOff[p];
          sOff[p] = (uint16_t)ex;
          ex += c;
        }
      }
      // (c) the tile's base in the output
      if (tid < 32) {
        const long long b = lookback_warp(a.ws.status, tile, tile_total, a.ctrl);
        if (tid == 0) sBase = b;
      }
      __syncthreads();
      if (tid == 0) {
        const long long b = sBase;
        if (tile == ntiles - 1) a.ws.sel->n_written = b + tile_total;
        if (b + tile_total > a.out->cap) set_error(a.ctrl, BASS_ERR_CAPACITY);
        if (a.prof) atomicAdd(reinterpret_cast<unsigned long long*>(&a.ctrl->prof_out[KIND * 5 + PASS]),
                              (unsigned long long)tile_total);
      }
      // (d) write the kept entries
      if (sBase + tile_total <= a.out->cap) {
        for (int p = tid; p < E; p += kThreads) {
          if (!sMask[p]) continue;
          const long long o = sBase + sOff[p];
          a.out->keys[o] = V.key(p);
          amp_put(a.out->amps, o, V.amp(p), C64);
        }
      }
    }
    __syncthreads();
  }
  pdl_trigger();
}

// The tile pass of one op on a state of complex64 (C64) or complex128 amplitudes.
template <int KIND, int PASS, bool C64>
__global__ void __launch_bounds__(kThreads, 4) k_tile(const __grid_constant__ OpArgs a) {
  pdl_wait();
  tile_body<KIND, PASS, C64>(a, whole_grid());
}

// Bulk copy of entries [lo, hi) of an array of `esz`-byte entries (esz 8 or
// 16) into shared memory at position (index - (lo & ~1)), so that both ends
// are 16-byte aligned (body_bytes: the bytes it copies).  For 8-byte entries
// the ragged entries lo (odd) and hi - 1 (even) are left to copy_ragged.
__device__ __forceinline__ unsigned body_bytes(long long lo, long long hi, unsigned esz) {
  const long long f = esz == 16 ? lo : (lo + 1) & ~1LL;
  const long long l = esz == 16 ? hi : hi & ~1LL;
  return (hi <= lo || l <= f) ? 0u : (unsigned)(esz * (l - f));
}
__device__ __forceinline__ void copy_body(void* dst, const void* src, long long lo, long long hi, unsigned esz,
                                          uint64_t* bar) {
  const unsigned nb = body_bytes(lo, hi, esz);
  if (nb == 0) return;
  const long long f = esz == 16 ? lo : (lo + 1) & ~1LL;
  const long long e0 = lo & ~1LL;
  bulk_load(static_cast<unsigned char*>(dst) + esz * (f - e0), static_cast<const unsigned char*>(src) + esz * f, nb,
            bar);
}
// The entry of [lo, hi) that copy_body leaves out at its start (last = false)
// or end (last = true), if any, by a plain load.
template <typename E>
__device__ __forceinline__ void copy_ragged(E* dst, const E* src, long long lo, long long hi, bool last) {
  if (sizeof(E) == 16 || hi <= lo) return;
  const long long f = (lo + 1) & ~1LL, l = hi & ~1LL, e0 = lo & ~1LL;
  if (last ? l < hi : lo < f) {
    const long long i = last ? l : lo;
    dst[i - e0] = src[i];
  }
}

// ---------------------------------------------------------------------------
// RDM moments of the qubits at low physical bits: one pass
// ---------------------------------------------------------------------------
// bass_simulator.py:441-470 for every qubit whose physical bit t is below
// kRdmLowBits, without a merge pass per qubit: the state is read in plain
// tiles of kTile entries (key order) plus the next kRdmHalo entries, which
// hold the partner x | 2^t of every tile entry x with bit t clear (the keys
// between x and x + 2^t are distinct integers, so at most 2^t - 1 of them
// come first); a binary search over at most 2^t positions finds it.  The four
// moments of each such qubit (|a|^2 of its bit-0 and bit-1 entries, re and im
// of a_x conj(a_{x | 2^t})) are the sums of k_tile's P_RDM pass, exact:
// each warp adds its lanes' sums into its own shared accumulators, and at the
// end every CTA adds its sums to the qubits' limbs (rdm_limbs; the workspace
// clear zeroed them).  Small states take smaller tiles, so that every CTA of the
// grid has one: what bounds them is the chain of one tile (16,384 entries of 40
// qubits: 27 us instead of 68 with tiles of kTile).
constexpr int kRdmSpan = kTile + kRdmHalo;
constexpr int kRdmSpanPad = kRdmSpan + 2;
constexpr size_t kRdmLowSmem = (size_t)kRdmSpanPad * (16 + 8);  // amplitudes, keys

// The low-bit pass's sums: four moments of four limbs per qubit, in ws.hist1.
__device__ __forceinline__ unsigned long long* rdm_limbs(const WsView& ws, int set) {
  return reinterpret_cast<unsigned long long*>(ws.hist1) + 16 * set;
}
static_assert(kMaxSets * 16 * 8 <= kHistBins * 4, "the limbs fit the histogram");

template <bool C64>
__global__ void __launch_bounds__(kThreads) k_rdm_low(const __grid_constant__ OpArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  double2* sA = reinterpret_cast<double2*>(smem);
  float2* sAf = reinterpret_cast<float2*>(sA);
  uint64_t* sK = reinterpret_cast<uint64_t*>(sA + kRdmSpanPad);
  __shared__ uint64_t sBar;
  __shared__ long long sItem;
  __shared__ i128 sAcc[kThreads / 32][kRdmLowBits][4];  // per warp, qubit and moment
  __shared__ int sSet[kRdmLowBits];  // the set of the qubit at physical bit t, or -1
  pdl_wait();
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  for (int i = lane; i < kRdmLowBits * 4; i += 32) sAcc[w][i >> 2][i & 3] = 0;
  const bass_state* in = a.in;
  const long long n = in->nnz;
  long long span = (n + gridDim.x - 1) / gridDim.x;  // entries of a tile: a multiple of kThreads
  span = span > kTile - kThreads ? kTile : (span + kThreads - 1) / kThreads * kThreads;
  if (span == 0) span = kThreads;
  const long long ntiles = (n + span - 1) / span;
  if (tid == 0) mbar_init(&sBar, 1);
  if (tid < kRdmLowBits) {
    int set = -1;
    if (tid < in->nq) {
      const int q = in->qat[tid] - a.q;
      if (q >= 0 && q < a.nsets) set = q;
    }
    sSet[tid] = set;
  }
  const double r0 = in->rscale[0], r1 = in->rscale[1];
  const bool scaled = !(r0 == 1.0 && r1 == 1.0);
  const uint64_t* keys = in->keys;
  const double2* amps = reinterpret_cast<const double2*>(in->amps);
  const float2* ampf = reinterpret_cast<const float2*>(in->amps);
  // bulk copies need both arrays 16-byte aligned; keys at an 8-byte offset
  // take plain loads
  const bool bulk = ((reinterpret_cast<uintptr_t>(keys) | reinterpret_cast<uintptr_t>(amps)) & 15) == 0;
  const bool bad = plain_tiles(n) > a.ws.max_tiles || (in->amp_type == BASS_AMP_C64) != C64;
  if (bad && blockIdx.x == 0 && tid == 0) set_error(a.ctrl, BASS_ERR_WORKSPACE);
  auto amp = [&](int p) {
    const double2 v = C64 ? f2d(sAf[p]) : sA[p];
    return scaled ? amp_scale(v, C64 ? 1 : 0, r0, r1) : v;
  };
  const long long lim = wait_limit(a.ctrl);
  __syncthreads();
  unsigned phase = 0;
  unsigned long long* item_ctr = &reinterpret_cast<unsigned long long*>(a.ws.counters)[a.counter];
  for (;;) {
    if (tid == 0) sItem = bad ? ntiles : (long long)atomicAdd(item_ctr, 1ULL);
    __syncthreads();
    const long long b = sItem;
    if (b >= ntiles) break;
    const long long lo = b * span;  // even: both arrays start on 16-byte words
    const long long own_end = (lo + span < n) ? lo + span : n;
    const long long hi = (own_end + kRdmHalo < n) ? own_end + kRdmHalo : n;
    const int own = (int)(own_end - lo), E = (int)(hi - lo);
    if (bulk) {
      if (tid == 0) {
        fence_proxy_async_smem();  // the previous tile's shared accesses (barrier above)
        mbar_arrive_expect(&sBar, body_bytes(lo, hi, 8) + body_bytes(lo, hi, C64 ? 8u : 16u));
        copy_body(sK, keys, lo, hi, 8, &sBar);
        if (C64) copy_body(sAf, ampf, lo, hi, 8, &sBar);
        else copy_body(sA, amps, lo, hi, 16, &sBar);
      }
      // an odd last entry of the 8-byte arrays (lo is even: no odd first one)
      if (tid == 0) copy_ragged(sK, keys, lo, hi, true);
      if (C64 && tid == 1) copy_ragged(sAf, ampf, lo, hi, true);
      bool done = false;
      for (long long sp = 0; sp < lim && !done; ++sp) done = mbar_try_wait(&sBar, phase);
      if (__syncthreads_or(!done)) {
        if (tid == 0) set_error(a.ctrl, BASS_ERR_WAIT);
        // (the block must not end with its copies in flight)
        for (long long sp = 0; sp < kSpinLimit && !done; ++sp) done = mbar_try_wait(&sBar, phase);
        __syncthreads();
        break;
      }
      phase ^= 1u;
    } else {
      for (int i = tid; i < E; i += kThreads) {
        sK[i] = keys[lo + i];
        if (C64) sAf[i] = ampf[lo + i];
        else sA[i] = amps[lo + i];
      }
      __syncthreads();
    }
    if (a.prof && tid == 0)
      atomicAdd(reinterpret_cast<unsigned long long*>(&a.ctrl->prof_in[K_RDM * 5 + P_HIST]), (unsigned long long)E);
    for (int t = 0; t < kRdmLowBits; ++t) {
      const int set = sSet[t];
      if (set < 0) continue;  // the same for every thread
      const uint64_t bit = 1ULL << t;
      const int reach = 1 << t;  // the partner lies at most this many positions on
      // at most kPerThread positions per thread: at most eight terms per
      // split accumulator (fx_acc96) before they are joined
      i128 v[4] = {0, 0, 0, 0};
      double dh[4] = {0.0, 0.0, 0.0, 0.0}, dl[4] = {0.0, 0.0, 0.0, 0.0};
      for (int e = tid; e < own; e += kThreads) {
        const uint64_t x = sK[e];
        const double2 ax = amp(e);
        if (x & bit) {
          fx_acc96(prob(ax), dh[1], dl[1], v[1]);
          continue;
        }
        fx_acc96(prob(ax), dh[0], dl[0], v[0]);
        const uint64_t y = x | bit;
        int L = e + 1;
        const int R0 = (e + reach < E - 1 ? e + reach : E - 1) + 1;  // search [e + 1, R0)
        int R = R0;
        while (L < R) {
          const int m = (L + R) >> 1;
          if (sK[m] < y) L = m + 1;
          else R = m;
        }
        if (L < R0 && sK[L] == y) {
          const double2 ay = amp(L);
          const double2 c = cmul(ax, make_double2(ay.x, -ay.y));
          fx_acc96(c.x, dh[2], dl[2], v[2]);
          fx_acc96(c.y, dh[3], dl[3], v[3]);
        }
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        v[k] += fx_join96s(dh[k], dl[k]);
        v[k] = warp_sum_i128(v[k]);
      }
      if (lane == 0) {
#pragma unroll
        for (int k = 0; k < 4; ++k) sAcc[w][t][k] += v[k];
      }
    }
    __syncthreads();  // the buffers are reused by the next tile
  }
  // the CTA's sums: thread (t, k) adds the warps' accumulators
  __syncthreads();
  if (tid < kRdmLowBits * 4) {
    const int t = tid >> 2, k = tid & 3, set = sSet[t];
    if (set >= 0 && !bad) {
      i128 sum = 0;
#pragma unroll
      for (int ww = 0; ww < kThreads / 32; ++ww) sum += sAcc[ww][t][k];
      limb_add(rdm_limbs(a.ws, set) + 4 * k, sum);
    }
  }
}

// Rotation step, after the write pass: keep the candidate if accepted.
__global__ void k_commit(bass_state* cur, bass_state* tmp, WsView ws, bass_ctrl* c, int j, int trace) {
  const SelState* sel = ws.sel;
  if (!sel->accept) return;
  bass_state t = *cur;
  *cur = *tmp;
  *tmp = t;
  c->pr_cur = sel->pr_new;
  const double frac = c->frac[j];
  c->gamma_running *= sqrt(frac > 1e-30 ? frac : 0.0);
  if (trace && c->trace) {
    const long long i = c->trace_len;
    if (i >= c->trace_cap) {
      set_error(c, BASS_ERR_CAPACITY);
      return;
    }
    uint64_t* e = c->trace + i * BASS_TRACE_WORDS;
    e[0] = 1;
    e[1] = (uint64_t)j;
    for (int k = 2; k < BASS_TRACE_WORDS; ++k) e[k] = 0;
    c->trace_len = i + 1;
  }
}

// low: the moments of qubits at physical bits below kRdmLowBits are k_rdm_low's
// limbs, the others the merge pass's partials (one per merge tile)
__global__ void k_rdm_final(const bass_state* st, double* rho, WsView ws, int first, int low) {
  __shared__ i128 sRed[4 * 8];
  const int set = blockIdx.x;
  const long long ntiles = merge_tiles(st->nnz);
  if (low && st->pos[first + set] < kRdmLowBits) {
    if (threadIdx.x < 4) rho[4 * (first + set) + threadIdx.x] = fx_to(limb_get(rdm_limbs(ws, set) + 4 * threadIdx.x));
    return;
  }
  i128 v[4] = {0, 0, 0, 0};
  for (long long t = threadIdx.x; t < ntiles; t += blockDim.x) {
    const Partial& p = ws.partials[(long long)set * ws.max_tiles + t];
    v[0] += p.s[0]; v[1] += p.s[1]; v[2] += p.s[2]; v[3] += p.s[3];
  }
  block_sum_i128<4>(v, sRed);
  if (threadIdx.x == 0) {
    double* r = rho + 4 * (first + set);
    r[0] = fx_to(v[0]);
    r[1] = fx_to(v[1]);
    r[2] = fx_to(v[2]);
    r[3] = fx_to(v[3]);
  }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
// Dynamic shared memory of a tile pass and its persistent grid (every CTA
// that fits at once, at most 1024), set up on first use.
template <int KIND, int PASS, bool C64>
static cudaError_t tile_grid(size_t* smem_out, int* grid_out) {
  const size_t smem = (size_t)kTilePad * (16 + 8 + 2 + (PASS == P_WRITE ? 3 : 0));
  static PerDevice cache;
  *smem_out = smem;
  return per_device(cache, grid_out, [smem](int* grid) {
    cudaError_t e = cudaFuncSetAttribute(k_tile<KIND, PASS, C64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int occ = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_tile<KIND, PASS, C64>, kThreads, smem);
    if (e != cudaSuccess) return e;
    *grid = device().sms * (occ > 0 ? occ : 1);
    if (*grid > 1024) *grid = 1024;
    return cudaSuccess;
  });
}

template <int KIND, int PASS, bool C64>
static cudaError_t launch_tile_t(OpArgs a, int counter, cudaStream_t s, int* grid_out) {
  size_t smem = 0;
  int grid = 0;
  cudaError_t e = tile_grid<KIND, PASS, C64>(&smem, &grid);
  if (e != cudaSuccess) return e;
  a.counter = counter;
  a.prof = prof_on() ? 1 : 0;
  KLAUNCH(KIND * 5 + PASS, s, launch_pdl(k_tile<KIND, PASS, C64>, dim3(grid), dim3(kThreads), smem, s, a));
  if (grid_out) *grid_out = grid;
  return cudaGetLastError();
}

// the tile pass for the op's amplitude type (a.c64, from the host's record of the state)
template <int KIND, int PASS>
static cudaError_t launch_tile(OpArgs a, int counter, cudaStream_t s, int* grid_out) {
  return a.c64 ? launch_tile_t<KIND, PASS, true>(a, counter, s, grid_out)
               : launch_tile_t<KIND, PASS, false>(a, counter, s, grid_out);
}

cudaError_t zero_small(const WsView& ws, cudaStream_t s) {
  // counters, hist1, hist2, sel and the look-back status words are contiguous
  const size_t bytes = (size_t)((char*)(ws.status + ws.max_tiles) - (char*)ws.counters);
  return cudaMemsetAsync(ws.counters, 0, bytes, s);
}

// Opts a kernel of kThreads threads in to `smem` bytes of dynamic shared
// memory and returns its resident grid (once per device).
template <typename K>
static cudaError_t smem_grid(PerDevice& cache, K kern, size_t smem, int* grid) {
  return per_device(cache, grid, [kern, smem](int* v) {
    cudaError_t e = cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int occ = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kThreads, smem);
    if (e != cudaSuccess) return e;
    *v = device().sms * (occ > 0 ? occ : 1);
    return cudaSuccess;
  });
}

cudaError_t run_commit(bass_state* cur, bass_state* tmp, bass_ctrl* ctrl, const WsView& ws, int j, int trace,
                       cudaStream_t s) {
  KLAUNCH(S_REDUCE, s, k_commit<<<1, 1, 0, s>>>(cur, tmp, ws, ctrl, j, trace));
  return cudaGetLastError();
}

// write pass only (keep everything the drop rule keeps); used by the guarded
// compaction after a 1-qubit diagonal gate.  The caller zeroed the small region.
cudaError_t run_ident_write(OpArgs a, cudaStream_t s) {
  return launch_tile<K_IDENT, P_WRITE>(a, 3, s, nullptr);
}

cudaError_t run_rdm(const bass_state* st, int nq, double* rho, bass_ctrl* ctrl, const WsView& ws,
                    cudaStream_t s, int c64) {
  cudaError_t e = cudaSuccess;
  OpArgs a{};
  a.c64 = c64;
  a.in = st;
  a.out = nullptr;
  a.ctrl = ctrl;
  a.ws = ws;
  a.q = 0;
  a.gb = 0;
  a.nsets = nq;
  a.rdm_low = 1;
  // the partition also clears the small workspace region; the qubits at
  // physical bits below kRdmLowBits take one pass of k_rdm_low instead of a
  // partition and a merge pass each
  // (no more blocks than the workspace's bound has boundaries, eight to a block:
  // the full grid for every qubit is 47,000 blocks)
  const long long want = (ws.max_tiles + 1 + 7) / 8;
  const int gp = want < device().grid_small ? (int)want : device().grid_small;
  KLAUNCH(S_PARTITION, s, launch_pdl(k_partition, dim3(gp, nq), dim3(256), 0, s, a, (int)K_RDM, 1));
  if ((e = launch_tile<K_RDM, P_RDM>(a, 0, s, nullptr)) != cudaSuccess) return e;
  {
    static PerDevice grid_c64, grid_c128;
    int gl = 0;
    if ((e = c64 ? smem_grid(grid_c64, k_rdm_low<true>, kRdmLowSmem, &gl)
                 : smem_grid(grid_c128, k_rdm_low<false>, kRdmLowSmem, &gl)) != cudaSuccess)
      return e;
    a.counter = 5;
    a.prof = prof_on() ? 1 : 0;
    if (c64)
      KLAUNCH(K_RDM * 5 + P_HIST, s, launch_pdl(k_rdm_low<true>, dim3(gl), dim3(kThreads), kRdmLowSmem, s, a));
    else
      KLAUNCH(K_RDM * 5 + P_HIST, s, launch_pdl(k_rdm_low<false>, dim3(gl), dim3(kThreads), kRdmLowSmem, s, a));
  }
  KLAUNCH(S_RDM_FINAL, s, k_rdm_final<<<nq, 256, 0, s>>>(st, rho, ws, 0, 1));
  return cudaGetLastError();
}

// 4x4 moments of the qubit pair (q1, q2): the first pass of a 2-qubit gate
// brings q2 to bit 0 (st -> tmp), then one moment pass over tmp groups the
// entries by every other bit with q1 at bit 1.  rho: 16 doubles, see k_tile's
// P_RDM pass for K_GATE2 (set s writes rho[4 s .. 4 s + 3]).
cudaError_t run_rdm_2q(const bass_state* st, bass_state* tmp, int q1, int q2, double* rho, bass_ctrl* ctrl,
                       const WsView& ws, cudaStream_t s, int c64) {
  OpArgs a{};
  a.c64 = c64;
  a.in = st; a.out = tmp; a.ctrl = ctrl; a.ws = ws; a.q = q2; a.gb = 0;
  bass_trunc none{};
  none.k_cond = -1;
  cudaError_t e = run_merge_op(K_PERM, a, none, 0, 0, s);
  if (e != cudaSuccess) return e;
  OpArgs b{};
  b.in = tmp; b.out = nullptr; b.ctrl = ctrl; b.ws = ws; b.q = q1; b.gb = 1; b.nsets = 4; b.c64 = c64;
  // the partition also clears the small workspace region
  KLAUNCH(S_PARTITION, s, launch_pdl(k_partition, dim3(device().grid_small, 1), dim3(256), 0, s, b, (int)K_GATE2, 1));
  if ((e = launch_tile<K_GATE2, P_RDM>(b, 0, s, nullptr)) != cudaSuccess) return e;
  KLAUNCH(S_RDM_FINAL, s, k_rdm_final<<<4, 256, 0, s>>>(tmp, rho, ws, 0, 0));
  return cudaGetLastError();
}

// RDM moments with a caller-prepared workspace view: the same kernels as
// run_rdm, without clearing any workspace region (the caller clears the tile
// counters) and with a final reduction that refuses states whose tile count
// exceeds the view's capacity.  Used by the no-allocation entry point.
__global__ void k_rdm_final_bounded(const bass_state* st, double* rho, WsView ws, bass_ctrl* c) {
  __shared__ i128 sRed[4 * 8];
  const int set = blockIdx.x;
  const long long ntiles = merge_tiles(st->nnz);
  if (ntiles > ws.max_tiles) {
    if (threadIdx.x == 0) {
      set_error(c, BASS_ERR_WORKSPACE);
      for (int k = 0; k < 4; ++k) rho[4 * set + k] = NAN;
    }
    return;
  }
  i128 v[4] = {0, 0, 0, 0};
  for (long long t = threadIdx.x; t < ntiles; t += blockDim.x) {
    const Partial& p = ws.partials[(long long)set * ws.max_tiles + t];
    v[0] += p.s[0]; v[1] += p.s[1]; v[2] += p.s[2]; v[3] += p.s[3];
  }
  block_sum_i128<4>(v, sRed);
  if (threadIdx.x == 0) {
    double* r = rho + 4 * set;
    r[0] = fx_to(v[0]);
    r[1] = fx_to(v[1]);
    r[2] = fx_to(v[2]);
    r[3] = fx_to(v[3]);
  }
}

cudaError_t run_rdm_prepared(const bass_state* st, int nq, double* rho, bass_ctrl* ctrl, const WsView& ws,
                             cudaStream_t s, int c64) {
  OpArgs a{};
  a.c64 = c64;
  a.in = st;
  a.out = nullptr;
  a.ctrl = ctrl;
  a.ws = ws;
  a.q = 0;
  a.gb = 0;
  a.nsets = nq;
  KLAUNCH(S_PARTITION, s, k_partition<<<dim3(device().grid_small, nq), 256, 0, s>>>(a, K_RDM, 0));
  cudaError_t e = launch_tile<K_RDM, P_RDM>(a, 0, s, nullptr);
  if (e != cudaSuccess) return e;
  KLAUNCH(S_RDM_FINAL, s, k_rdm_final_bounded<<<nq, 256, 0, s>>>(st, rho, ws, ctrl));
  return cudaGetLastError();
}


// ---------------------------------------------------------------------------
// segmented launches: one op on each of many states per launch
// ---------------------------------------------------------------------------
// The block groups of an op: work weight of state s = its input entries plus
// kSegPad (an RDM's: plus one tile, times its qubits).  One block.
__global__ void k_seg_plan(const OpArgs* ops, int nseg, int kind, SegPlan* plan) {
  __shared__ long long sW[kMaxSeg];
  for (int s = threadIdx.x; s < nseg; s += blockDim.x) {
    const long long n = ops[s].in->nnz;
    sW[s] = kind == K_RDM ? (n + kStep) * (long long)ops[s].nsets : n + kSegPad;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    long long run = 0;
    for (int s = 0; s < nseg; ++s) {
      plan->wp[s] = run;
      run += sW[s];
    }
    plan->wp[nseg] = run;
    plan->nseg = nseg;
    plan->kind = kind;
  }
}

cudaError_t run_seg_plan(const OpArgs* ops, int nseg, int kind, SegPlan* plan, cudaStream_t s) {
  KLAUNCH(S_SMALL, s, k_seg_plan<<<1, 1024, 0, s>>>(ops, nseg, kind, plan));
  return cudaGetLastError();
}

__global__ void k_partition_seg(const OpArgs* ops, const SegPlan* plan, int kind, int zero) {
  __shared__ OpArgs sa;
  const Grp g = seg_enter(ops, plan, &sa, nullptr);
  if (kind == K_RDM && (int)blockIdx.y >= sa.nsets) return;  // qubits this state does not have
  partition_body(sa, kind, zero, blockIdx.y, g);
}

template <int KIND, int PASS, bool C64>
__global__ void __launch_bounds__(kThreads, 4) k_tile_seg(const OpArgs* ops, const SegPlan* plan) {
  __shared__ OpArgs sa;
  const Grp g = seg_enter(ops, plan, &sa, nullptr);
  tile_body<KIND, PASS, C64>(sa, g);
}

// per state, the moments of each of its qubits (grid: qubit x state)
__global__ void k_rdm_final_seg(const OpArgs* ops) {
  __shared__ i128 sRed[4 * 8];
  const OpArgs& a = ops[blockIdx.y];
  const int set = blockIdx.x;
  if (set >= a.nsets) return;
  const long long ntiles = merge_tiles(a.in->nnz);
  if (ntiles > a.ws.max_tiles) {
    if (threadIdx.x == 0) set_error(a.ctrl, BASS_ERR_WORKSPACE);
    return;
  }
  i128 v[4] = {0, 0, 0, 0};
  for (long long t = threadIdx.x; t < ntiles; t += blockDim.x) {
    const Partial& p = a.ws.partials[(long long)set * a.ws.max_tiles + t];
    v[0] += p.s[0]; v[1] += p.s[1]; v[2] += p.s[2]; v[3] += p.s[3];
  }
  block_sum_i128<4>(v, sRed);
  if (threadIdx.x == 0) {
    double* r = a.rho + 4 * set;
    r[0] = fx_to(v[0]);
    r[1] = fx_to(v[1]);
    r[2] = fx_to(v[2]);
    r[3] = fx_to(v[3]);
  }
}


// Grid of a segmented kernel: every block of it that fits at once, and at
// least one block per state.
template <typename F>
static int seg_grid(F kern, int threads, size_t smem, int nseg) {
  int occ = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, threads, smem) != cudaSuccess || occ < 1) occ = 1;
  const int g = device().sms * occ;
  return g > nseg ? g : nseg;
}

template <bool C64>
static cudaError_t rdm_seg(const OpArgs* ops, int nseg, int max_nq, SegPlan* plan, cudaStream_t s) {
  KLAUNCH(S_SMALL, s, k_seg_plan<<<1, 1024, 0, s>>>(ops, nseg, K_RDM, plan));
  const int np = device().grid_small > nseg ? device().grid_small : nseg;
  KLAUNCH(S_PARTITION, s, k_partition_seg<<<dim3(np, max_nq), 256, 0, s>>>(ops, plan, K_RDM, 1));
  const size_t smem = (size_t)kTilePad * (16 + 8 + 2);
  static int nt = 0;
  if (nt == 0) {
    cudaError_t e = cudaFuncSetAttribute(k_tile_seg<K_RDM, P_RDM, C64>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem);
    if (e != cudaSuccess) return e;
    nt = seg_grid(k_tile_seg<K_RDM, P_RDM, C64>, kThreads, smem, 1);
  }
  const int gt = nt > nseg ? nt : nseg;
  KLAUNCH(K_RDM * 5 + P_RDM, s, k_tile_seg<K_RDM, P_RDM, C64><<<gt, kThreads, smem, s>>>(ops, plan));
  KLAUNCH(S_RDM_FINAL, s, k_rdm_final_seg<<<dim3(max_nq, nseg), 256, 0, s>>>(ops));
  return cudaGetLastError();
}

cudaError_t run_rdm_seg(const OpArgs* ops, int nseg, int max_nq, int c64, SegPlan* plan, cudaStream_t s) {
  if (nseg < 1 || nseg > kMaxSeg || max_nq < 1 || max_nq > kMaxSets) return cudaErrorInvalidValue;
  return c64 ? rdm_seg<true>(ops, nseg, max_nq, plan, s) : rdm_seg<false>(ops, nseg, max_nq, plan, s);
}

}  // namespace bass
