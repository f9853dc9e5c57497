// tile.cuh -- the pieces every tile kernel shares: tile boundaries in Z order
// (partition), a tile's load into shared memory, its merge into Z order and
// the evaluation of its groups.
//
// A state is sorted by physical key.  An op acting on qubit q (physical bit t)
// reads the state in "Z order": the order of zmove(key, t, gb), which brings
// bit t down to bit gb so that the entries a gate combines (keys that differ
// only in the gate's bits) become adjacent.  Within a block of keys sharing the
// bits above t, Z order is the merge of the block's bit-t-clear run and its
// bit-t-set run, so one merge pass pairs every entry with its partners.
#pragma once

#include <atomic>

#include "internal.h"

namespace bass {

// The blocks of a launch that work on one op.  A plain launch is one group
// (blockIdx.x of gridDim.x); a segmented launch (one op on each of many
// states) splits its grid into one group per state, see seg_enter.
struct Grp {
  int bid;   // block index within the group
  int nblk;  // blocks in the group
};
__device__ __forceinline__ Grp whole_grid() { return Grp{(int)blockIdx.x, (int)gridDim.x}; }

// The op's output qubit order: the input's, with the target qubit's
// position t = pos[q] moved down to gb (positions gb..t-1 move up by one) for
// the kinds that bring a target to the low bits.  One position per thread
// (threads 0-63 of the block); the caller synchronises before reading it.
__device__ __forceinline__ void out_order_par(const bass_state* in, int kind, int q, int gb, int8_t* qat_out) {
  const int p = threadIdx.x;
  if (p < 64) {
    int src = p;
    if (kind == K_GATE1 || kind == K_ROT1 || kind == K_GATE2 || kind == K_PERM) {
      const int t = in->pos[q];
      if (p > gb && p <= t) src = p - 1;
      if (p == gb) src = t;
    }
    qat_out[p] = in->qat[src];
  }
}

// The partition record of the tile boundary at Z position P, by one warp:
// r[0] the adjusted Z position (backed off to the start of its group unless
// the op keeps groups apart: back), r[1..3] the block's start, run split and
// end, r[4], r[5] the merge-path split inside it.  The block is found by
// warp-cooperative 32-ary searches; the record is the same in every lane.
template <int GB>
__device__ __forceinline__ void tile_boundary(const uint64_t* keys, long long n, long long P, int t, bool back,
                                              long long (&r)[6]) {
  if (P >= n) {
    r[0] = n; r[1] = n; r[2] = n; r[3] = n; r[4] = 0; r[5] = 0;
    return;
  }
  const int lane = threadIdx.x & 31;
  constexpr int sh = GB + 1;
  const ZMove<GB> zmove(t);
  const uint64_t y = keys[P];
  const uint64_t lo_key = (y >> (t + 1)) << (t + 1);
  const uint64_t mid_key = lo_key | (1ULL << t);
  const uint64_t hi_key = lo_key + (2ULL << t);
  const bool hi_ovf = hi_key <= lo_key;
  // block start, run split and block end in one lockstep search
  long long lo3[3] = {0, ((y >> t) & 1ULL) ? 0 : P + 1, hi_ovf ? n : P + 1};
  long long hi3[3] = {P + 1, ((y >> t) & 1ULL) ? P + 1 : n, n};
  const uint64_t thr3[3] = {lo_key, mid_key, hi_key};
  const bool back3[3] = {true, ((y >> t) & 1ULL) != 0, false};
  warp_bracket3(keys, P, lo3, hi3, thr3, back3);
  warp_lower_bound3(keys, lo3, hi3, thr3);
  const long long s = lo3[0], mid = lo3[1], e = lo3[2];
  const long long d = P - s, len0 = mid - s, len1 = e - mid;
  const long long lo = d - len1 > 0 ? d - len1 : 0;
  const long long hi = d < len0 ? d : len0;
  long long i = warp_first_false(lo, hi, [&](long long m) {
    return zmove(keys[s + m]) < zmove(keys[mid + d - 1 - m]);
  });
  long long j = d - i;
  if (back) {
    // back the boundary off to the start of its group: the two entries
    // at the split and the two before it in each run, fetched at once
    long long idx = -1;
    if (lane == 0 && i < len0) idx = s + i;
    if (lane == 1 && j < len1) idx = mid + j;
    if (lane == 2 && i >= 1) idx = s + i - 1;
    if (lane == 3 && i >= 2) idx = s + i - 2;
    if (lane == 4 && j >= 1) idx = mid + j - 1;
    if (lane == 5 && j >= 2) idx = mid + j - 2;
    const uint64_t zv = (idx >= 0) ? zmove(keys[idx]) : ~0ULL;
    const uint64_t z0 = __shfl_sync(0xffffffffu, zv, 0), z1 = __shfl_sync(0xffffffffu, zv, 1);
    const uint64_t a1 = __shfl_sync(0xffffffffu, zv, 2), a2 = __shfl_sync(0xffffffffu, zv, 3);
    const uint64_t c1 = __shfl_sync(0xffffffffu, zv, 4), c2 = __shfl_sync(0xffffffffu, zv, 5);
    const uint64_t gid = (z0 < z1 ? z0 : z1) >> sh;
    int b0 = 0, b1 = 0;
    if (i >= 1 && (a1 >> sh) == gid) b0 = (i >= 2 && (a2 >> sh) == gid) ? 2 : 1;
    if (j >= 1 && (c1 >> sh) == gid) b1 = (j >= 2 && (c2 >> sh) == gid) ? 2 : 1;
    i -= b0;
    j -= b1;
  }
  r[0] = s + i + j; r[1] = s; r[2] = mid; r[3] = e; r[4] = i; r[5] = j;
}

// tile_boundary when the target bit is already in its place (t == GB): a block is
// a group, at most 2 << GB entries around P, so one load replaces the searches.
template <int GB>
__device__ __forceinline__ void low_boundary(const uint64_t* keys, long long n, long long P, bool back,
                                             long long (&r)[6]) {
  if (P >= n) {
    r[0] = n; r[1] = n; r[2] = n; r[3] = n; r[4] = 0; r[5] = 0;
    return;
  }
  constexpr int kReach = (2 << GB) - 1;
  const int lane = threadIdx.x & 31;
  const uint64_t y = keys[P];
  const long long p = P - kReach + lane;
  const bool in = lane <= 2 * kReach && p >= 0 && p < n;
  const uint64_t k = in ? keys[p] : 0ULL;
  const bool mine = in && (k >> (GB + 1)) == (y >> (GB + 1));
  const unsigned m = __ballot_sync(0xffffffffu, mine), m1 = __ballot_sync(0xffffffffu, mine && ((k >> GB) & 1ULL));
  const long long s = P - kReach + (__ffs(m) - 1), e = s + __popc(m), mid = e - __popc(m1);
  long long i = 0, j = 0;
  if (!back) {
    const long long d = P - s, len0 = mid - s;
    i = d < len0 ? d : len0;
    j = d - i;
  }
  r[0] = s + i + j; r[1] = s; r[2] = mid; r[3] = e; r[4] = i; r[5] = j;
}

// ---------------------------------------------------------------------------
// a tile's input
// ---------------------------------------------------------------------------
// At most five contiguous input segments, packed into shared memory.  Segment
// k starts at its packed offset, or up to five positions later, so that its
// positions have the parity of its source entries (both ends of a bulk copy of
// 8-byte data are then 16-byte aligned).
struct TileSeg {
  long long lo[5];   // first source entry
  long long off[6];  // packed offset (off[5]: entries of the tile)
  long long zs;      // Z position of the tile's first entry
  int pos[5], gap[5];
};

struct TileSrc {
  const uint64_t* keys;
  const double2* amps;
  long long n;
  bool tma;  // both arrays 16-byte aligned
};

// One thread: the segments of the tile between the boundary records rc and rn
// (at most cap entries), and with bulk copies the copies of their 16-byte
// aligned bodies, which complete on bar.  An inconsistent partition leaves the
// tile empty and reports BASS_ERR_ARG.
template <bool C64>
__device__ __forceinline__ void tile_segments(TileSeg& T, const long long* rc, const long long* rn, const TileSrc& S,
                                              int cap, uint64_t* sZ, double2* sA, uint64_t* bar, bass_ctrl* ctrl) {
  long long lo[5] = {0, 0, 0, 0, 0}, len[5] = {0, 0, 0, 0, 0};
  const long long zs = rc[0];
  if (rc[1] == rn[1]) {
    lo[0] = rc[1] + rc[4]; len[0] = rn[4] - rc[4];
    lo[1] = rc[2] + rc[5]; len[1] = rn[5] - rc[5];
  } else {
    lo[0] = rc[1] + rc[4]; len[0] = rc[2] - lo[0];
    lo[1] = rc[2] + rc[5]; len[1] = rc[3] - lo[1];
    lo[2] = rc[3];         len[2] = rn[1] - rc[3];
    lo[3] = rn[1];         len[3] = rn[4];
    lo[4] = rn[2];         len[4] = rn[5];
  }
  long long o = 0;
  bool bad = false;
  for (int k = 0; k < 5; ++k) {
    if (len[k] < 0 || lo[k] < 0 || lo[k] + len[k] > S.n) { len[k] = 0; bad = true; }
    T.lo[k] = lo[k];
    T.off[k] = o;
    o += len[k];
  }
  if (o > cap || bad || zs < 0 || zs + o > S.n) {  // inconsistent partition: skip the tile, report
    set_error(ctrl, BASS_ERR_ARG);
    for (int k = 0; k < 5; ++k) T.off[k] = 0;
    o = 0;
  }
  T.off[5] = o;
  T.zs = zs;
  int gap = 0;
  for (int k = 0; k < 5; ++k) {
    const long long ln = T.off[k + 1] - T.off[k];
    if (S.tma && ln > 0 && ((T.off[k] + gap - T.lo[k]) & 1)) ++gap;
    T.gap[k] = gap;
    T.pos[k] = (int)T.off[k] + gap;
  }
  if (S.tma) {
    // the bulk copies of every segment's body [f, l): one arrival that expects
    // all their bytes, then the copies
    constexpr unsigned kAmpBytes = C64 ? 8u : 16u;
    unsigned bytes = 0;
    for (int k = 0; k < 5; ++k) {
      const long long l0 = T.lo[k], ln = T.off[k + 1] - T.off[k];
      if (ln > 0) bytes += (unsigned)(((l0 + ln) & ~1LL) - ((l0 + 1) & ~1LL)) * (8u + kAmpBytes);
    }
    fence_proxy_async_smem();  // the previous tile's shared accesses (all threads: the caller's barrier)
    mbar_arrive_expect(bar, bytes);
    for (int k = 0; k < 5; ++k) {
      const long long l0 = T.lo[k], ln = T.off[k + 1] - T.off[k];
      if (ln <= 0) continue;
      const long long f = (l0 + 1) & ~1LL, l = (l0 + ln) & ~1LL;
      if (l <= f) continue;
      const int p = T.pos[k] + (int)(f - l0);
      const unsigned nb = (unsigned)(l - f);
      bulk_load(sZ + p, S.keys + f, 8u * nb, bar);
      if (C64)
        bulk_load(reinterpret_cast<float2*>(sA) + p, reinterpret_cast<const float2*>(S.amps) + f, 8u * nb, bar);
      else
        bulk_load(sA + p, S.amps + f, 16u * nb, bar);
    }
  }
}

// The block waits until the tile's entries are in shared memory: bulk copies
// on bar (warp 0 fetches the at most two ragged entries of each segment, an odd
// first one and an even last one, with plain loads), or per-entry asynchronous
// copies for arrays at an 8-byte offset.  The wait is bounded by lim tries (the
// copies complete unless the byte count is wrong); false if it gave up, after
// another bounded wait for the copies in flight.
template <int PT, bool C64>
__device__ __forceinline__ bool tile_fetch(const TileSeg& T, const TileSrc& S, uint64_t* sZ, double2* sA, uint64_t* bar,
                                           unsigned* phase, bass_ctrl* ctrl, long long lim) {
  const int tid = threadIdx.x;
  if (S.tma) {
    if (tid < 10) {
      const int k = tid >> 1;
      const long long l0 = T.lo[k], ln = T.off[k + 1] - T.off[k];
      if (ln > 0) {
        const long long f = (l0 + 1) & ~1LL, l = (l0 + ln) & ~1LL;
        const bool last = tid & 1;
        if (last ? l < l0 + ln : l0 < f) {
          const long long i = last ? l : l0;
          const int p = T.pos[k] + (int)(i - l0);
          sZ[p] = S.keys[i];
          if (C64) reinterpret_cast<float2*>(sA)[p] = reinterpret_cast<const float2*>(S.amps)[i];
          else sA[p] = S.amps[i];
        }
      }
    }
    bool done = false;
    for (long long sp = 0; sp < lim && !done; ++sp) done = mbar_try_wait(bar, *phase);
    if (__syncthreads_or(!done)) {
      if (tid == 0) set_error(ctrl, BASS_ERR_WAIT);
      for (long long sp = 0; sp < kSpinLimit && !done; ++sp) done = mbar_try_wait(bar, *phase);
      __syncthreads();
      return false;
    }
    *phase ^= 1u;
  } else {
    // 8-byte aligned arrays: asynchronous per-entry copies (no gaps)
    const int E = (int)T.off[5];
    const int o1 = (int)T.off[1], o2 = (int)T.off[2], o3 = (int)T.off[3], o4 = (int)T.off[4];
    const unsigned zb = (unsigned)__cvta_generic_to_shared(sZ);
    const unsigned ab = (unsigned)__cvta_generic_to_shared(sA);
#pragma unroll
    for (int k = 0; k < PT; ++k) {
      const int e = k * kThreads + tid;
      if (e < E) {
        const int sg = (e >= o1) + (e >= o2) + (e >= o3) + (e >= o4);
        const long long src = T.lo[sg] + (e - T.off[sg]);
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(zb + 8u * e), "l"(S.keys + src) : "memory");
        if (C64)
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(ab + 8u * e),
                       "l"(reinterpret_cast<const float2*>(S.amps) + src)
                       : "memory");
        else
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(ab + 16u * e), "l"(S.amps + src) : "memory");
      }
    }
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
    __syncthreads();
  }
  return true;
}

// Z order of a loaded tile of at most 256 PT entries, as a permutation: sP[p]
// says where the entry at Z position p was loaded, and how it is grouped.
// Neither keys nor amplitudes move.  Z order is the merge of the bit-clear
// entries with the bit-set ones by the key without the target bit (and, for
// GB = 1, without the low bit, which the group's other qubit holds), the clear
// one first among equals, so the merge works on the raw keys: thread i finds
// where its PT positions start in both runs by a binary search and merges them
// from there.  When the tile lies within one block its two segments are the
// two runs; otherwise the entries are first split into two lists of places.
// (Moving Z keys through shared memory, split, merged and written back around
// its banks, made the reorder pass of a 2-qubit gate take 68 us instead of 52
// at 2^22 entries.)
constexpr unsigned kPlaceMask = 0xFFFu;       // bits 0-11: shared position of the entry
constexpr int kPlaceLocal = 12;               // bits 12-13: its index within its group
constexpr unsigned kPlaceNext = 1u << 14;     // the next position belongs to the same group
constexpr unsigned kPlaceStart = 1u << 15;    // the position starts a group
static_assert(kTilePad <= (int)kPlaceMask + 1, "places fit 12 bits");

template <int PT, int GB, bool LISTS>
__device__ __forceinline__ void tile_merge(const TileSeg& T, const uint64_t* sK, uint16_t* sP, int n0, int t) {
  const int tid = threadIdx.x;
  const int E = (int)T.off[5], n1 = E - n0;
  const uint64_t nmask = ~(1ULL << t);
  const int a0 = LISTS ? 0 : T.pos[0], b0 = LISTS ? n0 : T.pos[1];
  auto place = [&](int i) { return LISTS ? (int)sP[i] : i; };
  auto norm = [&](uint64_t k) { return (k & nmask) >> GB; };
  const int d = tid * PT < E ? tid * PT : E;
  int lo = d - n1 > 0 ? d - n1 : 0, hi = d < n0 ? d : n0;
  while (lo < hi) {
    const int m = (lo + hi) >> 1;
    if (norm(sK[place(a0 + m)]) <= norm(sK[place(b0 + d - 1 - m)])) lo = m + 1;
    else hi = m;
  }
  int i = lo, j = d - lo;
  // the key before position d (the larger of the two runs' last ones)
  uint64_t prev = ~0ULL;
  if (d > 0) {
    const uint64_t pa = i > 0 ? norm(sK[place(a0 + i - 1)]) : 0ULL, pb = j > 0 ? norm(sK[place(b0 + j - 1)]) : 0ULL;
    prev = pa > pb ? pa : pb;
  }
  int pa = i < n0 ? place(a0 + i) : 0, pb = j < n1 ? place(b0 + j) : 0;
  uint64_t ka = i < n0 ? sK[pa] : ~0ULL, kb = j < n1 ? sK[pb] : ~0ULL;
  uint64_t na = i < n0 ? norm(ka) : ~0ULL, nb = j < n1 ? norm(kb) : ~0ULL;
  unsigned rp[PT];
#pragma unroll
  for (int k = 0; k <= PT; ++k) {
    const bool take0 = na <= nb;
    const uint64_t cur = take0 ? na : nb;  // ~0 past the end
    const bool same = cur == prev;
    if (k > 0 && same) rp[k - 1] |= kPlaceNext;
    if (k == PT) break;
    prev = cur;
    const unsigned low = GB ? (unsigned)((take0 ? ka : kb) & 1ULL) : 0u;
    rp[k] = (unsigned)(take0 ? pa : pb) | (((take0 ? 0u : (GB ? 2u : 1u)) | low) << kPlaceLocal) |
            (same ? 0u : kPlaceStart);
    // the next entry of the run that was taken from (one load, no branch)
    const int ix = (take0 ? i : j) + 1;
    const bool more = ix < (take0 ? n0 : n1);
    const int px = more ? place((take0 ? a0 : b0) + ix) : 0;
    const uint64_t kx = sK[px];
    const uint64_t nx = more ? norm(kx) : ~0ULL;
    if (take0) {
      i = ix;
      pa = px;
      ka = kx;
      na = nx;
    } else {
      j = ix;
      pb = px;
      kb = kx;
      nb = nx;
    }
  }
  if (LISTS) __syncthreads();  // the lists are read before they are overwritten
  // consecutive positions in one store (what lies past E is never read)
  static_assert(PT == 8 || PT == 4 || PT == 2, "write-back of eight, four or two positions");
  if (tid * PT < E) {
    if (PT == 8)
      *reinterpret_cast<uint4*>(sP + d) = make_uint4(rp[0] | (rp[1] << 16), rp[2 % PT] | (rp[3 % PT] << 16),
                                                     rp[4 % PT] | (rp[5 % PT] << 16), rp[6 % PT] | (rp[7 % PT] << 16));
    else if (PT == 4)
      *reinterpret_cast<uint2*>(sP + d) = make_uint2(rp[0] | (rp[1] << 16), rp[2 % PT] | (rp[3 % PT] << 16));
    else
      *reinterpret_cast<unsigned*>(sP + d) = rp[0] | (rp[1] << 16);
  }
  __syncthreads();
}

// Z order of a tile when the target bit is already in its place (t == GB): the
// order of the keys, in which the segments were loaded.
template <int PT, int GB>
__device__ __forceinline__ void tile_in_order(const TileSeg& T, const uint64_t* sK, uint16_t* sP) {
  const int E = (int)T.off[5];
  const int o1 = (int)T.off[1], o2 = (int)T.off[2], o3 = (int)T.off[3], o4 = (int)T.off[4];
  auto place = [&](int e) { return e + T.gap[(e >= o1) + (e >= o2) + (e >= o3) + (e >= o4)]; };
#pragma unroll
  for (int k = 0; k < PT; ++k) {
    const int p = k * kThreads + (int)threadIdx.x;
    if (p >= E) break;
    const int q = place(p);
    const uint64_t key = sK[q], group = key >> (GB + 1);
    const bool same = p > 0 && (sK[place(p - 1)] >> (GB + 1)) == group;
    const bool next = p + 1 < E && (sK[place(p + 1)] >> (GB + 1)) == group;
    const unsigned local = (unsigned)key & ((2u << GB) - 1u);
    sP[p] = (uint16_t)((unsigned)q | (local << kPlaceLocal) | (next ? kPlaceNext : 0u) | (same ? 0u : kPlaceStart));
  }
  __syncthreads();
}

template <int PT, int GB>
__device__ __forceinline__ void tile_zorder(const TileSeg& T, const uint64_t* sK, uint16_t* sP, int* sWarp, int t) {
  const int E = (int)T.off[5];
  if (PT > 2 && t == GB) {  // (a chip tile's merge costs no more than the extra code)
    tile_in_order<PT, GB>(T, sK, sP);
    return;
  }
  if (T.off[2] == E) {  // two segments: the runs themselves
    tile_merge<PT, GB, false>(T, sK, sP, (int)T.off[1], t);
    return;
  }
  // lists of places: bit-clear entries first
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const unsigned lt = (1u << lane) - 1;
  constexpr int kWarpSpan = 32 * PT;
  unsigned m0[PT];
  int pe[PT];  // shared position of load position e
  int c0 = 0;
  const int o1 = (int)T.off[1], o2 = (int)T.off[2], o3 = (int)T.off[3], o4 = (int)T.off[4];
#pragma unroll
  for (int k = 0; k < PT; ++k) {
    const int e = w * kWarpSpan + k * 32 + lane;
    pe[k] = e + T.gap[(e >= o1) + (e >= o2) + (e >= o3) + (e >= o4)];
    const bool is0 = e < E && !((sK[e < E ? pe[k] : 0] >> t) & 1ULL);
    m0[k] = __ballot_sync(0xffffffffu, is0);
    c0 += __popc(m0[k]);
  }
  if (lane == 0) sWarp[w] = c0;
  __syncthreads();
  int wb0 = 0, n0 = 0;
#pragma unroll
  for (int i = 0; i < kThreads / 32; ++i) {
    const int v = sWarp[i];
    if (i < w) wb0 += v;
    n0 += v;
  }
  const int wstart = w * kWarpSpan < E ? w * kWarpSpan : E;
  int r0 = wb0, r1 = n0 + wstart - wb0;
#pragma unroll
  for (int k = 0; k < PT; ++k) {
    const int e = w * kWarpSpan + k * 32 + lane;
    const unsigned ones = __ballot_sync(0xffffffffu, e < E) & ~m0[k];
    if (e < E) sP[((m0[k] >> lane) & 1u) ? r0 + __popc(m0[k] & lt) : r1 + __popc(ones & lt)] = (uint16_t)pe[k];
    r0 += __popc(m0[k]);
    r1 += __popc(ones);
  }
  __syncthreads();
  tile_merge<PT, GB, true>(T, sK, sP, n0, t);
}

// ---------------------------------------------------------------------------
// groups -> children
// ---------------------------------------------------------------------------
// the position the target bit moves to, by kind
__host__ __device__ constexpr int group_bit(int kind) { return kind == K_GATE2 ? 1 : 0; }

// entries per group / children per group of each kind
template <int KIND>
struct KindTraits {
  static constexpr int kMaxChildren = (KIND == K_GATE2) ? 4 : (KIND == K_GATE1 || KIND == K_ROT1) ? 2 : 1;
};

// The rotation's drop rule hypot(re, im) > 1e-30 (bass_simulator.py:156-199),
// decided without calling hypot outside a narrow band: hypot lies between
// max(|re|, |im|) and sqrt(2) max(|re|, |im|) (within its last-place error),
// so the answer is known unless max is within [7e-31, 1e-30].
__device__ __forceinline__ bool above_drop(double2 c) {
  if (c.x != c.x || c.y != c.y) return hypot(c.x, c.y) > 1e-30;  // NaN: as hypot decides
  const double m = fmax(fabs(c.x), fabs(c.y));
  if (m > 1e-30) return true;
  if (m < 7e-31) return false;
  return hypot(c.x, c.y) > 1e-30;
}

// A loaded tile as the evaluation sees it: keys and amplitudes where they were
// loaded, read at Z position p through the merge's permutation (none: plain
// tiles, entry p at position p), with the state's pending renormalisation.
struct TileView {
  const uint64_t* sK;
  const double2* sA;   // complex128 amplitudes, or
  const float2* sAf;   // complex64 amplitudes (c64)
  const uint16_t* sP;  // tile_zorder's words, or nullptr
  double r0, r1;
  bool scaled;
  bool c64;
  __device__ __forceinline__ unsigned word(int p) const { return sP[p]; }
  __device__ __forceinline__ double2 amp_at(int q) const {  // by shared position
    const double2 v = c64 ? f2d(sAf[q]) : sA[q];
    return scaled ? amp_scale(v, c64 ? 1 : 0, r0, r1) : v;
  }
  __device__ __forceinline__ double2 amp(int p) const { return amp_at(sP ? (int)(sP[p] & kPlaceMask) : p); }
  __device__ __forceinline__ uint64_t key(int p) const { return sK[sP ? (int)(sP[p] & kPlaceMask) : p]; }
};
// The new physical key of child 0 of the group that starts at Z position p
// (child c: | c).
template <int KIND>
__device__ __forceinline__ uint64_t group_key(const TileView& V, int p, int t) {
  if (KIND == K_IDENT) return V.key(p);
  const ZMove<group_bit(KIND)> z(t);
  const uint64_t y = V.key(p);
  return KIND == K_PERM ? z(y) : (y & z.hi) | ((y & z.mid) << 1);
}

// The children of the group that starts at Z position p (0 if p does not
// start one): the mask of those that exist, child o with amplitude ca[o].
// Within a group, entries are in ascending local index, so the sums run over
// the local index in ascending order.  G is the op's gate matrix, read from
// the kernel's parameter block (the kernels take their arguments as a
// __grid_constant__), so every lane loads the same constant-bank words.
template <int KIND, bool F32>
__device__ __forceinline__ unsigned group_children(int p, const TileView& V, const double2* G, int drop_zero,
                                                   double2* ca) {
  constexpr int NC = KindTraits<KIND>::kMaxChildren;
  if (KIND == K_PERM || KIND == K_IDENT) {
    const double2 v = V.amp(p);
    if (KIND == K_IDENT && drop_zero && !cnz(v)) return 0u;
    ca[0] = v;
    return 1u;
  }
  unsigned w = V.word(p);
  if (!(w & kPlaceStart)) return 0u;
  double2 ar[NC];
  int lr[NC];
  bool in = true;
#pragma unroll
  for (int r = 0; r < NC; ++r) {
    if (r > 0) {
      in = in && (w & kPlaceNext);
      if (in) w = V.word(p + r);
    }
    lr[r] = in ? (int)((w >> kPlaceLocal) & 3u) : -1;
    ar[r] = in ? V.amp_at((int)(w & kPlaceMask)) : make_double2(0.0, 0.0);
  }
  unsigned mask = 0;
  if (F32) {
    // complex64: float gate entries and amplitudes, compensated FP32 sums
    // (Dot2); a contribution counts when neither factor is zero
    if (KIND == K_GATE1 || KIND == K_GATE2) {
#pragma unroll
      for (int o = 0; o < NC; ++o) {
        Dot2f re{0.f, 0.f}, im{0.f, 0.f};
        bool have = false;
#pragma unroll
        for (int r = 0; r < NC; ++r) {
          if (lr[r] < 0) continue;
          const float2 g = d2f(G[o * NC + lr[r]]), x = d2f(ar[r]);
          if (!((g.x != 0.f || g.y != 0.f) && (x.x != 0.f || x.y != 0.f))) continue;
          cdot2_add(re, im, g, x);
          have = true;
        }
        const double2 acc = make_double2((double)dot2_get(re), (double)dot2_get(im));
        ca[o] = acc;
        if (drop_zero == 2 ? above_drop(acc) : have) mask |= 1u << o;
      }
    } else if (KIND == K_ROT1) {
      const float2 zero = make_float2(0.f, 0.f);
      const float2 a0 = (lr[0] == 0) ? d2f(ar[0]) : zero;
      const float2 a1 = (lr[0] == 1) ? d2f(ar[0]) : (lr[1] == 1 ? d2f(ar[1]) : zero);
#pragma unroll
      for (int o = 0; o < 2; ++o) {
        Dot2f re{0.f, 0.f}, im{0.f, 0.f};
        cdot2_add(re, im, d2f(G[o * 2]), a0);
        cdot2_add(re, im, d2f(G[o * 2 + 1]), a1);
        const double2 c = make_double2((double)dot2_get(re), (double)dot2_get(im));
        ca[o] = c;
        if (above_drop(c)) mask |= 1u << o;
      }
    }
    return mask;
  }
  if (KIND == K_GATE1 || KIND == K_GATE2) {
#pragma unroll
    for (int o = 0; o < NC; ++o) {
      double2 acc = make_double2(0.0, 0.0);
      bool have = false;
#pragma unroll
      for (int r = 0; r < NC; ++r) {
        if (lr[r] < 0) continue;
        const double2 pr = cmul(G[o * NC + lr[r]], ar[r]);
        if (!cnz(pr)) continue;
        acc = have ? cadd(acc, pr) : pr;
        have = true;
      }
      ca[o] = acc;
      // drop_zero 2 (a 2-qubit rotation): the rotation's rule |a| > 1e-30
      // (bass_simulator.py:275) instead of "some product was non-zero"
      if (drop_zero == 2 ? above_drop(acc) : have) mask |= 1u << o;
    }
  } else if (KIND == K_ROT1) {
    const double2 zero = make_double2(0.0, 0.0);
    const double2 a0 = (lr[0] == 0) ? ar[0] : zero;
    const double2 a1 = (lr[0] == 1) ? ar[0] : (lr[1] == 1 ? ar[1] : zero);
#pragma unroll
    for (int o = 0; o < 2; ++o) {
      const double2 c = cadd(cmul(G[o * 2], a0), cmul(G[o * 2 + 1], a1));
      ca[o] = c;
      if (above_drop(c)) mask |= 1u << o;
    }
  }
  return mask;
}

// group_children for the state's amplitude type
template <int KIND>
__device__ __forceinline__ unsigned group_children_t(bool c64, int p, const TileView& V, const double2* G,
                                                     int drop_zero, double2* ca) {
  return c64 ? group_children<KIND, true>(p, V, G, drop_zero, ca) : group_children<KIND, false>(p, V, G, drop_zero, ca);
}

__host__ __device__ constexpr int slots_per_entry(int kind) {
  return kind == K_GATE2 ? 4 : (kind == K_GATE1 || kind == K_ROT1) ? 2 : 1;
}

// ---------------------------------------------------------------------------
// segmented launches: the block groups of a grid over many states
// ---------------------------------------------------------------------------
// Group g of a grid of N blocks over S states starts at
// start(s) = s + (N - S) * wp[s] / W, W = wp[S]: every state gets at least
// one block and the rest are shared in proportion to the work weights.
__device__ __forceinline__ long long seg_start(const SegPlan* plan, int s, long long N) {
  const int S = plan->nseg;
  const long long W = plan->wp[S] > 0 ? plan->wp[S] : 1;
  return (long long)s + ((N - S) * plan->wp[s]) / W;
}

// Blocks of state s's group in a grid of N blocks.
__device__ __forceinline__ int seg_size(const SegPlan* plan, int s, long long N) {
  return (int)(seg_start(plan, s + 1, N) - seg_start(plan, s, N));
}

// This block's state (the last s with start(s) <= blockIdx.x) and group; the
// state's op is copied into *sa.  Called by the whole block.
__device__ __forceinline__ Grp seg_enter(const OpArgs* ops, const SegPlan* plan, OpArgs* sa, int* seg_out) {
  __shared__ int sSeg, sBid, sN;
  if (threadIdx.x == 0) {
    const long long N = gridDim.x, b = blockIdx.x;
    int lo = 0, hi = plan->nseg - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (seg_start(plan, mid, N) <= b) lo = mid;
      else hi = mid - 1;
    }
    sSeg = lo;
    sBid = (int)(b - seg_start(plan, lo, N));
    sN = seg_size(plan, lo, N);
  }
  __syncthreads();
  constexpr int kWords = (int)(sizeof(OpArgs) / 8);
  static_assert(sizeof(OpArgs) % 8 == 0, "op words");
  const unsigned long long* src = reinterpret_cast<const unsigned long long*>(ops + sSeg);
  unsigned long long* dst = reinterpret_cast<unsigned long long*>(sa);
  for (int i = threadIdx.x; i < kWords; i += blockDim.x) dst[i] = src[i];
  __syncthreads();
  if (seg_out) *seg_out = sSeg;
  return Grp{sBid, sN};
}

// ---------------------------------------------------------------------------
// cooperative launches
// ---------------------------------------------------------------------------
// A cooperative launch (the runtime guarantees that every block of the grid
// is resident at once, or refuses the launch), as a programmatic dependent
// launch where the runtime accepts both attributes together; otherwise a
// plain cooperative launch.  The choice is made on the first launch and kept.
template <typename... K, typename... A>
inline cudaError_t launch_coop(void (*kern)(K...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                               A&&... args) {
  static std::atomic<int> with_pdl{1};
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  if (with_pdl.load(std::memory_order_relaxed)) {
    cfg.numAttrs = 2;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, args...);
    if (e == cudaSuccess) return e;
    cudaGetLastError();  // refused before launch: clear it and launch without PDL
    with_pdl.store(0, std::memory_order_relaxed);
  }
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...);
}

}  // namespace bass
