// op.cuh -- gates, rotation steps and truncations.
//
// An op reads a sorted state in Z order (tile.cuh), evaluates the children of
// every group, keeps the k of largest |a|^2 (ties: smaller true key) and writes
// them, sorted again, with the bookkeeping of the truncation.  Two routes:
//
//   chip    one cooperative launch.  Every block holds its tile in shared
//           memory from the load to the write, so nothing is staged, and the
//           threshold search works on |a|^2 held in registers, with a grid
//           barrier per step.  What bounds it is latency, so tiles are small
//           (252 to 508 entries; up to 1020 for gates and truncations of states
//           that only so fit), the grid is no larger than the bound asks, and
//           only blocks that have a tile take part in the barriers: a state of
//           up to 508 entries is one block's, without any.
//   staged  larger states: a sample of the children brackets the threshold
//           first; the evaluation then stages only the children at or above the
//           bracket (the ones certainly kept, and the few per cent inside it),
//           compacted per warp, and sums the certain ones as it goes; the
//           children inside the bracket are settled, and the write step copies.
//           What bounds it is instruction issue in the evaluation and memory
//           traffic in the copy; the passes are launches of their own so that
//           each has the registers it needs (as one kernel of barriers the
//           evaluation spilled: 142 us instead of 93 at 2^22 entries).  A bracket
//           that missed the threshold (seen from exact counts) is replaced by the
//           exact one and the evaluation repeated: the result never depends on
//           the sample.
//
// The host takes the chip route when the workspace bounds the state's entries by
// what it holds (launch_op); under a larger bound the staged route's first launch
// does the whole op if the state turns out small, and the others return at once.
//
// Measured on one B200 (us per op back to back, 40 qubits, complex128, top k =
// n, target at a high physical bit; before: a launch each for partition,
// evaluation of every child into 56 bytes of staging per entry, a selection of
// three histogram passes with grid barriers, and compaction):
//   n              64   508  16384  65536  300000  600000   2^20   2^22
//   1-qubit gate   14    17     31     35      48      60     89    198
//   before         38    43     60     64      69      75     91    221
//   2-qubit gate   30    39     54     58      87     121    147    350
//   before         55    62     99    113     124     141    171    429
//   rejected step  12    15     37     38      63      76     75    153
//   before         41    43     59     69      75      79     95    198
// (Between 620,000 and 2^20 entries a 1-qubit gate is 3 to 5 per cent slower than
// before, 9 on the lowest bit: its evaluation then has one tile for every second
// block.)
#pragma once

#include <math.h>

#include "tile.cuh"

namespace bass {

// Chip tiles of PT entries per thread: 2 (the smallest chains), or 4 for states
// that only so fit the chip.
template <int PT>
constexpr int kChipTile = PT * kThreads;         // 512, 1024
template <int PT>
constexpr int kChipStep = kChipTile<PT> - 4;     // a boundary backs off by at most 4
constexpr int kChipMin = 252;                    // smallest tile step when the grid would allow less
template <int PT>
constexpr int kChipPad = kChipTile<PT> + 8;
constexpr int kChipBins = 2048;                  // digits of the chip search: 11 bits (the first: the exponent)
constexpr int kChipLate = 32;                    // undecided children it stops at (one per lane of a warp)
constexpr int kSelMax = 256;                     // boundary children settled by ranking (one per thread)
constexpr int kSamples = 16384;                  // sampled entries of the bracket, at most
constexpr int kSampleRounds = 2;                 // ... per eight lanes of a group's blocks
constexpr int kRegion = 32 * kPerThread;         // Z positions of a warp's region of a tile
constexpr int kRegions = kThreads / 32;          // regions of a tile
// Blocks of a staged op's first launch: they do the whole op for a state of up
// to kFirstBlocks x kChipStep = 32,512 entries under a larger bound.  One per SM
// (148) would take states of 75,000 entries, but costs a gate at 2^22 entries
// 3 us (202 instead of 199), and at 65,536 entries its staged route is as fast.
// A truncation takes one per SM: staged it is slower there (65,536 entries: 51 us
// instead of 37), and at 2^22 no difference shows.
constexpr int kFirstBlocks = 64;
// |a|^2 bins of the sample: 128 per power of two over [2^-64, 1); what lies
// beyond (in the two outer bins) is also counted four bins to a power of two
constexpr int kSampleBase = (1023 - 64) << 7;
constexpr int kFarShift = 50;

// 8-byte words of the workspace counters, zeroed at the start of the op
enum OpCounter { C_TILE = 0, C_LIST = 1, C_OUT = 2, C_DEF = 3, C_STAGED = 4, C_TILE2 = 5, C_LIMB = 8 };
constexpr int kOpCounters = 16;  // C_LIMB: 2 sums x 4 words of 32 bits of the sum each
// ws.red as 8-byte words: the op's OpResult, its OpStage, then the undecided
// children's patterns, true keys and places
constexpr int kResultAt = 0, kStageAt = 16, kListAt = 64;
static_assert(kListAt + 3 * kSelMax <= 2 * 1024, "the list fits ws.red");

// dynamic shared memory: a staged tile; a chip tile plus the histogram (which
// the settled children share)
constexpr size_t kTileSmem = (size_t)kTilePad * (16 + 8 + 2);
template <int PT>
constexpr size_t kChipHistAt = ((size_t)kChipPad<PT> * (16 + 8 + 2) + 127) & ~(size_t)127;
template <int PT>
constexpr size_t kChipSmem = kChipHistAt<PT> + (size_t)kChipBins * 4;

// ---------------------------------------------------------------------------
// grid barriers
// ---------------------------------------------------------------------------
// One word of the control block (zero between ops): bits 0-19 arrivals of the
// op's barriers, bits 20-29 blocks that are done, bit 30 the launch was called
// off, bit 31 some block gave up.  The last block to finish resets it.
//
// Blocks that wait for one another have to be resident together: their launch
// is cooperative, or its first barrier may be called off.  A cooperative launch
// does not start beside the end of the kernel before it (4 us of every staged
// op at 2^20 entries), so the launch that only does the whole op for states
// that turn out small is a plain one: whoever waits too long at its first
// barrier calls the launch off, which nobody can once all blocks have arrived
// (and so are resident), and the staged launches that follow do the op.
constexpr unsigned kArriveMask = (1u << 20) - 1, kExitOne = 1u << 20, kExitMask = (1u << 10) - 1;
constexpr unsigned kOffBit = 1u << 30, kFailBit = 1u << 31;
constexpr long long kOffSpins = 512;  // polls (some 100 us) before a launch is called off

struct Gate {
  unsigned* word;
  int nact;         // blocks that take part
  int all;          // arrivals of the first barrier (every block of the launch may count there)
  unsigned passed;  // barriers entered
  bool off;         // the launch was called off
};

// Block-wide: arrive (everything written before is visible to the blocks that
// pass gate_wait).
__device__ __forceinline__ void gate_arrive(Gate& b) {
  __syncthreads();
  ++b.passed;
  if ((b.nact > 1 || b.passed == 1) && b.all > 1 && threadIdx.x == 0) {
    __threadfence();
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(b.word), "r"(1u) : "memory");
  }
}
// Block-wide: wait until every block has arrived (bounded; false on give-up,
// with BASS_ERR_WAIT recorded).  OFF: the launch's first barrier, which may be
// called off (false then too).
template <bool OFF = false>
__device__ __forceinline__ bool gate_wait(Gate& b, bass_ctrl* c) {
  __shared__ int sOk;  // 1 all arrived, 0 gave up, -1 called off
  if (b.nact > 1 || (b.passed == 1 && b.all > 1)) {
    if (threadIdx.x == 0) {
      const unsigned target = (unsigned)b.all + (b.passed - 1) * (unsigned)b.nact;
      long long lim = wait_limit(c);
      if (OFF && lim > kOffSpins) lim = kOffSpins;
      long long spins = 0;
      int ok = 1;
      for (;;) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(b.word) : "memory");
        if (OFF && (v & kOffBit)) {
          ok = -1;
          break;
        }
        if ((v & kArriveMask) >= target) break;
        if (++spins > lim) {
          if (!OFF) {
            set_error(c, BASS_ERR_WAIT);
            ok = 0;
            break;
          }
          atomicCAS(b.word, v, v | kOffBit);  // (or the word has changed: look again)
          continue;
        }
        __nanosleep(b.nact > 64 ? 100 : 20);  // (hundreds of pollers would hold up the arrivals)
      }
      __threadfence();
      sOk = ok;
    }
    __syncthreads();
    if (OFF) b.off = sOk < 0;
    return sOk > 0;
  }
  __syncthreads();
  return true;
}
__device__ __forceinline__ bool gate_sync(Gate& b, bass_ctrl* c) {
  gate_arrive(b);
  return gate_wait(b, c);
}
// Block-wide, once per block of the group, in the last block to call: 1, or 2
// if some block gave up, or 3 if the launch was called off; 0 in the others.
__device__ __forceinline__ int op_exit(bass_ctrl* c, int nblk, bool failed) {
  __shared__ int sLast;
  __syncthreads();
  if (nblk == 1) return failed ? 2 : 1;
  if (threadIdx.x == 0) {
    if (failed) atomicOr(&c->sync_counter, kFailBit);
    __threadfence();
    const unsigned old = atomicAdd(&c->sync_counter, kExitOne);
    const bool last = ((old >> 20) & kExitMask) == (unsigned)(nblk - 1);
    sLast = last ? ((old & kFailBit) ? 2 : (old & kOffBit) ? 3 : 1) : 0;
    if (last) *(volatile uint32_t*)&c->sync_counter = 0u;
    __threadfence();
  }
  __syncthreads();
  return sLast;
}

// ---------------------------------------------------------------------------
// exact sums
// ---------------------------------------------------------------------------
// Sums of fx_from(p) over terms 0 <= p < 1: the sum is carried in two doubles
// that stay within one binade, h in [16, 32) with unit 2^-48 and l in
// [2^-44, 2^-43) with unit 2^-96, and every addition rounds toward zero: h + p
// takes the term's multiple of 2^-48, what is left over (exact, below 2^-48)
// is truncated into l at 2^-96.  Four additions a term and no conversion: a
// run's (at most 16 terms) integers are the mantissa bits, added up in 64-bit
// words.  Larger terms take the integer path (fx_from_pbits).
struct Acc {
  double h, l;       // of the current run (at most 16 terms)
  long long ih, il;  // in units of 2^-48 and 2^-96
  __device__ __forceinline__ void clear() {
    h = 16.0;
    l = 0x1p-44;
    ih = il = 0;
  }
  __device__ __forceinline__ void add(double p) {  // 0 <= p < 1
    const double n = __dadd_rz(h, p);
    const double b = __dsub_rn(p, __dsub_rn(n, h));
    h = n;
    l = __dadd_rz(l, b);
  }
  __device__ __forceinline__ void fold() {  // after at most 16 terms
    constexpr long long kMant = (1LL << 52) - 1;
    ih += __double_as_longlong(h) & kMant;
    il += __double_as_longlong(l) & kMant;
    h = 16.0;
    l = 0x1p-44;
  }
  __device__ __forceinline__ i128 get() const { return (i128)ih * (i128)281474976710656LL + (i128)il; }
};
constexpr unsigned long long kOneBits = 0x3FF0000000000000ULL;  // the pattern of 1.0

// ---------------------------------------------------------------------------
// the threshold
// ---------------------------------------------------------------------------
// What survives: children are ranked by (|a|^2 bits descending, true key
// ascending).  The search narrows an undecided range [lo, hi] of bit patterns,
// then (when more than kSelMax children share one pattern) of inverted true
// keys, 13 bits at a time.
struct Cut {
  unsigned long long lo, hi;  // the undecided range, inclusive
  unsigned long long tie;     // C_KEYS: the pattern whose children are ranked by key
  long long need;             // children of the undecided range that are kept
  int mode;
  int all;   // the undecided range is kept whole
  int late;  // its (at most kSelMax) children are ranked one by one
};
enum CutMode { CUT_ALL = 0, CUT_NONE = 1, CUT_BITS = 2, CUT_KEYS = 3 };

// 1 kept, 0 dropped, 2 undecided
template <class KeyFn>
__device__ __forceinline__ int cut_class(const Cut& c, unsigned long long bits, KeyFn true_key_of) {
  if (c.mode == CUT_ALL) return 1;
  if (c.mode == CUT_NONE) return 0;
  unsigned long long x = bits;
  if (c.mode == CUT_KEYS) {
    if (bits != c.tie) return bits > c.tie ? 1 : 0;
    x = ~true_key_of();
  }
  if (x > c.hi) return 1;
  if (x < c.lo) return 0;
  return c.all ? 1 : 2;
}
template <int NB>
__device__ __forceinline__ int digit_shift(unsigned long long lo, unsigned long long hi) {
  constexpr int kBits = NB == 8192 ? 13 : 11;
  static_assert(NB == 1 << kBits, "digit size");
  const unsigned long long span = hi - lo;
  const int bits = span ? 64 - __clzll((long long)span) : 0;
  return bits > kBits ? bits - kBits : 0;
}
template <int NB>
__device__ __forceinline__ unsigned digit_of(unsigned long long x, unsigned long long lo, int shift) {
  const unsigned long long d = (x - lo) >> shift;
  return d < (unsigned long long)NB ? (unsigned)d : (unsigned)(NB - 1);
}
// After the bin of the undecided range's histogram that holds the need-th child
// is known (above: children in higher bins, cnt: in it).  false: search on, with
// the new range and shift.  The highest of the NB bins also holds what lies beyond
// the histogram's range; at most LATE children are left to be ranked.
template <int NB, int LATE>
__device__ __forceinline__ bool cut_narrow(Cut& c, int* shift, int bin, long long above, long long cnt) {
  constexpr int top = NB - 1;
  c.need -= above;
  const unsigned long long prev = c.hi;
  c.lo += (unsigned long long)bin << *shift;
  if (bin != top) {
    const unsigned long long end = c.lo + ((1ULL << *shift) - 1);
    c.hi = end < prev ? end : prev;
  }
  if (c.need >= cnt) {
    c.all = 1;
    return true;
  }
  if (cnt <= LATE) {
    c.late = 1;
    return true;
  }
  if (c.lo == c.hi) {
    if (c.mode == CUT_KEYS) {  // distinct keys: not reached
      c.all = 1;
      return true;
    }
    c.mode = CUT_KEYS;
    c.tie = c.lo;
    c.lo = 0ULL;
    c.hi = ~0ULL;
  }
  *shift = digit_shift<NB>(c.lo, c.hi);
  return false;
}

// Block-wide: per thread the count s of its NB / 256 bins (thread 0 the
// highest) and the inclusive count x from the top.
struct FindSh {
  unsigned long long w[kThreads / 32];
  long long above, cnt;
  int bin, owner;
};
template <bool GLOBAL, int NB>
__device__ __forceinline__ void top_scan(const unsigned* h, FindSh& F, unsigned long long* s, unsigned long long* x) {
  constexpr int PB = NB / kThreads;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const uint4* p = reinterpret_cast<const uint4*>(h + NB - PB * (tid + 1));
  unsigned long long v = 0;
#pragma unroll
  for (int q = 0; q < PB / 4; ++q) {
    const uint4 u = GLOBAL ? __ldcg(p + q) : p[q];
    v += (unsigned long long)u.x + u.y + u.z + u.w;
  }
  unsigned long long y = v;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const unsigned long long z = __shfl_up_sync(0xffffffffu, y, off);
    if (lane >= off) y += z;
  }
  __syncthreads();
  if (lane == 31) F.w[w] = y;
  __syncthreads();
  for (int i = 0; i < w; ++i) y += F.w[i];
  *s = v;
  *x = y;
}
// Block-wide: F.bin, F.above, F.cnt for the need-th count from the top
// (1 <= need <= total; beyond the total: bin 0).  Warp 0 reads the bins of the
// thread whose counts hold it, one per lane.
template <bool GLOBAL, int NB>
__device__ __forceinline__ void top_locate(const unsigned* h, FindSh& F, unsigned long long s, unsigned long long x,
                                           long long need) {
  constexpr int PB = NB / kThreads;
  const int tid = threadIdx.x;
  const bool beyond = tid == kThreads - 1 && (long long)x < need;
  if (((long long)(x - s) < need && need <= (long long)x) || beyond) {
    F.owner = tid;
    F.above = (long long)(x - s);
  }
  __syncthreads();
  if (tid < 32) {
    const int top = NB - PB * F.owner - 1;
    const long long above = F.above;
    const long long c = tid < PB ? (long long)(GLOBAL ? __ldcg(h + top - tid) : h[top - tid]) : 0;
    long long inc = c;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const long long y = __shfl_up_sync(0xffffffffu, inc, off);
      if (tid >= off) inc += y;
    }
    const unsigned m = __ballot_sync(0xffffffffu, above + inc >= need);
    const int l = m ? __ffs(m) - 1 : PB - 1;
    __syncwarp();
    if (tid == (l < PB ? l : PB - 1)) {
      F.bin = top - tid;
      F.above = above + inc - c;
      F.cnt = c;
    }
  }
  __syncthreads();
}
template <bool GLOBAL, int NB>
__device__ __forceinline__ void find_top(const unsigned* h, FindSh& F, long long need) {
  unsigned long long s, x;
  top_scan<GLOBAL, NB>(h, F, &s, &x);
  top_locate<GLOBAL, NB>(h, F, s, x, need);
}
// Block-wide, at most kSelMax listed children: thread i's child is kept if
// fewer than need rank above it.
struct CandSh {
  unsigned long long bits[kSelMax], key[kSelMax], code[kSelMax];
};
__device__ __forceinline__ bool rank_cand(const CandSh& C, int m, long long need) {
  const int i = threadIdx.x;
  if (i >= m) return false;
  const unsigned long long b = C.bits[i], k = C.key[i];
  int r = 0;
  for (int j = 0; j < m; ++j) r += C.bits[j] > b || (C.bits[j] == b && C.key[j] < k);
  return r < need;
}
// l: the list (ws.red from word kListAt on, or a CandSh).
__device__ __forceinline__ unsigned long long* cand_list(const OpArgs& a) {
  return reinterpret_cast<unsigned long long*>(a.ws.red) + kListAt;
}
__device__ __forceinline__ void list_cand(unsigned long long* l, unsigned long long* cn, unsigned long long bits,
                                          unsigned long long key, unsigned long long code) {
  const unsigned long long i = atomicAdd(cn + C_LIST, 1ULL);
  if (i < kSelMax) {
    l[i] = bits;
    l[kSelMax + i] = key;
    l[2 * kSelMax + i] = code;
  }
}
__device__ __forceinline__ int load_cands(const unsigned long long* l, const unsigned long long* cn, CandSh& C) {
  const unsigned long long n = *(const volatile unsigned long long*)(cn + C_LIST);
  const int m = n < kSelMax ? (int)n : kSelMax;
  const int i = threadIdx.x;
  if (l != C.bits && i < m) {
    C.bits[i] = __ldcg(l + i);
    C.key[i] = __ldcg(l + kSelMax + i);
    C.code[i] = __ldcg(l + 2 * kSelMax + i);
  }
  __syncthreads();
  return m;
}

// ---------------------------------------------------------------------------
// the result
// ---------------------------------------------------------------------------
struct OpResult {
  long long n_out, n_written;
  double kept, total, pr_new;
  int trunc, accept;
  int skip;    // a rejected rotation candidate is not written
  int failed;  // a wait gave up: no result (or kOver)
};
constexpr int kOver = 2;  // the op's first launch did the whole op, or refused it

// What a candidate's PR has to stay below (bass_simulator.py:795-814, with the
// relative tolerance).  Read before the first barrier: the op's end rewrites pr_cur.
__device__ __forceinline__ double pr_limit_of(const bass_ctrl* c) { return c->pr_cur * (1.0 - c->pr_tie_tol); }

// Every block computes the same: sums, and for a rotation step (mode 1) the
// decision of bass_simulator.py:795-814: the candidate's PR = kept^2 / sum |a|^4
// against pr_limit (pr_limit_of).
__device__ __forceinline__ void decide(const OpArgs& a, i128 v0, i128 v1, double pr_limit, OpResult& R) {
  R.kept = fx_to(v0);
  R.total = 0.0;
  R.pr_new = 0.0;
  R.accept = 0;
  R.skip = 0;
  if (a.fin_mode == 1) {
    const double p2 = fx_to(v1);
    const long long n_kept = R.trunc ? (a.k_keep > 0 ? a.k_keep : 0) : R.n_out;
    R.pr_new = (n_kept == 0 || !(p2 > 0.0)) ? INFINITY : __ddiv_rn(__dmul_rn(R.kept, R.kept), p2);
    const bool reject = R.pr_new >= pr_limit;
    R.accept = reject ? 0 : 1;
    R.skip = (reject && !a.tr.trace) ? 1 : 0;
  } else if (R.trunc) {
    R.total = fx_to(v1);
  }
}

// The last block to finish: the output descriptor, the gamma / truncation
// bookkeeping, and on a rotation step without a trace the swap that makes an
// accepted candidate the state.  ws.sel keeps what the traced commit and the
// event fingerprint read.
static __device__ void op_finalize(const OpArgs& a, int kind, const OpResult& R) {
  __shared__ int8_t sQo[64];
  const int tid = threadIdx.x;
  const bass_state* in = a.in;
  bass_state* out = a.out;
  bass_ctrl* c = a.ctrl;
  out_order_par(in, kind, a.q, a.gb, sQo);
  __syncthreads();
  if (tid == 0) {
    const long long n_in = in->nnz;
    long long nw = R.n_written;
    if (nw > out->cap) {
      set_error(c, BASS_ERR_CAPACITY);
      nw = 0;
    }
    out->nq = in->nq;
    out->amp_type = in->amp_type;
    out->nnz = nw;
    out->rscale[0] = 1.0;
    out->rscale[1] = 1.0;
    if (kind != K_PERM) {  // the first pass of a 2-qubit gate: no bookkeeping
      // an amplitude update is an input entry of a gate or a rotation step; a
      // plain truncation (K_IDENT) transforms nothing
      if (kind != K_IDENT) c->amp_updates += n_in;
      c->n_ops += 1;
      SelState* sel = a.ws.sel;
      sel->n_out = R.n_out;
      sel->k_keep = a.k_keep;
      sel->do_trunc = R.trunc;
      sel->kept = R.kept;
      sel->total = R.total;
      sel->n_written = R.n_written;
      sel->accept = R.accept;
      sel->pr_new = R.pr_new;
      const double nrm = sqrt(R.kept);
      if (a.fin_mode == 1) {
        c->frac[a.j] = R.kept;
        c->accept[a.j] = R.accept;
        if (nrm > 1e-30) out->rscale[0] = 1.0 / nrm;
      } else {
        c->last_truncated = R.trunc;
        if (R.trunc) {
          c->last_kept = R.kept;
          c->last_total = R.total;
          c->n_trunc += 1;
          if (a.tr.gamma_mode == 1) c->gamma_running *= (R.total > 1e-30 ? R.kept / R.total : 0.0);
          else if (a.tr.gamma_mode == 2) c->state_gamma *= (R.total > 1e-30 ? sqrt(R.kept / R.total) : 0.0);
          else if (a.tr.gamma_mode == 3) c->state_gamma *= nrm;
          if (a.tr.renorm == 1) {
            if (nrm > 1e-30) out->rscale[0] = 1.0 / nrm;
          } else if (a.tr.renorm == 2) {
            out->rscale[0] = 1.0 / nrm;
          }
          if (a.tr.mark_active) {
            c->truncation_active = 1;
            c->gates_since_trunc = 0;
          }
        }
      }
    }
  }
  if (tid < 64) {
    out->qat[tid] = sQo[tid];
    out->pos[sQo[tid]] = (int8_t)tid;
  }
  if (!a.commit || !R.accept) return;
  __syncthreads();
  constexpr int kWords = (int)(sizeof(bass_state) / 8);
  static_assert(sizeof(bass_state) % 8 == 0, "descriptor words");
  unsigned long long* pc = reinterpret_cast<unsigned long long*>(const_cast<bass_state*>(in));
  unsigned long long* pt = reinterpret_cast<unsigned long long*>(out);
  unsigned long long wc = 0, wt = 0;
  if (tid < kWords) {
    wc = pc[tid];
    wt = pt[tid];
  }
  __syncthreads();
  if (tid < kWords) {
    pc[tid] = wt;
    pt[tid] = wc;
  }
  if (tid == 0) {
    c->pr_cur = R.pr_new;
    const double frac = R.kept;
    c->gamma_running *= sqrt(frac > 1e-30 ? frac : 0.0);
  }
}

// ---------------------------------------------------------------------------
// the op
// ---------------------------------------------------------------------------
struct Bracket {
  unsigned long long lo, hi;  // certainly kept from hi on, undecided in [lo, hi), dropped below lo
  int shift;                  // of the undecided children's histogram
  int pad;
};
// What one pass of the staged route leaves for the next.
struct OpStage {
  Bracket B;
  Cut cut;
  long long n_out;
  int trunc;
  int state;  // StageState
};
enum StageState { ST_OK = 0, ST_MISSED = 1 /* the threshold is outside the bracket */, ST_GAVE_UP = 2,
                  ST_OVER = 3 /* as kOver */ };
static_assert(sizeof(OpResult) % 8 == 0 && sizeof(OpResult) <= 8 * (kStageAt - kResultAt), "result words");
static_assert(sizeof(OpStage) % 8 == 0 && sizeof(OpStage) <= 8 * (kListAt - kStageAt), "stage words");

struct OpSh {
  TileSeg T;
  long long rec[2][6];
  FindSh F;
  OpResult R;
  OpStage St;
  unsigned long long cn[kOpCounters];  // the counters of a one-block op
  unsigned long long limb[8];
  i128 red[2 * kRegions];
  long long sum[5 * kRegions];  // block_sum's
  int warp[4 * kRegions];
  uint64_t bar;
  long long item;
  int8_t qat[64];  // output qubit order
  uint64_t* okeys;  // the output's arrays
  double* oamps;
  long long ocap;
  double pr_limit;
};
// One thread, at the start of a kernel: what the op's end may rewrite.
__device__ __forceinline__ void op_preload(const OpArgs& a, OpSh& sh) {
  sh.okeys = a.out->keys;
  sh.oamps = a.out->amps;
  sh.ocap = a.out->cap;
  sh.pr_limit = pr_limit_of(a.ctrl);
}
// Block-wide copies between shared memory and ws.red (a __syncthreads before
// store_words and after load_words is the caller's).
template <typename T>
__device__ __forceinline__ void store_words(const OpArgs& a, int at, const T& v) {
  if (threadIdx.x < sizeof(T) / 8)
    (reinterpret_cast<unsigned long long*>(a.ws.red) + at)[threadIdx.x] =
        reinterpret_cast<const unsigned long long*>(&v)[threadIdx.x];
}
template <typename T>
__device__ __forceinline__ void load_words(const OpArgs& a, int at, T& v) {
  if (threadIdx.x < sizeof(T) / 8)
    reinterpret_cast<unsigned long long*>(&v)[threadIdx.x] =
        __ldcg(reinterpret_cast<const unsigned long long*>(a.ws.red) + at + threadIdx.x);
}

__device__ __forceinline__ OpStage* stage_of(const OpArgs& a) {
  return reinterpret_cast<OpStage*>(reinterpret_cast<unsigned long long*>(a.ws.red) + kStageAt);
}
__device__ __forceinline__ OpResult* result_of(const OpArgs& a) {
  return reinterpret_cast<OpResult*>(reinterpret_cast<unsigned long long*>(a.ws.red) + kResultAt);
}

constexpr long long kMaxEntries = 1LL << 31;  // an op takes fewer
// The op's input, the same in every thread.
struct OpCtx {
  TileSrc S;
  double r0, r1;
  int t;
  bool may_trunc;
  bool bad;  // refused (amplitude type, workspace)
  long long ntiles;
  long long lim;  // tries of a bounded wait
};
template <int KIND, bool C64>
__device__ __forceinline__ OpCtx op_ctx(const OpArgs& a) {
  constexpr int NS = slots_per_entry(KIND);
  const bass_state* in = a.in;
  OpCtx X;
  X.S.keys = in->keys;
  X.S.amps = reinterpret_cast<const double2*>(in->amps);
  const long long n = in->nnz;
  X.S.n = n;
  X.S.tma = ((reinterpret_cast<uintptr_t>(X.S.keys) | reinterpret_cast<uintptr_t>(X.S.amps)) & 15) == 0;
  X.r0 = in->rscale[0];
  X.r1 = in->rscale[1];
  X.t = KIND == K_IDENT ? 0 : in->pos[a.q];
  X.lim = wait_limit(a.ctrl);
  const long long children = (long long)NS * n;
  X.may_trunc = KIND != K_PERM && a.k_cond >= 0 && children > a.k_cond && children > a.k_keep;
  X.ntiles = KIND == K_IDENT ? plain_tiles(n) : merge_tiles(n);
  X.bad = (in->amp_type == BASS_AMP_C64) != C64 || X.ntiles > a.ws.max_tiles || children > a.ws.max_n ||
          n >= kMaxEntries;
  return X;
}
// One thread: the refusal's error bits.
__device__ __forceinline__ void op_refuse(const OpArgs& a, bool c64) {
  if ((a.in->amp_type == BASS_AMP_C64) != c64) set_error(a.ctrl, BASS_ERR_ARG);
  set_error(a.ctrl, BASS_ERR_WORKSPACE);
}

// Block sums of N longs (every thread gets all); sh: 8 N words.
template <int N>
__device__ __forceinline__ void block_sum(long long (&v)[N], long long* sh) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < N; ++k)
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], off);
  __syncthreads();
  if (lane == 0) {
#pragma unroll
    for (int k = 0; k < N; ++k) sh[k * kRegions + w] = v[k];
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < N; ++k) {
    v[k] = 0;
#pragma unroll
    for (int i = 0; i < kRegions; ++i) v[k] += sh[k * kRegions + i];
  }
}

// Block-wide: adds the threads' two sums to the counters' limbs.
__device__ __forceinline__ void flush_sums(OpSh& sh, unsigned long long* cn, i128 v0, i128 v1) {
  i128 v[2] = {v0, v1};
  block_sum_i128<2>(v, sh.red);
  if (threadIdx.x == 0) {
    limb_add(cn + C_LIMB, v[0]);
    limb_add(cn + C_LIMB + 4, v[1]);
  }
}

// ---- chip route -------------------------------------------------------------
// Block b of nact holds tile b (step Z positions).  Returns false if a wait
// gave up; otherwise sh.R is the op's result.
template <int KIND, bool C64, bool OFF, int PT>
__device__ __forceinline__ bool op_chip(const OpArgs& a, const Grp& g, OpSh& sh, const OpCtx& X, Gate& gate, int step,
                                        unsigned char* smem) {
  constexpr int NS = slots_per_entry(KIND);
  constexpr bool P2 = KIND == K_ROT1;  // rotation steps: sums of |a|^2 and |a|^4; others: kept and total |a|^2
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  double2* sA = reinterpret_cast<double2*>(smem);
  uint64_t* sZ = reinterpret_cast<uint64_t*>(sA + kChipPad<PT>);
  uint16_t* sIdx = reinterpret_cast<uint16_t*>(sZ + kChipPad<PT>);
  unsigned* sHist = reinterpret_cast<unsigned*>(smem + kChipHistAt<PT>);
  CandSh& sCand = *reinterpret_cast<CandSh*>(sHist);                              // after the search
  uint8_t* sKeep = reinterpret_cast<uint8_t*>(sHist) + ((sizeof(CandSh) + 15) & ~15);  // per position, settled children
  static_assert(((sizeof(CandSh) + 15) & ~15) + kChipTile<PT> <= 4 * kChipBins, "the settled children fit the histogram");
  const bool multi = gate.nact > 1;
  const int nact = gate.nact;
  const long long n = X.S.n;
  unsigned long long* cn = multi ? reinterpret_cast<unsigned long long*>(a.ws.counters) : sh.cn;
  if (KIND != K_PERM) {
    // cleared for the first use after the first barrier
    if (multi) {
      const int i0 = g.bid * kThreads + tid, st = nact * kThreads;
      if (X.may_trunc) {
        for (int i = i0; i < kChipBins; i += st) a.ws.hist1[i] = a.ws.hist2[i] = 0u;
      }
      if (i0 < kOpCounters) cn[i0] = 0ULL;
    } else if (tid < kOpCounters) {
      cn[tid] = 0ULL;
    }
    gate_arrive(gate);
  }
  // the tile
  if (KIND == K_IDENT) {
    if (tid < 12) {
      const long long lo = (long long)(g.bid + (tid >= 6)) * step;
      const long long P = lo < n ? lo : n;
      const int f = tid % 6;
      // one segment: a block [0, n) without bit-set entries
      sh.rec[tid / 6][f] = f == 0 ? P : f == 1 ? 0 : f == 2 ? n : f == 3 ? n : f == 4 ? P : 0;
    }
  } else if (!multi) {
    // the whole state: whole blocks only, no boundary to search for
    if (tid < 12) sh.rec[tid / 6][tid % 6] = tid >= 6 && tid < 10 ? n : 0;
  } else if (w < 2) {
    long long r[6];
    tile_boundary<group_bit(KIND)>(X.S.keys, n, (long long)(g.bid + w) * step, X.t, KIND != K_PERM, r);
    if (lane == 0)
      for (int q = 0; q < 6; ++q) sh.rec[w][q] = r[q];
  }
  __syncthreads();
  if (tid == 0)
    tile_segments<C64>(sh.T, sh.rec[0], sh.rec[1], X.S, kChipTile<PT>, sZ, sA, &sh.bar, a.ctrl);
  if (KIND != K_PERM && X.may_trunc)
    for (int i = tid; i < kChipBins; i += kThreads) sHist[i] = 0u;
  __syncthreads();
  unsigned phase = 0;
  if (!tile_fetch<PT, C64>(sh.T, X.S, sZ, sA, &sh.bar, &phase, a.ctrl, X.lim)) return false;
  const int E = (int)sh.T.off[5];
  if (KIND != K_IDENT) tile_zorder<PT, group_bit(KIND)>(sh.T, sZ, sIdx, sh.warp, X.t);
  const bool scaled = !(X.r0 == 1.0 && X.r1 == 1.0);
  const TileView V{sZ, sA, reinterpret_cast<const float2*>(sA), KIND == K_IDENT ? nullptr : sIdx, X.r0, X.r1, scaled, C64};
  double2 ca[NS];

  if (KIND == K_PERM) {  // a reorder: every entry to its Z position
    const long long zs = sh.T.zs;
    if (n <= sh.ocap) {
      for (int p = tid; p < E; p += kThreads) {
        sh.okeys[zs + p] = group_key<K_PERM>(V, p, X.t);
        amp_put(sh.oamps, zs + p, V.amp(p), C64);
      }
    }
    if (tid == 0) {
      sh.R = OpResult{};
      sh.R.n_written = n;
    }
    __syncthreads();
    return true;
  }

  // the children's |a|^2 patterns (~0: no such child)
  unsigned long long bits[PT][NS];
  int nex = 0;
#pragma unroll
  for (int r = 0; r < PT; ++r) {
    const int p = r * kThreads + tid;
    unsigned cm = 0;
    if (p < E) cm = group_children_t<KIND>(C64, p, V, a.G, a.drop_zero, ca);
#pragma unroll
    for (int c = 0; c < NS; ++c) {
      const bool on = (cm >> c) & 1u;
      bits[r][c] = on ? (unsigned long long)__double_as_longlong(prob(ca[c])) : ~0ULL;
      // the search's first digit: the exponent, counted in shared memory (few
      // bins hold most children)
      if (X.may_trunc && on) atomicAdd(&sHist[digit_of<kChipBins>(bits[r][c], 0ULL, 52)], 1u);
    }
    nex += __popc(cm);
  }
  nex = (int)__reduce_add_sync(0xffffffffu, (unsigned)nex);
  if (!gate_wait<OFF>(gate, a.ctrl)) return false;
  if (lane == 0 && nex) atomicAdd(cn + C_OUT, (unsigned long long)nex);

  // the threshold
  Cut cut{0ULL, ~0ULL - 1, 0ULL, a.k_keep, CUT_ALL, 0, 0};
  long long n_out = 0;
  int trunc = 0;
  if (X.may_trunc) {
    if (multi)
      for (int i = tid; i < kChipBins; i += kThreads)
        if (sHist[i]) atomicAdd(a.ws.hist1 + i, sHist[i]);
    if (!gate_sync(gate, a.ctrl)) return false;
    n_out = (long long)*(volatile unsigned long long*)(cn + C_OUT);
    trunc = !(n_out <= a.k_cond || a.k_keep >= n_out);
    if (trunc) cut.mode = a.k_keep <= 0 ? CUT_NONE : CUT_BITS;
    if (cut.mode == CUT_BITS) {
      int shift = 52;
      if (multi) find_top<true, kChipBins>(a.ws.hist1, sh.F, cut.need);
      else find_top<false, kChipBins>(sHist, sh.F, cut.need);
      bool found = cut_narrow<kChipBins, kChipLate>(cut, &shift, sh.F.bin, sh.F.above, sh.F.cnt);
      __syncthreads();
      for (int level = 1; !found; ++level) {
        unsigned* gh = multi ? ((level & 1) ? a.ws.hist2 : a.ws.hist1) : sHist;
        if (multi && level >= 2) {
          // the buffer's last readers passed the previous level's barrier
          for (int i = g.bid * kThreads + tid; i < kChipBins; i += nact * kThreads) gh[i] = 0u;
          if (!gate_sync(gate, a.ctrl)) return false;
        } else if (!multi) {
          for (int i = tid; i < kChipBins; i += kThreads) gh[i] = 0u;
          __syncthreads();
        }
#pragma unroll
        for (int r = 0; r < PT; ++r) {
#pragma unroll
          for (int c = 0; c < NS; ++c) {
            const unsigned long long b = bits[r][c];
            if (b == ~0ULL) continue;
            const int p = r * kThreads + tid;
            auto tk = [&]() { return true_key(group_key<KIND>(V, p, X.t) | (uint64_t)c, sh.qat, 64); };
            if (cut_class(cut, b, tk) != 2) continue;
            atomicAdd(gh + digit_of<kChipBins>(cut.mode == CUT_KEYS ? ~tk() : b, cut.lo, shift), 1u);
          }
        }
        if (!gate_sync(gate, a.ctrl)) return false;
        if (multi) find_top<true, kChipBins>(gh, sh.F, cut.need);
        else find_top<false, kChipBins>(gh, sh.F, cut.need);
        found = cut_narrow<kChipBins, kChipLate>(cut, &shift, sh.F.bin, sh.F.above, sh.F.cnt);
        __syncthreads();
      }
    }
  }

  // who is kept, the sums, the undecided ones' list
  unsigned long long* list = multi ? cand_list(a) : sCand.bits;
  const bool sums = P2 || trunc;
  unsigned kept[PT];
  int nkeep = 0;
  Acc s0, s1;
  s0.clear();
  s1.clear();
#pragma unroll
  for (int r = 0; r < PT; ++r) {
    kept[r] = 0;
    const int p = r * kThreads + tid;
#pragma unroll
    for (int c = 0; c < NS; ++c) {
      const unsigned long long b = bits[r][c];
      if (b == ~0ULL) continue;
      auto tk = [&]() { return true_key(group_key<KIND>(V, p, X.t) | (uint64_t)c, sh.qat, 64); };
      const int cl = cut_class(cut, b, tk);
      if (cl == 2) list_cand(list, cn, b, tk(), ((unsigned long long)g.bid << 32) | ((unsigned)p << 2) | (unsigned)c);
      const bool kp = cl == 1;
      if (kp) kept[r] |= 1u << c;
      if (sums && (kp || !P2)) {
        const double pv = __longlong_as_double((long long)b);
        const double p2 = P2 ? __dmul_rn(pv, pv) : pv;  // what the second sum adds
        if (b < kOneBits) {  // and p2 too
          if (kp) s0.add(pv);
          s1.add(p2);
        } else {
          if (kp) limb_add(cn + C_LIMB, fx_from_pbits(b));
          limb_add(cn + C_LIMB + 4, fx_from_pbits((unsigned long long)__double_as_longlong(p2)));
        }
      }
    }
    nkeep += __popc(kept[r]);
  }
  s0.fold();
  s1.fold();
  // at most 16 terms below 1 per thread: the block's integers fit 64 bits
  long long bs[5] = {nkeep, s0.ih, s0.il, s1.ih, s1.il};
  if (sums) {
    block_sum<5>(bs, sh.sum);
    if (tid == 0) {
      s0.ih = bs[1], s0.il = bs[2], s1.ih = bs[3], s1.il = bs[4];
      if (multi) {
        limb_add(cn + C_LIMB, s0.get());
        limb_add(cn + C_LIMB + 4, s1.get());
      }
    }
  } else {
    long long b1[1] = {nkeep};
    block_sum<1>(b1, sh.sum);
    bs[0] = b1[0];
  }
  const long long blk = bs[0];
  long long* counts = a.ws.part;  // per block (the partition records are not used on this route)
  if (multi && tid == 0) counts[g.bid] = blk;
  if (!gate_sync(gate, a.ctrl)) return false;
  if (!X.may_trunc) n_out = (long long)*(volatile unsigned long long*)(cn + C_OUT);

  // settle, offsets, decision: the same in every block
  i128 v0 = 0, v1 = 0;
  long long before = 0, total = 0;
  if (tid < 8) sh.limb[tid] = *(volatile unsigned long long*)(cn + C_LIMB + tid);
  if (multi) {
    for (int i = tid; i < nact; i += kThreads) {
      const long long c = __ldcg(counts + i);
      total += c;
      if (i < g.bid) before += c;
    }
  } else if (tid == 0) {
    total = blk;
  }
  if (cut.late) {
    const int m = load_cands(list, cn, sCand);
    for (int i = tid; i < kChipTile<PT> / 4; i += kThreads) reinterpret_cast<unsigned*>(sKeep)[i] = 0u;
    __syncthreads();
    if (rank_cand(sCand, m, cut.need)) {
      const unsigned long long b = sCand.bits[tid];
      if (sums) {
        v0 += fx_from_pbits(b);
        const double pv = __longlong_as_double((long long)b);
        if (P2) v1 += fx_from_pbits((unsigned long long)__double_as_longlong(__dmul_rn(pv, pv)));
      }
      const int owner = (int)(sCand.code[tid] >> 32);
      const unsigned at = (unsigned)sCand.code[tid];
      total += 1;
      if (owner < g.bid) before += 1;
      if (owner == g.bid) {
        const int p = (int)(at >> 2);
        atomicOr(reinterpret_cast<unsigned*>(sKeep) + (p >> 2), (1u << (at & 3)) << (8 * (p & 3)));
      }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < PT; ++r) kept[r] |= sKeep[r * kThreads + tid];
    if (sums && w == 0) {  // (at most kChipLate of them: warp 0's)
      v0 = warp_sum_i128(v0);
      v1 = warp_sum_i128(v1);
    }
  }
  long long bt[2] = {before, total};
  block_sum<2>(bt, sh.sum);
  before = bt[0];
  total = bt[1];
  if (tid == 0 && (P2 || g.bid == 0)) {  // (block 0 closes the op)
    OpResult& R = sh.R;
    R.n_out = n_out;
    R.n_written = total;
    R.trunc = trunc;
    if (sums) {  // (one block: the terms of 1 and above are in the limbs, the others still here)
      v0 += limb_get(sh.limb) + (multi ? (i128)0 : s0.get());
      v1 += limb_get(sh.limb + 4) + (multi ? (i128)0 : s1.get());
    }
    decide(a, v0, v1, sh.pr_limit, R);
  }
  // write: the survivors in position order
#pragma unroll
  for (int r = 0; r < PT; ++r) {
    const int c = (int)__reduce_add_sync(0xffffffffu, (unsigned)__popc(kept[r]));
    if (lane == 0) sh.warp[r * kRegions + w] = c;
  }
  __syncthreads();
  if ((P2 && sh.R.skip) || total > sh.ocap) return true;
  const int* wc = sh.warp;
  uint64_t* okeys = sh.okeys;
  double* oamps = sh.oamps;
#pragma unroll
  for (int r = 0; r < PT; ++r) {
    int roff = 0;  // survivors before this warp's in the tile
#pragma unroll
    for (int i = 0; i < PT * kRegions; ++i)
      if (i < r * kRegions + w) roff += wc[i];
    int x = __popc(kept[r]);
    const int own = x;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, off);
      if (lane >= off) x += y;
    }
    long long o = before + roff + x - own;
    if (kept[r]) {
      const int p = r * kThreads + tid;
      group_children_t<KIND>(C64, p, V, a.G, a.drop_zero, ca);
      const uint64_t kb = group_key<KIND>(V, p, X.t);
#pragma unroll
      for (int c = 0; c < NS; ++c) {
        if ((kept[r] >> c) & 1u) {
          okeys[o] = kb | (uint64_t)c;
          amp_put(oamps, o, ca[c], C64);
          ++o;
        }
      }
    }
  }
  return true;
}

// The tile step of a chip op on nblk blocks, or 0 if they cannot hold it.
template <int PT>
__device__ __forceinline__ int chip_step(long long n, int nblk) {
  if (n <= kChipStep<PT>) return kChipStep<PT>;
  const long long step = ((n + nblk - 1) / nblk + 3) & ~3LL;
  return step > kChipStep<PT> ? 0 : step < kChipMin ? kChipMin : (int)step;
}

// ---- staged route -------------------------------------------------------------
__device__ __forceinline__ unsigned sample_bin(unsigned long long bits) {
  if (bits >= 0x3FF0000000000000ULL) return kHistBins - 1;  // 1 and above
  const unsigned v = (unsigned)(bits >> 45);
  return v < (unsigned)kSampleBase ? 0u : v - (unsigned)kSampleBase;
}
__device__ __forceinline__ unsigned long long sample_edge(int b) {  // lowest pattern of bin b
  if (b <= 0) return 0ULL;
  if (b >= kHistBins) return ~0ULL;
  return (unsigned long long)(b + kSampleBase) << 45;
}

// first index in [lo, hi) with keys[i] >= y, by eight lanes together (the lanes
// of an aligned group of eight, which all call with the same arguments): eight
// probes per round instead of a chain of single ones
__device__ __forceinline__ long long lower_bound8(const uint64_t* keys, long long lo, long long hi, uint64_t y) {
  const int lane = threadIdx.x & 31, l = lane & 7, base = lane & 24;
  const unsigned group = 0xFFu << base;
  while (hi - lo > 8) {
    const long long span = hi - lo;
    const bool t = keys[lo + span * (l + 1) / 9] < y;
    const int c = __popc(__ballot_sync(group, t));
    const long long nlo = c == 0 ? lo : lo + span * c / 9 + 1;
    hi = c == 8 ? hi : lo + span * (c + 1) / 9;
    lo = nlo;
  }
  const bool t = lo + l < hi && keys[lo + l] < y;
  return lo + __popc(__ballot_sync(group, t));
}

// By eight lanes together (see lower_bound8); lane 0 of the eight adds the
// children of entry i to the sample's histogram.  A group's children
// are shared out: child o belongs to entry o of the group, those without an
// entry to the group's first, so that every child has one owner and the sampled
// entries' children are a fair sample of all children.
template <int KIND, bool C64>
__device__ __forceinline__ void sample_entry(const OpArgs& a, const OpCtx& X, long long i, unsigned* hist) {
  const uint64_t* keys = X.S.keys;
  const long long n = X.S.n;
  const double* amps = reinterpret_cast<const double*>(X.S.amps);
  auto at = [&](long long k) { return amp_get(amps, k, C64, X.r0, X.r1); };
  auto put = [&](double2 c) {
    const unsigned long long bits = (unsigned long long)__double_as_longlong(prob(c)) & 0x7FFFFFFFFFFFFFFFULL;
    const unsigned b = sample_bin(bits);
    atomicAdd(hist + b, 1u);
    if (b == 0 || b == kHistBins - 1) atomicAdd(a.ws.hist3 + (bits >> kFarShift), 1u);
  };
  if (KIND == K_IDENT) {
    if ((threadIdx.x & 7) == 0) put(at(i));
    return;
  }
  const uint64_t y = keys[i];
  const uint64_t bt = 1ULL << X.t;
  const uint64_t low = KIND == K_GATE2 ? 1ULL : 0ULL;
  const uint64_t other = (y ^ bt) & ~low;
  // the partner lies fewer than 2^(t + 1) positions away
  long long lo = 0, hi = n;
  if (X.t < 40) {
    const long long reach = 2LL << X.t;
    if (y & bt) lo = i - reach > 0 ? i - reach : 0;
    else hi = i + reach < n ? i + reach : n;
  }
  if (y & bt) hi = i;
  else lo = i;
  const long long j = lower_bound8(keys, lo, hi, other);
  if (threadIdx.x & 7) return;
  if (KIND != K_GATE2) {
    const bool pair = j < n && keys[j] == other;
    const double2 zero = make_double2(0.0, 0.0);
    const double2 mine = at(i), theirs = pair ? at(j) : zero;
    const int b = (int)((y >> X.t) & 1);
    const double2 x0 = b ? theirs : mine, x1 = b ? mine : theirs;
#pragma unroll
    for (int o = 0; o < 2; ++o)
      if (o == b || !pair) put(cadd(cmul(a.G[2 * o], x0), cmul(a.G[2 * o + 1], x1)));
  } else {
    double2 x[4];
    unsigned have = 0;
#pragma unroll
    for (int o = 0; o < 4; ++o) x[o] = make_double2(0.0, 0.0);
    const int side = (int)((y >> X.t) & 1), idx = 2 * side + (int)(y & 1);
    auto take = [&](int o, long long k) {
      const double2 v = at(k);
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (q == o) x[q] = v;
      have |= 1u << o;
    };
    take(idx, i);
    const long long near = (y & 1) ? i - 1 : i + 1;
    if (near >= 0 && near < n && keys[near] == (y ^ 1ULL)) take(idx ^ 1, near);
    for (long long k = j; k < n && k < j + 2; ++k)
      if ((keys[k] & ~1ULL) == other) take(2 * (side ^ 1) + (int)(keys[k] & 1), k);
    const bool first = (__ffs(have) - 1) == idx;
#pragma unroll
    for (int o = 0; o < 4; ++o) {
      if (!(o == idx || (first && !((have >> o) & 1u)))) continue;
      double2 acc = make_double2(0.0, 0.0);
#pragma unroll
      for (int q = 0; q < 4; ++q) acc = cadd(acc, cmul(a.G[4 * o + q], x[q]));
      put(acc);
    }
  }
}

// Sampled entries: no more than two rounds of the group's eights of lanes.  A
// small group of a segmented op spends longer on a full sample's chains of loads
// than a wider bracket costs (64 states of 32,768 entries: 204 us per gate with
// two rounds, 208 with four, 224 with eight, summed over the launches).
__device__ __forceinline__ long long sample_count(long long n, int nblk) {
  const long long room = (long long)nblk * (kThreads / 8) * kSampleRounds;
  const long long s = room < kSamples ? room : kSamples;
  return n < s ? n : s;
}
__device__ __forceinline__ bool is_bracketed(const OpArgs& a, const OpCtx& X) { return X.may_trunc && a.k_keep > 0; }

// Clears the counters, both histograms and the tiles' counts.
__device__ __forceinline__ void staged_zero(const OpArgs& a, const Grp& g, long long ntiles) {
  const long long gthreads = (long long)g.nblk * kThreads, gtid = (long long)g.bid * kThreads + threadIdx.x;
  for (long long i = gtid; i < kHistBins / 4; i += gthreads) {
    reinterpret_cast<uint4*>(a.ws.hist1)[i] = make_uint4(0, 0, 0, 0);
    reinterpret_cast<uint4*>(a.ws.hist2)[i] = make_uint4(0, 0, 0, 0);
    reinterpret_cast<uint4*>(a.ws.hist3)[i] = make_uint4(0, 0, 0, 0);
  }
  for (long long i = gtid; i < ntiles; i += gthreads) a.ws.status[i] = 0ULL;
  if (gtid < kOpCounters) reinterpret_cast<unsigned long long*>(a.ws.counters)[gtid] = 0ULL;
}

// Tile boundaries, one warp each from the front of the grid, and the sample's
// histogram, eight lanes per entry from its end (both are chains of dependent
// loads, so they run side by side).
template <int KIND, bool C64>
__device__ __forceinline__ void staged_prep(const OpArgs& a, const Grp& g, const OpCtx& X) {
  const long long gthreads = (long long)g.nblk * kThreads, gtid = (long long)g.bid * kThreads + threadIdx.x;
  const long long n = X.S.n;
  if (KIND != K_IDENT) {
    for (long long b = gtid >> 5; b <= X.ntiles; b += gthreads >> 5) {
      long long r[6];
      if (X.t == group_bit(KIND)) low_boundary<group_bit(KIND)>(X.S.keys, n, b * kStep, KIND != K_PERM, r);
      else tile_boundary<group_bit(KIND)>(X.S.keys, n, b * kStep, X.t, KIND != K_PERM, r);
      if ((threadIdx.x & 31) == 0)
        for (int q = 0; q < 6; ++q) a.ws.part[b * 6 + q] = r[q];
    }
  }
  if (KIND != K_PERM && is_bracketed(a, X)) {
    const long long S = sample_count(n, g.nblk);
    for (long long s = (gthreads - 1 - gtid) >> 3; s < S; s += gthreads >> 3) {
      // one entry of each of S equal ranges, at a hashed place in it
      const long long lo = s * n / S, hi = (s + 1) * n / S;
      sample_entry<KIND, C64>(a, X, lo + (long long)(fmix64((uint64_t)s + 1) % (uint64_t)(hi - lo)), a.ws.hist1);
    }
  }
}

// Block-wide: the edges of the sample's bin that holds the r-th child (s, x: the
// sample's top_scan).  One of the two outer bins is replaced by the quarter of a
// power of two in it: as a whole it would leave every child of a state with all
// |a|^2 below 2^-64 undecided (us per 1-qubit gate and truncation of 2^20 entries:
// 678 and 336 instead of 113 and 83; of 2^22 2164 and 1184 instead of 217 and 146).
__device__ __forceinline__ void sample_range(const OpArgs& a, FindSh& F, unsigned long long s, unsigned long long x,
                                             long long r, unsigned long long* lo, unsigned long long* hi) {
  top_locate<true, kHistBins>(a.ws.hist1, F, s, x, r);
  const int bin = F.bin;
  const long long above = F.above;
  const bool held = above + F.cnt >= r;  // (otherwise fewer children than r)
  __syncthreads();
  *lo = held ? sample_edge(bin) : 0ULL;
  *hi = sample_edge(bin + 1);
  if (!held || (bin != 0 && bin != kHistBins - 1)) return;
  // (the highest bin's children come before the lowest one's there)
  const long long skip = bin == 0 ? (long long)__ldcg(a.ws.hist1 + kHistBins - 1) : 0;
  find_top<true, kHistBins>(a.ws.hist3, F, skip + r - above);
  const unsigned long long l = (unsigned long long)F.bin << kFarShift, h = (unsigned long long)(F.bin + 1) << kFarShift;
  __syncthreads();
  if (l > *lo) *lo = l;
  if (h < *hi) *hi = h;
}

// Block-wide: the bracket, from the sample's histogram (every thread gets it).
__device__ __forceinline__ Bracket staged_bracket(const OpArgs& a, const Grp& g, const OpCtx& X, FindSh& F) {
  Bracket B{0ULL, 0ULL, 0, 0};  // nothing is dropped: every child certain
  if (!is_bracketed(a, X)) return B;
  const long long n = X.S.n, S = sample_count(n, g.nblk);
  // ranks k S / n -+ the margin of the sampled children
  unsigned long long s, x;
  top_scan<true, kHistBins>(a.ws.hist1, F, &s, &x);
  const long long r = (long long)(((unsigned __int128)a.k_keep * (unsigned long long)S) / (unsigned long long)n);
  const long long margin = S < n ? (long long)(4.0f * sqrtf((float)S)) : 0;  // four deviations of a rank
  const long long rh = r - margin, rl = r + margin + (S < n ? 1 : 0);
  B.hi = ~0ULL;
  unsigned long long unused;
  if (rh >= 1) sample_range(a, F, s, x, rh, &unused, &B.hi);
  sample_range(a, F, s, x, rl, &B.lo, &unused);
  B.shift = digit_shift<kHistBins>(B.lo, B.hi - 1);
  return B;
}

// Loads tile `tile` and brings it into Z order; false on a give-up.  The next
// tile of the loop (sh.item) is claimed while this one loads.
template <int KIND, bool C64>
__device__ __forceinline__ bool staged_tile(const OpArgs& a, OpSh& sh, const OpCtx& X, long long tile, uint64_t* sZ,
                                            double2* sA, uint16_t* sIdx, unsigned* phase, unsigned long long* next) {
  const int tid = threadIdx.x;
  if (tid == 0) {
    if (KIND == K_IDENT) {
      const long long lo = tile * kTile, hi = lo + kTile < X.S.n ? lo + kTile : X.S.n;
      const long long rc[6] = {lo, 0, X.S.n, X.S.n, lo, 0}, rn[6] = {hi, 0, X.S.n, X.S.n, hi, 0};
      tile_segments<C64>(sh.T, rc, rn, X.S, kTile, sZ, sA, &sh.bar, a.ctrl);
    } else {
      const long long* rc = a.ws.part + tile * 6;
      tile_segments<C64>(sh.T, rc, rc + 6, X.S, kTile, sZ, sA, &sh.bar, a.ctrl);
    }
    sh.item = (long long)atomicAdd(next, 1ULL);
  }
  __syncthreads();
  if (!tile_fetch<kPerThread, C64>(sh.T, X.S, sZ, sA, &sh.bar, phase, a.ctrl, X.lim)) return false;
  if (KIND != K_IDENT) tile_zorder<kPerThread, group_bit(KIND)>(sh.T, sZ, sIdx, sh.warp, X.t);
  return true;
}

// The first pass of a 2-qubit gate: every entry to its Z position.
template <bool C64>
__device__ __forceinline__ bool staged_perm(const OpArgs& a, OpSh& sh, const OpCtx& X, unsigned* phase,
                                            unsigned char* smem) {
  const int tid = threadIdx.x;
  double2* sA = reinterpret_cast<double2*>(smem);
  uint64_t* sZ = reinterpret_cast<uint64_t*>(sA + kTilePad);
  uint16_t* sIdx = reinterpret_cast<uint16_t*>(sZ + kTilePad);
  unsigned long long* cn = reinterpret_cast<unsigned long long*>(a.ws.counters);
  const bool fits = X.S.n <= a.out->cap;
  const TileView V{sZ, sA, reinterpret_cast<const float2*>(sA), sIdx, X.r0, X.r1, !(X.r0 == 1.0 && X.r1 == 1.0), C64};
  if (tid == 0) {
    sh.item = (long long)atomicAdd(cn + C_TILE, 1ULL);
    sh.R = OpResult{};
    sh.R.n_written = X.S.n;
  }
  __syncthreads();
  for (long long tile = sh.item; tile < X.ntiles; tile = sh.item) {
    __syncthreads();
    if (!staged_tile<K_PERM, C64>(a, sh, X, tile, sZ, sA, sIdx, phase, cn + C_TILE)) return false;
    const int E = (int)sh.T.off[5];
    const long long zs = sh.T.zs;
    if (fits) {
      for (int p = tid; p < E; p += kThreads) {
        a.out->keys[zs + p] = group_key<K_PERM>(V, p, X.t);
        amp_put(a.out->amps, zs + p, V.amp(p), C64);
      }
    }
    __syncthreads();
  }
  return true;
}

// What the passes keep per region (in ws.partials): the staged children (low
// half) and the undecided ones, and, from the settling on, the kept ones.
__device__ __forceinline__ unsigned* region_counts(const OpArgs& a) { return reinterpret_cast<unsigned*>(a.ws.partials); }
__device__ __forceinline__ uint16_t* region_kept(const OpArgs& a) {
  return reinterpret_cast<uint16_t*>(region_counts(a) + a.ws.max_tiles * kRegions);
}

// The evaluation: every tile's children at or above the bracket are staged, one
// region per warp (compacted in child order); the undecided ones are listed per
// region (|a|^2 pattern, place in the region) and counted in the histogram
// ws.hist2; counts and the certain ones' sums go to the counters.  False on a
// give-up.
template <int KIND, bool C64>
__device__ __forceinline__ bool staged_eval(const OpArgs& a, OpSh& sh, const OpCtx& X, const Bracket& B,
                                            unsigned* phase, unsigned char* smem) {
  constexpr int NS = slots_per_entry(KIND);
  constexpr bool P2 = KIND == K_ROT1;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const unsigned lt = (1u << lane) - 1;
  double2* sA = reinterpret_cast<double2*>(smem);
  uint64_t* sZ = reinterpret_cast<uint64_t*>(sA + kTilePad);
  uint16_t* sIdx = reinterpret_cast<uint16_t*>(sZ + kTilePad);
  unsigned long long* cn = reinterpret_cast<unsigned long long*>(a.ws.counters);
  const TileView V{sZ, sA, reinterpret_cast<const float2*>(sA), KIND == K_IDENT ? nullptr : sIdx, X.r0, X.r1, !(X.r0 == 1.0 && X.r1 == 1.0), C64};
  const bool sums = P2 || X.may_trunc;
  double2 ca[NS];
  const unsigned lo32 = (unsigned)(B.lo >> 32), hi32 = (unsigned)(B.hi >> 32);
  // the region's undecided children: how many so far, and the first ones' places
  constexpr int kQueue = 48;
  __shared__ int sUnd[kRegions];
  __shared__ uint16_t sQueue[kRegions][kQueue];
  // lists the child staged at place q as the region's u-th undecided one (its
  // amplitude, written by this warp, is read back from L2)
  auto undecided = [&](long long sbase, int u, int q) {
    const double2 v = C64 ? f2d(__ldcg(reinterpret_cast<const float2*>(a.ws.tmp_amps) + sbase + q))
                          : __ldcg(a.ws.tmp_amps + sbase + q);
    const unsigned long long bits = (unsigned long long)__double_as_longlong(prob(v));
    a.ws.cand_bits[sbase + u] = bits;
    reinterpret_cast<uint16_t*>(a.ws.cand_key)[sbase + u] = (uint16_t)q;
    atomicAdd(a.ws.hist2 + digit_of<kHistBins>(bits, B.lo, B.shift), 1u);
  };
  int c_out = 0, c_def = 0, c_staged = 0, folded = 0;
  Acc s0, s1;
  s0.clear();
  s1.clear();
  if (tid == 0) sh.item = (long long)atomicAdd(cn + C_TILE, 1ULL);
  __syncthreads();
  for (long long tile = sh.item; tile < X.ntiles; tile = sh.item) {
    __syncthreads();
    if (!staged_tile<KIND, C64>(a, sh, X, tile, sZ, sA, sIdx, phase, cn + C_TILE)) return false;
    const int E = (int)sh.T.off[5];
    const long long region = tile * kRegions + w;
    const long long sbase = region * (NS * kRegion);
    if (lane == 0) sUnd[w] = 0;
    __syncwarp();
    int run = 0;  // staged children of the region so far
    for (int r = 0; r < kPerThread; ++r) {
      const int p = w * kRegion + r * 32 + lane;
      if (w * kRegion + r * 32 >= E) break;
      unsigned cm = 0;
      if (p < E) cm = group_children_t<KIND>(C64, p, V, a.G, a.drop_zero, ca);
      unsigned st = 0, um = 0, big = 0;  // children staged, the undecided ones among them, |a|^2 of 1 and above
      double pv[NS];
      int at = run;
#pragma unroll
      for (int c = 0; c < NS; ++c) {
        pv[c] = prob(ca[c]);
        // (the bracket's edges are multiples of 2^32: the high words decide)
        const unsigned hb = (unsigned)__double2hiint(pv[c]);
        const bool exists = (cm >> c) & 1u;
        const bool on = exists && hb >= lo32, def = exists && hb >= hi32;
        c_out += exists;
        if (on) st |= 1u << c;
        if (on && !def) um |= 1u << c;
        const unsigned m = __ballot_sync(0xffffffffu, on);
        at += __popc(m & lt);
        run += __popc(m);
        if (sums) {
          // the kept sum's term, and the second sum's (no branch: 0 adds nothing)
          const bool small = hb < (unsigned)(kOneBits >> 32);
          const double q = def && small ? pv[c] : 0.0;
          s0.add(q);
          s1.add(P2 ? __dmul_rn(q, q) : exists && small ? pv[c] : 0.0);
          if (exists && !small) big |= 1u << c;
        }
      }
      if (sums && big) {
#pragma unroll
        for (int c = 0; c < NS; ++c) {
          if (!((big >> c) & 1u)) continue;
          const bool def = ((st & ~um) >> c) & 1u;
          const double p2 = P2 ? __dmul_rn(pv[c], pv[c]) : pv[c];
          if (def) limb_add(cn + C_LIMB, fx_from_pbits((unsigned long long)__double_as_longlong(pv[c])));
          if (def || !P2) limb_add(cn + C_LIMB + 4, fx_from_pbits((unsigned long long)__double_as_longlong(p2)));
        }
      }
      if (st) {
        const uint64_t kb = group_key<KIND>(V, p, X.t);
        uint64_t* const sk = a.ws.stage_keys + sbase + at;
#pragma unroll
        for (int c = 0; c < NS; ++c)
          if ((st >> c) & 1u) sk[__popc(st & ((1u << c) - 1u))] = kb | (uint64_t)c;
        if (C64) {
          float2* const sa = reinterpret_cast<float2*>(a.ws.tmp_amps) + sbase + at;
#pragma unroll
          for (int c = 0; c < NS; ++c)
            if ((st >> c) & 1u) sa[__popc(st & ((1u << c) - 1u))] = d2f(ca[c]);
        } else {
          double2* const sa = a.ws.tmp_amps + sbase + at;
#pragma unroll
          for (int c = 0; c < NS; ++c)
            if ((st >> c) & 1u) sa[__popc(st & ((1u << c) - 1u))] = ca[c];
        }
      }
      for (; um; um &= um - 1) {  // few: at most one per lane in most rounds; their order does not matter
        const int c = __ffs(um) - 1;
        const int q = at + __popc(st & ((1u << c) - 1u));
        const int u = atomicAdd(&sUnd[w], 1);
        if (u < kQueue) sQueue[w][u] = (uint16_t)q;  // listed after the last round
        else undecided(sbase, u, q);
      }
      if (NS == 4 && r == 3) {  // at most 16 terms between folds
        s0.fold();
        s1.fold();
      }
    }
    __syncwarp();
    const int und = sUnd[w];
    for (int u = lane; u < und && u < kQueue; u += 32) undecided(sbase, u, sQueue[w][u]);
    s0.fold();
    s1.fold();
    if (++folded == 512) {  // the 64-bit integers hold 2^10 tiles of terms below 1 (32 a thread at most)
      limb_add(cn + C_LIMB, s0.get());
      limb_add(cn + C_LIMB + 4, s1.get());
      s0.clear();
      s1.clear();
      folded = 0;
    }
    if (lane == 0) {
      region_counts(a)[region] = (unsigned)run | ((unsigned)und << 16);
      c_staged += run;
      c_def += run - und;
    }
    __syncthreads();
  }
  if (sums) flush_sums(sh, cn, s0.get(), s1.get());
  long long ct[3] = {c_out, c_def, c_staged};
  block_sum<3>(ct, sh.sum);
  if (tid == 0) {
    atomicAdd(cn + C_OUT, (unsigned long long)ct[0]);
    atomicAdd(cn + C_DEF, (unsigned long long)ct[1]);
    atomicAdd(cn + C_STAGED, (unsigned long long)ct[2]);
  }
  return true;
}

// Block-wide, after every block's evaluation: does the op truncate, did the
// bracket hold the threshold, and the first step of the search inside it
// (sh.St, with B).
__device__ __forceinline__ void staged_plan(const OpArgs& a, OpSh& sh, const OpCtx& X, const Bracket& B) {
  const unsigned long long* cn = reinterpret_cast<const unsigned long long*>(a.ws.counters);
  const long long n_out = (long long)*(const volatile unsigned long long*)(cn + C_OUT);
  const long long n_def = (long long)*(const volatile unsigned long long*)(cn + C_DEF);
  const long long n_staged = (long long)*(const volatile unsigned long long*)(cn + C_STAGED);
  const int trunc = X.may_trunc && !(n_out <= a.k_cond || a.k_keep >= n_out);
  Cut cut{0ULL, 0ULL, 0ULL, 0, CUT_ALL, 0, 0};
  int state = ST_OK;
  Bracket Bn = B;
  if (trunc && a.k_keep <= 0) {
    cut.mode = CUT_NONE;
  } else if (!(trunc ? (n_def <= a.k_keep && n_staged >= a.k_keep) : n_staged == n_out)) {
    state = ST_MISSED;
  } else if (trunc) {
    cut.mode = CUT_BITS;
    cut.lo = B.lo;
    cut.hi = B.hi - 1;
    cut.need = a.k_keep - n_def;
    if (cut.need >= n_staged - n_def) {
      cut.all = 1;  // every staged child
    } else if (cut.need <= 0) {
      cut.lo = cut.hi + 1;  // none of the undecided ones
    } else {
      find_top<true, kHistBins>(a.ws.hist2, sh.F, cut.need);
      const bool done = cut_narrow<kHistBins, kSelMax>(cut, &Bn.shift, sh.F.bin, sh.F.above, sh.F.cnt);
      if (!done) Bn.pad = 1;  // search on (staged_settle)
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    sh.St.B = Bn;
    sh.St.cut = cut;
    sh.St.n_out = n_out;
    sh.St.trunc = trunc;
    sh.St.state = state;
  }
  __syncthreads();
}

// Every child's sample bin into ws.hist1 (the exact bracket after a miss).
template <int KIND, bool C64>
__device__ __forceinline__ bool staged_count(const OpArgs& a, OpSh& sh, const OpCtx& X, unsigned* phase,
                                             unsigned char* smem) {
  constexpr int NS = slots_per_entry(KIND);
  const int tid = threadIdx.x;
  double2* sA = reinterpret_cast<double2*>(smem);
  uint64_t* sZ = reinterpret_cast<uint64_t*>(sA + kTilePad);
  uint16_t* sIdx = reinterpret_cast<uint16_t*>(sZ + kTilePad);
  unsigned long long* cn = reinterpret_cast<unsigned long long*>(a.ws.counters);
  const TileView V{sZ, sA, reinterpret_cast<const float2*>(sA), KIND == K_IDENT ? nullptr : sIdx, X.r0, X.r1, !(X.r0 == 1.0 && X.r1 == 1.0), C64};
  double2 ca[NS];
  if (tid == 0) sh.item = (long long)atomicAdd(cn + C_TILE2, 1ULL);
  __syncthreads();
  for (long long tile = sh.item; tile < X.ntiles; tile = sh.item) {
    __syncthreads();
    if (!staged_tile<KIND, C64>(a, sh, X, tile, sZ, sA, sIdx, phase, cn + C_TILE2)) return false;
    const int E = (int)sh.T.off[5];
    for (int p = tid; p < E; p += kThreads) {
      const unsigned cm = group_children_t<KIND>(C64, p, V, a.G, a.drop_zero, ca);
#pragma unroll
      for (int c = 0; c < NS; ++c)
        if ((cm >> c) & 1u)
          atomicAdd(a.ws.hist1 + sample_bin((unsigned long long)__double_as_longlong(prob(ca[c]))), 1u);
    }
    __syncthreads();
  }
  return true;
}

// Visits the regions, four per warp and round (eight lanes each, so that four
// chains of dependent loads run side by side), and the undecided children listed
// for each: begin(staged), fn(bits, place in the region, stage index) for each,
// done(region).  All lanes call begin and done; live is false past the end.
template <int NS, class Begin, class Fn, class Done>
__device__ __forceinline__ void visit_regions(const OpArgs& a, const Grp& g, long long nregions, Begin begin, Fn fn,
                                              Done done) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, l8 = lane & 7;
  const uint16_t* place = reinterpret_cast<const uint16_t*>(a.ws.cand_key);
  const long long stride = 4LL * g.nblk * kRegions;
  for (long long rb = 4LL * (g.bid * kRegions + w); rb < nregions; rb += stride) {
    const long long r = rb + (lane >> 3);
    const bool live = r < nregions;
    const unsigned rc = live ? __ldcg(region_counts(a) + r) : 0u;
    const int staged = (int)(rc & 0xFFFFu), und = (int)(rc >> 16);
    const long long s0 = r * (NS * kRegion);
    begin(staged);
    for (int j = l8; j < und; j += 8) {
      const int at = (int)__ldcg(place + s0 + j);
      fn(__ldcg(a.ws.cand_bits + s0 + j), at, s0 + at);
    }
    done(r, live);
  }
}

// The undecided children's threshold, found and applied: masks, counts per tile,
// sums, and the list of the (at most kSelMax) children still to be ranked.  All
// blocks of the launch resident.  A bracket that missed (ST_MISSED) is
// replaced first.  False on a give-up.
template <int KIND, bool C64>
__device__ __forceinline__ bool staged_settle(const OpArgs& a, const Grp& g, OpSh& sh, const OpCtx& X, Gate& gate,
                                              unsigned* phase, unsigned char* smem) {
  constexpr int NS = slots_per_entry(KIND);
  constexpr int W = NS * kRegion / 32;
  constexpr bool P2 = KIND == K_ROT1;
  const int tid = threadIdx.x, lane = tid & 31;
  const long long gthreads = (long long)g.nblk * kThreads, gtid = (long long)g.bid * kThreads + tid;
  const long long nregions = X.ntiles * kRegions;
  unsigned long long* cn = reinterpret_cast<unsigned long long*>(a.ws.counters);
  auto clear = [&](unsigned* h) {
    for (long long i = gtid; i < kHistBins / 4; i += gthreads) reinterpret_cast<uint4*>(h)[i] = make_uint4(0, 0, 0, 0);
  };
  if (sh.St.state == ST_MISSED) {
    // the exact bracket, from the histogram of all children, and the
    // evaluation again
    clear(a.ws.hist1);
    clear(a.ws.hist2);
    if (!gate_sync(gate, a.ctrl)) return false;
    if (gtid < kOpCounters && gtid != C_TILE2) cn[gtid] = 0ULL;
    const int trunc = sh.St.trunc;
    if (trunc && !staged_count<KIND, C64>(a, sh, X, phase, smem)) return false;
    if (!gate_sync(gate, a.ctrl)) return false;
    Bracket B{0ULL, 0ULL, 0, 0};
    if (trunc) {
      find_top<true, kHistBins>(a.ws.hist1, sh.F, a.k_keep);
      B.lo = sample_edge(sh.F.bin);
      B.hi = sample_edge(sh.F.bin + 1);
      B.shift = digit_shift<kHistBins>(B.lo, B.hi - 1);
      __syncthreads();
    }
    if (!staged_eval<KIND, C64>(a, sh, X, B, phase, smem)) return false;
    if (!gate_sync(gate, a.ctrl)) return false;
    staged_plan(a, sh, X, B);
  }
  Cut cut = sh.St.cut;
  const bool trunc = sh.St.trunc != 0;
  const uint64_t* skeys = a.ws.stage_keys;
  auto key_at = [&](long long i) { return true_key(__ldcg(skeys + i), sh.qat, 64); };
  if (sh.St.B.pad) {
    int shift = sh.St.B.shift;
    for (int level = 1;; ++level) {
      unsigned* gh = (level & 1) ? a.ws.hist1 : a.ws.hist2;
      // the buffer's readers of two levels ago passed the previous barrier
      clear(gh);
      if (!gate_sync(gate, a.ctrl)) return false;
      visit_regions<NS>(
          a, g, nregions, [](int) {},
          [&](unsigned long long b, int, long long i) {
            if (cut_class(cut, b, [&]() { return key_at(i); }) == 2)
              atomicAdd(gh + digit_of<kHistBins>(cut.mode == CUT_KEYS ? ~key_at(i) : b, cut.lo, shift), 1u);
          },
          [](long long, bool) {});
      if (!gate_sync(gate, a.ctrl)) return false;
      find_top<true, kHistBins>(gh, sh.F, cut.need);
      const int bin = sh.F.bin;
      const long long above = sh.F.above, cnt = sh.F.cnt;
      __syncthreads();
      if (cut_narrow<kHistBins, kSelMax>(cut, &shift, bin, above, cnt)) break;
    }
  }
  i128 v0 = 0, v1 = 0;
  // the region's kept bits, one per staged child (the tile's memory is free)
  unsigned* mask = reinterpret_cast<unsigned*>(smem) + (tid >> 3) * W;
  const int l8 = lane & 7;
  visit_regions<NS>(
      a, g, nregions,
      [&](int staged) {
        for (int l = l8; l < W; l += 8) {
          const int nv = cut.mode == CUT_NONE ? 0 : staged - 32 * l;
          mask[l] = nv >= 32 ? ~0u : nv <= 0 ? 0u : (1u << nv) - 1u;
        }
        __syncwarp();
      },
      [&](unsigned long long b, int at, long long i) {
        const int cl = cut_class(cut, b, [&]() { return key_at(i); });
        if (cl == 2) list_cand(cand_list(a), cn, b, key_at(i), (unsigned long long)i);
        if (cl != 1) {
          atomicAnd(mask + (at >> 5), ~(1u << (at & 31)));
        } else if (trunc || P2) {
          v0 += fx_from_pbits(b);
          const double pv = __longlong_as_double((long long)b);
          if (P2) v1 += fx_from_pbits((unsigned long long)__double_as_longlong(__dmul_rn(pv, pv)));
        }
      },
      [&](long long r, bool live) {
        __syncwarp();
        int kc = 0;
        for (int l = l8; l < W; l += 8) {
          const unsigned word = mask[l];
          kc += __popc(word);
          if (live) reinterpret_cast<unsigned*>(a.ws.kmask)[r * W + l] = word;
        }
#pragma unroll
        for (int off = 1; off < 8; off <<= 1) kc += __shfl_xor_sync(0xffffffffu, kc, off);
        if (l8 == 0 && live) {
          region_kept(a)[r] = (uint16_t)kc;
          if (kc) atomicAdd(a.ws.status + r / kRegions, (unsigned long long)kc);
        }
        __syncwarp();
      });
  if (trunc || P2) flush_sums(sh, cn, v0, v1);
  __syncthreads();
  if (tid == 0) sh.St.cut = cut;
  return true;
}

// One block, after every block's staged_settle: ranks the listed children, adds
// the kept ones to the masks, counts and sums, scans the tiles' counts (into
// ws.status: where each tile's survivors go) and decides.  sh.R is the result.
template <int KIND>
__device__ __forceinline__ void staged_final(const OpArgs& a, OpSh& sh, const OpCtx& X, unsigned char* smem) {
  constexpr int NS = slots_per_entry(KIND);
  constexpr int W = NS * kRegion / 32;
  constexpr bool P2 = KIND == K_ROT1;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  CandSh& sCand = *reinterpret_cast<CandSh*>(smem);
  unsigned long long* cn = reinterpret_cast<unsigned long long*>(a.ws.counters);
  const bool trunc = sh.St.trunc != 0, sums = P2 || trunc;
  i128 v0 = 0, v1 = 0;
  if (tid < 8) sh.limb[tid] = *(volatile unsigned long long*)(cn + C_LIMB + tid);
  if (sh.St.cut.late) {
    const int m = load_cands(cand_list(a), cn, sCand);
    if (rank_cand(sCand, m, sh.St.cut.need)) {
      const unsigned long long b = sCand.bits[tid], i = sCand.code[tid];
      v0 += fx_from_pbits(b);
      const double pv = __longlong_as_double((long long)b);
      if (P2) v1 += fx_from_pbits((unsigned long long)__double_as_longlong(__dmul_rn(pv, pv)));
      const unsigned long long r = i / (NS * kRegion), j = i % (NS * kRegion);
      atomicOr(reinterpret_cast<unsigned*>(a.ws.kmask) + r * W + j / 32, 1u << (j & 31));
      atomicAdd(a.ws.status + r / kRegions, 1ULL);
      atomicAdd(reinterpret_cast<unsigned*>(region_kept(a)) + r / 2, 1u << (16 * (r & 1)));
    }
    __threadfence();
    i128 v[2] = {v0, v1};
    block_sum_i128<2>(v, sh.red);
    v0 = v[0];
    v1 = v[1];
  }
  __syncthreads();
  // exclusive scan of the tiles' counts: every thread a contiguous run of tiles
  const long long C = (X.ntiles + kThreads - 1) / kThreads;
  const long long lo = (long long)tid * C, hi = lo + C < X.ntiles ? lo + C : X.ntiles;
  constexpr int kRun = 12;
  long long cr[kRun];
  long long run = 0;
  if (C <= kRun) {
#pragma unroll
    for (int q = 0; q < kRun; ++q) {
      cr[q] = lo + q < hi ? (long long)__ldcg(a.ws.status + lo + q) : 0;
      run += cr[q];
    }
  } else {
    for (long long b = lo; b < hi; ++b) run += (long long)__ldcg(a.ws.status + b);
  }
  long long x = run;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const long long y = __shfl_up_sync(0xffffffffu, x, off);
    if (lane >= off) x += y;
  }
  long long* sW = sh.sum;
  if (lane == 31) sW[w] = x;
  __syncthreads();
  long long ex = x - run, total = 0;
#pragma unroll
  for (int i = 0; i < kRegions; ++i) {
    if (i < w) ex += sW[i];
    total += sW[i];
  }
  if (C <= kRun) {
#pragma unroll
    for (int q = 0; q < kRun; ++q) {
      if (lo + q < hi) a.ws.status[lo + q] = (unsigned long long)ex;
      ex += cr[q];
    }
  } else {
    for (long long b = lo; b < hi; ++b) {
      const long long c = (long long)__ldcg(a.ws.status + b);
      a.ws.status[b] = (unsigned long long)ex;
      ex += c;
    }
  }
  if (tid == 0) {
    OpResult& R = sh.R;
    R.n_out = sh.St.n_out;
    R.n_written = total;
    R.trunc = sh.St.trunc;
    R.failed = 0;
    if (sums) {
      // (when nothing is kept the limbs hold sums over children that are not)
      if (sh.St.cut.mode != CUT_NONE) v0 += limb_get(sh.limb);
      if (sh.St.cut.mode != CUT_NONE || !P2) v1 += limb_get(sh.limb + 4);
    }
    decide(a, v0, v1, sh.pr_limit, R);
  }
  __syncthreads();
}

// The write: every region's survivors, copied to their place, one region per
// warp and round.  Where they go: the tile's offset plus what the tile's
// earlier regions keep (its eight counts are one 16-byte load), so warps need
// no barrier.  Staged children are read and survivors written once: streaming
// accesses (202 -> 194 us per gate at 2^22 entries for the stores).  Four loads in
// flight per lane at four blocks per SM; two (206 us) or eight (225) are slower.
template <int KIND, bool C64>
__device__ __forceinline__ void staged_write(const OpArgs& a, const Grp& g, OpSh& sh, const OpCtx& X) {
  constexpr int NS = slots_per_entry(KIND);
  constexpr int W = NS * kRegion / 32;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1;
  if (sh.R.skip || sh.R.n_written > sh.ocap) return;
  const long long nregions = X.ntiles * kRegions, stride = (long long)g.nblk * kRegions;
  uint64_t* okeys = sh.okeys;
  double2* oamps = reinterpret_cast<double2*>(sh.oamps);
  float2* oampf = reinterpret_cast<float2*>(sh.oamps);
  const float2* stf = reinterpret_cast<const float2*>(a.ws.tmp_amps);
  unsigned nword = 0, nc = 0;
  uint4 nk = make_uint4(0, 0, 0, 0);
  long long nbase = 0;
  auto fetch = [&](long long r) {
    nword = lane < W ? __ldcg(reinterpret_cast<const unsigned*>(a.ws.kmask) + r * W + lane) : 0u;
    nc = __ldcg(region_counts(a) + r);
    nk = __ldcg(reinterpret_cast<const uint4*>(region_kept(a)) + r / kRegions);
    nbase = (long long)__ldcg(a.ws.status + r / kRegions);
  };
  long long r = (long long)g.bid * kRegions + w;
  if (r < nregions) fetch(r);
  for (; r < nregions; r += stride) {
    const unsigned word = nword;
    const int c = (int)(nc & 0xFFFFu);
    const unsigned kw[4] = {nk.x, nk.y, nk.z, nk.w};
    long long o0 = nbase;
#pragma unroll
    for (int i = 0; i < kRegions - 1; ++i)
      if (i < (int)(r % kRegions)) o0 += (kw[i >> 1] >> (16 * (i & 1))) & 0xFFFFu;
    if (r + stride < nregions) fetch(r + stride);  // the next region's words, while this one is copied
    const int pc = __popc(word);
    int inc = pc;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, inc, off);
      if (lane >= off) inc += y;
    }
    const long long s0 = r * (NS * kRegion);
    constexpr int U = 4;
    for (int l0 = 0; 32 * l0 < c; l0 += U) {
      uint64_t kk[U];
      double2 aa[U];
      float2 af[U];
      unsigned mw[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int l = l0 + u;
        mw[u] = __shfl_sync(0xffffffffu, word, l & 31);
        if (l >= W) mw[u] = 0;
        if ((mw[u] >> lane) & 1u) {
          kk[u] = __ldcs(a.ws.stage_keys + s0 + 32 * l + lane);
          if (C64) af[u] = __ldcs(stf + s0 + 32 * l + lane);
          else aa[u] = __ldcs(a.ws.tmp_amps + s0 + 32 * l + lane);
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int ob = __shfl_sync(0xffffffffu, inc - pc, (l0 + u) & 31);
        if ((mw[u] >> lane) & 1u) {
          const long long o = o0 + ob + __popc(mw[u] & lt);
          __stcs(okeys + o, kk[u]);
          if (C64) __stcs(oampf + o, af[u]);
          else __stcs(oamps + o, aa[u]);
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// kernels
// ---------------------------------------------------------------------------
__device__ __forceinline__ void prof_add(int64_t* slots, int slot, long long v) {
  atomicAdd(reinterpret_cast<unsigned long long*>(slots + slot), (unsigned long long)v);
}
// The op's last block: the result, its bookkeeping and profile counts (pass_in:
// the kernel that read the entries, pass_out: the one that wrote the survivors).
__device__ __forceinline__ void op_close(const OpArgs& a, int kind, int pass_in, int pass_out, const OpResult& R,
                                         long long n) {
  if (a.prof && threadIdx.x == 0) {
    prof_add(a.ctrl->prof_in, kind * 5 + pass_in, n);
    if (!R.skip) prof_add(a.ctrl->prof_out, kind * 5 + pass_out, R.n_written);
  }
  __syncthreads();
  op_finalize(a, kind, R);
}

// The first launch of an op: the whole op on the chip route if the group's
// blocks can hold the state, otherwise (a.staged) the staged route's clearing.
// The later launches of an op that is over return at once.
// STAGED: launches of the staged route follow.  OFF: the launch may be called off.
template <int KIND, bool C64, bool STAGED, bool OFF, int PT>
__device__ __forceinline__ void op_first(const OpArgs& a, const Grp& g) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ OpSh sh;
  const int tid = threadIdx.x;
  if (STAGED && a.staged) {
    // too large for the chip route and accepted: as little code as can be (its
    // lines come from DRAM after an op on a large state)
    const long long n = a.in->nnz, nt = KIND == K_IDENT ? plain_tiles(n) : merge_tiles(n);
    if (n > (long long)g.nblk * kChipStep<PT> && n * slots_per_entry(KIND) <= a.ws.max_n && nt <= a.ws.max_tiles &&
        n < kMaxEntries && (a.in->amp_type == BASS_AMP_C64) == C64) {
      pdl_trigger();
      staged_zero(a, g, nt);
      if (g.bid == 0 && tid == 0) stage_of(a)->state = ST_OK;
      return;
    }
  }
  const OpCtx X = op_ctx<KIND, C64>(a);
  const long long n = X.S.n;
  const int step = X.bad ? 0 : chip_step<PT>(n, g.nblk);
  if (tid == 0) mbar_init(&sh.bar, 1);
  out_order_par(a.in, KIND, a.q, a.gb, sh.qat);
  __syncthreads();
  if (tid == 0) op_preload(a, sh);
  __syncthreads();
  bool ok = true, off = false;
  unsigned* word = reinterpret_cast<unsigned*>(&a.ctrl->sync_counter);
  if (step) {
    // every block counts at the first barrier (it has then read the
    // descriptors, which block 0 rewrites at the end), the ones with a tile
    // at the others
    const int nact = n > 0 ? (int)((n + step - 1) / step) : 1;
    Gate gate{word, nact, g.nblk, 0u, false};
    if (g.bid < nact) ok = op_chip<KIND, C64, OFF, PT>(a, g, sh, X, gate, step, smem);
    else if (KIND != K_PERM) gate_arrive(gate);
    off = gate.off;
  } else {
    if (tid == 0) sh.R = OpResult{};
    if (g.bid == 0 && tid == 0) op_refuse(a, C64);
    // block 0 closes the op below: the others must have read its descriptors
    Gate gate{word, 1, g.nblk, 0u, false};
    gate_arrive(gate);
    if (g.bid == 0) ok = gate_wait(gate, a.ctrl);
  }
  pdl_trigger();
  if (g.bid == 0 && !off) {
    if (STAGED && a.staged && tid == 0) {  // for the launches that follow
      stage_of(a)->state = ST_OVER;
      result_of(a)->failed = kOver;
    }
    // every block knows the result; the last one out only resets the barrier
    if (ok) op_close(a, KIND, P_GATHER, P_GATHER, sh.R, n);
  }
  if (g.nblk > 1 && op_exit(a.ctrl, g.nblk, !ok && !off) == 3 && OFF) {
    // called off: the staged launches do the op
    staged_zero(a, Grp{0, 1}, X.ntiles);
    if (tid == 0) stage_of(a)->state = ST_OK;
  }
}

// The staged route's later passes, each a launch.
template <int KIND, bool C64>
__device__ __forceinline__ void op_prep(const OpArgs& a, const Grp& g) {
  __shared__ FindSh F;
  __shared__ OpStage St;
  const bool first = KIND == K_PERM && !a.seg;  // a plain reorder has no launch before this one
  const int state = first ? ST_OK : __ldcg(&stage_of(a)->state);
  const OpCtx X = op_ctx<KIND, C64>(a);
  if (state != ST_OK) return;
  if (KIND == K_PERM) {
    if (g.bid == 0 && threadIdx.x < kOpCounters)
      reinterpret_cast<unsigned long long*>(a.ws.counters)[threadIdx.x] = 0ULL;
    if (X.bad && g.bid == 0 && threadIdx.x == 0) op_refuse(a, C64);
    if (!X.bad) staged_prep<KIND, C64>(a, g, X);
    pdl_trigger();
    return;
  }
  staged_prep<KIND, C64>(a, g, X);
  pdl_trigger();
  if (!op_exit(a.ctrl, g.nblk, false)) return;
  const Bracket B = staged_bracket(a, g, X, F);
  if (threadIdx.x == 0) {
    St = OpStage{};
    St.B = B;
  }
  __syncthreads();
  store_words(a, kStageAt, St);
}
template <int KIND, bool C64>
__device__ __forceinline__ void op_eval(const OpArgs& a, const Grp& g) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ OpSh sh;
  if (threadIdx.x == 0) mbar_init(&sh.bar, 1);
  const OpCtx X = op_ctx<KIND, C64>(a);
  unsigned phase = 0;
  bool ok = true;
  if constexpr (KIND == K_PERM) {
    if (a.seg && __ldcg(&stage_of(a)->state) != ST_OK) return;
    __syncthreads();
    if (threadIdx.x == 0) sh.R = OpResult{};
    if (!X.bad) ok = staged_perm<C64>(a, sh, X, &phase, smem);
    pdl_trigger();
    if (op_exit(a.ctrl, g.nblk, !ok) == 1) op_close(a, KIND, P_HIST, P_HIST, sh.R, X.S.n);
  } else {
    load_words(a, kStageAt, sh.St);
    __syncthreads();
    if (sh.St.state != ST_OK) return;
    const Bracket B = sh.St.B;
    ok = staged_eval<KIND, C64>(a, sh, X, B, &phase, smem);
    pdl_trigger();
    const int last = op_exit(a.ctrl, g.nblk, !ok);
    if (!last) return;
    if (last == 1) {
      staged_plan(a, sh, X, B);
    } else {
      if (threadIdx.x == 0) sh.St.state = ST_GAVE_UP;
      __syncthreads();
    }
    store_words(a, kStageAt, sh.St);
  }
}
template <int KIND, bool C64>
__device__ __forceinline__ void op_settle(const OpArgs& a, const Grp& g) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ OpSh sh;
  if (threadIdx.x == 0) mbar_init(&sh.bar, 1);
  const OpCtx X = op_ctx<KIND, C64>(a);
  if (threadIdx.x == 0) op_preload(a, sh);
  load_words(a, kStageAt, sh.St);
  out_order_par(a.in, KIND, a.q, a.gb, sh.qat);
  __syncthreads();
  if (sh.St.state == ST_OVER) return;
  Gate gate{reinterpret_cast<unsigned*>(&a.ctrl->sync_counter), g.nblk, g.nblk, 0u, false};
  unsigned phase = 0;
  const bool ok = sh.St.state != ST_GAVE_UP && staged_settle<KIND, C64>(a, g, sh, X, gate, &phase, smem);
  pdl_trigger();
  const int last = op_exit(a.ctrl, g.nblk, !ok);
  if (!last) return;
  if (last == 1) {
    staged_final<KIND>(a, sh, X, smem);
  } else {
    if (threadIdx.x == 0) {
      sh.R = OpResult{};
      sh.R.failed = 1;
    }
    __syncthreads();
  }
  store_words(a, kResultAt, sh.R);
}
template <int KIND, bool C64>
__device__ __forceinline__ void op_write(const OpArgs& a, const Grp& g) {
  __shared__ OpSh sh;
  const OpCtx X = op_ctx<KIND, C64>(a);
  if (threadIdx.x == 0) op_preload(a, sh);
  if (X.bad) {
    if (threadIdx.x == 0) sh.R = OpResult{};
  } else {
    load_words(a, kResultAt, sh.R);
  }
  __syncthreads();
  if (!X.bad && !sh.R.failed) staged_write<KIND, C64>(a, g, sh, X);
  pdl_trigger();
  if (sh.R.failed == kOver) return;
  if (op_exit(a.ctrl, g.nblk, sh.R.failed != 0) == 1) op_close(a, KIND, P_HIST, P_WRITE, sh.R, X.S.n);
}

template <int KIND, bool C64>
__global__ void __launch_bounds__(kThreads, 4) k_op(const __grid_constant__ OpArgs a) {
  pdl_wait();
  op_first<KIND, C64, false, false, 2>(a, whole_grid());
}
template <int KIND, bool C64>
__global__ void __launch_bounds__(kThreads, 4) k_op4(const __grid_constant__ OpArgs a) {
  pdl_wait();
  op_first<KIND, C64, false, false, 4>(a, whole_grid());
}
template <int KIND, bool C64>
__global__ void __launch_bounds__(kThreads, 4) k_op_try(const __grid_constant__ OpArgs a) {
  pdl_wait();
  op_first<KIND, C64, true, true, 2>(a, whole_grid());
}
template <int KIND, bool C64>
__global__ void __launch_bounds__(kThreads) k_op_prep(const __grid_constant__ OpArgs a) {
  pdl_wait();
  op_prep<KIND, C64>(a, whole_grid());
}
template <int KIND, bool C64>
__global__ void __launch_bounds__(kThreads, 4) k_op_eval(const __grid_constant__ OpArgs a) {
  pdl_wait();
  op_eval<KIND, C64>(a, whole_grid());
}
template <int KIND, bool C64>
__global__ void __launch_bounds__(kThreads, 4) k_op_settle(const __grid_constant__ OpArgs a) {
  pdl_wait();
  op_settle<KIND, C64>(a, whole_grid());
}
template <int KIND, bool C64>
__global__ void __launch_bounds__(kThreads, 4) k_op_write(const __grid_constant__ OpArgs a) {
  pdl_wait();
  op_write<KIND, C64>(a, whole_grid());
}

// One op on each of many states: every state's block group runs the same passes
// with the state's own workspace and control block (and so its own barriers).
// (As one kernel of both routes they spilled 700 to 2,300 bytes a thread and
// waited at grid barriers between the passes: 64 states of 32,768 entries took
// 431 us per 1-qubit gate.)
template <int KIND, bool C64>
__global__ void __launch_bounds__(kThreads, 4) k_op_seg(const OpArgs* ops, const SegPlan* plan) {
  __shared__ OpArgs sa;
  pdl_wait();  // the plan is the kernel before's
  const Grp g = seg_enter(ops, plan, &sa, nullptr);
  op_first<KIND, C64, false, false, 2>(sa, g);
}
// (states that need larger tiles, or the launches after this one)
template <int KIND, bool C64>
__global__ void __launch_bounds__(kThreads, 4) k_op4_seg(const OpArgs* ops, const SegPlan* plan) {
  __shared__ OpArgs sa;
  pdl_wait();
  const Grp g = seg_enter(ops, plan, &sa, nullptr);
  op_first<KIND, C64, true, false, 4>(sa, g);
}
template <int KIND, bool C64>
__global__ void __launch_bounds__(kThreads) k_op_prep_seg(const OpArgs* ops, const SegPlan* plan) {
  __shared__ OpArgs sa;
  pdl_wait();
  const Grp g = seg_enter(ops, plan, &sa, nullptr);
  op_prep<KIND, C64>(sa, g);
}
// (three blocks per SM: with the op's arguments in shared memory four spill; 148
// states of 2048 entries 52 -> 40 us, 64 of 32,768 81 -> 75)
template <int KIND, bool C64>
__global__ void __launch_bounds__(kThreads, 3) k_op_eval_seg(const OpArgs* ops, const SegPlan* plan) {
  __shared__ OpArgs sa;
  pdl_wait();
  const Grp g = seg_enter(ops, plan, &sa, nullptr);
  op_eval<KIND, C64>(sa, g);
}
template <int KIND, bool C64>
__global__ void __launch_bounds__(kThreads, 4) k_op_settle_seg(const OpArgs* ops, const SegPlan* plan) {
  __shared__ OpArgs sa;
  pdl_wait();
  const Grp g = seg_enter(ops, plan, &sa, nullptr);
  op_settle<KIND, C64>(sa, g);
}
template <int KIND, bool C64>
__global__ void __launch_bounds__(kThreads, 4) k_op_write_seg(const OpArgs* ops, const SegPlan* plan) {
  __shared__ OpArgs sa;
  pdl_wait();
  const Grp g = seg_enter(ops, plan, &sa, nullptr);
  op_write<KIND, C64>(sa, g);
}

// ---------------------------------------------------------------------------
// launch
// ---------------------------------------------------------------------------
// op_exit counts the blocks in 10 bits; a chip op keeps a count per block in
// the smallest workspace's partition records (3 x 6 words per set)
constexpr int kOpMaxBlocks = 1023;
static_assert(kOpMaxBlocks <= (int)kExitMask && kOpMaxBlocks <= kMaxSets * 3 * 6, "block counts");

// Resident grid of a kernel of kThreads threads (at most kOpMaxBlocks).  carveout:
// the share of an SM's memory preferred as shared memory, in per cent.
template <typename K>
static cudaError_t op_grid(PerDevice& cache, K kern, size_t smem, int* grid, int carveout = -1) {
  return per_device(cache, grid, [kern, smem, carveout](int* g) {
    cudaError_t e = cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess && carveout >= 0)
      e = cudaFuncSetAttribute((const void*)kern, cudaFuncAttributePreferredSharedMemoryCarveout, carveout);
    if (e != cudaSuccess) return e;
    int occ = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kThreads, smem);
    if (e != cudaSuccess) return e;
    if (occ < 1) return cudaErrorInvalidConfiguration;
    *g = device().sms * occ;
    if (*g > kOpMaxBlocks) *g = kOpMaxBlocks;
    return cudaSuccess;
  });
}

// The kinds that take states of up to 592 x 1020 entries on chip, in larger tiles
// (us per op of 400,000 entries, staged and on chip: 1-qubit gate 73 and 56,
// 2-qubit gate 119 and 107, truncation 52 and 39; of 600,000: 81 and 60, 130 and
// 124, 58 and 52).  A rotation step that is rejected writes nothing, and the
// larger tiles' chain costs more than the staging: 67 and 71, 74 and 79.
template <int KIND>
constexpr bool kChip4 = KIND != K_PERM && KIND != K_ROT1;

// The grids of a kind's launches.
struct OpGrids {
  int first, first4, prep, eval, settle, write;
};
// (A staged op's first launch follows the write of the op before: the same split
// of an SM's memory between L1 and shared memory spares it a change, 1 to 2 us
// per op at 2^22 entries.)
constexpr int kCarveout = 28;  // per cent: 64 KB
template <int KIND, bool C64>
static cudaError_t op_grids(OpGrids* g) {
  static PerDevice cf, c4, ct, cp, ce, cs, cw;
  int unused = 0;
  cudaError_t e = op_grid(cf, k_op<KIND, C64>, kChipSmem<2>, &g->first);
  if constexpr (kChip4<KIND>)
    if (e == cudaSuccess) e = op_grid(c4, k_op4<KIND, C64>, kChipSmem<4>, &g->first4);
  if constexpr (KIND != K_PERM) {
    if (e == cudaSuccess) e = op_grid(ct, k_op_try<KIND, C64>, kChipSmem<2>, &unused, kCarveout);
  }
  if (e == cudaSuccess) e = op_grid(cp, k_op_prep<KIND, C64>, 0, &g->prep);
  if (e == cudaSuccess) e = op_grid(ce, k_op_eval<KIND, C64>, kTileSmem, &g->eval);
  if constexpr (KIND != K_PERM) {
    if (e == cudaSuccess) e = op_grid(cs, k_op_settle<KIND, C64>, kTileSmem, &g->settle);
    if (e == cudaSuccess) e = op_grid(cw, k_op_write<KIND, C64>, 0, &g->write, kCarveout);
  }
  return e;
}

template <int KIND, bool C64>
static cudaError_t launch_op(OpArgs a, cudaStream_t s) {
  OpGrids g{};
  cudaError_t e = op_grids<KIND, C64>(&g);
  if (e != cudaSuccess) return e;
  // the workspace bounds the entries (the kernels refuse more); the reorder of a
  // 2-qubit gate is bounded by the gate after it, which holds a quarter
  const long long bound = a.entries ? a.entries : a.ws.max_n / slots_per_entry(KIND);
  const bool larger = bound > (long long)g.first * kChipStep<2>;
  a.staged = larger && (!kChip4<KIND> || bound > (long long)g.first4 * kChipStep<4>);
  const long long want = bound <= kChipStep<2> ? 1 : (bound + kChipMin - 1) / kChipMin;
  if (a.staged) g.first = KIND == K_IDENT ? device().sms : kFirstBlocks;
  else if (want < g.first) g.first = (int)want;
  if (a.staged) {
    if constexpr (KIND != K_PERM)  // (a staged reorder has nothing to clear)
      KLAUNCH(KIND * 5 + P_GATHER, s,
              e = launch_pdl(k_op_try<KIND, C64>, dim3(g.first), dim3(kThreads), kChipSmem<2>, s, a));
  } else if (larger) {
    if constexpr (kChip4<KIND>)
      KLAUNCH(KIND * 5 + P_GATHER, s,
              e = launch_coop(k_op4<KIND, C64>, dim3(g.first4), dim3(kThreads), kChipSmem<4>, s, a));
  } else if (g.first == 1) {  // no barrier
    KLAUNCH(KIND * 5 + P_GATHER, s, e = launch_pdl(k_op<KIND, C64>, dim3(1), dim3(kThreads), kChipSmem<2>, s, a));
  } else {
    KLAUNCH(KIND * 5 + P_GATHER, s, e = launch_coop(k_op<KIND, C64>, dim3(g.first), dim3(kThreads), kChipSmem<2>, s, a));
  }
  if (e != cudaSuccess || !a.staged) return e;
  KLAUNCH(S_PARTITION, s, e = launch_pdl(k_op_prep<KIND, C64>, dim3(g.prep), dim3(kThreads), 0, s, a));
  if (e != cudaSuccess) return e;
  KLAUNCH(KIND * 5 + P_HIST, s, e = launch_pdl(k_op_eval<KIND, C64>, dim3(g.eval), dim3(kThreads), kTileSmem, s, a));
  if constexpr (KIND != K_PERM) {
    if (e != cudaSuccess) return e;
    KLAUNCH(KIND * 5 + P_HIST2, s,
            e = launch_coop(k_op_settle<KIND, C64>, dim3(g.settle), dim3(kThreads), kTileSmem, s, a));
    if (e != cudaSuccess) return e;
    KLAUNCH(KIND * 5 + P_WRITE, s, e = launch_pdl(k_op_write<KIND, C64>, dim3(g.write), dim3(kThreads), 0, s, a));
  }
  return e;
}

template <int KIND>
cudaError_t merge_op(const OpArgs& a, cudaStream_t s) {
  return a.c64 ? launch_op<KIND, true>(a, s) : launch_op<KIND, false>(a, s);
}

// ---- segmented ------------------------------------------------------------------
// Resident grid of the segmented op (at least one block per segment).
template <int KIND, bool C64>
static cudaError_t seg_op_grid(int* grid) {
  static PerDevice cache;
  return op_grid(cache, k_op_seg<KIND, C64>, kChipSmem<2>, grid);
}

// Do the staged launches have to follow the first one?  Not if every state fits
// its blocks however many entries it holds: with work weights n + kSegPad a
// state gets more than (grid - nseg) (n + kSegPad) / W blocks, so W <= (grid -
// nseg) kChipStep, which the workspaces' bounds show, is enough: 0 for the small
// tiles, 1 for the larger ones; 2 otherwise.  slots: children per entry that the
// workspaces are sized for.
template <int KIND>
cudaError_t seg_stages_t(OpArgs* ops, int nseg, int slots, int* staged) {
  int grid = 0;
  const cudaError_t e = ops[0].c64 ? seg_op_grid<KIND, true>(&grid) : seg_op_grid<KIND, false>(&grid);
  if (e != cudaSuccess) return e;
  long long w = 0;
  for (int i = 0; i < nseg; ++i) w += ops[i].ws.max_n / slots + kSegPad;
  const long long fit = w / (grid - nseg > 0 ? grid - nseg : 1);
  *staged = fit < kChipStep<2> ? 0 : fit < kChipStep<4> ? 1 : 2;
  for (int i = 0; i < nseg; ++i) ops[i].staged = *staged == 2, ops[i].seg = 1;
  return cudaSuccess;
}

// The first launch is cooperative, since states that stay on chip share it.
template <int KIND, bool C64>
static cudaError_t merge_op_seg(const OpArgs* ops, int nseg, int staged, SegPlan* plan, cudaStream_t s) {
  static PerDevice c4, cp, ce, cs, cw;
  OpGrids g{};
  cudaError_t e = seg_op_grid<KIND, C64>(&g.first);
  if (e == cudaSuccess) e = op_grid(c4, k_op4_seg<KIND, C64>, kChipSmem<4>, &g.first4);
  if (e == cudaSuccess) e = op_grid(cp, k_op_prep_seg<KIND, C64>, 0, &g.prep);
  if (e == cudaSuccess) e = op_grid(ce, k_op_eval_seg<KIND, C64>, kTileSmem, &g.eval);
  if constexpr (KIND != K_PERM) {
    if (e == cudaSuccess) e = op_grid(cs, k_op_settle_seg<KIND, C64>, kTileSmem, &g.settle);
    if (e == cudaSuccess) e = op_grid(cw, k_op_write_seg<KIND, C64>, 0, &g.write);
  }
  if (e != cudaSuccess) return e;
  int most = g.first;  // the groups' barriers need every block resident
  if (KIND != K_PERM && most > device().sms) most = device().sms;  // (seg_max_segments)
  if (nseg > most) return cudaErrorInvalidValue;
  if ((e = run_seg_plan(ops, nseg, KIND, plan, s)) != cudaSuccess) return e;
  const SegPlan* p = plan;
  if (staged == 0)
    KLAUNCH(KIND * 5 + P_GATHER, s,
            e = launch_coop(k_op_seg<KIND, C64>, dim3(g.first), dim3(kThreads), kChipSmem<2>, s, ops, p));
  else
    KLAUNCH(KIND * 5 + P_GATHER, s,
            e = launch_coop(k_op4_seg<KIND, C64>, dim3(g.first4), dim3(kThreads), kChipSmem<4>, s, ops, p));
  if (e != cudaSuccess || staged < 2) return e;
  KLAUNCH(S_PARTITION, s, e = launch_pdl(k_op_prep_seg<KIND, C64>, dim3(g.prep), dim3(kThreads), 0, s, ops, p));
  if (e != cudaSuccess) return e;
  KLAUNCH(KIND * 5 + P_HIST, s,
          e = launch_pdl(k_op_eval_seg<KIND, C64>, dim3(g.eval), dim3(kThreads), kTileSmem, s, ops, p));
  if constexpr (KIND != K_PERM) {
    if (e != cudaSuccess) return e;
    KLAUNCH(KIND * 5 + P_HIST2, s,
            e = launch_coop(k_op_settle_seg<KIND, C64>, dim3(g.settle), dim3(kThreads), kTileSmem, s, ops, p));
    if (e != cudaSuccess) return e;
    KLAUNCH(KIND * 5 + P_WRITE, s,
            e = launch_pdl(k_op_write_seg<KIND, C64>, dim3(g.write), dim3(kThreads), 0, s, ops, p));
  }
  return e;
}

template <int KIND>
cudaError_t merge_op_seg_t(const OpArgs* ops, int nseg, int c64, int staged, SegPlan* plan, cudaStream_t s) {
  return c64 ? merge_op_seg<KIND, true>(ops, nseg, staged, plan, s)
             : merge_op_seg<KIND, false>(ops, nseg, staged, plan, s);
}

}  // namespace bass
