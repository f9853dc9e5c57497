// sort.cu -- the stable LSD radix sort of (key, amplitude) entries
// (sparse_state.py:150-172 sorts 16-bit digits; any stable LSD order gives
// the same result) and the export of a state as sorted true keys.
//
// One cooperative launch sorts: the keys are read once for the histograms of
// every 8-bit digit, then one pass per digit moves (key, 32-bit index) pairs,
// and the last pass fetches each entry's amplitude by its index straight to
// its final place.  What bounds it is memory traffic, so a pass moves 12 bytes
// per entry each way instead of the 24 of a whole entry, and reads nothing
// twice: a tile's offsets come from its predecessors' counts while they run
// (decoupled look-back per digit, tiles taken in order from a counter) instead
// of a histogram pass and a scan per digit.  Tiles of 4096 entries go through
// shared memory, so that a digit's run (16 entries on average) is written
// contiguously.  At 2^22 entries of 40 bits the export takes 0.48 ms on the
// device (5 passes); three launches per digit with a one-CTA scan and 24-byte
// moves took 6.4 ms (150,001 complex64 entries of 30 bits: 0.10 and 0.22 ms).
// Up to kSortTile entries are sorted by one CTA without leaving shared memory:
// 19 us instead of 65 at 256 entries of 12 bits.
#include <math.h>

#include "internal.h"

namespace bass {

constexpr int kSortThreads = 512;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSortItems = 8;                          // per thread
constexpr int kSortTile = kSortThreads * kSortItems;   // 4096
constexpr int kDigits = 256;
constexpr int kMaxPasses = 8;
constexpr int kSortCounters = kMaxPasses + 2;

struct SortArgs {
  const bass_state* st;      // export: the source state (n = its nnz), or nullptr
  const long long* n_dev;    // entry count on the device, or nullptr: n_host
  long long n_host;
  uint64_t* keys;            // result keys (the source too, without st)
  void* amps;                // result amplitudes
  const void* src_amps;      // amplitudes in source order (without st)
  uint64_t* tkeys;           // second key buffer
  unsigned int* idx0;        // index buffers
  unsigned int* idx1;
  unsigned int* hist;        // kMaxPasses x kDigits counts, zeroed before the launch
  unsigned long long* ctr;   // zeroed: [p] tile counter of pass p, [kMaxPasses] barrier arrivals, [kMaxPasses + 1] give-ups
  unsigned long long* status;  // per tile and digit: pass tag and count, see look_back
  long long max_n;
  long long max_tiles;       // tiles the status array holds
  int passes;
  int amp_type;              // export: the type the caller expects
  bass_ctrl* ctrl;           // may be nullptr (the plain array sort)
};

// Status words: bits 62-63 flag (1 the tile's count, 2 the inclusive prefix),
// bits 56-61 the pass, so that a word of an earlier pass counts as not written
// and the array is cleared once per sort.
__device__ __forceinline__ unsigned long long sort_word(int pass, int flag, unsigned long long v) {
  return ((unsigned long long)flag << 62) | ((unsigned long long)(pass + 1) << 56) | v;
}

__device__ __forceinline__ void sort_error(const SortArgs& a) {
  if (a.ctrl) set_error(a.ctrl, BASS_ERR_WAIT);
  else atomicAdd(a.ctr + kMaxPasses + 1, 1ULL);
}

// Barrier of the launch's nblk working blocks (all resident: a cooperative
// launch); false if the bounded wait gave up.
__device__ bool sort_sync(const SortArgs& a, int nblk, unsigned long long target, long long lim) {
  __shared__ int sOk;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    red_release_add(a.ctr + kMaxPasses, 1ULL);
    int ok = 1;
    long long spins = 0;
    while (ld_acquire(a.ctr + kMaxPasses) < target * (unsigned long long)nblk) {
      if (++spins > lim) {
        sort_error(a);
        ok = 0;
        break;
      }
      __nanosleep(32);
    }
    __threadfence();
    sOk = ok;
  }
  __syncthreads();
  return sOk != 0;
}

struct SortSmem {
  uint64_t key[kSortTile];
  unsigned int idx[kSortTile];
  unsigned int cnt[kSortWarps][kDigits];  // per warp: count, then first rank of the digit
  unsigned int start[kDigits];            // local position of the digit's run
  unsigned int scan[kDigits / 32];
  long long base[kDigits];                // global position of the digit's run minus start
};

// Exclusive scan of one value per thread 0..255 (all threads call).
__device__ __forceinline__ unsigned scan256(unsigned v, unsigned* sw) {
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  unsigned x = v;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const unsigned y = __shfl_up_sync(0xffffffffu, x, off);
    if (lane >= off) x += y;
  }
  if (t < kDigits && lane == 31) sw[w] = x;
  __syncthreads();
  unsigned add = 0;
  if (t < kDigits)
    for (int i = 0; i < w; ++i) add += sw[i];
  __syncthreads();
  return x - v + add;
}

// Ranks the tile's entries by the digit (stable: entry j of lane l of warp w is
// position 256 w + 32 j + l) and leaves them in digit order in S.key / S.idx.
// S.start: local start per digit; the returned value is digit threadIdx.x's
// count in the tile (threads 0-255).
__device__ __forceinline__ unsigned tile_rank(SortSmem& S, const uint64_t (&k)[kSortItems],
                                              const unsigned (&ix)[kSortItems], int m, int shift) {
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const unsigned lt = (1u << lane) - 1;
  for (int d = lane; d < kDigits; d += 32) S.cnt[w][d] = 0;
  __syncwarp();
  unsigned rk[kSortItems];
#pragma unroll
  for (int j = 0; j < kSortItems; ++j) {
    const int p = w * (32 * kSortItems) + 32 * j + lane;
    const bool live = p < m;
    const unsigned d = (unsigned)(k[j] >> shift) & 255u;
    unsigned peers = __ballot_sync(0xffffffffu, live);
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const unsigned o = __ballot_sync(0xffffffffu, (d >> b) & 1u);
      peers &= ((d >> b) & 1u) ? o : ~o;
    }
    const unsigned before = __popc(peers & lt);
    unsigned old = 0;
    if (live) old = S.cnt[w][d];
    __syncwarp();
    if (live && before == 0) S.cnt[w][d] = old + __popc(peers);
    __syncwarp();
    rk[j] = old + before;
  }
  __syncthreads();
  unsigned tot = 0;
  if (t < kDigits) {
#pragma unroll
    for (int i = 0; i < kSortWarps; ++i) {
      const unsigned c = S.cnt[i][t];
      S.cnt[i][t] = tot;
      tot += c;
    }
  }
  const unsigned st = scan256(t < kDigits ? tot : 0u, S.scan);
  if (t < kDigits) S.start[t] = st;
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kSortItems; ++j) {
    const int p = w * (32 * kSortItems) + 32 * j + lane;
    if (p < m) {
      const unsigned d = (unsigned)(k[j] >> shift) & 255u;
      const unsigned q = S.start[d] + S.cnt[w][d] + rk[j];
      S.key[q] = k[j];
      S.idx[q] = ix[j];
    }
  }
  __syncthreads();
  return tot;
}

// Digit threadIdx.x (threads 0-255): publishes the tile's count and returns
// the count in the tiles before it (bounded wait; *ok cleared on give-up).
__device__ __forceinline__ unsigned long long look_back(const SortArgs& a, long long tile, int pass,
                                                        unsigned cnt, long long lim, bool* ok) {
  unsigned long long* col = a.status + threadIdx.x;
  const unsigned long long vmask = (1ULL << 56) - 1;
  if (tile == 0) {
    st_release(col, sort_word(pass, 2, cnt));
    return 0;
  }
  st_release(col + tile * kDigits, sort_word(pass, 1, cnt));
  unsigned long long excl = 0;
  long long spins = 0;
  for (long long k = tile - 1; k >= 0;) {
    const unsigned long long s = ld_acquire(col + k * kDigits);
    if (((s >> 56) & 63) != (unsigned long long)(pass + 1) || (s >> 62) == 0) {
      if (++spins > lim) {
        *ok = false;
        break;
      }
      continue;
    }
    excl += s & vmask;
    if ((s >> 62) == 2) break;
    --k;
  }
  st_release(col + tile * kDigits, sort_word(pass, 2, excl + cnt));
  return excl;
}

// The amplitude of source entry i to result entry o: scaled (export) or moved.
template <typename P>
__device__ __forceinline__ void put_amp(const SortArgs& a, long long o, unsigned i, bool c64, double r0, double r1) {
  if (a.st)
    amp_put(static_cast<double*>(a.amps), o, amp_get(a.st->amps, i, c64, r0, r1), c64);
  else
    static_cast<P*>(a.amps)[o] = static_cast<const P*>(a.src_amps)[i];
}

template <typename P>
__global__ void __launch_bounds__(kSortThreads, 2) k_sort(const __grid_constant__ SortArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  SortSmem& S = *reinterpret_cast<SortSmem*>(smem);
  __shared__ int8_t qat[64];
  __shared__ long long sTile;
  __shared__ int sBad;
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const long long n = a.n_dev ? *a.n_dev : a.n_host;
  const long long ntiles = (n + kSortTile - 1) / kSortTile;
  if (n > a.max_n || ntiles > a.max_tiles) return;
  double r0 = 1.0, r1 = 1.0;
  if (a.st) {
    if (a.st->amp_type != a.amp_type) {
      if (blockIdx.x == 0 && t == 0) set_error(a.ctrl, BASS_ERR_ARG);
      return;
    }
    if (t < 64) qat[t] = a.st->qat[t];
    r0 = a.st->rscale[0];
    r1 = a.st->rscale[1];
  }
  if (n <= 0) return;
  const bool c64 = sizeof(P) == 8;
  const uint64_t* in = a.st ? a.st->keys : a.keys;
  auto first_key = [&](long long i) { return a.st ? true_key(in[i], qat, 64) : in[i]; };
  __syncthreads();
  const long long lim = a.ctrl ? wait_limit(a.ctrl) : kSpinLimit;

  if (ntiles == 1) {
    // one tile: every pass in block 0's shared memory
    if (blockIdx.x != 0) return;
    const int m = (int)n;
    uint64_t k[kSortItems];
    unsigned ix[kSortItems];
#pragma unroll
    for (int j = 0; j < kSortItems; ++j) {
      const int p = w * (32 * kSortItems) + 32 * j + lane;
      k[j] = p < m ? first_key(p) : 0;
      ix[j] = (unsigned)p;
    }
    for (int pass = 0; pass < a.passes; ++pass) {
      tile_rank(S, k, ix, m, 8 * pass);
      if (pass + 1 == a.passes) break;
#pragma unroll
      for (int j = 0; j < kSortItems; ++j) {
        const int p = w * (32 * kSortItems) + 32 * j + lane;
        k[j] = p < m ? S.key[p] : 0;
        ix[j] = p < m ? S.idx[p] : 0;
      }
      __syncthreads();
    }
    for (int p = t; p < m; p += kSortThreads) {
      a.keys[p] = S.key[p];
      put_amp<P>(a, p, S.idx[p], c64, r0, r1);
    }
    return;
  }

  // the working blocks; every key buffer alternates, the last pass writes a.keys
  const int nblk = (long long)gridDim.x < ntiles ? (int)gridDim.x : (int)ntiles;
  if ((int)blockIdx.x >= nblk) return;
  unsigned long long bars = 0;
  uint64_t* src = (a.passes & 1) ? a.tkeys : a.keys;
  uint64_t* dst = (a.passes & 1) ? a.keys : a.tkeys;
  // histograms of every digit; the true keys (or a copy, when the first pass
  // must not read a.keys) to src; the status words cleared
  {
    unsigned* h = &S.cnt[0][0];  // passes x 256
    for (int i = t; i < kMaxPasses * kDigits; i += kSortThreads) h[i] = 0;
    const long long gs = (long long)nblk * kSortThreads;
    const long long g0 = (long long)blockIdx.x * kSortThreads + t;
    for (long long i = g0; i < ntiles * kDigits; i += gs) a.status[i] = 0ULL;
    __syncthreads();
    for (long long i = g0; i < n; i += gs) {
      const uint64_t k = first_key(i);
      if (src != in) src[i] = k;
      for (int p = 0; p < a.passes; ++p) atomicAdd(&h[p * kDigits + ((unsigned)(k >> (8 * p)) & 255u)], 1u);
    }
    __syncthreads();
    for (int i = t; i < a.passes * kDigits; i += kSortThreads)
      if (h[i]) atomicAdd(a.hist + i, h[i]);
  }
  if (!sort_sync(a, nblk, ++bars, lim)) return;
  for (int pass = 0; pass < a.passes; ++pass) {
    const int shift = 8 * pass;
    const bool last = pass + 1 == a.passes;
    const unsigned int* isrc = (pass & 1) ? a.idx1 : a.idx0;
    unsigned int* idst = (pass & 1) ? a.idx0 : a.idx1;
    // the digits' first positions in the sorted order
    const unsigned gstart = scan256(t < kDigits ? __ldcg(a.hist + pass * kDigits + t) : 0u, S.scan);
    for (;;) {
      if (t == 0) {
        sTile = (long long)atomicAdd(a.ctr + pass, 1ULL);
        sBad = 0;
      }
      __syncthreads();
      const long long tile = sTile;
      if (tile >= ntiles) break;
      const long long lo = tile * kSortTile;
      const int m = (int)(n - lo < kSortTile ? n - lo : kSortTile);
      uint64_t k[kSortItems];
      unsigned ix[kSortItems];
#pragma unroll
      for (int j = 0; j < kSortItems; ++j) {
        const int p = w * (32 * kSortItems) + 32 * j + lane;
        k[j] = p < m ? __ldcg(src + lo + p) : 0;
        ix[j] = pass == 0 ? (unsigned)(lo + p) : (p < m ? __ldcg(isrc + lo + p) : 0u);
      }
      const unsigned cnt = tile_rank(S, k, ix, m, shift);
      if (t < kDigits) {
        bool ok = true;
        const unsigned long long before = look_back(a, tile, pass, cnt, lim, &ok);
        S.base[t] = (long long)gstart + (long long)before - (long long)S.start[t];
        if (!ok) sBad = 1;
      }
      __syncthreads();
      if (sBad) {  // a wait gave up: nothing of this tile is written
        if (t == 0) sort_error(a);
      } else {
        for (int p = t; p < m; p += kSortThreads) {
          const uint64_t key = S.key[p];
          const long long o = S.base[(unsigned)(key >> shift) & 255u] + p;
          if (o < 0 || o >= n) continue;  // only after another tile's give-up
          dst[o] = key;
          if (!last) idst[o] = S.idx[p];
          else if (S.idx[p] < n) put_amp<P>(a, o, S.idx[p], c64, r0, r1);  // (as above)
        }
      }
      __syncthreads();
    }
    if (last) break;
    if (!sort_sync(a, nblk, ++bars, lim)) return;
    uint64_t* tk = src;
    src = dst;
    dst = tk;
  }
}

// After a sort without a control block: a give-up leaves keys out of place and
// nothing else would say so, so every amplitude of the result becomes NaN.
__global__ void k_sort_check(SortArgs a, int c64) {
  if (a.ctr[kMaxPasses + 1] == 0ULL) return;
  const long long step = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < 2 * a.n_host; i += step) {
    if (c64) static_cast<float*>(a.amps)[i] = NAN;
    else static_cast<double*>(a.amps)[i] = NAN;
  }
}

template <typename P>
static cudaError_t launch_sort(SortArgs a, const WsView& ws, cudaStream_t s) {
  static PerDevice cache;
  int grid = 0;
  const size_t smem = sizeof(SortSmem);
  cudaError_t e = per_device(cache, &grid, [smem](int* g) {
    cudaError_t e2 = cudaFuncSetAttribute(k_sort<P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e2 != cudaSuccess) return e2;
    int occ = 0;
    e2 = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_sort<P>, kSortThreads, smem);
    if (e2 != cudaSuccess) return e2;
    if (occ < 1) return cudaErrorInvalidConfiguration;
    *g = device().sms * occ;
    return cudaSuccess;
  });
  if (e != cudaSuccess) return e;
  // the digit histograms and counters share the selection's histogram area
  a.hist = ws.hist1;
  a.ctr = reinterpret_cast<unsigned long long*>(ws.hist1 + kMaxPasses * kDigits);
  static_assert(kMaxPasses * kDigits + 2 * kSortCounters <= kHistBins, "sort counters fit the histogram area");
  e = cudaMemsetAsync(a.hist, 0, (kMaxPasses * kDigits + 2 * kSortCounters) * sizeof(unsigned int), s);
  if (e != cudaSuccess) return e;
  a.tkeys = ws.tmp_keys;
  a.idx0 = reinterpret_cast<unsigned int*>(ws.cand_key);
  a.idx1 = a.idx0 + ws.max_n;
  a.status = reinterpret_cast<unsigned long long*>(ws.sort_hist);
  a.max_n = ws.max_n < (1LL << 32) ? ws.max_n : (1LL << 32) - 1;
  a.max_tiles = ws.sort_tiles / 2;  // 256 eight-byte words per tile of 4096
  void* args[] = {&a};
  KLAUNCH(S_SORT, s, e = cudaLaunchCooperativeKernel((const void*)k_sort<P>, dim3(grid), dim3(kSortThreads), args,
                                                     smem, s));
  if (e == cudaSuccess && !a.ctrl) {
    KLAUNCH(S_SORT, s, k_sort_check<<<device().sms, 256, 0, s>>>(a, sizeof(P) == 8));
    e = cudaGetLastError();
  }
  return e;
}

// Sorts n entries in place by the low key_bits bits (amps: complex128 pairs,
// or complex64 pairs when c64).
cudaError_t run_radix_sort(uint64_t* keys, double* amps, long long n, int key_bits, const WsView& ws,
                           bass_ctrl* ctrl, cudaStream_t s, int c64) {
  if (n <= 0) return cudaSuccess;
  SortArgs a{};
  a.n_host = n;
  a.keys = keys;
  a.amps = amps;
  a.src_amps = ws.tmp_amps;
  a.passes = (key_bits + 7) / 8;
  a.ctrl = ctrl;
  // the last pass reads the amplitudes by index: from a copy
  cudaError_t e = cudaMemcpyAsync(ws.tmp_amps, amps, (size_t)n * (c64 ? 8 : 16), cudaMemcpyDeviceToDevice, s);
  if (e != cudaSuccess) return e;
  return c64 ? launch_sort<unsigned long long>(a, ws, s) : launch_sort<ulonglong2>(a, ws, s);
}

// The state's entries as true keys in ascending order with the pending
// renormalisation applied.
cudaError_t run_export(const bass_state* st, uint64_t* ok, double* oa, int key_bits, const WsView& ws,
                       bass_ctrl* ctrl, cudaStream_t s, int amp_type) {
  SortArgs a{};
  a.st = st;
  a.n_dev = reinterpret_cast<const long long*>(&st->nnz);
  a.keys = ok;
  a.amps = oa;
  a.passes = (key_bits + 7) / 8;
  a.amp_type = amp_type;
  a.ctrl = ctrl;
  return amp_type == BASS_AMP_C64 ? launch_sort<unsigned long long>(a, ws, s) : launch_sort<ulonglong2>(a, ws, s);
}

}  // namespace bass
