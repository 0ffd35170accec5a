// Pivot retrieval: for every pool head, the pivots of the queried voxels ordered by weight W
// (descending), the first R of them copied out with bias log C.
//
// Replaces VoxelKVMerger.retrieve on the reference's Python path (stac/merger.py:1377-1482:
// gather of all [H, Q*P] pivots, argsort by W, three more gathers, index_put compaction) and
// MergerWrapper.retrieve_seg with its torch sort (merger-cuda/csrc/merger_wrapper.cu:3148-3221).
//
// retrieve_select_kernel  one CTA per head: radix select of the weight threshold over the
//                         (voxel, slot) candidates of the queried voxels, the candidates at or
//                         above it collected in shared memory (64-bit keys = weight bits |
//                         inverted candidate index, so equal weights resolve to the earlier
//                         candidate) and put in order: by their places in the range of keys where
//                         they are few and spread, else thinned out to the power of two above R and
//                         sorted in registers.
// retrieve_gather_kernel  copies K/V of the selected pivots with 16-byte vectors, writes mask
//                         and bias, zero-fills the padding.
#include "common.cuh"
#include "stac_internal.h"

namespace stac {
namespace {

constexpr int kSelCap = 8192;     // shared-memory candidate buffer (64-bit keys)
constexpr int kFineKeys = 128;    // keys in whose places 256 counters lie
constexpr int kSelBins = 8192;    // counters of one radix digit (13 + 11 + 8 bits, most significant first)
constexpr int kRankKeys = 3072;   // collected keys that are ranked by their places in the range of keys: two copies of them and
constexpr int kRankBins = 4096;   // so many counters fill the buffer
constexpr int kRankPairs = 1 << 18;    // comparisons of keys of one counter with one another
static_assert(2 * kRankKeys * 8 + kRankBins * 4 <= kSelCap * 8, "ranking in the candidate buffer");
constexpr int kSelUnroll = 2;     // queried voxels per thread in flight
// Threads of the selection kernel.  With more heads than SMs three CTAs of 512 share an SM and hide each
// other's loads; a launch of one CTA per SM or fewer (one layer's memory, a stream whose heads are shared
// by several GPUs) has only its own threads for that.  (5000 voxels, R = 2048, 512 and 1024 threads: 16 heads 57 and 54 us, 148
// heads 94 and 88 us, 149 heads 114 and 131 us, 384 heads 194 and 245 us.  With a few hundred voxels the smaller
// shape is ahead by up to 3 us at any number of heads, but how many there are is known on the device only.
// Four voxels per thread in flight there made the code
// that every call walks through longer and were slower at all sizes: 16 heads, 300 voxels, R = 64 22.9 us
// against 21.2 us with two; 5000 voxels, R = 2048 55.8 against 53.8 us.)
template <bool kFew> struct SelShape {
  static constexpr int kThreads = kFew ? 1024 : 512, kCtas = kFew ? 1 : 3;
};

__device__ __forceinline__ unsigned int wkey(float f) {
  const unsigned int u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ void bitonic_desc(unsigned long long* a, int n) {
  for (int k = 2; k <= n; k <<= 1) {
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int ixj = i ^ j;
        if (ixj > i) {
          const unsigned long long x = a[i], y = a[ixj];
          const bool desc = (i & k) == 0;
          if ((x < y) == desc) {
            a[i] = y;
            a[ixj] = x;
          }
        }
      }
      __syncthreads();
    }
  }
}

// Descending sort of kE * kT keys in shared memory by kT threads: thread t holds keys t * kE ... of the
// bitonic network in registers, partners nearer than that are its own registers, partners inside the
// warp come by shuffle, and only the stages that cross warps (10 of 78 at 4096 keys and 512 threads)
// go through shared memory, one value per bank.
template <int kE, int kT>
__device__ __forceinline__ void sort_desc(unsigned long long* a) {
  const int t = threadIdx.x;
  unsigned long long v[kE];
#pragma unroll
  for (int e = 0; e < kE; ++e) v[e] = a[e * kT + t];        // any assignment will do: the input has no order
#pragma unroll 1
  for (int k = 2; k <= kE * kT; k <<= 1) {
#pragma unroll 1
    for (int j = k >> 1; j >= kE; j >>= 1) {
      const int x = j / kE;                                 // partner thread: t ^ x, same register
      const bool take_max = ((t & x) == 0) == (((t * kE) & k) == 0);
      if (x >= 32) {
        __syncthreads();
#pragma unroll
        for (int e = 0; e < kE; ++e) a[e * kT + t] = v[e];
        __syncthreads();
#pragma unroll
        for (int e = 0; e < kE; ++e) {
          const unsigned long long o = a[e * kT + (t ^ x)];
          if ((o > v[e]) == take_max) v[e] = o;
        }
      } else {
#pragma unroll
        for (int e = 0; e < kE; ++e) {
          const unsigned long long o = __shfl_xor_sync(0xffffffffu, v[e], x);
          if ((o > v[e]) == take_max) v[e] = o;
        }
      }
    }
#pragma unroll
    for (int j = kE / 2; j > 0; j >>= 1) {
      if (j < k) {
#pragma unroll
        for (int e = 0; e < kE; ++e) {
          if ((e & j) == 0) {
            const bool desc = ((t * kE + e) & k) == 0;
            const unsigned long long lo = v[e], hi = v[e + j];
            if ((lo < hi) == desc) {
              v[e] = hi;
              v[e + j] = lo;
            }
          }
        }
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int e = 0; e < kE; ++e) a[t * kE + e] = v[e];
  __syncthreads();
}

struct RetrieveParams {
  int heads, D, P, voxel_cap, voxel_used, R;
  int seg_vec;             // 1: the pivot segments of a row are one aligned 16-byte vector
  const int* query_ids;    // ascending voxel ids
  const int* query_count;  // device scalar
  const int* piv_row_seg;
  const int* piv_row_cnt;
  const void* piv_K;
  const void* piv_V;
  const float* piv_W;
  const float* piv_C;
  int* sel;        // [heads][R] candidate index q*P + slot, -1 = padding
  void* out_K;     // [heads][R][D]
  void* out_V;
  unsigned char* out_mask;  // [heads][R]
  float* out_bias;          // [heads][R]
  int* out_idx;             // [heads][R][2] (voxel, slot) or nullptr
};

// Calls f(weight key, candidate index) for every pivot of the queried voxels of head h: one
// pass over the candidates, kSelUnroll voxels per thread in flight.  Every thread of the CTA
// must call it (no barrier inside).  A voxel's segments are requested together with its count: the
// chain id -> (count, segments) -> weights is what a pass waits for.
template <int kThreads, typename F>
__device__ __forceinline__ void for_each_candidate(const RetrieveParams& p, int h, int Q, F f) {
  const long long hrow = static_cast<long long>(h) * p.voxel_cap;
  for (int base = 0; base < Q; base += kThreads * kSelUnroll) {
    int v[kSelUnroll], n[kSelUnroll];
    int4 seg[kSelUnroll];
#pragma unroll
    for (int u = 0; u < kSelUnroll; ++u) {
      const int q = base + u * kThreads + threadIdx.x;
      v[u] = q < Q ? p.query_ids[q] : -1;
    }
#pragma unroll
    for (int u = 0; u < kSelUnroll; ++u) {
      n[u] = 0;
      seg[u] = make_int4(0, 0, 0, 0);
      if (v[u] >= 0 && v[u] < p.voxel_used) {
        const long long r = hrow + v[u];
        n[u] = min(p.piv_row_cnt[r], 4);
        const int* sr = p.piv_row_seg + r * p.P;
        if (p.seg_vec) {
          seg[u] = *reinterpret_cast<const int4*>(sr);
        } else {
          seg[u].x = sr[0];
          if (p.P > 1) seg[u].y = sr[1];
          if (p.P > 2) seg[u].z = sr[2];
          if (p.P > 3) seg[u].w = sr[3];
        }
      }
    }
    float w[kSelUnroll][4];
#pragma unroll
    for (int u = 0; u < kSelUnroll; ++u) {
      w[u][0] = n[u] > 0 ? p.piv_W[seg[u].x] : 0.f;
      w[u][1] = n[u] > 1 ? p.piv_W[seg[u].y] : 0.f;
      w[u][2] = n[u] > 2 ? p.piv_W[seg[u].z] : 0.f;
      w[u][3] = n[u] > 3 ? p.piv_W[seg[u].w] : 0.f;
    }
#pragma unroll
    for (int u = 0; u < kSelUnroll; ++u) {
      if (base + u * kThreads >= Q) break;      // the same for the whole CTA
      const int q = base + u * kThreads + threadIdx.x;
#pragma unroll
      for (int s = 0; s < 4; ++s)
        if (s < n[u]) f(wkey(w[u][s]), static_cast<unsigned int>(q * p.P + s));
    }
  }
}

// One slot of a shared list per calling lane (slots of one warp are consecutive).
__device__ __forceinline__ int list_push(int* counter) {
  const unsigned int m = __activemask();
  const unsigned int lane = threadIdx.x & 31;
  const int leader = __ffs(m) - 1;
  int base = 0;
  if (static_cast<int>(lane) == leader) base = atomicAdd(counter, __popc(m));
  base = __shfl_sync(m, base, leader);
  return base + __popc(m & ((1u << lane) - 1u));
}

// Top R candidates of one head by (weight desc, candidate index asc).  A radix select on the
// weight key finds the threshold digit by digit (13 + 11 + 8 bits, one pass over the candidates
// per digit) and stops as soon as the candidates at or above the current prefix fit the
// shared-memory buffer, which is then sorted; with the usual spread of weights that is after the
// first digit, i.e. two passes.  Only when more than kSelCap - R candidates share one exact
// weight is the last group taken in candidate order by an ordered pass.
//
// The digit at which the collection stops leaves up to kSelCap keys of which R are wanted, and the
// sort costs more than the passes: the select goes on over the collected keys in shared memory,
// eight bits at a time, until at most the power of two above R are left.  The sort is as wide as what
// was collected, which may be much less than R (16 heads, one voxel queried, R = 4000: 67 us with a sort of
// 4096 keys, 48 us).
// (One layer's memory, 16 heads, R = 2048: insert and retrieval 338 -> 285 us with the 1024-thread shape
// and the register sort; 384 heads, R = 2048: 1170 -> 1139 us.)
template <bool kFew>
__global__ void __launch_bounds__(SelShape<kFew>::kThreads, SelShape<kFew>::kCtas)
retrieve_select_kernel(const RetrieveParams p) {
  constexpr int kSelThreads = SelShape<kFew>::kThreads;
  grid_dep_wait();   // launched with programmatic serialization behind the previous kernel in the stream
  // kSelCap keys; the digit counters live in the same 64 KB (they are dead once the threshold is
  // known and the keys are collected), so three CTAs fit one SM and 384 heads run in one wave
  extern __shared__ unsigned long long cand[];
  int* hist = reinterpret_cast<int*>(cand);
  static_assert(kSelBins * 4 <= kSelCap * 8, "digit counters must fit the candidate buffer");
  __shared__ int warp_sums[kSelThreads / 32];
  __shared__ int sh_count, sh_bin, sh_above, sh_ties;
  // Counters of the select over the collected keys: the last places of the buffer, which that select
  // leaves alone where they are taken (a sort of all of it then).  With a KB of their own three CTAs needed
  // 198 KB, and the SM set aside 228 instead of 196 KB as shared memory: with half the L1 cache left, 384
  // heads, 5000 voxels and scattered segments took 113 instead of 79 us at R = 1, 259 instead of 219 us at
  // R = 2048.
  int* fine = reinterpret_cast<int*>(cand + kSelCap - kFineKeys);
  static_assert(kFew || 3 * (kSelCap * 8 + 1024 + (kSelThreads / 32 + 4 + 63) / 64 * 256) <= 196 * 1024,
                "shared memory of three CTAs (each with the 1 KB that the system takes, in steps of 256 bytes)");
  const int h = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int Q = *p.query_count;
  const int R = p.R;
  // prefix of the threshold found so far: candidates with (key >> shift) > prefix are in for
  // certain, those with (key >> shift) == prefix are undecided
  unsigned int prefix = 0;
  int shift = 32, need = R;       // need = how many of the undecided ones are wanted
  bool take_all = false, ordered_ties = false;
  const int widths[3] = {13, 11, 8};
  for (int level = 0; level < 3; ++level) {
    const int width = widths[level];
    const int new_shift = shift - width;
    for (int i = threadIdx.x; i < kSelBins; i += kSelThreads) hist[i] = 0;
    __syncthreads();
    const unsigned int pf = prefix;
    const int sh_old = shift;
    for_each_candidate<kSelThreads>(p, h, Q, [&](unsigned int wk, unsigned int) {
      // a plain increment: the shared-memory unit adds up the lanes of one address.  (The lanes that have the first one's digit
      // counted together by a ballot first: selection and gather of 16 heads, 6512 voxels 56.3 against 50.1 us, with one weight
      // for all 71.5 against 62.4; 384 heads 247 against 235, one weight 282 against 268.)
      if (sh_old == 32 || (wk >> sh_old) == pf) atomicAdd(&hist[(wk >> new_shift) & ((1u << width) - 1u)], 1);
    });
    __syncthreads();
    // the digit at which the count from the top reaches `need`: every thread sums a few counters, thread 0 the highest
    // (found by one warp, 32 counters at a time from the top: 64 rounds for weights around 1; selection of 16 heads
    // 37.7 against 31.2 us, of 384 heads 72.2 against 51.5)
    const int per = max(1, (1 << width) / kSelThreads);
    const int low = (1 << width) - (static_cast<int>(threadIdx.x) + 1) * per;
    int sum = 0;
    if (low >= 0)
      for (int e = 0; e < per; ++e) sum += hist[low + e];
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) warp_sums[warp] = incl;
    if (threadIdx.x == 0) sh_bin = -1;                  // fewer than `need` undecided candidates exist
    __syncthreads();
    int before = lane < warp ? warp_sums[lane] : 0;     // (at most 32 warps)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
    int above = before + incl - sum;
    if (above < need && above + sum >= need) {          // one thread at most
      for (int e = per - 1;; --e) {
        const int c = hist[low + e];
        if (above + c >= need) {
          sh_bin = low + e;
          sh_above = above;
          sh_ties = c;
          break;
        }
        above += c;
      }
    }
    __syncthreads();
    if (sh_bin < 0) {
      take_all = true;                  // everything undecided is wanted
      break;
    }
    prefix = (prefix << width) | static_cast<unsigned int>(sh_bin);
    shift = new_shift;
    const int decided = (R - need) + sh_above;      // candidates strictly above the new prefix
    need -= sh_above;
    if (decided + sh_ties <= kSelCap) break;        // they all fit: sort settles the rest
    if (level == 2) ordered_ties = true;            // one exact weight, more copies than fit
    __syncthreads();
  }
  // ---- collect (the counters are no longer needed: their memory becomes the key buffer)
  __syncthreads();
  if (threadIdx.x == 0) sh_count = 0;
  __syncthreads();
  if (!ordered_ties) {
    const unsigned int pf = prefix;
    const int sh = shift;
    for_each_candidate<kSelThreads>(p, h, Q, [&](unsigned int wk, unsigned int idx) {
      if (take_all || sh == 32 || (wk >> sh) >= pf) {
        const int pos = list_push(&sh_count);
        if (pos < kSelCap) cand[pos] = (static_cast<unsigned long long>(wk) << 32) | (0xFFFFFFFFu - idx);
      }
    });
  } else {
    // weights above the threshold in any order, then the first `need` candidates that carry the
    // threshold weight itself, in candidate order (batches of one voxel per thread, block scan)
    const unsigned int T = prefix;
    for_each_candidate<kSelThreads>(p, h, Q, [&](unsigned int wk, unsigned int idx) {
      if (wk > T) {
        const int pos = list_push(&sh_count);
        cand[pos] = (static_cast<unsigned long long>(wk) << 32) | (0xFFFFFFFFu - idx);
      }
    });
    __syncthreads();
    int taken = 0;                    // ties accepted so far (same value in every thread)
    for (int base = 0; base < Q && taken < need; base += kSelThreads) {
      const int q = base + threadIdx.x;
      unsigned int mine[4];
      int n_mine = 0;
      if (q < Q) {
        const int v = p.query_ids[q];
        if (v >= 0 && v < p.voxel_used) {
          const long long r = static_cast<long long>(h) * p.voxel_cap + v;
          const int n = min(p.piv_row_cnt[r], 4);
          for (int s = 0; s < n; ++s)
            if (wkey(p.piv_W[p.piv_row_seg[r * p.P + s]]) == T) mine[n_mine++] = static_cast<unsigned int>(q * p.P + s);
        }
      }
      int incl = n_mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
      }
      if (lane == 31) warp_sums[warp] = incl;
      __syncthreads();
      if (warp == 0) {
        int w = lane < kSelThreads / 32 ? warp_sums[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int t = __shfl_up_sync(0xffffffffu, w, o);
          if (lane >= o) w += t;
        }
        if (lane < kSelThreads / 32) warp_sums[lane] = w;
      }
      __syncthreads();
      const int off = taken + (warp > 0 ? warp_sums[warp - 1] : 0) + incl - n_mine;
      for (int s = 0; s < n_mine; ++s) {
        if (off + s < need) {
          const int pos = atomicAdd(&sh_count, 1);
          cand[pos] = (static_cast<unsigned long long>(T) << 32) | (0xFFFFFFFFu - mine[s]);
        }
      }
      taken += warp_sums[kSelThreads / 32 - 1];
      __syncthreads();
    }
  }
  __syncthreads();
  int cnt = min(sh_count, kSelCap);
  int* const out = p.sel + static_cast<long long>(h) * R;
  if (cnt <= kRankKeys) {
    // Few keys: the range that they span is cut into equal pieces, the keys are scattered to the places of their pieces (counters and a
    // scan of them), and a key's place among those of its piece is the number of larger ones.  Where weights crowd in one piece,
    // many equal ones or a few far above the others, the keys are sorted instead, below.
    // (us per retrieval with select and sort for all, and now: 16 heads, R = 2048 34.5 -> 22.8, 384 heads 60.3 -> 45.8, with 12.9 thousand queried
    // voxels 119 -> 94, 48 heads, R = 2082 51 -> 39.  About 2800 keys with 190, 400, 600 equal ones per head: 16 heads 16.1, 19.8, 27.1, sorted
    // 26.9; 384 heads 111, 121, 130 and 130.  The sort behind an attempt takes 0.3 to 1.0 us more than without it.  Twice as many comparisons: 384 heads
    // with 800 equal keys of 1200 75 against 56, sorted 53.)
    unsigned long long lo = ~0ull, hi = 0ull;
    for (int i = threadIdx.x; i < cnt; i += kSelThreads) {
      const unsigned long long x = cand[i];
      lo = min(lo, x);
      hi = max(hi, x);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    unsigned long long* const placed = cand + kRankKeys;      // (first the warps' ends: a word more than the buffer costs L1 cache, see above)
    if (lane == 0) {
      placed[warp] = lo;
      placed[32 + warp] = hi;
    }
    int* const piece = reinterpret_cast<int*>(cand + 2 * kRankKeys);
    for (int i = threadIdx.x; i < kRankBins; i += kSelThreads) piece[i] = 0;
    if (threadIdx.x == 0) sh_above = 0;
    __syncthreads();
    lo = placed[lane % (kSelThreads / 32)];
    hi = placed[32 + lane % (kSelThreads / 32)];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    // piece 0 holds the largest keys
    const int drop = cnt > 0 ? max(0, 64 - __clzll(static_cast<long long>(hi - lo)) - 12) : 0;
    static_assert(kRankBins == 1 << 12, "piece of a key");
    auto piece_of = [&](unsigned long long x) { return static_cast<int>((hi - x) >> drop); };
    for (int i = threadIdx.x; i < cnt; i += kSelThreads) atomicAdd(&piece[piece_of(cand[i])], 1);
    __syncthreads();
    constexpr int kPer = kRankBins / kSelThreads;
    int c[kPer], sum = 0, pairs = 0;
#pragma unroll
    for (int e = 0; e < kPer; ++e) {
      c[e] = piece[threadIdx.x * kPer + e];
      sum += c[e];
      pairs += c[e] * c[e];
    }
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) warp_sums[warp] = incl;
    pairs = __reduce_add_sync(0xffffffffu, pairs);
    if (lane == 0) atomicAdd(&sh_above, pairs);      // (the square of kRankKeys at most)
    __syncthreads();
    if (sh_above <= kRankPairs) {
      int run = lane < warp ? warp_sums[lane] : 0;     // (at most 32 warps)
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) run += __shfl_xor_sync(0xffffffffu, run, o);
      run += incl - sum;
#pragma unroll
      for (int e = 0; e < kPer; ++e) {
        piece[threadIdx.x * kPer + e] = run;
        run += c[e];
      }
      __syncthreads();
      for (int i = threadIdx.x; i < cnt; i += kSelThreads) {
        const unsigned long long x = cand[i];
        placed[atomicAdd(&piece[piece_of(x)], 1)] = x;
      }
      __syncthreads();
      // (the counter of a piece has become the place behind its last key, the one before it the place of its first)
      for (int i = threadIdx.x; i < cnt; i += kSelThreads) {
        const unsigned long long x = placed[i];
        const int b = piece_of(x), first = b > 0 ? piece[b - 1] : 0, end = piece[b];
        int rank = first;
        for (int j = first; j < end; ++j) rank += placed[j] > x ? 1 : 0;
        if (rank < R) out[rank] = static_cast<int>(0xFFFFFFFFu - static_cast<unsigned int>(x & 0xFFFFFFFFull));
      }
      for (int i = cnt + threadIdx.x; i < R; i += kSelThreads) out[i] = -1;
      return;
    }
  }
  int limit = kSelThreads;
  while (limit < R) limit <<= 1;
  if (cnt > limit && cnt <= kSelCap - kFineKeys) {
    // the R-th largest key, eight bits at a time (keys are distinct, so this ends with R of them at
    // the latest); R <= limit < cnt, so there is one
    unsigned long long pre = 0;       // leading bits of that key found so far
    int sh = 64, want = R;            // want: its rank among the keys that share them
    for (;;) {
      sh -= 8;
      for (int i = threadIdx.x; i < 256; i += kSelThreads) fine[i] = 0;
      __syncthreads();
      for (int i = threadIdx.x; i < cnt; i += kSelThreads) {
        const unsigned long long x = cand[i];
        if (sh == 56 || (x >> (sh + 8)) == pre) atomicAdd(&fine[static_cast<unsigned>(x >> sh) & 255u], 1);
      }
      __syncthreads();
      if (warp == 0) {
        // lane l counts bins 8 l' .. 8 l' + 7 with l' = 31 - l: lane 0 holds the highest
        int c[8], sum = 0;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          c[e] = fine[(31 - lane) * 8 + 7 - e];
          sum += c[e];
        }
        int incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int t = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += t;
        }
        int above = incl - sum;
        if (above < want && incl >= want) {       // exactly one lane
          bool found = false;
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            if (!found) {
              if (above + c[e] >= want) {
                found = true;
                sh_bin = (31 - lane) * 8 + 7 - e;
                sh_above = above;
                sh_ties = c[e];
              }
              above += found ? 0 : c[e];
            }
          }
        }
      }
      __syncthreads();
      pre = (pre << 8) | static_cast<unsigned>(sh_bin);
      want -= sh_above;
      const int left = (R - want) + sh_ties;      // keys at or above the new prefix
      __syncthreads();
      if (left <= limit || sh == 0) break;
    }
    // keep the keys at or above the prefix, in place: a batch is read before any of it is written,
    // and what is written never lies past the batches that have been read
    if (threadIdx.x == 0) sh_count = 0;
    __syncthreads();
    for (int base = 0; base < cnt; base += kSelThreads) {
      const int i = base + threadIdx.x;
      const unsigned long long x = i < cnt ? cand[i] : 0ull;
      __syncthreads();
      if (i < cnt && (x >> sh) >= pre) cand[list_push(&sh_count)] = x;
    }
    __syncthreads();
    cnt = sh_count;
  }
  int np2 = 1;
  while (np2 < cnt) np2 <<= 1;
  for (int i = cnt + threadIdx.x; i < np2; i += kSelThreads) cand[i] = 0ull;
  __syncthreads();
  if (np2 == kSelThreads) sort_desc<1, kSelThreads>(cand);
  else if (np2 == 2 * kSelThreads) sort_desc<2, kSelThreads>(cand);
  else if (np2 == 4 * kSelThreads) sort_desc<4, kSelThreads>(cand);
  else if (np2 == 8 * kSelThreads) sort_desc<8, kSelThreads>(cand);
  else if (np2 > 1) bitonic_desc(cand, np2);       // (16 keys per thread would not fit three CTAs' registers)
  const int keep = min(cnt, R);
  for (int i = threadIdx.x; i < R; i += kSelThreads) {
    int c = -1;
    if (i < keep) c = static_cast<int>(0xFFFFFFFFu - static_cast<unsigned int>(cand[i] & 0xFFFFFFFFull));
    out[i] = c;
  }
}

__global__ void retrieve_gather_kernel(const RetrieveParams p, int vec_per_token) {
  grid_dep_wait();   // launched with programmatic serialization behind the previous kernel in the stream
  const long long gid = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int h = blockIdx.y;
  const long long tok = gid / vec_per_token;
  const int part = static_cast<int>(gid % vec_per_token);
  if (tok >= p.R) return;
  const long long o = static_cast<long long>(h) * p.R + tok;
  const int c = p.sel[o];
  uint4 kv = make_uint4(0, 0, 0, 0), vv = make_uint4(0, 0, 0, 0);
  int seg = -1, v = -1, slot = -1;
  if (c >= 0) {
    v = p.query_ids[c / p.P];
    slot = c % p.P;
    seg = p.piv_row_seg[(static_cast<long long>(h) * p.voxel_cap + v) * p.P + slot];
    kv = static_cast<const uint4*>(p.piv_K)[static_cast<long long>(seg) * vec_per_token + part];
    vv = static_cast<const uint4*>(p.piv_V)[static_cast<long long>(seg) * vec_per_token + part];
  }
  static_cast<uint4*>(p.out_K)[o * vec_per_token + part] = kv;
  static_cast<uint4*>(p.out_V)[o * vec_per_token + part] = vv;
  if (part == 0) {
    p.out_mask[o] = c >= 0 ? 1 : 0;
    p.out_bias[o] = c >= 0 ? logf(fmaxf(p.piv_C[seg], 1e-9f)) : -INFINITY;
    if (p.out_idx != nullptr) {
      p.out_idx[2 * o] = v;
      p.out_idx[2 * o + 1] = slot;
    }
  }
}

}  // namespace
}  // namespace stac

extern "C" {

int stac_retrieve(const stac_pool* pool, const int* query_ids, const int* query_count, int retrieve_size, int* sel,
                  void* out_K, void* out_V, uint8_t* out_mask, float* out_bias, int* out_idx, stac_stream_t stream) {
  if (pool == nullptr || query_ids == nullptr || query_count == nullptr || sel == nullptr || out_K == nullptr ||
      out_V == nullptr || out_mask == nullptr || out_bias == nullptr)
    return STAC_ERR_BAD_ARG;
  if (retrieve_size <= 0 || retrieve_size > stac::kSelCap || pool->pivot_cap > 4) return STAC_ERR_BAD_ARG;
  const int token_bytes = pool->head_dim * pool->elem_bytes;
  if (token_bytes % 16 != 0) return STAC_ERR_BAD_ARG;
  stac::RetrieveParams rp;
  rp.heads = pool->heads; rp.D = pool->head_dim; rp.P = pool->pivot_cap; rp.voxel_cap = pool->voxel_cap;
  rp.voxel_used = pool->voxel_used; rp.R = retrieve_size;
  rp.query_ids = query_ids; rp.query_count = query_count;
  rp.piv_row_seg = pool->piv_row_seg; rp.piv_row_cnt = pool->piv_row_cnt;
  rp.seg_vec = rp.P == 4 && (reinterpret_cast<uintptr_t>(rp.piv_row_seg) & 15) == 0 ? 1 : 0;
  rp.piv_K = pool->piv_K; rp.piv_V = pool->piv_V; rp.piv_W = pool->piv_W; rp.piv_C = pool->piv_C;
  rp.sel = sel; rp.out_K = out_K; rp.out_V = out_V; rp.out_mask = out_mask; rp.out_bias = out_bias;
  rp.out_idx = out_idx;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  int dev = 0;
  if (stac::current_device(&dev) != STAC_OK) return STAC_ERR_CUDA;
  int n_sm = 0;
  if (stac::device_sm_count(dev, &n_sm) != STAC_OK) return STAC_ERR_CUDA;
  static stac::PerDeviceFlag attr_done;   // the shared-memory opt-in is made once per device
  const int smem = stac::kSelCap * 8;
  if (attr_done.needs_setup(dev)) {
    if (cudaFuncSetAttribute(stac::retrieve_select_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) !=
            cudaSuccess ||
        cudaFuncSetAttribute(stac::retrieve_select_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) !=
            cudaSuccess)
      return STAC_ERR_CUDA;
    attr_done.mark(dev);
  }
  const bool few = pool->heads <= n_sm;
  if (stac::launch_behind(few ? stac::retrieve_select_kernel<true> : stac::retrieve_select_kernel<false>,
                          dim3(pool->heads), dim3(few ? stac::SelShape<true>::kThreads : stac::SelShape<false>::kThreads),
                          smem, st, rp) != cudaSuccess)
    return STAC_ERR_CUDA;
  const int vpt = token_bytes / 16;
  const long long total = static_cast<long long>(retrieve_size) * vpt;
  dim3 grid(static_cast<unsigned>((total + 255) / 256), pool->heads);
  if (stac::launch_behind(stac::retrieve_gather_kernel, grid, dim3(256), 0, st, rp, vpt) != cudaSuccess) return STAC_ERR_CUDA;
  return cudaGetLastError() == cudaSuccess ? STAC_OK : STAC_ERR_CUDA;
}

}  // extern "C"
