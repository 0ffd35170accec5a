// Eviction into the voxel memory: deterministic segmented merge of evicted K/V into the
// per-(head, voxel) pools.
//
// Replaces VoxelKVMerger.insert_and_merge and its helpers on the reference's Python path
// (stac/merger.py:1157-1255 filter + stable sort by row, :765-918 order of operations,
// :586-760 token -> pivot merge, :408-461 full buffer -> one pivot, :462-582 pivot insert /
// victim re-merge) together with the Top-B append and the segment allocator
// (stac/allocator.py:559-723, :2237-2345, :2306-2319), and the merger-cuda pipeline that the
// reference uses on the GPU (merger-cuda/csrc/kernels/merger_kernels.cu).
//
// Every output is a pure function of the inputs: per-(head, voxel) work is done in token order by one
// thread, eight lanes or a warp, and everything that depends on an order across rows (which
// segment id a row gets, where its overflow lands, where freed ids go) is computed from
// exclusive scans over the rows in (head, voxel) order.  No floating-point atomics and no slot pops by
// atomics, so keys, slot maps and merged values repeat bit for bit from run to run.
//
// Kernels, in launch order:
//   sort_tokens_kernel   one CTA per pool head: list the head's valid evicted tokens followed
//                        by its carried overflow tokens, in the order of their voxels (a counter per voxel, a stable LSD radix
//                        sort in shared memory, or one in global memory), emit the unique rows (CSR).
//   tokens_sim_merge_kernel  token-parallel (a thread per token, four lanes per token and pivot of its row, 16-byte
//                        loads): cosine of the token with the pivots of its row, best pivot; then
//                        eight lanes per pivot of a row of up to eight tokens: fold the tokens that reach the merge threshold
//                        into it in token order (exp(sim) weights), publish the new pivot weights.
//   rows_merge_kernel    the same folding for longer rows, which the kernel above queues.
//   rows_rank_kernel     one thread per row: score gate of the row's pivots, selection, ranking of
//                        the buffered tokens + selected tokens by (score desc, arrival order),
//                        counts of new segments / overflow / full; rows with many tokens, which
//                        sort_tokens_kernel has listed, by a warp each (same result).
//   scan_rows_kernel     exclusive scans of those counts inside every head; the CTA that finishes
//                        last scans the heads and makes the allocation plan (k ids from the top of
//                        the free list, the rest fresh) and the capacity checks.  Launched twice:
//                        the second launch does something only if bounded pools were too small,
//                        and then skips the rows that do not fit before it scans again.
//   rows_phase_b1a_kernel one thread per row: hand out segment ids, publish occupancy, queue rows
//                        whose buffered tokens change column / whose buffer filled up.
//   rows_phase_b1m_kernel one warp per queued row: move buffered tokens to their new column
//                        (or to the overflow list), last column first, in place.
//   tokens_place_kernel  token-parallel 16-byte-vector copy of every selected token to its
//                        column's segment or overflow slot.
//   rows_phase_b2_kernel a warp or eight lanes per full row: turn the buffer into a pivot, insert it (folding
//                        the lowest-weight pivot into its nearest neighbour when the row is
//                        saturated), stage the freed segment ids.
//   finalize_kernel      append staged ids to the free list (or carry the overflow list over when the
//                        call had no valid token).
// (Eleven launches and one memset; with the long rows, the plan, the skipping and the carried list in launches
// of their own they were sixteen and two: bounded memory of 384 heads 1381 -> 1282 us per insert and
// retrieval.)
#include <cuda_bf16.h>

#include "common.cuh"
#include "stac_internal.h"

namespace stac {
namespace {

constexpr int kMaxB = 8;
constexpr int kMaxP = 4;
constexpr int kLongRow = 32;   // rows with more tokens are ranked by a warp each
constexpr unsigned kFull = 0xffffffffu;

// ------------------------------------------------------------------------------------ helpers
template <typename T> struct Elem;
template <> struct Elem<float> {
  static __device__ __forceinline__ float load(const float* p) { return *p; }
  static __device__ __forceinline__ void store(float* p, float v) { *p = v; }
  static __device__ __forceinline__ float round(float v) { return v; }
  static constexpr bool kIsBf16 = false;
};
template <> struct Elem<__nv_bfloat16> {
  static __device__ __forceinline__ float load(const __nv_bfloat16* p) { return __bfloat162float(*p); }
  static __device__ __forceinline__ void store(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }
  static __device__ __forceinline__ float round(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
  static constexpr bool kIsBf16 = true;
};

// One slot of a global work list per calling lane: the lanes of a warp that push at the same time
// take consecutive slots with ONE atomic (the order of a list never reaches an output).
__device__ __forceinline__ int list_push(int* counter) {
  const unsigned m = __activemask();
  const unsigned lane = threadIdx.x & 31;
  const int leader = __ffs(m) - 1;
  int base = 0;
  if (static_cast<int>(lane) == leader) base = atomicAdd(counter, __popc(m));
  base = __shfl_sync(m, base, leader);
  return base + __popc(m & ((1u << lane) - 1u));
}

struct MergeParams {
  // geometry
  int heads, D, P, B, voxel_cap, voxel_used;
  float sim_thresh, replace_thresh, score_thresh;
  // evicted tokens: token j of head h lives at position pos = idx ? idx[h*n_new + j] : j
  const void* k_src;
  const void* v_src;
  const float* s_src;
  const int* vx_src;
  const int* idx;
  long long src_head_stride;   // elements between heads in k_src / v_src
  long long src_row_stride;    // elements between positions
  long long meta_head_stride;  // elements between heads in s_src / vx_src
  int n_new;                   // tokens per head
  // pools
  void* buf_K; void* buf_V; float* buf_S;
  int* buf_row_seg; int* buf_row_cnt; int* buf_free; int buf_cap;
  void* piv_K; void* piv_V; float* piv_W; float* piv_S; float* piv_C;
  int* piv_row_seg; int* piv_row_cnt; int piv_cap;
  // overflow lists
  const void* over_K_in; const void* over_V_in; const float* over_S_in; const int* over_hv_in;
  const int* over_start_in;  // [heads + 1]
  void* over_K_out; void* over_V_out; float* over_S_out; int* over_hv_out;
  int* over_start_out;
  int over_cap;
  int* meta;  // device ints, see STAC_META_*
  const int* voxel_count;  // device scalar or nullptr
  // scratch
  int ncap;            // per-head capacity of the token lists
  unsigned int* keys_a; unsigned int* keys_b;  // [heads][ncap]
  int* vals_a; int* vals_b;                    // [heads][ncap]
  int* n_tok;          // [heads]
  int* n_rows;         // [heads]
  int* row_vx;         // [heads][ncap]
  int* row_start;      // [heads][ncap + 1]
  int4* row_info;      // [heads][ncap]: add_cnt, over_cnt, flags, n_sel
  int4* row_pref;      // [heads][ncap]: exclusive prefixes inside the head
  int* old_dest;       // [heads][ncap][8] new rank of each buffered token (>= B: goes to the overflow list)
  int* tok_dest;       // [heads][ncap]
  float* tok_sim;      // [heads][ncap]
  float* tok_score;    // [heads][ncap]
  int4* head_tot;      // [heads]
  int4* head_base;     // [heads]
  int* plan;           // device ints, see kPlan*
  int* free_stage;     // [buf_cap]
  int2* full_list;     // [heads*ncap] rows whose buffer filled up in this call
  int2* long_list;     // rows with more than kLongRow tokens: the memory of full_list, which is filled later
  int2* move_list;     // [heads*ncap] rows in which buffered tokens change column
  int* tok_row;        // [heads][ncap] row index of each sorted token
  int* tok_best;       // [heads][ncap] index of the most similar pivot of the token's row (rows of more than kShortRow tokens)
  int* row_flag;       // [heads][ncap] cleared with the row list: set once the row is in merge_list
  int2* merge_list;    // [heads*ncap] rows (head, row index) of more than kShortRow tokens with at least one merging token
  int passes;          // radix passes (8 bits each)
  int counted;         // 1: a counter per voxel id of the call fits the shared memory of the sort, and pays
  float minus_zero;    // -0, unknown to the compiler
  int seg_vec;         // 1: the pivot segments of a row are one aligned 16-byte vector
  int buf_seg_vec;     // 1: the buffer segments of a row are two of them
  int* err;
};

enum { kPlanK = 0, kPlanFreeLen, kPlanBufTop, kPlanPivTop, kPlanTotalAdd, kPlanTotalFull, kPlanTotalOver,
       kPlanAnyValid, kPlanAbort, kPlanFullCount, kPlanMoveCount, kPlanShort, kPlanAvailBuf, kPlanAvailPiv,
       kPlanMergeCount, kPlanTicket, kPlanTicket2, kPlanLongCount, kPlanSize = 32 };

// Block-wide exclusive scan over kWarps warps.
template <int kWarps = 32>
__device__ __forceinline__ int block_scan(int v, int* warp_sums, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) warp_sums[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    int w = lane < kWarps ? warp_sums[lane] : 0;
#pragma unroll
    for (int o = 1; o < kWarps; o <<= 1) {
      const int t = __shfl_up_sync(kFull, w, o);
      if (lane >= o) w += t;
    }
    if (lane < kWarps) warp_sums[lane] = w;
  }
  __syncthreads();
  const int excl = (warp > 0 ? warp_sums[warp - 1] : 0) + incl - v;
  if (threadIdx.x == 0) *total = warp_sums[kWarps - 1];
  __syncthreads();
  return excl;
}

__device__ __forceinline__ int4 add4(int4 a, int4 b) { return make_int4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
__device__ __forceinline__ int4 shfl_up4(int4 v, int o) {
  return make_int4(__shfl_up_sync(kFull, v.x, o), __shfl_up_sync(kFull, v.y, o), __shfl_up_sync(kFull, v.z, o),
                   __shfl_up_sync(kFull, v.w, o));
}
// Block-wide exclusive scan of four values at once, kWarps warps; every thread gets the total.
template <int kWarps>
__device__ __forceinline__ int4 block_scan4(int4 v, int4* warp_sums, int4* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int4 incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int4 t = shfl_up4(incl, o);
    if (lane >= o) incl = add4(incl, t);
  }
  if (lane == 31) warp_sums[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    int4 w = lane < kWarps ? warp_sums[lane] : make_int4(0, 0, 0, 0);
#pragma unroll
    for (int o = 1; o < kWarps; o <<= 1) {
      const int4 t = shfl_up4(w, o);
      if (lane >= o) w = add4(w, t);
    }
    if (lane < kWarps) warp_sums[lane] = w;
  }
  __syncthreads();
  const int4 before = warp > 0 ? warp_sums[warp - 1] : make_int4(0, 0, 0, 0);
  *total = warp_sums[kWarps - 1];
  __syncthreads();
  return make_int4(before.x + incl.x - v.x, before.y + incl.y - v.y, before.z + incl.z - v.z, before.w + incl.w - v.w);
}

// ------------------------------------------------------------------------------------ sort
// A CTA per head: a chain of latencies and barriers, so that a second wave of CTAs costs as much as the first.  The
// number of heads decides how many have to share an SM (see launch_merge).
// (Digits are counted with shared-memory adds; matching the lanes of a warp first cost more than the adds' conflicts.)
// Lanes of the warp that are `in` and have this lane's digit, by eight ballots.  (__match_any_sync takes longer the more digits
// there are: 16 heads of 8328 tokens, the first scatter 16.3 thousand cycles with it, 9.2 with ballots.)
__device__ __forceinline__ unsigned same_digit(bool in, unsigned digit) {
  unsigned peers = __ballot_sync(kFull, in);
#pragma unroll
  for (int bit = 0; bit < 8; ++bit) {
    const bool set = (digit >> bit) & 1u;
    const unsigned m = __ballot_sync(kFull, set);
    peers &= set ? m : ~m;
  }
  return peers;
}

// Lists of up to kThreads * kItems tokens and voxel ids of 16 bits are sorted in shared memory (sort_tokens_shared), others
// through the lists in global memory (the rest of this kernel).
__device__ __forceinline__ int warp_scan_sum(int v, int lane) {      // inclusive
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(kFull, v, o);
    if (lane >= o) v += t;
  }
  return v;
}

// One word per token, voxel id above its place in the list (evicted tokens by position, then carried ones), in one array: a
// warp takes its part of it into registers before a pass scatters.  Tokens that are not valid take the id 0xFFFF and end
// up behind the others, so nothing is compacted first; rows are found in one sweep.
// (8328 tokens each: 16 heads 34.5 -> 21.4 us, 384 heads 105.5 -> 70.3; 4164 each, 384 heads 54.5 -> 44.5; 1041 each, 384 heads
// 19.4 -> 14.1.  The lists in global memory cost a scattered 4-byte write per key, value and pass, and a round trip
// to L2 around every block scan, one per 4 kThreads tokens.)
// False, with nothing written, if a carried token's id does not fit: carried tokens may lie above this call's voxel count.
// `known`: the items' voxel ids in shared memory (0xFFFF: none), which is written over, or nullptr.
template <int kThreads, int kItems>
__device__ __forceinline__ bool sort_tokens_shared(const MergeParams& p, int h, int os, int n_items, unsigned* buf, int* hist,
                                                   const unsigned short* known) {
  constexpr int kWarps = kThreads / 32, kHistRow = 257;
  constexpr unsigned kNone = 0xFFFFu;
  __shared__ int counts[kWarps];
  __shared__ int scan_sums[32];
  __shared__ int scan_total, n_new_valid, n_valid;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int chunk = ((n_items + kWarps - 1) / kWarps + 31) / 32 * 32;    // items per warp, at most 32 kItems
  const int c0 = warp * chunk, c1 = min(n_items, c0 + chunk);
  if (threadIdx.x == 0) n_new_valid = n_valid = 0;
  const int n_it = (max(c1 - c0, 0) + 31) / 32;        // rounds of 32 items in which this warp has any
  unsigned item[kItems];
  if (known != nullptr) {
#pragma unroll
    for (int t = 0; t < kItems; ++t)
      if (t < n_it) item[t] = c0 + t * 32 + lane < c1 ? known[c0 + t * 32 + lane] : kNone;
    __syncthreads();
  } else {
#pragma unroll
    for (int t = 0; t < kItems; ++t) {       // positions first, so that all loads of a thread are in flight together
      const int i = c0 + t * 32 + lane;
      item[t] = i;
      if (t < n_it && p.idx != nullptr && i < c1 && i < p.n_new) item[t] = p.idx[static_cast<long long>(h) * p.n_new + i];
    }
#pragma unroll
    for (int t = 0; t < kItems; ++t) {
      if (t < n_it) {
        const int i = c0 + t * 32 + lane;
        int vx = -1;
        if (i < c1) {
          vx = i < p.n_new ? p.vx_src[h * p.meta_head_stride + static_cast<int>(item[t])]
                           : p.over_hv_in[2 * (os + i - p.n_new) + 1];
        }
        item[t] = vx;
      }
    }
  }
  int* my_hist = hist + warp * kHistRow;
  auto clear_hist = [&] {
    for (int i = lane; i < 256; i += 32) my_hist[i] = 0;
    __syncwarp();
  };
  auto count = [&](unsigned w, int shift) { atomicAdd(&my_hist[(w >> shift) & 255u], 1); };
  clear_hist();
  __syncthreads();
  int new_valid = 0, valid = 0;
#pragma unroll
  for (int t = 0; t < kItems; ++t) {
    if (t < n_it) {
      const int i = c0 + t * 32 + lane;
      // (carried tokens are valid whatever the voxel count of this call is)
      const bool ok = item[t] < (i < p.n_new ? static_cast<unsigned>(p.voxel_used) : kNone);
      new_valid += __popc(__ballot_sync(kFull, ok && i < p.n_new));
      valid += __popc(__ballot_sync(kFull, ok));
      item[t] = (ok ? item[t] << 16 : kNone << 16) | static_cast<unsigned>(i);
      if (i < c1) {
        buf[i] = item[t];
        count(item[t], 16);
      }
    }
  }
  if (lane == 0) {
    atomicAdd(&n_new_valid, new_valid);
    atomicAdd(&n_valid, valid);
  }
#pragma unroll 1
  for (int shift = 16; shift < 32; shift += 8) {
    if (shift > 16) {
      clear_hist();
      for (int t = 0; t < n_it; ++t)
        if (c0 + t * 32 + lane < c1) count(buf[c0 + t * 32 + lane], shift);
    }
    __syncthreads();
    if (shift == 16 && n_valid - n_new_valid != n_items - p.n_new) return false;      // a carried token's id is too wide
    // exclusive scan of the counters in (digit, warp) order: 8 consecutive entries per thread
    int loc[8];
    int sum = 0;
    constexpr int kParts = kWarps / 8;      // threads per digit
    int* of_thread = hist + (threadIdx.x % kParts) * 8 * kHistRow + threadIdx.x / kParts;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      loc[e] = of_thread[e * kHistRow];
      sum += loc[e];
    }
    int run = block_scan<kWarps>(sum, scan_sums, &scan_total);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      of_thread[e * kHistRow] = run;
      run += loc[e];
    }
#pragma unroll
    for (int t = 0; t < kItems; ++t)
      if (t < n_it && c0 + t * 32 + lane < c1) item[t] = buf[c0 + t * 32 + lane];
    __syncthreads();
#pragma unroll
    for (int t = 0; t < kItems; ++t) {
      if (t < n_it) {                       // warp-uniform
        const bool in = c0 + t * 32 + lane < c1;
        const unsigned d = (item[t] >> shift) & 255u;
        const unsigned peers = same_digit(in, d);
        const unsigned before = peers & ((1u << lane) - 1);
        if (in) buf[my_hist[d] + __popc(before)] = item[t];
        __syncwarp();
        if (in && before == 0) my_hist[d] += __popc(peers);
        __syncwarp();
      }
    }
    __syncthreads();
  }
  // rows of the sorted list: a bit per item that starts one, then everything that is known about the items
  const int n = n_valid, c1_valid = min(c1, n);
  unsigned starts = 0;
  int n_starts = 0;
  for (int t = 0; t < n_it; ++t) {
    const int i = c0 + t * 32 + lane;
    const bool start = i < c1_valid && (i == 0 || buf[i - 1] >> 16 != buf[i] >> 16);
    starts |= (start ? 1u : 0u) << t;
    n_starts += __popc(__ballot_sync(kFull, start));
  }
  if (lane == 0) counts[warp] = n_starts;
  __syncthreads();
  const int incl = warp_scan_sum(lane < kWarps ? counts[lane] : 0, lane);
  int r0 = warp > 0 ? __shfl_sync(kFull, incl, warp - 1) : 0;      // rows that start before this warp's items
  const int n_rows = __shfl_sync(kFull, incl, kWarps - 1);
  const long long hb = static_cast<long long>(h) * p.ncap;
  unsigned int* keys = ((p.passes & 1) ? p.keys_b : p.keys_a) + hb;
  int* codes = ((p.passes & 1) ? p.vals_b : p.vals_a) + hb;
  int* rst = p.row_start + static_cast<long long>(h) * (p.ncap + 1);
  for (int t = 0; t < n_it; ++t) {
    const int i = c0 + t * 32 + lane;
    const unsigned m = __ballot_sync(kFull, (starts >> t) & 1u);
    if (i < c1_valid) {
      const int r = r0 + __popc(m & (0xffffffffu >> (31 - lane))) - 1;
      const unsigned key = buf[i] >> 16;
      const int at = static_cast<int>(buf[i] & 0xFFFFu);
      keys[i] = key;
      codes[i] = at < p.n_new ? at : ~(os + at - p.n_new);
      p.tok_row[hb + i] = r;
      if ((starts >> t) & 1u) {
        p.row_vx[hb + r] = static_cast<int>(key);
        rst[r] = i;
        p.row_flag[hb + r] = 0;
      }
      // the token behind kLongRow others of its row lists it
      if (i >= kLongRow && buf[i - kLongRow] >> 16 == key && (i == kLongRow || buf[i - kLongRow - 1] >> 16 != key))
        p.long_list[list_push(&p.plan[kPlanLongCount])] = make_int2(h, r);
    }
    r0 += __popc(m);
  }
  if (threadIdx.x == 0) {
    rst[n_rows] = n;
    p.n_rows[h] = n_rows;
    p.n_tok[h] = n;
    if (n_new_valid > 0) atomicOr(&p.plan[kPlanAnyValid], 1);
  }
  return true;
}

// Comparisons that the rows of more than kLongCounted tokens take, of all threads (`comparisons`: zero before).  A function of its own: in line, its code
// made calls without such rows up to 2 us longer.
constexpr int kLongCounted = 64;
__device__ __noinline__ int comparisons_of_long_rows(const unsigned* cnt, int w0, int w1, int* comparisons) {
  int squares = 0;                        // (9216 squared at most)
  for (int w = w0; w < w1; ++w) {
    const int lo = static_cast<int>(cnt[w] & 0xffffu), hi = static_cast<int>(cnt[w] >> 16);
    squares += (lo > kLongCounted ? lo * lo : 0) + (hi > kLongCounted ? hi * hi : 0);
  }
  if (squares > 0) atomicAdd(comparisons, squares);
  __syncthreads();
  return *comparisons;
}
// A counter per voxel id of the call instead of digits: tokens are scattered to the places of their voxel in any order, and a token's
// place in its row is the number of the row's tokens before it.  Two 16-bit counters per word.
// (The digits of sort_tokens_shared against counters: 16 heads of 8328 tokens, 4000 voxels 21.4 -> 12.8 us, 384 heads 64.5 -> 30.9, 384 heads of
// 4164 44.1 -> 20.9, 100 heads of 1200 9.5 -> 7.4.)
// That takes the square of a row's tokens in comparisons: with too many in rows of more than kLongCounted tokens the list is sorted by digits, from the
// voxel ids that are in shared memory already.  (One voxel of 65, 300 and 1000 tokens among 4000: 16 heads of 8328 tokens 13.5, 18.3, 24.9 us, by digits
// alone 21.1; 384 heads 31.0, 38, 67 and 68; 384 heads of 1041 tokens 13.7, 17.2, 17.4 and 14.4.  Sent back for any row above 64, and loaded
// again, it was 25.1, 72 and 18 for all of them.)
// kWide, kCrowded: nothing is written; a carried token's id has no counter, or those rows are too long (`vox`: the voxel ids).
enum { kCounted, kWide, kCrowded };
template <int kThreads, int kItems>
__device__ __forceinline__ int sort_tokens_counted(const MergeParams& p, int h, int os, int n_items, unsigned* smem,
                                                   const unsigned short** ids) {
  constexpr int kWarps = kThreads / 32, kComparisons = 16;      // (of tokens of long rows, per token of the list)
  __shared__ int scan_sums[32];
  __shared__ int scan_total, n_new_valid, n_valid, comparisons;
  const int V = p.voxel_used, words = (V + 1) / 2;
  unsigned* cnt = smem;                                                       // [words]
  unsigned short* row_of = reinterpret_cast<unsigned short*>(smem + words);   // [V]: rows before a voxel's
  unsigned short* vox = reinterpret_cast<unsigned short*>(smem + 2 * words);  // [n_items]: a token's voxel id, kNone: it has none
  unsigned short* buf = vox + kThreads * kItems;                              // [n_items]: tokens in the order of their voxels
  *ids = vox;
  constexpr unsigned short kNone = 0xFFFFu;
  const int tid = threadIdx.x, lane = tid & 31;
  for (int w = tid; w < words; w += kThreads) cnt[w] = 0u;
  if (tid == 0) n_new_valid = n_valid = comparisons = 0;
  int item[kItems];                  // voxel id, -1: none
#pragma unroll
  for (int t = 0; t < kItems; ++t) {       // positions first, so that all loads of a thread are in flight together
    const int i = t * kThreads + tid;
    item[t] = i;
    if (p.idx != nullptr && i < p.n_new) item[t] = p.idx[static_cast<long long>(h) * p.n_new + i];
  }
#pragma unroll
  for (int t = 0; t < kItems; ++t) {
    const int i = t * kThreads + tid;
    int vx = -1;
    if (i < n_items)
      vx = i < p.n_new ? p.vx_src[h * p.meta_head_stride + item[t]] : p.over_hv_in[2 * (os + i - p.n_new) + 1];
    item[t] = vx;
  }
  __syncthreads();
  bool wide = false;
  int new_valid = 0, valid = 0;
#pragma unroll
  for (int t = 0; t < kItems; ++t) {
    const int i = t * kThreads + tid;
    const bool ok = static_cast<unsigned>(item[t]) < static_cast<unsigned>(V);
    wide = wide || (!ok && i >= p.n_new && i < n_items);      // (carried tokens are valid whatever the voxel count of this call is)
    if (ok) atomicAdd(&cnt[item[t] >> 1], 1u << ((item[t] & 1) * 16));
    vox[i] = ok ? static_cast<unsigned short>(item[t]) : kNone;
    new_valid += __popc(__ballot_sync(kFull, ok && i < p.n_new));
    valid += __popc(__ballot_sync(kFull, ok));
  }
  if (lane == 0 && valid > 0) {
    atomicAdd(&n_new_valid, new_valid);
    atomicAdd(&n_valid, valid);
  }
  if (__syncthreads_or(wide)) return kWide;
  // exclusive scan over the voxels of (rows << 16 | tokens); an odd number of words per thread: no bank conflicts
  const int per = ((words + kThreads - 1) / kThreads) | 1, w0 = min(words, tid * per), w1 = min(words, w0 + per);
  int sum = 0, most = 0;
  for (int w = w0; w < w1; ++w) {
    const int lo = static_cast<int>(cnt[w] & 0xffffu), hi = static_cast<int>(cnt[w] >> 16);
    sum += lo + hi + ((lo > 0 ? 1 : 0) + (hi > 0 ? 1 : 0)) * 65536;
    most = max(most, max(lo, hi));
  }
  if (__builtin_expect(__syncthreads_or(most > kLongCounted), 0) &&
      comparisons_of_long_rows(cnt, w0, w1, &comparisons) > kComparisons * n_items)
    return kCrowded;
  int run = block_scan<kWarps>(sum, scan_sums, &scan_total);
  for (int w = w0; w < w1; ++w) {
    const int lo = static_cast<int>(cnt[w] & 0xffffu), hi = static_cast<int>(cnt[w] >> 16);
    const int run_hi = run + lo + (lo > 0 ? 65536 : 0);
    cnt[w] = static_cast<unsigned>(run & 0xffff) | static_cast<unsigned>(run_hi & 0xffff) << 16;
    reinterpret_cast<unsigned*>(row_of)[w] = static_cast<unsigned>(run >> 16) | static_cast<unsigned>(run_hi >> 16) << 16;
    run = run_hi + hi + (hi > 0 ? 65536 : 0);
  }
  __syncthreads();
#pragma unroll 4
  for (int i = tid; i < n_items; i += kThreads) {
    const int v = vox[i];
    if (v != kNone) {
      const int shift = (v & 1) * 16;
      buf[(atomicAdd(&cnt[v >> 1], 1u << shift) >> shift) & 0xffffu] = static_cast<unsigned short>(i);
    }
  }
  __syncthreads();
  // a voxel's counter has become the place behind its last token, the one before it the place of its first
  const unsigned short* end_of = reinterpret_cast<const unsigned short*>(cnt);
  const int n = n_valid, n_rows = scan_total >> 16;
  const long long hb = static_cast<long long>(h) * p.ncap;
  int* rst = p.row_start + static_cast<long long>(h) * (p.ncap + 1);
  for (int v = tid; v < V; v += kThreads) {
    const int s = v > 0 ? end_of[v - 1] : 0, e = end_of[v];
    if (e > s) {
      const int r = row_of[v];
      p.row_vx[hb + r] = v;
      rst[r] = s;
      p.row_flag[hb + r] = 0;
      if (e - s > kLongRow) p.long_list[list_push(&p.plan[kPlanLongCount])] = make_int2(h, r);
    }
  }
  unsigned int* keys = ((p.passes & 1) ? p.keys_b : p.keys_a) + hb;
  int* codes = ((p.passes & 1) ? p.vals_b : p.vals_a) + hb;
#pragma unroll 2
  for (int i = tid; i < n; i += kThreads) {
    const int at = buf[i], v = vox[at], s = v > 0 ? end_of[v - 1] : 0, e = end_of[v];
    int place = s;
    for (int j = s; j < e; ++j) place += buf[j] < at ? 1 : 0;
    keys[place] = static_cast<unsigned>(v);
    codes[place] = at < p.n_new ? at : ~(os + at - p.n_new);
    p.tok_row[hb + place] = row_of[v];
  }
  if (tid == 0) {
    rst[n_rows] = n;
    p.n_rows[h] = n_rows;
    p.n_tok[h] = n;
    if (n_new_valid > 0) atomicOr(&p.plan[kPlanAnyValid], 1);
  }
  return kCounted;
}

template <int kThreads, int kMinCtas, int kItems>
__global__ void __launch_bounds__(kThreads, kMinCtas) sort_tokens_kernel(const __grid_constant__ MergeParams p) {
  constexpr int kWarps = kThreads / 32;
  grid_dep_wait();   // launched with programmatic serialization behind the previous kernel of the call
  // Digit counters, [warp][digit]: a warp's lanes count different digits of the same warp, so neighbouring
  // digits lie in neighbouring banks; rows of 257 words let the scan, which walks them digit by
  // digit, read without conflicts too.  ([digit][warp] put all of a warp's counters in one bank.)
  // (384 heads, 8328 tokens each: insert + retrieval 1112 -> 1068 us; 16 heads, fp32: 278 -> 263 us.)
  constexpr int kHistRow = 257;
  extern __shared__ int sort_smem[];
  int* hist = sort_smem;               // [kHistRow * kWarps]
  __shared__ int warp_sums[32];
  __shared__ int sh_total;
  __shared__ int sh_carry;
  __shared__ int n_passes;
  const int h = blockIdx.x;
  if constexpr (kItems > 0) {
    const int os = p.over_start_in[h], n_items = p.n_new + p.over_start_in[h + 1] - os;
    const unsigned short* known = nullptr;
    if (p.counted && n_items <= min(p.ncap, kThreads * kItems)) {
      const int how = sort_tokens_counted<kThreads, kItems>(p, h, os, n_items, reinterpret_cast<unsigned*>(sort_smem), &known);
      if (__builtin_expect(how == kCounted, 1)) return;
      if (how == kWide) known = nullptr;
      __syncthreads();
    }
    if (n_items <= min(p.ncap, kThreads * kItems) && p.voxel_used <= 0xFFFF &&
        sort_tokens_shared<kThreads, kItems>(p, h, os, n_items, reinterpret_cast<unsigned*>(sort_smem + kHistRow * kWarps), hist, known))
      return;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned int* ka = p.keys_a + static_cast<long long>(h) * p.ncap;
  unsigned int* kb = p.keys_b + static_cast<long long>(h) * p.ncap;
  int* va = p.vals_a + static_cast<long long>(h) * p.ncap;
  int* vb = p.vals_b + static_cast<long long>(h) * p.ncap;

  // 1. valid evicted tokens in position order
  if (threadIdx.x == 0) sh_carry = 0;
  __syncthreads();
  // four consecutive positions per thread: one block scan per 4 kThreads tokens, loads issued together
  for (int base = 0; base < p.n_new; base += 4 * kThreads) {
    const int j0 = base + threadIdx.x * 4;
    int vxs[4];
    int sum = 0;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int j = j0 + t;
      int vx = -1;
      if (j < p.n_new) {
        const int pos = p.idx ? p.idx[static_cast<long long>(h) * p.n_new + j] : j;
        vx = p.vx_src[h * p.meta_head_stride + pos];
      }
      vxs[t] = (vx >= 0 && vx < p.voxel_used) ? vx : -1;
      sum += vxs[t] >= 0 ? 1 : 0;
    }
    int off = sh_carry + block_scan<kWarps>(sum, warp_sums, &sh_total);
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      if (vxs[t] >= 0) {
        ka[off] = static_cast<unsigned int>(vxs[t]);
        va[off] = j0 + t;
        ++off;
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) sh_carry += sh_total;
    __syncthreads();
  }
  const int n_valid = sh_carry;
  if (n_valid > 0 && threadIdx.x == 0) atomicOr(&p.plan[kPlanAnyValid], 1);
  // 2. carried overflow tokens of this head, in list order
  const int os = p.over_start_in[h], oe = p.over_start_in[h + 1];
  int n = n_valid + (oe - os);
  if (n > p.ncap) {
    if (threadIdx.x == 0) report_error(p.err, DEV_SORT_CAPACITY);
    n = p.ncap;
  }
  unsigned int top = 0u;
  for (int o = os + threadIdx.x; o < oe; o += kThreads) {
    const int dst = n_valid + (o - os);
    if (dst < n) {
      const unsigned int id = static_cast<unsigned int>(p.over_hv_in[2 * o + 1]);
      ka[dst] = id;
      va[dst] = ~o;
      top = max(top, id);
    }
  }
  // Carried tokens may lie above this call's voxel count: all digits then, one more pass where that keeps their number odd (the
  // kernels behind take the list from where p.passes leaves it).
  const bool wide = __syncthreads_or(p.passes < 4 && (top >> (8 * p.passes)) != 0u);
  if (threadIdx.x == 0) n_passes = wide ? 4 + (p.passes & 1) : p.passes;
  __syncthreads();
  // 3. stable LSD radix sort by voxel id.  Each warp owns a contiguous chunk of the list so
  //    that (warp, position in chunk) preserves the input order.
  const int chunk = ((n + kWarps - 1) / kWarps + 31) / 32 * 32;  // items per warp, multiple of 32
  const int c0 = warp * chunk;
  const int c1 = min(n, c0 + chunk);
  unsigned int* kin = ka; int* vin = va; unsigned int* kout = kb; int* vout = vb;
  // The first kRegIt * 32 items of a warp's chunk (all of it in lists of up to 8 kThreads tokens) are read into
  // registers once per pass: one round trip to L2 instead of one per 32 items in each of the two
  // loops.
  constexpr int kRegIt = 8;
  int* my_hist = hist + warp * kHistRow;
  for (int pass = 0; pass < n_passes; ++pass) {
    const int shift = min(pass, 3) * 8;      // (a fifth pass moves the sorted list)
    for (int i = threadIdx.x; i < kHistRow * kWarps; i += kThreads) hist[i] = 0;
    unsigned int kreg[kRegIt];
    int vreg[kRegIt];
#pragma unroll
    for (int t = 0; t < kRegIt; ++t) {
      const int i = c0 + t * 32 + lane;
      kreg[t] = i < c1 ? kin[i] : 0u;
      vreg[t] = i < c1 ? vin[i] : 0;
    }
    __syncthreads();
    auto count = [&](bool in, unsigned int key) {
      if (in) atomicAdd(&my_hist[(key >> shift) & 255u], 1);
    };
#pragma unroll
    for (int t = 0; t < kRegIt; ++t) {
      const int base = c0 + t * 32;
      if (base < c1) count(base + lane < c1, kreg[t]);       // warp-uniform
    }
    for (int base = c0 + kRegIt * 32; base < c1; base += 32) count(base + lane < c1, base + lane < c1 ? kin[base + lane] : 0u);
    __syncthreads();
    // exclusive scan of the counters in (digit, warp) order: 8 consecutive entries per thread
    int loc[8];
    int sum = 0;
    constexpr int kParts = kWarps / 8;      // threads per digit
    int* of_thread = hist + (threadIdx.x % kParts) * 8 * kHistRow + threadIdx.x / kParts;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      loc[e] = of_thread[e * kHistRow];
      sum += loc[e];
    }
    int run = block_scan<kWarps>(sum, warp_sums, &sh_total);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      of_thread[e * kHistRow] = run;
      run += loc[e];
    }
    __syncthreads();
    auto scatter = [&](bool in, unsigned int key, int val) {
      const unsigned int d = in ? ((key >> shift) & 255u) : (256u + lane);
      const unsigned int peers = __match_any_sync(kFull, d);
      const unsigned int before = peers & ((1u << lane) - 1);
      if (in) {
        const int dst = my_hist[d] + __popc(before);
        kout[dst] = key;
        vout[dst] = val;
      }
      __syncwarp();
      if (in && before == 0) my_hist[d] += __popc(peers);
      __syncwarp();
    };
#pragma unroll
    for (int t = 0; t < kRegIt; ++t) {
      const int base = c0 + t * 32;
      if (base < c1) scatter(base + lane < c1, kreg[t], vreg[t]);
    }
    for (int base = c0 + kRegIt * 32; base < c1; base += 32) {
      const int i = base + lane;
      scatter(i < c1, i < c1 ? kin[i] : 0u, i < c1 ? vin[i] : 0);
    }
    __syncthreads();
    unsigned int* tk = kin; kin = kout; kout = tk;
    int* tv = vin; vin = vout; vout = tv;
  }
  // 4. unique rows of the sorted list (kin / vin now hold the result)
  if (threadIdx.x == 0) sh_carry = 0;
  __syncthreads();
  int* rvx = p.row_vx + static_cast<long long>(h) * p.ncap;
  int* rst = p.row_start + static_cast<long long>(h) * (p.ncap + 1);
  for (int base = 0; base < n; base += 4 * kThreads) {
    const int i0 = base + threadIdx.x * 4;
    unsigned int key[4];
    int hf[4];
    int sum = 0;
    const unsigned int prev = (i0 > 0 && i0 - 1 < n) ? kin[i0 - 1] : 0u;
    const unsigned int back = i0 >= kLongRow - 3 && i0 < n ? kin[i0 - (kLongRow - 3)] : ~0u;   // (no voxel has this id)
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int i = i0 + t;
      key[t] = i < n ? kin[i] : 0u;
      hf[t] = 0;
      if (i < n) hf[t] = (i == 0 || key[t] != (t == 0 ? prev : key[t - 1])) ? 1 : 0;
      sum += hf[t];
    }
    int r = sh_carry + block_scan<kWarps>(sum, warp_sums, &sh_total);    // rows that begin before this thread's tokens
    if (back == key[0]) {      // the first token's row reaches far back: the token behind kLongRow others lists it
      for (int t = 0; t < 4; ++t) {
        const int s0 = i0 + t - kLongRow;
        if (s0 >= 0 && s0 + kLongRow < n && kin[s0 + kLongRow] == key[0] && kin[s0] == key[0] &&
            (s0 == 0 || kin[s0 - 1] != key[0]))
          p.long_list[list_push(&p.plan[kPlanLongCount])] = make_int2(h, r - 1);
      }
    }
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int i = i0 + t;
      if (i < n) {
        if (hf[t]) {
          rvx[r] = static_cast<int>(key[t]);
          rst[r] = i;
          p.row_flag[static_cast<long long>(h) * p.ncap + r] = 0;
        }
        p.tok_row[static_cast<long long>(h) * p.ncap + i] = r + hf[t] - 1;
        r += hf[t];
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) sh_carry += sh_total;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    rst[sh_carry] = n;
    p.n_rows[h] = sh_carry;
    p.n_tok[h] = n;
  }
}

// ------------------------------------------------------------------------------------ phase A
// Eight consecutive lanes work on one token: each holds eight of its 64 values (16 bytes of a
// bf16 row, 32 of an fp32 row).  Raw8: those values as they were loaded, in flight while others are worked on.
template <typename T> struct Raw8;
template <> struct Raw8<__nv_bfloat16> {
  uint4 u;
  __device__ __forceinline__ void load(const __nv_bfloat16* row, int sub) { u = reinterpret_cast<const uint4*>(row)[sub]; }
  __device__ __forceinline__ void values(float (&x)[8]) const {
    x[0] = __uint_as_float(u.x << 16); x[1] = __uint_as_float(u.x & 0xffff0000u);
    x[2] = __uint_as_float(u.y << 16); x[3] = __uint_as_float(u.y & 0xffff0000u);
    x[4] = __uint_as_float(u.z << 16); x[5] = __uint_as_float(u.z & 0xffff0000u);
    x[6] = __uint_as_float(u.w << 16); x[7] = __uint_as_float(u.w & 0xffff0000u);
  }
};
template <> struct Raw8<float> {
  float4 a, b;
  __device__ __forceinline__ void load(const float* row, int sub) {
    a = reinterpret_cast<const float4*>(row)[2 * sub];
    b = reinterpret_cast<const float4*>(row)[2 * sub + 1];
  }
  __device__ __forceinline__ void values(float (&x)[8]) const {
    x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
  }
};
template <typename T>
__device__ __forceinline__ void row8_load(const T* row, int sub, float (&x)[8]) {
  Raw8<T> r;
  r.load(row, sub);
  r.values(x);
}
__device__ __forceinline__ void row8_store(__nv_bfloat16* row, int sub, const float (&x)[8]) {
  uint4 u;
  u.x = pack_bf16x2(x[0], x[1]); u.y = pack_bf16x2(x[2], x[3]);
  u.z = pack_bf16x2(x[4], x[5]); u.w = pack_bf16x2(x[6], x[7]);
  reinterpret_cast<uint4*>(row)[sub] = u;
}
__device__ __forceinline__ void row8_store(float* row, int sub, const float (&x)[8]) {
  reinterpret_cast<float4*>(row)[2 * sub] = make_float4(x[0], x[1], x[2], x[3]);
  reinterpret_cast<float4*>(row)[2 * sub + 1] = make_float4(x[4], x[5], x[6], x[7]);
}

// sum over the eight lanes of a group (every lane gets it; same order in every group)
__device__ __forceinline__ float group8_sum(float v, unsigned gmask) {
  v += __shfl_xor_sync(gmask, v, 4);
  v += __shfl_xor_sync(gmask, v, 2);
  v += __shfl_xor_sync(gmask, v, 1);
  return v;
}

// Source position of an evicted token (code >= 0) in its head's cache.
__device__ __forceinline__ int token_pos(const MergeParams& p, int h, int code) {
  return p.idx ? p.idx[static_cast<long long>(h) * p.n_new + code] : code;
}
// K or V row of a token whose position (evicted) or list index (carried overflow) is known.
template <typename T>
__device__ __forceinline__ const T* token_row_at(const MergeParams& p, int h, int code, int pos, bool want_v) {
  if (code >= 0) return static_cast<const T*>(want_v ? p.v_src : p.k_src) + h * p.src_head_stride + pos * p.src_row_stride;
  return static_cast<const T*>(want_v ? p.over_V_in : p.over_K_in) + static_cast<long long>(~code) * p.D;
}

// What the tokens of a row that merge into one pivot add up to, in token order, held by eight lanes.
struct MergeSums {
  float K[8], V[8], A, S, C;
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int e = 0; e < 8; ++e) K[e] = V[e] = 0.f;
    A = S = C = 0.f;
  }
  __device__ __forceinline__ void add(float a, float s, const float (&k)[8], const float (&v)[8]) {
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      K[e] = __fadd_rn(K[e], __fmul_rn(a, k[e]));
      V[e] = __fadd_rn(V[e], __fmul_rn(a, v[e]));
    }
    A = __fadd_rn(A, a);
    S = __fadd_rn(S, s);
    C = __fadd_rn(C, 1.f);
  }
};
// K <- (W K + sum a k) / (W + sum a), same for V, W += sum a, S += sum of the scores, C += count; stored in
// the pool dtype (stac/merger.py:660-760).
template <typename T>
__device__ __forceinline__ void merge_into_pivot(const MergeParams& p, int seg, float W, const MergeSums& m, int sub) {
  T* kb = static_cast<T*>(p.piv_K) + static_cast<long long>(seg) * p.D;
  T* vb = static_cast<T*>(p.piv_V) + static_cast<long long>(seg) * p.D;
  const float denom = fmaxf(__fadd_rn(W, m.A), 1e-8f);
  const float fo = __fdiv_rn(W, denom), fn = __fdiv_rn(1.0f, denom);
  Raw8<T> k_old, v_old;
  k_old.load(kb, sub);
  v_old.load(vb, sub);
  const float S = sub == 0 ? p.piv_S[seg] : 0.f, C = sub == 0 ? p.piv_C[seg] : 0.f;
  float o[8];
  k_old.values(o);
#pragma unroll
  for (int e = 0; e < 8; ++e) o[e] = __fadd_rn(__fmul_rn(fo, o[e]), __fmul_rn(fn, m.K[e]));
  row8_store(kb, sub, o);
  v_old.values(o);
#pragma unroll
  for (int e = 0; e < 8; ++e) o[e] = __fadd_rn(__fmul_rn(fo, o[e]), __fmul_rn(fn, m.V[e]));
  row8_store(vb, sub, o);
  if (sub == 0) {
    p.piv_W[seg] = denom;
    p.piv_S[seg] = __fadd_rn(S, m.S);
    p.piv_C[seg] = __fadd_rn(C, m.C);
  }
}

// Tokens against the pivots of their row (stac/merger.py:586-660): cosine with every pivot key
// (both L2-normalised, norms clamped at 1e-6), clamped to [-1, 1]; the first largest wins.  All
// similarities are taken against the pivots as they are BEFORE this call's merges, as the
// reference's vectorised code does.  Then the tokens whose best similarity reaches the threshold are folded
// into that pivot in token order with weights exp(sim).
//
// A CTA takes 256 consecutive tokens of a head (sorted by row) in five steps, each with the number of lanes that suits it:
//   1. a thread per token fetches what is known about it (coalesced; the sorted key is the voxel id), settles the tokens whose
//      row has no pivot and lists the others, once per pivot of their row;
//   2. four lanes per (token, pivot) pair: dot product and squared norms;
//   3. a thread per token: roots, divisions, the best pivot, the weight exp(sim) of a token that merges; the (row, pivot)
//      pairs that tokens merge into are listed;
//   4. a thread per listed pair: what the tokens add up to in weight, score and count, the new weight of the pivot;
//   5. eight lanes per listed pair add up the tokens' rows and fold them into the pivot's.
// Steps 3 to 5 are for rows of up to eight tokens.  Such a row belongs to the CTA in which it starts, which fetches eight tokens
// more than its own; only that CTA looks at its pivots, so all of its similarities are taken before.  Longer rows are
// queued for rows_merge_kernel.
// Most rows have none, one or two pivots (of 384 heads' rows late in a stream 67, 23 and 10 %), so what is done around the 64 products of a
// pair decides: eight lanes that walked a token's pivots and then its row's tokens repeated roots, divisions and
// look-ups in every lane and diverged between their rows.  (us per call, late in a stream, before and now: 384 heads of 8328 tokens in a bounded
// memory 374 -> 206, 384 heads of 4164 tokens 496 -> 244, of 1041 163 -> 100, 48 heads of 8328 89 -> 46, 16 heads of 8328 fp32 tokens 60 -> 43;
// 384 heads of 8328 tokens, 700 voxels, rows of 12 tokens, 582 -> 416.)  Now the rows that are fetched and written decide, 128 bytes each
// wherever they lie: rows are asked for as soon as they are known to be needed (206 against 232 us without that), a pivot's together
// with the first token's.  Five CTAs per SM against four and six: 384 heads of 1041 tokens 100, 95 and 109 us, of 8328 206, 232 and 206.
// Pairs whose next rows are requested ahead, one or two, were no faster.
template <typename T>
__device__ __forceinline__ void prefetch_row(uintptr_t row) {     // a row of 64 values, into L2
  asm volatile("prefetch.global.L2 [%0];" ::"l"(row));
  if (sizeof(T) == 4) asm volatile("prefetch.global.L2 [%0];" ::"l"(row + 128));
}
constexpr int kTokBlock = 256;
constexpr int kShortRow = 8;           // tokens; their pairs are listed as a first token and a bit per token
template <typename T>
__global__ void __launch_bounds__(kTokBlock, sizeof(T) == 2 ? 5 : 4) tokens_sim_merge_kernel(const MergeParams p) {
  grid_dep_wait();   // launched with programmatic serialization behind the previous kernel of the call
  constexpr int kAll = kTokBlock + kShortRow;
  constexpr int kNoKey = -1;           // not a voxel id
  __shared__ int key_s[kAll + 2 * kShortRow];    // voxel ids from eight tokens before to eight behind, and eight of none
  __shared__ uintptr_t krow_s[kAll];             // address of the token's key row (16-byte aligned); bit 0: a carried token
  __shared__ float score_s[kAll];
  __shared__ __align__(16) int segs[kTokBlock][kMaxP];
  __shared__ float dot_s[kAll][kMaxP], nrm_s[kAll][kMaxP], kk_s[kAll];   // step 2; then kk_s: weight of a token that merges
  constexpr int kQueued = -2;
  __shared__ signed char best_s[kAll];           // pivot that the token merges into, -1 = none, kQueued = its row is a longer one
  __shared__ unsigned char npiv_s[kTokBlock], len_s[kTokBlock];   // len: tokens of the short row that starts here
  __shared__ unsigned char before_s[kAll];       // tokens of its row before a token of a short row; kShortRow: of a longer one
  __shared__ unsigned short list[kAll * kMaxP];  // pairs: token | pivot << 9; then first token of a row | pivot << 9
  __shared__ unsigned pair_mask[kTokBlock / 8];  // four bits per token: a token of the row that starts there merges into pivot q
  __shared__ int n_list, n_pairs;
  const int h = blockIdx.y;
  if (p.plan[kPlanAnyValid] == 0) return;
  const int n_tok = p.n_tok[h];
  const int i0 = blockIdx.x * kTokBlock;
  if (i0 >= n_tok) return;
  const int t = threadIdx.x, lane = t & 31;
  const long long hb = static_cast<long long>(h) * p.ncap;
  const unsigned* keys = ((p.passes & 1) ? p.keys_b : p.keys_a) + hb;
  const int* codes = ((p.passes & 1) ? p.vals_b : p.vals_a) + hb;
  if (t == 0) n_list = n_pairs = 0;
  if (t < kTokBlock / 8) pair_mask[t] = 0u;
  // ---- 1. Key, source and score of token t and, by the first threads, of one of the tokens behind the CTA's: both
  // chains of loads go out side by side.
  const int i = i0 + t;
  const bool mine = i < n_tok, extra = t < kShortRow && i + kTokBlock < n_tok;
  const int key = mine ? static_cast<int>(keys[i]) : kNoKey, key_x = extra ? static_cast<int>(keys[i + kTokBlock]) : kNoKey;
  const int code = mine ? codes[i] : 0, code_x = extra ? codes[i + kTokBlock] : 0;
  int npiv = 0;
  int4 sg = make_int4(0, 0, 0, 0);
  if (mine) {
    const long long r = static_cast<long long>(h) * p.voxel_cap + key;
    npiv = p.piv_row_cnt[r];
    if (p.seg_vec) {
      sg = reinterpret_cast<const int4*>(p.piv_row_seg)[r];
    } else if (npiv > 0) {
      sg.x = p.piv_row_seg[r * p.P];
      if (npiv > 1) sg.y = p.piv_row_seg[r * p.P + 1];
      if (npiv > 2) sg.z = p.piv_row_seg[r * p.P + 2];
      if (npiv > 3) sg.w = p.piv_row_seg[r * p.P + 3];
    }
  }
  const int pos = mine && code >= 0 ? token_pos(p, h, code) : 0, pos_x = extra && code_x >= 0 ? token_pos(p, h, code_x) : 0;
  auto score_of = [&](int code, int pos) { return code >= 0 ? p.s_src[h * p.meta_head_stride + pos] : p.over_S_in[~code]; };
  const float score = mine ? score_of(code, pos) : 0.f, score_x = extra ? score_of(code_x, pos_x) : 0.f;
  auto keep = [&](int t, int key, int code, int pos, float score) {
    key_s[kShortRow + t] = key;
    krow_s[t] = reinterpret_cast<uintptr_t>(token_row_at<T>(p, h, code, pos, false)) | (code < 0 ? 1u : 0u);
    score_s[t] = score;
    best_s[t] = -1;
  };
  keep(t, key, code, pos, score);
  npiv_s[t] = static_cast<unsigned char>(npiv);
  *reinterpret_cast<int4*>(segs[t]) = sg;
  if (t < kShortRow) {
    keep(t + kTokBlock, key_x, code_x, pos_x, score_x);
    key_s[t] = i0 > 0 ? static_cast<int>(keys[i0 - kShortRow + t]) : kNoKey;
    key_s[kShortRow + kAll + t] = kNoKey;
  }
  if (mine) {
    p.tok_score[hb + i] = score;
    if (npiv == 0) {
      p.tok_sim[hb + i] = -INFINITY;
    }
  }
  const int seg_t[kMaxP] = {sg.x, sg.y, sg.z, sg.w};
#pragma unroll
  for (int q = 0; q < kMaxP; ++q)
    if (q < npiv) prefetch_row<T>(reinterpret_cast<uintptr_t>(static_cast<const T*>(p.piv_K) + static_cast<long long>(seg_t[q]) * p.D));
  if (!__syncthreads_or(npiv > 0)) return;
  // Lists the pairs of token t: tokens of a short row with pivots where the row starts in this CTA, tokens of a longer one in the
  // CTA that they lie in.  The number of pivots, 0 if it is not listed.
  auto enlist = [&](int t) {
    const int* k = key_s + kShortRow + t;
    const int key = k[0];
    if (key == kNoKey || (t < kTokBlock && npiv_s[t] == 0)) return 0;
    // tokens of the row on either side, up to eight: equal keys lie side by side
    auto run = [&](int dir) {
      if (k[8 * dir] == key) return 8;
      int n = k[4 * dir] == key ? 4 : 0;
      if (k[(n + 2) * dir] == key) n += 2;
      return k[(n + 1) * dir] == key ? n + 1 : n;
    };
    const int before = run(-1), behind = 1 + run(1);
    const bool is_short = before + behind <= kShortRow;
    const int first = is_short ? t - before : t;
    if (first < 0 || first >= kTokBlock || npiv_s[first] == 0) return 0;
    if (is_short && before == 0) len_s[t] = static_cast<unsigned char>(behind);
    before_s[t] = static_cast<unsigned char>(is_short ? before : kShortRow);
    const int np = npiv_s[first];
    prefetch_row<T>(krow_s[t] & ~static_cast<uintptr_t>(1));
    for (int q = 0; q < np; ++q) list[list_push(&n_list)] = static_cast<unsigned short>(t | (q << 9));
    return np;
  };
  const int np_t = enlist(t), np_x = t < kShortRow ? enlist(kTokBlock + t) : 0;
  auto first_of = [&](int t) {
    const int before = before_s[t];
    return before < kShortRow ? t - before : t;
  };
  __syncthreads();
  // ---- 2. Lane j of four holds the 16-byte (fp32: 32-byte) pieces j and j + 4 of both rows.  The sums have the order
  // of eight lanes with a piece each that add with the lane four, two and one away.
  {
    const int gl = t & 3, n = n_list;
    const unsigned gmask = 0xfu << (lane & 28);
    for (int e = t >> 2; e < n; e += kTokBlock / 4) {
      const int entry = list[e], tk = entry & 0x1ff, q = entry >> 9;
      const T* kr = reinterpret_cast<const T*>(krow_s[tk] & ~static_cast<uintptr_t>(1));
      const T* pr = static_cast<const T*>(p.piv_K) + static_cast<long long>(segs[first_of(tk)][q]) * p.D;
      Raw8<T> rk[2], rp[2];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        rk[c].load(kr, gl + 4 * c);
        rp[c].load(pr, gl + 4 * c);
      }
      float k[2][8], pk[2][8];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        rk[c].values(k[c]);
        rp[c].values(pk[c]);
      }
      uint64_t d2 = 0ull, kk2 = 0ull, pp2 = 0ull;
#pragma unroll
      for (int x = 0; x < 8; ++x) {
        const uint64_t k2 = pack_f32x2(k[0][x], k[1][x]), p2 = pack_f32x2(pk[0][x], pk[1][x]);
        d2 = fma_f32x2(k2, p2, d2);
        kk2 = fma_f32x2(k2, k2, kk2);
        pp2 = fma_f32x2(p2, p2, pp2);
      }
      auto sum4 = [&](uint64_t v) {
        float lo, hi;
        unpack_f32x2(v, lo, hi);
        float s = lo + hi;
        s += __shfl_xor_sync(gmask, s, 2);
        return s + __shfl_xor_sync(gmask, s, 1);
      };
      const float d = sum4(d2), kk = sum4(kk2), pp = sum4(pp2);
      if (gl == 0) {
        dot_s[tk][q] = d;
        nrm_s[tk][q] = pp;
        if (q == 0) kk_s[tk] = kk;
      }
    }
  }
  __syncthreads();
  // ---- 3.
  const long long to_v = static_cast<const char*>(p.v_src) - static_cast<const char*>(p.k_src);
  const long long to_v_over = static_cast<const char*>(p.over_V_in) - static_cast<const char*>(p.over_K_in);
  auto decide = [&](int t, int np) {
    if (np == 0) return;
    const float den_k = fmaxf(sqrtf(kk_s[t]), 1e-6f);
    int best = 0;
    float best_sim = -INFINITY;
    for (int q = 0; q < np; ++q) {
      const float den_p = fmaxf(sqrtf(nrm_s[t][q]), 1e-6f);
      const float sim = fminf(1.f, fmaxf(-1.f, __fdiv_rn(dot_s[t][q], __fmul_rn(den_k, den_p))));
      if (sim > best_sim) {
        best_sim = sim;
        best = q;
      }
    }
    const long long o = hb + i0 + t;
    const bool is_short = before_s[t] < kShortRow;
    p.tok_sim[o] = best_sim;
    if (!is_short) p.tok_best[o] = best;
    if (!(best_sim >= p.sim_thresh)) return;
    best_s[t] = static_cast<signed char>(is_short ? best : kQueued);
    if (is_short) {
      const uintptr_t a = krow_s[t];
      prefetch_row<T>((a & ~static_cast<uintptr_t>(1)) + ((a & 1) ? to_v_over : to_v));
      kk_s[t] = expf(best_sim);
      const int first = first_of(t);
      const unsigned bit = 1u << ((first & 7) * 4 + best);
      if ((atomicOr(&pair_mask[first >> 3], bit) & bit) == 0u) {
        const long long at = static_cast<long long>(segs[first][best]) * p.D;
        prefetch_row<T>(reinterpret_cast<uintptr_t>(static_cast<const T*>(p.piv_V) + at));
        list[list_push(&n_pairs)] = static_cast<unsigned short>(first | (best << 9));
      }
    }
  };
  decide(t, np_t);
  if (t < kShortRow) decide(kTokBlock + t, np_x);
  __syncthreads();
  // Longer rows are queued by the first of several neighbouring tokens: with many heads the steps above
  // are bound by their instructions.  (384 heads of 8328 tokens, rows of 12: 652 -> 606 us against every token for itself;
  // the runs of equal keys counted in four looks instead of a loop: -> 582.)
  if (best_s[t] == kQueued && !(t > 0 && best_s[t - 1] == kQueued && key_s[kShortRow + t - 1] == key)) {
    const int ri = p.tok_row[hb + i];
    if (atomicExch(&p.row_flag[hb + ri], 1) == 0) p.merge_list[list_push(&p.plan[kPlanMergeCount])] = make_int2(h, ri);
  }
  const int n = n_pairs;
  if (n == 0) return;
  // ---- 4.  (A row has at least as many tokens as pairs: at most kAll of them.)
  float* const fo_s = &dot_s[0][0];                       // the pivot's old rows and the tokens' sums are weighted with these
  float* const fn_s = fo_s + kAll;
  unsigned* const tokens_s = reinterpret_cast<unsigned*>(fn_s + kAll);      // a bit per token of the row that merges into the pivot
  for (int e = t; e < n; e += kTokBlock) {
    const int entry = list[e], t0 = entry & 0x1ff, q = entry >> 9, seg = segs[t0][q], len = len_s[t0];
    const float W = p.piv_W[seg], S0 = p.piv_S[seg], C0 = p.piv_C[seg];
    float A = 0.f, S = 0.f, C = 0.f;
    unsigned tokens = 0u;
    for (int j = 0; j < len; ++j) {
      if (best_s[t0 + j] == q) {
        tokens |= 1u << j;
        A = __fadd_rn(A, kk_s[t0 + j]);
        S = __fadd_rn(S, fmaxf(score_s[t0 + j], 1e-6f));
        C = __fadd_rn(C, 1.f);
      }
    }
    const float denom = fmaxf(__fadd_rn(W, A), 1e-8f);
    fo_s[e] = __fdiv_rn(W, denom);
    fn_s[e] = __fdiv_rn(1.0f, denom);
    tokens_s[e] = tokens;
    p.piv_W[seg] = denom;
    p.piv_S[seg] = __fadd_rn(S0, S);
    p.piv_C[seg] = __fadd_rn(C0, C);
  }
  __syncthreads();
  // ---- 5.
  // Products that are rounded for themselves, two at a time: mul.rn.f32x2 and the add.rn.f32x2 behind it, and a fused operation with a -0
  // that the compiler sees, come out as one fused operation, which rounds once.
  const uint64_t minus_zero = pack_f32x2(p.minus_zero, p.minus_zero);
  auto times = [&](uint64_t a, uint64_t b) { return fma_f32x2(a, b, minus_zero); };
  const int sub = t & 7;
  for (int e = t >> 3; e < n; e += kTokBlock / 8) {
    const int entry = list[e], t0 = entry & 0x1ff, seg = segs[t0][entry >> 9];
    unsigned todo = tokens_s[e];
    T* kb = static_cast<T*>(p.piv_K) + static_cast<long long>(seg) * p.D;
    T* vb = static_cast<T*>(p.piv_V) + static_cast<long long>(seg) * p.D;
    uint64_t K[4] = {0ull, 0ull, 0ull, 0ull}, V[4] = {0ull, 0ull, 0ull, 0ull};      // two values each
    Raw8<T> nk, nv, pk, pv;      // the next token's rows, in flight while one is added, and the pivot's
    int j = __ffs(todo) - 1;
    auto load = [&] {
      const uintptr_t a = krow_s[t0 + j], kr = a & ~static_cast<uintptr_t>(1);
      nk.load(reinterpret_cast<const T*>(kr), sub);
      nv.load(reinterpret_cast<const T*>(kr + ((a & 1) ? to_v_over : to_v)), sub);
    };
    load();
    pk.load(kb, sub);
    pv.load(vb, sub);
    while (todo) {
      todo &= todo - 1;
      float k[8], v[8];
      nk.values(k);
      nv.values(v);
      const uint64_t a2 = pack_f32x2(kk_s[t0 + j], kk_s[t0 + j]);
      if (todo) {
        j = __ffs(todo) - 1;
        load();
      }
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        K[x] = add_f32x2(K[x], times(a2, pack_f32x2(k[2 * x], k[2 * x + 1])));
        V[x] = add_f32x2(V[x], times(a2, pack_f32x2(v[2 * x], v[2 * x + 1])));
      }
    }
    const uint64_t fo2 = pack_f32x2(fo_s[e], fo_s[e]), fn2 = pack_f32x2(fn_s[e], fn_s[e]);
    auto fold = [&](const Raw8<T>& old, const uint64_t (&sums)[4], T* row) {
      float o[8];
      old.values(o);
#pragma unroll
      for (int x = 0; x < 4; ++x)
        unpack_f32x2(add_f32x2(times(fo2, pack_f32x2(o[2 * x], o[2 * x + 1])), times(fn2, sums[x])), o[2 * x], o[2 * x + 1]);
      row8_store(row, sub, o);
    };
    fold(pk, K, kb);
    fold(pv, V, vb);
  }
}

// The same for the queued rows, those with more than kShortRow tokens.
// What a row waits for is its chain of dependent loads, so the number of rows in flight decides:
// eight lanes per row (16 bytes of a bf16 row each), what is known about a row's tokens fetched eight at a
// time (a lane per token), and one pivot after the other, so that only one pair of accumulators is live.
template <typename T>
__global__ void __launch_bounds__(256, 4) rows_merge_kernel(const MergeParams p) {
  grid_dep_wait();   // launched with programmatic serialization behind the previous kernel of the call
  const int lane = threadIdx.x & 31, sub = threadIdx.x & 7, gbase = lane & 24;
  const unsigned gmask = 0xffu << gbase;
  if (p.plan[kPlanAnyValid] == 0) return;
  const int n = p.plan[kPlanMergeCount];
  const int groups = (gridDim.x * blockDim.x) >> 3;
  for (int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 3; w < n; w += groups) {
    const int2 hr = p.merge_list[w];
    const int h = hr.x, ri = hr.y;
    const long long hb = static_cast<long long>(h) * p.ncap;
    const int vx = p.row_vx[hb + ri];
    const int* rst = p.row_start + static_cast<long long>(h) * (p.ncap + 1);
    const int s0 = rst[ri], s1 = rst[ri + 1];
    const int* codes = ((p.passes & 1) ? p.vals_b : p.vals_a) + hb;
    const long long r = static_cast<long long>(h) * p.voxel_cap + vx;
    const int npiv = p.piv_row_cnt[r];
    int seg_l = 0;                           // lane q < npiv: segment and weight of pivot q
    float W_l = 0.f;
    if (sub < npiv) {
      seg_l = p.piv_row_seg[r * p.P + sub];
      W_l = p.piv_W[seg_l];
    }
    float a_l = 0.f, s_l = 0.f;
    int code_l = 0, best_l = -1, pos_l = 0;  // best_l: pivot that this lane's token merges into, -1 = none
    auto fetch = [&](int i) {
      best_l = -1;
      if (i < s1) {
        const float sim = p.tok_sim[hb + i];
        code_l = codes[i];
        const int best = p.tok_best[hb + i];
        s_l = fmaxf(p.tok_score[hb + i], 1e-6f);
        if (sim >= p.sim_thresh) {
          best_l = best;
          a_l = expf(sim);
          pos_l = code_l >= 0 ? token_pos(p, h, code_l) : 0;
        }
      }
    };
    for (int q = 0; q < npiv; ++q) {
      MergeSums m;
      m.clear();
      for (int base = s0; base < s1; base += 8) {
        fetch(base + sub);
        unsigned todo = __ballot_sync(gmask, best_l == q) >> gbase & 0xffu;
        while (todo) {
          const int src = gbase + __ffs(todo) - 1;
          todo &= todo - 1;
          const int code = __shfl_sync(gmask, code_l, src), pos = __shfl_sync(gmask, pos_l, src);
          const float a = __shfl_sync(gmask, a_l, src), s_t = __shfl_sync(gmask, s_l, src);
          float k[8], v[8];
          row8_load(token_row_at<T>(p, h, code, pos, false), sub, k);
          row8_load(token_row_at<T>(p, h, code, pos, true), sub, v);
          m.add(a, s_t, k, v);
        }
      }
      if (!(m.A > 0.f)) continue;
      merge_into_pivot<T>(p, __shfl_sync(gmask, seg_l, gbase + q), __shfl_sync(gmask, W_l, gbase + q), m, sub);
    }
  }
}

// Score gate of a row with pivots (after this call's merges): mean score per merged token of
// the row's pivots times score_thresh (stac/merger.py:735-745).
__device__ __forceinline__ float row_gate(const MergeParams& p, long long r, int npiv) {
  float sumS = 0.f, sumC = 0.f;
  if (p.seg_vec) {       // all loads side by side
    const int4 sg = reinterpret_cast<const int4*>(p.piv_row_seg)[r];
    const int seg[kMaxP] = {sg.x, sg.y, sg.z, sg.w};
    float S[kMaxP], C[kMaxP];
#pragma unroll
    for (int q = 0; q < kMaxP; ++q) {
      S[q] = q < npiv ? p.piv_S[seg[q]] : 0.f;
      C[q] = q < npiv ? p.piv_C[seg[q]] : 0.f;
    }
#pragma unroll
    for (int q = 0; q < kMaxP; ++q) {
      if (q < npiv) {
        sumS = __fadd_rn(sumS, S[q]);
        sumC = __fadd_rn(sumC, C[q]);
      }
    }
  } else {
    for (int q = 0; q < npiv; ++q) {
      const int seg = p.piv_row_seg[r * p.P + q];
      sumS = __fadd_rn(sumS, p.piv_S[seg]);
      sumC = __fadd_rn(sumC, p.piv_C[seg]);
    }
  }
  return __fmul_rn(__fdiv_rn(sumS, fmaxf(sumC, 1e-6f)), p.score_thresh);
}

// Selection and ranking of one row by one warp (rows with many tokens).  A token of a row with
// pivots is selected for the buffer if it did not come close to a pivot (sim < replace) and its
// score passes the gate; every token of a row without pivots is selected.  Candidates = buffered
// tokens (in column order) then selected tokens (in list order), ranked by (score desc,
// candidate order); rank < B = new column, the rest overflows (stac/allocator.py:559-723).
__device__ __forceinline__ void rank_row_warp(const MergeParams& p, const int h, const int ri, const int lane) {
  const long long hb = static_cast<long long>(h) * p.ncap;
  const int vx = p.row_vx[hb + ri];
  const int* rst = p.row_start + static_cast<long long>(h) * (p.ncap + 1);
  const int s0 = rst[ri], s1 = rst[ri + 1];
  const long long r = static_cast<long long>(h) * p.voxel_cap + vx;
  const int npiv = p.piv_row_cnt[r];
  const int nbuf = p.buf_row_cnt[r];
  float* tsim = p.tok_sim + hb;
  float* tscore = p.tok_score + hb;
  int* tdest = p.tok_dest + hb;
  if (npiv > 0) {
    const float gate = row_gate(p, r, npiv);
    for (int i = s0 + lane; i < s1; i += 32) {
      const bool sel = (tsim[i] < p.replace_thresh) && (fmaxf(tscore[i], 1e-6f) > gate);
      tdest[i] = sel ? 0 : -1;
    }
  } else {
    for (int i = s0 + lane; i < s1; i += 32) tdest[i] = 0;
  }
  __syncwarp();
  // ---- rank existing buffer tokens and selected tokens by (score desc, arrival order)
  float ex_s = 0.f;
  if (lane < nbuf) ex_s = p.buf_S[p.buf_row_seg[r * p.B + lane]];
  int n_sel = 0;
  for (int base = s0; base < s1; base += 32) {
    const int i = base + lane;
    const bool sel = i < s1 && tdest[i] >= 0;
    n_sel += __popc(__ballot_sync(kFull, sel));
  }
  // existing tokens
  int ex_rank = 0;
  for (int c = 0; c < nbuf; ++c) {
    const float sc = __shfl_sync(kFull, ex_s, c);
    if (lane < nbuf && (sc > ex_s || (sc == ex_s && c < lane))) ++ex_rank;
  }
  for (int base = s0; base < s1; base += 32) {
    const int i = base + lane;
    const bool sel = i < s1 && tdest[i] >= 0;
    const float sc = sel ? tscore[i] : 0.f;
    const unsigned m = __ballot_sync(kFull, sel);
    for (unsigned mm = m; mm; mm &= mm - 1) {
      const int src = __ffs(mm) - 1;
      const float s2 = __shfl_sync(kFull, sc, src);
      if (lane < nbuf && s2 > ex_s) ++ex_rank;  // tokens arrive after every existing entry
    }
  }
  int* od = p.old_dest + (hb + ri) * kMaxB;
  if (lane < nbuf) od[lane] = ex_rank;
  // selected tokens
  for (int base = s0; base < s1; base += 32) {
    const int i = base + lane;
    const bool sel = i < s1 && tdest[i] >= 0;
    if (!__any_sync(kFull, sel)) continue;
    const float mine = sel ? tscore[i] : 0.f;
    int rank = 0;
    for (int c = 0; c < nbuf; ++c) {
      const float sc = __shfl_sync(kFull, ex_s, c);
      if (sc >= mine) ++rank;  // existing entries win ties
    }
    for (int base2 = s0; base2 < s1; base2 += 32) {
      const int i2 = base2 + lane;
      const bool sel2 = i2 < s1 && tdest[i2] >= 0;
      if (!__any_sync(kFull, sel2)) continue;
      const float sc = sel2 ? tscore[i2] : __int_as_float(0x7fffffff);      // NaN: not counted
      if (base2 < base) {                    // earlier tokens win ties
#pragma unroll
        for (int t = 0; t < 32; ++t) rank += __shfl_sync(kFull, sc, t) >= mine ? 1 : 0;
      } else {
#pragma unroll
        for (int t = 0; t < 32; ++t) {
          const float s2 = __shfl_sync(kFull, sc, t);
          rank += (s2 > mine || (s2 == mine && base2 + t < i)) ? 1 : 0;
        }
      }
    }
    __syncwarp();
    if (sel) tdest[i] = rank;
  }
  if (lane == 0) {
    const int n_cand = nbuf + n_sel;
    const int newcnt = min(p.B, n_cand);
    const int full = (n_sel > 0 && newcnt == p.B) ? 1 : 0;
    int4 info;
    info.x = newcnt - nbuf;
    info.y = max(0, n_cand - p.B);
    info.z = full | ((full && npiv < p.P) ? 2 : 0) | (nbuf << 4);
    info.w = n_sel;
    p.row_info[hb + ri] = info;
  }
}

// The same for a short row, by one thread.
__device__ __forceinline__ void rank_row_thread(const MergeParams& p, const int h, const int ri, const int vx,
                                                const int s0, const int s1) {
  const long long hb = static_cast<long long>(h) * p.ncap;
  const long long r = static_cast<long long>(h) * p.voxel_cap + vx;
  const int npiv = p.piv_row_cnt[r];
  const int nbuf = p.buf_row_cnt[r];
  const float* tscore = p.tok_score + hb;
  int* tdest = p.tok_dest + hb;
  int* od = p.old_dest + (hb + ri) * kMaxB;
  auto publish = [&](int n_sel) {
    const int n_cand = nbuf + n_sel;
    const int newcnt = min(p.B, n_cand);
    const int full = (n_sel > 0 && newcnt == p.B) ? 1 : 0;
    int4 info;
    info.x = newcnt - nbuf;
    info.y = max(0, n_cand - p.B);
    info.z = full | ((full && npiv < p.P) ? 2 : 0) | (nbuf << 4);
    info.w = n_sel;
    p.row_info[hb + ri] = info;
  };
  if (s1 - s0 <= kShortRow) {
    // Most rows: all tokens in registers; similarities become bits before the gate is there, and the buffer's segments are read only where a
    // token is selected, so that few values are spilled.  (Token by token, as below, with scores read again for every comparison:
    // 80.6 against 49.6 us in this kernel with 384 heads of 8328 tokens, 15.2 against 10.0 with 16 heads.)
    const int n = s1 - s0;
    float sc[kShortRow];
    unsigned sel = npiv == 0 ? (1u << n) - 1u : 0u;
    if (npiv > 0) {
#pragma unroll
      for (int j = 0; j < kShortRow; ++j)
        if (j < n && p.tok_sim[hb + s0 + j] < p.replace_thresh) sel |= 1u << j;
    }
#pragma unroll
    for (int j = 0; j < kShortRow; ++j) sc[j] = j < n ? tscore[s0 + j] : 0.f;
    if (npiv > 0) {
      const float gate = row_gate(p, r, npiv);
#pragma unroll
      for (int j = 0; j < kShortRow; ++j)
        if (!(fmaxf(sc[j], 1e-6f) > gate)) sel &= ~(1u << j);
    }
    if (sel == 0u) {           // nothing to buffer: everything stays in its place
#pragma unroll
      for (int j = 0; j < kShortRow; ++j)
        if (j < n) tdest[s0 + j] = -1;
#pragma unroll
      for (int c = 0; c < kMaxB; c += 4)      // (places behind the buffered ones are not read)
        if (c < nbuf) *reinterpret_cast<int4*>(od + c) = make_int4(c, c + 1, c + 2, c + 3);
      publish(0);
      return;
    }
    float ex[kMaxB];           // buffered tokens are stored in rank order
#pragma unroll
    for (int c = 0; c < kMaxB; c += 4) {
      int4 sg = make_int4(0, 0, 0, 0);
      if (p.buf_seg_vec) {
        if (c < nbuf) sg = reinterpret_cast<const int4*>(p.buf_row_seg)[r * 2 + c / 4];
      } else {
        const int* row_seg = p.buf_row_seg + r * p.B;
        if (c < nbuf) sg.x = row_seg[c];
        if (c + 1 < nbuf) sg.y = row_seg[c + 1];
        if (c + 2 < nbuf) sg.z = row_seg[c + 2];
        if (c + 3 < nbuf) sg.w = row_seg[c + 3];
      }
      ex[c] = c < nbuf ? p.buf_S[sg.x] : 0.f;
      ex[c + 1] = c + 1 < nbuf ? p.buf_S[sg.y] : 0.f;
      ex[c + 2] = c + 2 < nbuf ? p.buf_S[sg.z] : 0.f;
      ex[c + 3] = c + 3 < nbuf ? p.buf_S[sg.w] : 0.f;
    }
#pragma unroll
    for (int c = 0; c < kMaxB; c += 4) {
      if (c < nbuf) {
        int old_rank[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          old_rank[e] = c + e;
#pragma unroll
          for (int j = 0; j < kShortRow; ++j) old_rank[e] += ((sel >> j) & 1u) && sc[j] > ex[c + e] ? 1 : 0;
        }
        *reinterpret_cast<int4*>(od + c) = make_int4(old_rank[0], old_rank[1], old_rank[2], old_rank[3]);
      }
    }
#pragma unroll
    for (int j = 0; j < kShortRow; ++j) {
      if (j < n) {
        int rank = 0;
#pragma unroll
        for (int c = 0; c < kMaxB; ++c) rank += c < nbuf && ex[c] >= sc[j] ? 1 : 0;
#pragma unroll
        for (int j2 = 0; j2 < kShortRow; ++j2)
          rank += ((sel >> j2) & 1u) && (j2 < j ? sc[j2] >= sc[j] : sc[j2] > sc[j]) ? 1 : 0;
        tdest[s0 + j] = (sel >> j) & 1u ? rank : -1;
      }
    }
    publish(__popc(sel));
    return;
  }
  unsigned sel_mask = 0u;      // bit j: token s0 + j goes to the buffer
  if (npiv > 0) {
    const float gate = row_gate(p, r, npiv);
    for (int i = s0; i < s1; ++i)
      if ((p.tok_sim[hb + i] < p.replace_thresh) && (fmaxf(tscore[i], 1e-6f) > gate)) sel_mask |= 1u << (i - s0);
  } else {
    sel_mask = (s1 - s0) == 32 ? 0xffffffffu : ((1u << (s1 - s0)) - 1u);
  }
  float ex[kMaxB];
#pragma unroll
  for (int c = 0; c < kMaxB; ++c) ex[c] = (c < nbuf) ? p.buf_S[p.buf_row_seg[r * p.B + c]] : 0.f;
#pragma unroll
  for (int c = 0; c < kMaxB; ++c) {
    if (c < nbuf) {
      int rank = c;  // buffered tokens are stored in rank order
      for (unsigned mm = sel_mask; mm; mm &= mm - 1) rank += (tscore[s0 + __ffs(mm) - 1] > ex[c]) ? 1 : 0;
      od[c] = rank;
    }
  }
  for (int i = s0; i < s1; ++i) {
    if (!((sel_mask >> (i - s0)) & 1u)) {
      tdest[i] = -1;
      continue;
    }
    const float mine = tscore[i];
    int rank = 0;
#pragma unroll
    for (int c = 0; c < kMaxB; ++c) rank += (c < nbuf && ex[c] >= mine) ? 1 : 0;
    for (unsigned mm = sel_mask; mm; mm &= mm - 1) {
      const int i2 = s0 + __ffs(mm) - 1;
      const float s2 = tscore[i2];
      rank += (s2 > mine || (s2 == mine && i2 < i)) ? 1 : 0;
    }
    tdest[i] = rank;
  }
  publish(__popc(sel_mask));
}

// One thread per row; the rows with more than kLongRow tokens are listed and ranked by a warp each, which
// may be any warp of the grid: their ranking is quadratic in their tokens, and with few, large voxels
// there are few CTAs with rows.  The list is dealt out one row per CTA first, CTAs without rows of their
// own in front.  (8328 tokens a head, fourth to seventh call: 16 heads on 60
// voxels 1490 us per insert when the warps of the CTA that held a long row had to rank it, 767 us with
// the list, 572 us with the scores passed between lanes instead of read one by one; 48 heads on 20 voxels 4966,
// 2910 and 1938 us; 384 heads on 200 voxels 2816, 2378 and 2240 us.)
// kMinCtas: four CTAs per SM let the rows of up to kShortRow tokens have 64 registers, six 40.  Six are better wherever they find work,
// most of all with longer rows, which wait for more loads.  (us in this kernel with four and six, tokens and voxels of a head: 384
// heads 8328, 6500 63, 50, 8328, 300 of 70000 721, 621; 148 heads 4164, 200 of 70000 260, 234; 16 heads 8328, 6500 9.9, 11.2.)
template <int kMinCtas>
__global__ void __launch_bounds__(256, kMinCtas) rows_rank_kernel(const MergeParams p) {
  grid_dep_wait();   // launched with programmatic serialization behind the previous kernel of the call
  const int h = blockIdx.y;
  const int r0 = blockIdx.x * 256;
  const int n_long = p.plan[kPlanLongCount];
  if (p.plan[kPlanAnyValid] == 0) return;
  const int n_rows = p.n_rows[h];
  if (r0 >= n_rows && n_long == 0) return;
  const int ri = r0 + threadIdx.x;
  if (ri < n_rows) {
    const int* rst = p.row_start + static_cast<long long>(h) * (p.ncap + 1);
    const int s0 = rst[ri], s1 = rst[ri + 1];
    const int vx = p.row_vx[static_cast<long long>(h) * p.ncap + ri];
    if (s1 - s0 <= kLongRow) rank_row_thread(p, h, ri, vx, s0, s1);
  }
  __syncwarp();
  const int cta = (gridDim.x - 1 - blockIdx.x) * gridDim.y + h, n_cta = gridDim.x * gridDim.y;
  for (int w = cta + (threadIdx.x >> 5) * n_cta; w < n_long; w += 8 * n_cta) {
    const int2 hr = p.long_list[w];
    rank_row_warp(p, hr.x, hr.y, threadIdx.x & 31);
  }
}

// ------------------------------------------------------------------------------------ scans
// Bounded pools: a row that would open new buffer columns, or need a new pivot segment, beyond
// what is left is skipped as a whole (its selected tokens are dropped, the row stays as it
// was).  The cut follows the allocation order, i.e. (head, voxel) ascending, so it is
// deterministic; merges into existing pivots done before stay.  A skipped row is left with no
// selected token (info.w = 0): tokens_place_kernel looks at that.  Returns the tokens dropped.
__device__ __forceinline__ int skip_row_that_does_not_fit(const MergeParams& p, int4& info, int4 pref, int4 hbase) {
  if (info.w == 0) return 0;
  const bool no_buf = info.x > 0 && hbase.x + pref.x + info.x > p.plan[kPlanAvailBuf];
  const bool no_piv = (info.z & 2) && hbase.w + pref.w + 1 > p.plan[kPlanAvailPiv];
  if (!no_buf && !no_piv) return 0;
  const int dropped = info.w;
  info = make_int4(0, 0, info.z & ~3, 0);
  return dropped;
}

// Scan over the heads and allocation plan, by one CTA of kThreads threads.
template <int kThreads>
__device__ __forceinline__ void make_plan(const MergeParams& p, const int pass, int4* warp_sums) {
  int4 carry = make_int4(0, 0, 0, 0);
  for (int base = 0; base < p.heads; base += kThreads) {
    const int h = base + threadIdx.x;
    int4 t = make_int4(0, 0, 0, 0), total;
    if (h < p.heads) t = __ldcg(&p.head_tot[h]);
    const int4 b = add4(carry, block_scan4<kThreads / 32>(t, warp_sums, &total));
    if (h < p.heads) {
      p.head_base[h] = b;
      p.over_start_out[h] = b.y;
    }
    carry = add4(carry, total);
  }
  if (threadIdx.x == 0) {
    if (pass == 0 && p.voxel_count != nullptr) p.meta[STAC_META_VOXELS] = max(p.meta[STAC_META_VOXELS], *p.voxel_count);
    const int any = p.plan[kPlanAnyValid];
    const int total_add = carry.x, total_over = carry.y, total_full = carry.z, total_piv = carry.w;
    const int free_len = p.meta[STAC_META_BUF_FREE_LEN];
    const int buf_top = p.meta[STAC_META_BUF_TOP];
    const int piv_top = p.meta[STAC_META_PIV_TOP];
    const int k = min(total_add, free_len);
    p.plan[kPlanK] = k;
    p.plan[kPlanFreeLen] = free_len;
    p.plan[kPlanBufTop] = buf_top;
    p.plan[kPlanPivTop] = piv_top;
    p.plan[kPlanTotalAdd] = total_add;
    p.plan[kPlanTotalFull] = total_full;
    p.plan[kPlanTotalOver] = total_over;
    int abort = 0;
    if (any) {
      const int avail_buf = free_len + (p.buf_cap - buf_top);
      const int avail_piv = p.piv_cap - piv_top;
      if (pass == 0 && (total_add > avail_buf || total_piv > avail_piv)) {
        // The pools are bounded and this call does not fit: rows are skipped in (head, voxel)
        // order by the second launch, which makes the plan again.
        p.plan[kPlanShort] = 1;
        p.plan[kPlanAvailBuf] = avail_buf;
        p.plan[kPlanAvailPiv] = avail_piv;
        return;
      }
      if (buf_top + (total_add - k) > p.buf_cap || piv_top + total_piv > p.piv_cap || total_over > p.over_cap ||
          free_len - k + total_full * p.B > p.buf_cap)
        abort = 1;
    }
    p.plan[kPlanAbort] = abort;
    if (abort) report_error(p.err, DEV_POOL_CAPACITY);
    if (any && !abort) {
      p.over_start_out[p.heads] = total_over;
      p.meta[STAC_META_BUF_TOP] = buf_top + (total_add - k);
      p.meta[STAC_META_PIV_TOP] = piv_top + total_piv;
      p.meta[STAC_META_OVER_COUNT] = total_over;
      p.meta[STAC_META_BUF_FREE_LEN] = free_len - k + total_full * p.B;
      p.meta[STAC_META_BUF_USED] += total_add - total_full * p.B;
      p.meta[STAC_META_PIV_USED] += total_piv;
    }
  }
}

// pass 0 always runs; pass 1 only when pass 0 found the pools too small
template <int kThreads>
__global__ void __launch_bounds__(kThreads, 2048 / kThreads) scan_rows_kernel(const MergeParams p, const int pass) {
  grid_dep_wait();   // launched with programmatic serialization behind the previous kernel of the call
  __shared__ int4 warp_sums[32];
  __shared__ int sh_last;
  if (pass == 1 && p.plan[kPlanShort] == 0) return;
  const int h = blockIdx.x;
  const long long hb = static_cast<long long>(h) * p.ncap;
  const int n = p.plan[kPlanAnyValid] ? p.n_rows[h] : 0;
  int4 hbase = make_int4(0, 0, 0, 0), carry = make_int4(0, 0, 0, 0);
  if (pass == 1) hbase = p.head_base[h];
  int dropped = 0;
  for (int base = 0; base < n; base += kThreads) {
    const int i = base + threadIdx.x;
    int4 info = make_int4(0, 0, 0, 0), total;
    if (i < n) {
      info = p.row_info[hb + i];
      if (pass == 1) {
        const int d = skip_row_that_does_not_fit(p, info, p.row_pref[hb + i], hbase);
        if (d > 0) p.row_info[hb + i] = info;
        dropped += d;
      }
    }
    const int4 v = make_int4(info.x, info.y, info.z & 1, (info.z >> 1) & 1);
    const int4 pref = add4(carry, block_scan4<kThreads / 32>(v, warp_sums, &total));
    if (i < n) p.row_pref[hb + i] = pref;
    carry = add4(carry, total);
  }
  if (pass == 1) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dropped += __shfl_xor_sync(kFull, dropped, o);
    if ((threadIdx.x & 31) == 0 && dropped > 0) atomicAdd(&p.meta[STAC_META_DROPPED], dropped);
  }
  // the CTA that arrives last sees every head's total
  if (threadIdx.x == 0) {
    p.head_tot[h] = carry;
    __threadfence();
    sh_last = atomicAdd(&p.plan[pass == 0 ? kPlanTicket : kPlanTicket2], 1) == p.heads - 1;
    __threadfence();
  }
  __syncthreads();
  if (sh_last) make_plan<kThreads>(p, pass, warp_sums);
}

// ------------------------------------------------------------------------------------ phase B
// Phase B, step 1 (one thread per row): hand out the segment ids of the new columns in
// (row, column) order from the allocation plan, publish the new occupancy, and queue the rows
// whose buffered tokens change column or whose buffer filled up.
__global__ void __launch_bounds__(256) rows_phase_b1a_kernel(const MergeParams p) {
  grid_dep_wait();   // launched with programmatic serialization behind the previous kernel of the call
  const int h = blockIdx.y;
  const int ri = blockIdx.x * blockDim.x + threadIdx.x;
  if (p.plan[kPlanAnyValid] == 0 || p.plan[kPlanAbort] != 0) return;
  if (ri >= p.n_rows[h]) return;
  const long long hb = static_cast<long long>(h) * p.ncap;
  const int4 info = p.row_info[hb + ri];
  if (info.w == 0) return;  // nothing selected: the buffer is untouched
  const int vx = p.row_vx[hb + ri];
  const long long r = static_cast<long long>(h) * p.voxel_cap + vx;
  const int add_off = p.head_base[h].x + p.row_pref[hb + ri].x;
  const int nbuf = info.z >> 4;
  const int newcnt = nbuf + info.x;
  const int k_take = p.plan[kPlanK], free_len = p.plan[kPlanFreeLen], buf_top = p.plan[kPlanBufTop];
  for (int col = nbuf; col < newcnt; ++col) {
    const int q = add_off + (col - nbuf);
    p.buf_row_seg[r * p.B + col] = q < k_take ? p.buf_free[free_len - k_take + q] : buf_top + (q - k_take);
  }
  const int* od = p.old_dest + (hb + ri) * kMaxB;
  bool moves = false;
  for (int c = 0; c < nbuf; ++c) moves = moves || (od[c] != c);
  if (moves) p.move_list[list_push(&p.plan[kPlanMoveCount])] = make_int2(h, ri);
  if (info.z & 1) p.full_list[list_push(&p.plan[kPlanFullCount])] = make_int2(h, ri);
  else p.buf_row_cnt[r] = newcnt;
}

// Phase B, step 2 (one warp per queued row): buffered tokens only ever move to a higher column
// (new tokens push them down the ranking), so walking them from the last column to the first
// moves each one into a slot whose old content has already left.
template <typename T, int EPL>
__global__ void __launch_bounds__(256) rows_phase_b1m_kernel(const MergeParams p) {
  grid_dep_wait();   // launched with programmatic serialization behind the previous kernel of the call
  const int lane = threadIdx.x & 31;
  const int warps_per_block = blockDim.x >> 5;
  if (p.plan[kPlanAnyValid] == 0 || p.plan[kPlanAbort] != 0) return;
  const int n_move = p.plan[kPlanMoveCount];
  const int B = p.B, D = p.D;
  T* bK = static_cast<T*>(p.buf_K);
  T* bV = static_cast<T*>(p.buf_V);
  T* oK = static_cast<T*>(p.over_K_out);
  T* oV = static_cast<T*>(p.over_V_out);
  for (int wi = blockIdx.x * warps_per_block + (threadIdx.x >> 5); wi < n_move; wi += gridDim.x * warps_per_block) {
    const int2 hr = p.move_list[wi];
    const int h = hr.x, ri = hr.y;
    const long long hb = static_cast<long long>(h) * p.ncap;
    const int4 info = p.row_info[hb + ri];
    const int vx = p.row_vx[hb + ri];
    const long long r = static_cast<long long>(h) * p.voxel_cap + vx;
    const int over_off = p.head_base[h].y + p.row_pref[hb + ri].y;
    const int nbuf = info.z >> 4;
    const int newcnt = nbuf + info.x;
    const int* od = p.old_dest + (hb + ri) * kMaxB;
    int my_seg = -1, ex_dest = -1;
    if (lane < newcnt) my_seg = p.buf_row_seg[r * B + lane];
    if (lane < nbuf) ex_dest = od[lane];
    for (int c = nbuf - 1; c >= 0; --c) {
      const int d = __shfl_sync(kFull, ex_dest, c);
      if (d == c) continue;
      const int sg = __shfl_sync(kFull, my_seg, c);
      float k[EPL], v[EPL];
#pragma unroll
      for (int e = 0; e < EPL; ++e) {
        k[e] = Elem<T>::load(bK + static_cast<long long>(sg) * D + lane * EPL + e);
        v[e] = Elem<T>::load(bV + static_cast<long long>(sg) * D + lane * EPL + e);
      }
      const float sc = p.buf_S[sg];
      __syncwarp();
      if (d < B) {
        const int dg = __shfl_sync(kFull, my_seg, d);
#pragma unroll
        for (int e = 0; e < EPL; ++e) {
          Elem<T>::store(bK + static_cast<long long>(dg) * D + lane * EPL + e, k[e]);
          Elem<T>::store(bV + static_cast<long long>(dg) * D + lane * EPL + e, v[e]);
        }
        if (lane == 0) p.buf_S[dg] = sc;
      } else {
        const long long o = over_off + (d - B);
#pragma unroll
        for (int e = 0; e < EPL; ++e) {
          Elem<T>::store(oK + o * D + lane * EPL + e, k[e]);
          Elem<T>::store(oV + o * D + lane * EPL + e, v[e]);
        }
        if (lane == 0) {
          p.over_S_out[o] = sc;
          p.over_hv_out[2 * o] = h;
          p.over_hv_out[2 * o + 1] = vx;
        }
      }
      __syncwarp();
    }
  }
}

// Phase B, step 3 (token-parallel): every selected token is copied to its column's segment or
// to its overflow slot.  A CTA takes 256 consecutive tokens of a head: one thread per token finds
// where it goes (most tokens of a bounded memory go nowhere, and that is then all they cost), the
// selected ones are listed in shared memory and copied by eight lanes each, 16 (bf16) or 32 (fp32)
// bytes of K and of V per lane, the next token's loads in flight before this one's stores.
// (1.6 M tokens, all placed: 174 -> 128 us against eight lanes per token throughout; 3.2 M tokens of a
// bounded memory: 82 -> 19 us.)
template <typename T>
__global__ void __launch_bounds__(kTokBlock) tokens_place_kernel(const MergeParams p) {
  grid_dep_wait();   // launched with programmatic serialization behind the previous kernel of the call
  constexpr int kVec = static_cast<int>(sizeof(T)) * 8 / 16;   // 16-byte vectors per lane and row
  __shared__ int4 list[kTokBlock];   // code, position, destination row, 1 = overflow list
  __shared__ int n_list;
  const int h = blockIdx.y;
  if (p.plan[kPlanAnyValid] == 0 || p.plan[kPlanAbort] != 0) return;
  const int n_tok = p.n_tok[h];
  const int i0 = blockIdx.x * kTokBlock;
  if (i0 >= n_tok) return;
  if (threadIdx.x == 0) n_list = 0;
  __syncthreads();
  const long long hb = static_cast<long long>(h) * p.ncap;
  const int i = i0 + threadIdx.x;
  const bool short_of_room = p.plan[kPlanShort] != 0;     // rows may have been skipped since their tokens were ranked
  if (i < n_tok) {
    const int d = p.tok_dest[hb + i];
    if (d >= 0 && (!short_of_room || p.row_info[hb + p.tok_row[hb + i]].w != 0)) {
      const int code = (((p.passes & 1) ? p.vals_b : p.vals_a) + hb)[i];
      const int vx = static_cast<int>((((p.passes & 1) ? p.keys_b : p.keys_a) + hb)[i]);
      const float sc = p.tok_score[hb + i];
      const int pos = code >= 0 ? token_pos(p, h, code) : 0;
      int dst;
      if (d < p.B) {
        dst = p.buf_row_seg[(static_cast<long long>(h) * p.voxel_cap + vx) * p.B + d];
        p.buf_S[dst] = sc;
      } else {
        dst = p.head_base[h].y + p.row_pref[hb + p.tok_row[hb + i]].y + (d - p.B);
        p.over_S_out[dst] = sc;
        p.over_hv_out[2 * dst] = h;
        p.over_hv_out[2 * dst + 1] = vx;
      }
      list[list_push(&n_list)] = make_int4(code, pos, dst, d < p.B ? 0 : 1);
    }
  }
  __syncthreads();
  const int n = n_list;
  const int sub = threadIdx.x & 7;
  constexpr int kStep = kTokBlock / 8;
  uint4 kv[2][kVec], vv[2][kVec];
  auto fetch = [&](int e, uint4 (&k)[kVec], uint4 (&v)[kVec]) {
    const int4 tk = list[e];
    const uint4* src_k = reinterpret_cast<const uint4*>(token_row_at<T>(p, h, tk.x, tk.y, false)) + sub * kVec;
    const uint4* src_v = reinterpret_cast<const uint4*>(token_row_at<T>(p, h, tk.x, tk.y, true)) + sub * kVec;
#pragma unroll
    for (int j = 0; j < kVec; ++j) {
      k[j] = src_k[j];
      v[j] = src_v[j];
    }
  };
  auto put = [&](int e, const uint4 (&k)[kVec], const uint4 (&v)[kVec]) {
    const int4 tk = list[e];
    uint4* dst_k = reinterpret_cast<uint4*>(static_cast<T*>(tk.w ? p.over_K_out : p.buf_K) + static_cast<long long>(tk.z) * p.D);
    uint4* dst_v = reinterpret_cast<uint4*>(static_cast<T*>(tk.w ? p.over_V_out : p.buf_V) + static_cast<long long>(tk.z) * p.D);
#pragma unroll
    for (int j = 0; j < kVec; ++j) {
      dst_k[sub * kVec + j] = k[j];
      dst_v[sub * kVec + j] = v[j];
    }
  };
  int e = threadIdx.x >> 3;
  for (; e + kStep < n; e += 2 * kStep) {
    fetch(e, kv[0], vv[0]);
    fetch(e + kStep, kv[1], vv[1]);
    put(e, kv[0], vv[0]);
    put(e + kStep, kv[1], vv[1]);
  }
  if (e < n) {
    fetch(e, kv[0], vv[0]);
    put(e, kv[0], vv[0]);
  }
}

// Two of a row's 64 values per lane, as they were loaded.
template <typename T> struct Pair;
template <> struct Pair<__nv_bfloat16> {
  uint32_t u;
  __device__ __forceinline__ void load(const __nv_bfloat16* row, int lane) { u = reinterpret_cast<const uint32_t*>(row)[lane]; }
  __device__ __forceinline__ float2 values() const { return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u)); }
  static __device__ __forceinline__ void store(__nv_bfloat16* row, int lane, float2 x) {
    reinterpret_cast<uint32_t*>(row)[lane] = pack_bf16x2(x.x, x.y);
  }
};
template <> struct Pair<float> {
  float2 u;
  __device__ __forceinline__ void load(const float* row, int lane) { u = reinterpret_cast<const float2*>(row)[lane]; }
  __device__ __forceinline__ float2 values() const { return u; }
  static __device__ __forceinline__ void store(float* row, int lane, float2 x) { reinterpret_cast<float2*>(row)[lane] = x; }
};

// Full buffers -> one pivot each, inserted into the row's pivot slots; the buffer row is released.
// A row is a chain of loads, sums, roots and divisions.
// Few rows: a warp per row, because the kernel takes as long as one of them.  The warp's four groups of eight lanes compare two of the
// buffered tokens each with the seed, and one pivot each with the victim (eight values per lane, 16-byte loads, sums over
// eight lanes), and the weighted means are taken by all lanes, two values each.
template <typename T>
__device__ __forceinline__ void full_rows_by_warps(const MergeParams& p, const int n_full) {
  const int lane = threadIdx.x & 31, sub = lane & 7, group = lane >> 3;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  for (int wi = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; wi < n_full; wi += warps) {
    const int2 hr = p.full_list[wi];
    const int h = hr.x, ri = hr.y;
    const long long hb = static_cast<long long>(h) * p.ncap;
    const int vx = p.row_vx[hb + ri];
    const long long r = static_cast<long long>(h) * p.voxel_cap + vx;
    const int4 pref = p.row_pref[hb + ri];
    const int4 hbase = p.head_base[h];
    const int full_off = hbase.z + pref.z, piv_off = hbase.w + pref.w;
    const int B = p.B, D = p.D;
    const T* bK = static_cast<const T*>(p.buf_K);
    const T* bV = static_cast<const T*>(p.buf_V);
    T* pK = static_cast<T*>(p.piv_K);
    T* pV = static_cast<T*>(p.piv_V);
    const int npiv = p.piv_row_cnt[r];
    // (asked for as soon as its place is known, a lane per buffered token and per pivot)
    int my_seg = -1, ps_l = -1;        // lane c < B of every group: segment of column c; lane q < P: of pivot q
    if (sub < B) my_seg = p.buf_row_seg[r * B + sub];
    if (npiv >= p.P && sub < p.P) ps_l = p.piv_row_seg[r * p.P + sub];
    // ---- the buffer is full: B tokens -> one pivot (stac/merger.py:408-461)
    float ts = 0.f, pw_l = INFINITY;   // lane q < P of a saturated row: weight of pivot q
    if (sub < B) {
      ts = fmaxf(p.buf_S[my_seg], 1e-6f);
      const T* rows = group & 1 ? bV : bK;
      if (group < 2) prefetch_row<T>(reinterpret_cast<uintptr_t>(rows + static_cast<long long>(my_seg) * D));
    }
    if (ps_l >= 0) {
      pw_l = p.piv_W[ps_l];
      const T* rows = group & 1 ? pV : pK;
      if (group >= 2) prefetch_row<T>(reinterpret_cast<uintptr_t>(rows + static_cast<long long>(ps_l) * D));
    }
    int seed = 0;
    float seed_s = -INFINITY, sumS = 0.f;
    for (int c = 0; c < B; ++c) {
      const float sc = __shfl_sync(kFull, ts, c);
      if (sc > seed_s) {
        seed_s = sc;
        seed = c;
      }
      sumS = __fadd_rn(sumS, sc);
    }
    float kn_seed[8];
    {
      const int sg = __shfl_sync(kFull, my_seg, seed);
      float k[8];
      row8_load(bK + static_cast<long long>(sg) * D, sub, k);
      float ss = 0.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) ss += k[e] * k[e];
      const float den = fmaxf(sqrtf(group8_sum(ss, kFull)), 1e-6f);
#pragma unroll
      for (int e = 0; e < 8; ++e) kn_seed[e] = __fdiv_rn(k[e], den);
    }
    // pass 1 over the keys, tokens `group` and group + 4: w_c = exp(cos(k_c, seed))
    float w_own[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int c = group + 4 * i;
      const int sg = __shfl_sync(kFull, my_seg, c < B ? c : 0);
      float k[8];
      row8_load(bK + static_cast<long long>(sg) * D, sub, k);
      float ss = 0.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) ss += k[e] * k[e];
      const float den = fmaxf(sqrtf(group8_sum(ss, kFull)), 1e-6f);
      float d = 0.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) d += __fdiv_rn(k[e], den) * kn_seed[e];
      w_own[i] = expf(fminf(1.f, fmaxf(-1.f, group8_sum(d, kFull))));
    }
    // pass 2: the weighted means of keys and values, two values per lane
    Pair<T> tk[kMaxB], tv[kMaxB];
#pragma unroll
    for (int c = 0; c < kMaxB; ++c) {
      const int sg = __shfl_sync(kFull, my_seg, c < B ? c : 0);
      tk[c].load(bK + static_cast<long long>(sg) * D, lane);
      tv[c].load(bV + static_cast<long long>(sg) * D, lane);
    }
    float w[kMaxB], Wsum = 0.f;
#pragma unroll
    for (int c = 0; c < kMaxB; ++c) {
      w[c] = __shfl_sync(kFull, w_own[c / 4], (c % 4) * 8);
      if (c < B) Wsum = __fadd_rn(Wsum, w[c]);
    }
    float2 nk = make_float2(0.f, 0.f), nv = make_float2(0.f, 0.f);
    const float wden = __fadd_rn(Wsum, 1e-8f);
#pragma unroll
    for (int c = 0; c < kMaxB; ++c) {
      if (c < B) {
        const float cn = __fdiv_rn(w[c], wden);
        const float2 k = tk[c].values(), v = tv[c].values();
        nk.x = __fadd_rn(nk.x, __fmul_rn(cn, k.x));
        nk.y = __fadd_rn(nk.y, __fmul_rn(cn, k.y));
        nv.x = __fadd_rn(nv.x, __fmul_rn(cn, v.x));
        nv.y = __fadd_rn(nv.y, __fmul_rn(cn, v.y));
      }
    }
    // ---- insert the pivot (stac/merger.py:462-582)
    int pseg;
    if (npiv < p.P) {
      pseg = p.plan[kPlanPivTop] + piv_off;
      if (lane == 0) {
        p.piv_row_seg[r * p.P + npiv] = pseg;
        p.piv_row_cnt[r] = npiv + 1;
      }
    } else {
      // saturated: fold the lowest-weight pivot into its most similar neighbour, reuse its slot
      int victim = 0;
      float wmin = INFINITY;
      for (int q = 0; q < p.P; ++q) {
        const float wq = __shfl_sync(kFull, pw_l, q);
        if (wq < wmin) {
          wmin = wq;
          victim = q;
        }
      }
      // keys normalised in the pool dtype, as the reference does here (stac/merger.py:493-495)
      auto load_normalised = [&](int seg, float (&out)[8]) {
        float pk[8];
        row8_load(pK + static_cast<long long>(seg) * D, sub, pk);
        float ss = 0.f;
#pragma unroll
        for (int e = 0; e < 8; ++e) ss += pk[e] * pk[e];
        float nrm = Elem<T>::round(sqrtf(group8_sum(ss, kFull)));
        nrm = fmaxf(nrm, Elem<T>::round(1e-6f));
#pragma unroll
        for (int e = 0; e < 8; ++e) out[e] = Elem<T>::round(__fdiv_rn(pk[e], nrm));
      };
      const int vseg = __shfl_sync(kFull, ps_l, victim);
      const float Wv = __shfl_sync(kFull, pw_l, victim);
      float vn[8], pkn[8];
      load_normalised(vseg, vn);
      load_normalised(__shfl_sync(kFull, ps_l, group < p.P ? group : victim), pkn);      // pivot `group`
      float d = 0.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) d += pkn[e] * vn[e];
      d = Elem<T>::round(group8_sum(d, kFull));
      int nb = 0;
      float best = -INFINITY;
      for (int q = 0; q < p.P; ++q) {
        const float dq = __shfl_sync(kFull, d, 8 * q);
        if (q != victim && dq > best) {
          best = dq;
          nb = q;
        }
      }
      if (p.P == 1) nb = victim;   // no neighbour to fold into: the victim is simply replaced
      float scale;
      if (Elem<T>::kIsBf16) scale = Elem<T>::round(expf(Elem<T>::round(best - 1.0f)));
      else scale = expf(best - 1.0f);
      const int nseg = __shfl_sync(kFull, ps_l, nb);
      const float Wn = __shfl_sync(kFull, pw_l, nb);
      if (p.P > 1) {
        const float Wj = __fmul_rn(Wv, scale);
        const float denom = fmaxf(__fadd_rn(Wj, Wn), 1e-8f);
        const float fj = __fdiv_rn(Wj, denom), fk = __fdiv_rn(Wn, denom);
        auto fold = [&](T* rows) {
          Pair<T> a, b;
          a.load(rows + static_cast<long long>(vseg) * D, lane);
          b.load(rows + static_cast<long long>(nseg) * D, lane);
          const float2 x = a.values(), y = b.values();
          Pair<T>::store(rows + static_cast<long long>(nseg) * D, lane,
                         make_float2(__fadd_rn(__fmul_rn(fj, x.x), __fmul_rn(fk, y.x)), __fadd_rn(__fmul_rn(fj, x.y), __fmul_rn(fk, y.y))));
        };
        fold(pK);
        fold(pV);
        if (lane == 0) {
          p.piv_W[nseg] = denom;
          p.piv_S[nseg] = __fadd_rn(p.piv_S[vseg], p.piv_S[nseg]);
          p.piv_C[nseg] = __fadd_rn(p.piv_C[vseg], p.piv_C[nseg]);
        }
      }
      pseg = vseg;
      __syncwarp();        // all lanes have read the victim's rows that are written over now
    }
    Pair<T>::store(pK + static_cast<long long>(pseg) * D, lane, nk);
    Pair<T>::store(pV + static_cast<long long>(pseg) * D, lane, nv);
    if (lane == 0) {
      p.piv_W[pseg] = Wsum;
      p.piv_S[pseg] = sumS;
      p.piv_C[pseg] = static_cast<float>(B);
    }
    // ---- release the buffer row: segment ids go to the staging area in column order
    if (lane < B) {
      p.free_stage[full_off * B + lane] = my_seg;
      p.buf_row_seg[r * B + lane] = -1;
    }
    if (lane == 0) p.buf_row_cnt[r] = 0;
  }
}

// Many rows: eight lanes per row, each holding eight of the 64 values of a token (16-byte loads), so a warp
// works on four rows at once.  Tokens are streamed (keys twice: once for the weights, once for
// the weighted mean; the second read hits the cache) so that few registers are live and many
// rows are in flight per SM.  With more bf16 rows than are resident at once, theirs are asked for as soon as their places are known
// (60 thousand rows 80, 116 -> 73, 107.5 us; fewer, or fp32, took up to 12 % longer with that).
// (holding all eight key rows of a row in registers, at four CTAs per SM, measured 15 % slower for
// the whole merge than streaming them at eight CTAs per SM: these per-row kernels want threads)
template <typename T>
__device__ __forceinline__ void full_rows_by_groups(const MergeParams& p, const int n_full) {
  const int lane = threadIdx.x & 31, sub = threadIdx.x & 7;
  const int gbase = lane & 24;                       // first lane of this group
  const unsigned gmask = 0xffu << gbase;
  const int groups = (gridDim.x * blockDim.x) >> 3;
  const bool ahead = sizeof(T) == 2 && n_full > groups / 2;      // (half of the CTAs are resident at once, see launch_merge)
  for (int wi = (blockIdx.x * blockDim.x + threadIdx.x) >> 3; wi < n_full; wi += groups) {
    const int2 hr = p.full_list[wi];
    const int h = hr.x, ri = hr.y;
    const long long hb = static_cast<long long>(h) * p.ncap;
    const int vx = p.row_vx[hb + ri];
    const long long r = static_cast<long long>(h) * p.voxel_cap + vx;
    const int4 pref = p.row_pref[hb + ri];
    const int4 hbase = p.head_base[h];
    const int full_off = hbase.z + pref.z, piv_off = hbase.w + pref.w;
    const int B = p.B, D = p.D;
    const T* bK = static_cast<const T*>(p.buf_K);
    const T* bV = static_cast<const T*>(p.buf_V);
    T* pK = static_cast<T*>(p.piv_K);
    T* pV = static_cast<T*>(p.piv_V);
    // (asked for as soon as its place is known, a lane per buffered token and per pivot)
    const int npiv = p.piv_row_cnt[r];
    int my_seg = -1, ps_l = -1;        // lane c < B: segment of column c; lane q < P: of pivot q
    if (sub < B) my_seg = p.buf_row_seg[r * B + sub];
    if (npiv >= p.P && sub < p.P) ps_l = p.piv_row_seg[r * p.P + sub];
    // ---- the buffer is full: B tokens -> one pivot (stac/merger.py:408-461)
    float ts = 0.f, pw_l = INFINITY;   // lane q < P of a saturated row: weight of pivot q
    if (sub < B) {
      ts = fmaxf(p.buf_S[my_seg], 1e-6f);
      if (ahead) prefetch_row<T>(reinterpret_cast<uintptr_t>(bK + static_cast<long long>(my_seg) * D));
      if (ahead) prefetch_row<T>(reinterpret_cast<uintptr_t>(bV + static_cast<long long>(my_seg) * D));
    }
    if (ps_l >= 0) {
      pw_l = p.piv_W[ps_l];
      if (ahead) prefetch_row<T>(reinterpret_cast<uintptr_t>(pK + static_cast<long long>(ps_l) * D));
      if (ahead) prefetch_row<T>(reinterpret_cast<uintptr_t>(pV + static_cast<long long>(ps_l) * D));
    }
    int seed = 0;
    float seed_s = -INFINITY, sumS = 0.f;
    for (int c = 0; c < B; ++c) {
      const float sc = __shfl_sync(gmask, ts, gbase + c);
      if (sc > seed_s) {
        seed_s = sc;
        seed = c;
      }
      sumS = __fadd_rn(sumS, sc);
    }
    float kn_seed[8];
    {
      const int sg = __shfl_sync(gmask, my_seg, gbase + seed);
      float k[8];
      row8_load(bK + static_cast<long long>(sg) * D, sub, k);
      float ss = 0.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) ss += k[e] * k[e];
      const float den = fmaxf(sqrtf(group8_sum(ss, gmask)), 1e-6f);
#pragma unroll
      for (int e = 0; e < 8; ++e) kn_seed[e] = __fdiv_rn(k[e], den);
    }
    // pass 1 over the keys: w_c = exp(cos(k_c, seed))
    float w[kMaxB];
    float Wsum = 0.f;
#pragma unroll
    for (int c = 0; c < kMaxB; ++c) {
      w[c] = 0.f;
      if (c < B) {
        const int sg = __shfl_sync(gmask, my_seg, gbase + c);
        float k[8];
        row8_load(bK + static_cast<long long>(sg) * D, sub, k);
        float ss = 0.f;
#pragma unroll
        for (int e = 0; e < 8; ++e) ss += k[e] * k[e];
        const float den = fmaxf(sqrtf(group8_sum(ss, gmask)), 1e-6f);
        float d = 0.f;
#pragma unroll
        for (int e = 0; e < 8; ++e) d += __fdiv_rn(k[e], den) * kn_seed[e];
        d = fminf(1.f, fmaxf(-1.f, group8_sum(d, gmask)));
        w[c] = expf(d);
        Wsum = __fadd_rn(Wsum, w[c]);
      }
    }
    // pass 2: the weighted means of keys and values
    float nk[8], nv[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) nk[e] = nv[e] = 0.f;
    const float wden = __fadd_rn(Wsum, 1e-8f);
#pragma unroll
    for (int c = 0; c < kMaxB; ++c) {
      if (c < B) {
        const float cn = __fdiv_rn(w[c], wden);
        const int sg = __shfl_sync(gmask, my_seg, gbase + c);
        float tk[8], tv[8];
        row8_load(bK + static_cast<long long>(sg) * D, sub, tk);
        row8_load(bV + static_cast<long long>(sg) * D, sub, tv);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          nk[e] = __fadd_rn(nk[e], __fmul_rn(cn, tk[e]));
          nv[e] = __fadd_rn(nv[e], __fmul_rn(cn, tv[e]));
        }
      }
    }
    // ---- insert the pivot (stac/merger.py:462-582)
    int pseg;
    if (npiv < p.P) {
      pseg = p.plan[kPlanPivTop] + piv_off;
      if (sub == 0) {
        p.piv_row_seg[r * p.P + npiv] = pseg;
        p.piv_row_cnt[r] = npiv + 1;
      }
    } else {
      // saturated: fold the lowest-weight pivot into its most similar neighbour, reuse its slot
      int victim = 0;
      float wmin = INFINITY;
      for (int q = 0; q < p.P; ++q) {
        const float wq = __shfl_sync(gmask, pw_l, gbase + q);
        if (wq < wmin) {
          wmin = wq;
          victim = q;
        }
      }
      // keys normalised in the pool dtype, as the reference does here (stac/merger.py:493-495)
      auto load_normalised = [&](int seg, float (&out)[8]) {
        float pk[8];
        row8_load(pK + static_cast<long long>(seg) * D, sub, pk);
        float ss = 0.f;
#pragma unroll
        for (int e = 0; e < 8; ++e) ss += pk[e] * pk[e];
        float nrm = Elem<T>::round(sqrtf(group8_sum(ss, gmask)));
        nrm = fmaxf(nrm, Elem<T>::round(1e-6f));
#pragma unroll
        for (int e = 0; e < 8; ++e) out[e] = Elem<T>::round(__fdiv_rn(pk[e], nrm));
      };
      const int vseg = __shfl_sync(gmask, ps_l, gbase + victim);
      const float Wv = __shfl_sync(gmask, pw_l, gbase + victim);
      float vn[8];
      load_normalised(vseg, vn);
      int nb = 0;
      float best = -INFINITY;
      for (int q = 0; q < p.P; ++q) {
        if (q == victim) continue;
        const int qseg = __shfl_sync(gmask, ps_l, gbase + q);
        float pkn[8];
        load_normalised(qseg, pkn);
        float d = 0.f;
#pragma unroll
        for (int e = 0; e < 8; ++e) d += pkn[e] * vn[e];
        d = Elem<T>::round(group8_sum(d, gmask));
        if (d > best) {
          best = d;
          nb = q;
        }
      }
      if (p.P == 1) nb = victim;   // no neighbour to fold into: the victim is simply replaced
      float scale;
      if (Elem<T>::kIsBf16) scale = Elem<T>::round(expf(Elem<T>::round(best - 1.0f)));
      else scale = expf(best - 1.0f);
      const int nseg = __shfl_sync(gmask, ps_l, gbase + nb);
      const float Wn = __shfl_sync(gmask, pw_l, gbase + nb);
      if (p.P > 1) {
        const float Wj = __fmul_rn(Wv, scale);
        const float denom = fmaxf(__fadd_rn(Wj, Wn), 1e-8f);
        const float fj = __fdiv_rn(Wj, denom), fk = __fdiv_rn(Wn, denom);
        float a[8], b[8];
        row8_load(pK + static_cast<long long>(vseg) * D, sub, a);
        row8_load(pK + static_cast<long long>(nseg) * D, sub, b);
#pragma unroll
        for (int e = 0; e < 8; ++e) b[e] = __fadd_rn(__fmul_rn(fj, a[e]), __fmul_rn(fk, b[e]));
        row8_store(pK + static_cast<long long>(nseg) * D, sub, b);
        row8_load(pV + static_cast<long long>(vseg) * D, sub, a);
        row8_load(pV + static_cast<long long>(nseg) * D, sub, b);
#pragma unroll
        for (int e = 0; e < 8; ++e) b[e] = __fadd_rn(__fmul_rn(fj, a[e]), __fmul_rn(fk, b[e]));
        row8_store(pV + static_cast<long long>(nseg) * D, sub, b);
        if (sub == 0) {
          p.piv_W[nseg] = denom;
          p.piv_S[nseg] = __fadd_rn(p.piv_S[vseg], p.piv_S[nseg]);
          p.piv_C[nseg] = __fadd_rn(p.piv_C[vseg], p.piv_C[nseg]);
        }
      }
      pseg = vseg;
    }
    row8_store(pK + static_cast<long long>(pseg) * D, sub, nk);
    row8_store(pV + static_cast<long long>(pseg) * D, sub, nv);
    if (sub == 0) {
      p.piv_W[pseg] = Wsum;
      p.piv_S[pseg] = sumS;
      p.piv_C[pseg] = static_cast<float>(B);
    }
    // ---- release the buffer row: segment ids go to the staging area in column order
    if (sub < B) {
      p.free_stage[full_off * B + sub] = my_seg;
      p.buf_row_seg[r * B + sub] = -1;
    }
    if (sub == 0) p.buf_row_cnt[r] = 0;
  }
}

// A warp per row while those are two waves of warps at most (9472 on 148 SMs).  (us, eight lanes and a warp per row, rows with room for the pivot
// and, behind the comma, without: 960 rows 15.5, 20.8 and 7.1, 10.0; 4800 16.3, 21.9 and 11.7, 17.7; 12000 17.5, 25.7 and 19.1, 30.3; 16000 19.5, 28.9
// and 24.0, 39.4; 38400 52.8, 76.5 and 57.5, 90; fp32, 4800 16.5, 22.6 and 12.9, 19.5; 16000 24.5, 34.7 and 29.9, 45.6.  Rows that a stream
// of 48 heads has left in DRAM: 8911 25.1 and 22.9, a stream of 384 heads: 27 thousand 49 and 44, 34 thousand 93 and 101.)
constexpr int kManyFullRows = 9472;
template <typename T>
__global__ void __launch_bounds__(128, 8) rows_phase_b2_kernel(const MergeParams p) {
  grid_dep_wait();   // launched with programmatic serialization behind the previous kernel of the call
  if (p.plan[kPlanAnyValid] == 0 || p.plan[kPlanAbort] != 0) return;
  const int n_full = p.plan[kPlanFullCount];
  if (n_full < kManyFullRows) full_rows_by_warps<T>(p, n_full);
  else full_rows_by_groups<T>(p, n_full);
}

// Freed ids are appended after the part of the free list that was not handed out.  Without a valid
// evicted token in the whole call the reference returns before touching the carried overflow
// (stac/merger.py:1203-1208), so the list is carried over unchanged.
template <typename T>
__global__ void finalize_kernel(const MergeParams p) {
  grid_dep_wait();   // launched with programmatic serialization behind the previous kernel of the call
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
  const long long first = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (p.plan[kPlanAnyValid] != 0 && p.plan[kPlanAbort] == 0) {
    const int n_freed = p.plan[kPlanTotalFull] * p.B;
    const int base = p.plan[kPlanFreeLen] - p.plan[kPlanK];
    for (long long i = first; i < n_freed; i += stride) p.buf_free[base + i] = p.free_stage[i];
    return;
  }
  const int n = p.over_start_in[p.heads];
  const long long total = static_cast<long long>(n) * p.D;
  for (long long i = first; i < total; i += stride) {
    static_cast<T*>(p.over_K_out)[i] = static_cast<const T*>(p.over_K_in)[i];
    static_cast<T*>(p.over_V_out)[i] = static_cast<const T*>(p.over_V_in)[i];
  }
  for (long long i = first; i < n; i += stride) {
    p.over_S_out[i] = p.over_S_in[i];
    p.over_hv_out[2 * i] = p.over_hv_in[2 * i];
    p.over_hv_out[2 * i + 1] = p.over_hv_in[2 * i + 1];
  }
  for (long long i = first; i <= p.heads; i += stride) p.over_start_out[i] = p.over_start_in[i];
}

size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

struct ScratchLayout {
  size_t keys_a, keys_b, vals_a, vals_b, n_tok, n_rows, row_vx, row_start, row_info, row_pref, old_dest, tok_dest,
      tok_sim, tok_score, head_tot, head_base, plan, free_stage, full_list, move_list, tok_row, tok_best, row_flag, merge_list, total;
};

ScratchLayout scratch_layout(int heads, int ncap, int buf_cap) {
  ScratchLayout L;
  size_t off = 0;
  const size_t hn = static_cast<size_t>(heads) * ncap;
  auto take = [&](size_t bytes) {
    const size_t o = off;
    off = align_up(off + bytes, 256);
    return o;
  };
  L.keys_a = take(hn * 4); L.keys_b = take(hn * 4); L.vals_a = take(hn * 4); L.vals_b = take(hn * 4);
  L.n_tok = take(static_cast<size_t>(heads) * 4); L.n_rows = take(static_cast<size_t>(heads) * 4);
  L.row_vx = take(hn * 4); L.row_start = take(static_cast<size_t>(heads) * (ncap + 1) * 4);
  L.row_info = take(hn * 16); L.row_pref = take(hn * 16); L.old_dest = take(hn * kMaxB * 4);
  L.tok_dest = take(hn * 4); L.tok_sim = take(hn * 4); L.tok_score = take(hn * 4);
  L.head_tot = take(static_cast<size_t>(heads) * 16); L.head_base = take(static_cast<size_t>(heads) * 16);
  L.plan = take(kPlanSize * 4); L.free_stage = take(static_cast<size_t>(buf_cap) * 4);
  L.full_list = take(hn * 8);
  L.move_list = take(hn * 8); L.tok_row = take(hn * 4);
  L.tok_best = take(hn * 4); L.row_flag = take(hn * 4); L.merge_list = take(hn * 8);
  L.total = off;
  return L;
}

// One wave of CTAs wherever there can be one, a second wave costs as much as the first: a head has an SM to itself or shares it
// with one other head (9216 tokens: what 32 warps hold in nine registers per lane, and twice that with the counters in an SM's shared
// memory), with two (8704), or with three (2048, of which 1536 evicted and the rest carried ones).  Lists beyond that, voxel
// ids above 16 bits and more heads with longer lists are sorted in global memory by the same CTAs, and take what they took before
// there was a sort in shared memory (us, before and now: 16 heads, 9216 and 260 carried tokens 41.7, 41.6; 12492 58.6, 56.7; 16
// heads, 8328 of 70000 voxels 44.3, 41.7; 384 heads, 12492 172, 173; 500 heads, 4164 104, 104; 768 heads, 2082 50.6, 50.5).
cudaError_t launch_sort(MergeParams& mp, int dev, int n_sm, cudaStream_t st) {
  auto launch = [&](auto* kernel, int threads, int items, int per_sm) {
    const int digits = (257 * (threads / 32) + threads * items) * 4, counters = ((mp.voxel_used + 1) / 2 * 2 + threads * items) * 4;
    // A counter per voxel where they fit and there are neither many more voxels than tokens, for whose counters the scan
    // walks, nor so few that rows are long.  (us, 16 and 384 heads of 1041 tokens: 3600 voxels 9.0 -> 7.4 and 14.5 -> 11.4, 5500 8.9 -> 8.4 and 14.5 -> 13.1,
    // 7200 level; 20 voxels, rows of 52, 384 heads 16.8 -> 19.7.)
    mp.counted = items > 0 && mp.voxel_used < 0xFFFF && mp.voxel_used <= 6ll * mp.n_new && 8ll * mp.voxel_used >= mp.n_new &&
                 (counters + 2048) * per_sm <= 220 * 1024 ? 1 : 0;
    return launch_behind(kernel, dim3(mp.heads), dim3(threads), mp.counted && counters > digits ? counters : digits, st, mp);
  };
  static PerDeviceFlag attr_done;       // the shared-memory opt-in is made once per device
  if (attr_done.needs_setup(dev)) {
    for (auto* kernel : {sort_tokens_kernel<1024, 1, 9>, sort_tokens_kernel<1024, 2, 9>, sort_tokens_kernel<512, 3, 17>,
                         sort_tokens_kernel<512, 4, 4>}) {
      const cudaError_t rc = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
      if (rc != cudaSuccess) return rc;
    }
    attr_done.mark(dev);
  }
  if (mp.heads <= n_sm) return launch(sort_tokens_kernel<1024, 1, 9>, 1024, 9, 1);
  if (mp.heads <= 2 * n_sm) return launch(sort_tokens_kernel<1024, 2, 9>, 1024, 9, 2);
  if (mp.heads <= 4 * n_sm && mp.n_new <= 1536) return launch(sort_tokens_kernel<512, 4, 4>, 512, 4, 4);   // (512 carried ones)
  if (mp.heads <= 3 * n_sm) return launch(sort_tokens_kernel<512, 3, 17>, 512, 17, 3);
  return launch(sort_tokens_kernel<512, 4, 0>, 512, 0, 4);
}

template <typename T>
int launch_merge(MergeParams& mp, cudaStream_t st) {
  if (cudaMemsetAsync(mp.plan, 0, kPlanSize * 4, st) != cudaSuccess) return STAC_ERR_CUDA;
  int dev, n_sm;
  if (current_device(&dev) != STAC_OK || device_sm_count(dev, &n_sm) != STAC_OK) return STAC_ERR_CUDA;
  if (launch_sort(mp, dev, n_sm, st) != cudaSuccess) return STAC_ERR_CUDA;
  dim3 grid_a1((mp.ncap + 255) / 256, mp.heads);
  dim3 grid_tok((mp.ncap + kTokBlock - 1) / kTokBlock, mp.heads);
  if (launch_behind(tokens_sim_merge_kernel<T>, grid_tok, dim3(kTokBlock), 0, st, mp) != cudaSuccess) return STAC_ERR_CUDA;
  if (launch_behind(rows_merge_kernel<T>, dim3(n_sm * 4), dim3(256), 0, st, mp) != cudaSuccess) return STAC_ERR_CUDA;
  // (four CTAs per SM hold a thread per token: no row waits for a place)
  const bool few_rows = static_cast<long long>(mp.heads) * mp.n_new <= 4ll * 256 * n_sm;
  if (launch_behind(few_rows ? rows_rank_kernel<4> : rows_rank_kernel<6>, dim3(grid_a1), dim3(256), 0, st, mp) != cudaSuccess)
    return STAC_ERR_CUDA;
  // (a CTA per head: with more than two per SM those of 512 threads are one wave; 384 heads, both launches
  // 55.1 -> 38.3 us in a bounded memory, 21.5 -> 15.6 in a stream of chunks of four frames)
  const bool two_per_sm = mp.heads <= 2 * n_sm;
  for (int pass = 0; pass < 2; ++pass)
    if (launch_behind(two_per_sm ? scan_rows_kernel<1024> : scan_rows_kernel<512>, dim3(mp.heads), dim3(two_per_sm ? 1024 : 512), 0, st,
                      mp, pass) != cudaSuccess)
      return STAC_ERR_CUDA;
  if (launch_behind(rows_phase_b1a_kernel, dim3(grid_a1), dim3(256), 0, st, mp) != cudaSuccess) return STAC_ERR_CUDA;
  if (launch_behind(rows_phase_b1m_kernel<T, 2>, dim3(n_sm * 6), dim3(256), 0, st, mp) != cudaSuccess) return STAC_ERR_CUDA;
  if (launch_behind(tokens_place_kernel<T>, grid_tok, dim3(kTokBlock), 0, st, mp) != cudaSuccess) return STAC_ERR_CUDA;
  // (two waves: eight CTAs per SM are resident)
  if (launch_behind(rows_phase_b2_kernel<T>, dim3(n_sm * 16), dim3(128), 0, st, mp) != cudaSuccess) return STAC_ERR_CUDA;
  // (grid-stride over the freed ids, whose number only the device knows)
  if (launch_behind(finalize_kernel<T>, dim3(n_sm * 4), dim3(256), 0, st, mp) != cudaSuccess) return STAC_ERR_CUDA;
  return cudaGetLastError() == cudaSuccess ? STAC_OK : STAC_ERR_CUDA;
}

}  // namespace
}  // namespace stac

extern "C" {

size_t stac_merge_scratch_bytes(int heads, int tokens_per_head, int buf_cap) {
  if (heads <= 0 || tokens_per_head <= 0 || buf_cap < 0) return 0;
  return stac::scratch_layout(heads, tokens_per_head, buf_cap).total;
}

int stac_merge_insert(const stac_pool* pool, const stac_evicted* ev, void* scratch, size_t scratch_bytes,
                      int list_cap_per_head, int* dev_status, stac_stream_t stream) {
  if (pool == nullptr || ev == nullptr || scratch == nullptr) return STAC_ERR_BAD_ARG;
  if (pool->head_dim != 64 || (pool->elem_bytes != 2 && pool->elem_bytes != 4)) return STAC_ERR_BAD_ARG;
  if (pool->pivot_cap < 1 || pool->pivot_cap > stac::kMaxP || pool->budget_cap < 1 ||
      pool->budget_cap > stac::kMaxB)
    return STAC_ERR_BAD_ARG;
  if (pool->heads <= 0 || pool->voxel_cap <= 0 || pool->voxel_used < 0 || pool->voxel_used > pool->voxel_cap)
    return STAC_ERR_BAD_ARG;
  if (ev->tokens_per_head <= 0 || list_cap_per_head < ev->tokens_per_head || list_cap_per_head > STAC_MERGE_MAX_LIST)
    return STAC_ERR_BAD_ARG;
  const stac::ScratchLayout L = stac::scratch_layout(pool->heads, list_cap_per_head, pool->buf_cap);
  if (scratch_bytes < L.total) return STAC_ERR_CAPACITY;
  stac::MergeParams mp;
  mp.heads = pool->heads; mp.D = pool->head_dim; mp.P = pool->pivot_cap; mp.B = pool->budget_cap;
  mp.voxel_cap = pool->voxel_cap; mp.voxel_used = pool->voxel_used;
  mp.sim_thresh = pool->sim_thresh; mp.replace_thresh = pool->replace_thresh; mp.score_thresh = pool->score_thresh;
  mp.k_src = ev->k; mp.v_src = ev->v; mp.s_src = ev->scores; mp.vx_src = ev->voxel_ids; mp.idx = ev->positions;
  mp.src_head_stride = ev->kv_head_stride; mp.src_row_stride = ev->kv_row_stride;
  mp.meta_head_stride = ev->meta_head_stride; mp.n_new = ev->tokens_per_head;
  mp.buf_K = pool->buf_K; mp.buf_V = pool->buf_V; mp.buf_S = pool->buf_S;
  mp.buf_row_seg = pool->buf_row_seg; mp.buf_row_cnt = pool->buf_row_cnt; mp.buf_free = pool->buf_free;
  mp.buf_cap = pool->buf_cap;
  mp.piv_K = pool->piv_K; mp.piv_V = pool->piv_V; mp.piv_W = pool->piv_W; mp.piv_S = pool->piv_S;
  mp.piv_C = pool->piv_C; mp.piv_row_seg = pool->piv_row_seg; mp.piv_row_cnt = pool->piv_row_cnt;
  mp.piv_cap = pool->piv_cap;
  mp.over_K_in = pool->over_K_in; mp.over_V_in = pool->over_V_in; mp.over_S_in = pool->over_S_in;
  mp.over_hv_in = pool->over_hv_in; mp.over_start_in = pool->over_start_in;
  mp.over_K_out = pool->over_K_out; mp.over_V_out = pool->over_V_out; mp.over_S_out = pool->over_S_out;
  mp.over_hv_out = pool->over_hv_out; mp.over_start_out = pool->over_start_out; mp.over_cap = pool->over_cap;
  mp.meta = pool->meta;
  mp.voxel_count = pool->voxel_count;
  mp.ncap = list_cap_per_head;
  char* base = static_cast<char*>(scratch);
  mp.keys_a = reinterpret_cast<unsigned int*>(base + L.keys_a);
  mp.keys_b = reinterpret_cast<unsigned int*>(base + L.keys_b);
  mp.vals_a = reinterpret_cast<int*>(base + L.vals_a);
  mp.vals_b = reinterpret_cast<int*>(base + L.vals_b);
  mp.n_tok = reinterpret_cast<int*>(base + L.n_tok);
  mp.n_rows = reinterpret_cast<int*>(base + L.n_rows);
  mp.row_vx = reinterpret_cast<int*>(base + L.row_vx);
  mp.row_start = reinterpret_cast<int*>(base + L.row_start);
  mp.row_info = reinterpret_cast<int4*>(base + L.row_info);
  mp.row_pref = reinterpret_cast<int4*>(base + L.row_pref);
  mp.old_dest = reinterpret_cast<int*>(base + L.old_dest);
  mp.tok_dest = reinterpret_cast<int*>(base + L.tok_dest);
  mp.tok_sim = reinterpret_cast<float*>(base + L.tok_sim);
  mp.tok_score = reinterpret_cast<float*>(base + L.tok_score);
  mp.head_tot = reinterpret_cast<int4*>(base + L.head_tot);
  mp.head_base = reinterpret_cast<int4*>(base + L.head_base);
  mp.plan = reinterpret_cast<int*>(base + L.plan);
  mp.free_stage = reinterpret_cast<int*>(base + L.free_stage);
  mp.full_list = reinterpret_cast<int2*>(base + L.full_list);
  mp.long_list = mp.full_list;
  mp.move_list = reinterpret_cast<int2*>(base + L.move_list);
  mp.tok_row = reinterpret_cast<int*>(base + L.tok_row);
  mp.tok_best = reinterpret_cast<int*>(base + L.tok_best);
  mp.row_flag = reinterpret_cast<int*>(base + L.row_flag);
  mp.merge_list = reinterpret_cast<int2*>(base + L.merge_list);
  int bits = 1;
  while ((1ll << bits) < pool->voxel_used) ++bits;
  mp.passes = (bits + 7) / 8;
  mp.buf_seg_vec = mp.B == stac::kMaxB && (reinterpret_cast<uintptr_t>(mp.buf_row_seg) & 15) == 0 ? 1 : 0;
  mp.minus_zero = -0.f;
  mp.seg_vec = mp.P == 4 && (reinterpret_cast<uintptr_t>(mp.piv_row_seg) & 15) == 0 ? 1 : 0;
  mp.err = dev_status;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (pool->elem_bytes == 2) return stac::launch_merge<__nv_bfloat16>(mp, st);
  return stac::launch_merge<float>(mp, st);
}

}  // extern "C"
