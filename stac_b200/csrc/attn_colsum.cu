// Window + pivot attention with per-key softmax column sums (H2O scores), head_dim 64, bf16.
//
// Replaces the reference's attn_cuda.flash_attn_bias_colsum (attn-cuda/csrc/launch.cu:87-158,
// kernels fwd_kernel.h:78-485 and colsum_kernel.h:22-325) and its Triton twin
// (stac/flash_attn_triton.py:900-1006).  Semantics: S = q k^T * scale + bias[n], softmax over
// the keys, O = P v, lse = logsumexp, colsum[n] = sum over (optionally strided) query rows of
// exp(S - lse) times M / M_sub.  Keys come from two segments that are never concatenated in
// memory: the hot cache rows [0, T_hot) of a head and the retrieved pivots [0, T_ret) with a
// per-key bias (log C, or -inf for padding).
//
// Two kernels, both tcgen05 + TMA:
//   attn_fwd_fast_kernel  items (128 query rows, head): S = Q K^T into TMEM, probabilities relative
//                       to one fixed reference per row back into TMEM, O += P V there.
//   attn_colsum_kernel  items (up to three 128-key tiles, head): S^T = K Q^T into TMEM so that each thread
//                       owns one key (TMEM lane) and sums exp2(S^T - lse[m]) over the query
//                       columns in registers: no shuffles, no atomics, deterministic.
#include <type_traits>

#include "common.cuh"
#include "stac_internal.h"

namespace stac {

namespace {

constexpr int kD = 64;
constexpr int kBM = 128;
constexpr int kBN = 128;
constexpr int kTileBytes = 128 * 128;  // 128 rows x 64 bf16
constexpr int kColGroup = 3;           // key tiles per item = exponent warpgroups of the column-sum kernel (two or one in short calls)
constexpr int kColStages = 4;
constexpr int col_threads(int group) { return 128 + group * 128; }   // warpgroup 0 control (warp 0 TMA, warp 1 MMA issue), then exponent
#ifndef STAC_COL_PAIR_MASK
#define STAC_COL_PAIR_MASK 0x88
#endif
// which of 8 consecutive PAIRS of exponentials of the column-sum kernel run on the FMA pipes
constexpr unsigned kColPairMask = STAC_COL_PAIR_MASK;
#ifndef STAC_COL_FOLD_LSE
#define STAC_COL_FOLD_LSE 1
#endif
// 1: the row term -lse2[m] of the exponent is added to the score tile by the tensor core (a fifth
// K = 16 step whose operands are a tile of ones and the row values split into three bf16), so the
// exponent warps read nothing from shared memory; 0: they read it per score (LDS.128 per four).
constexpr bool kColFoldLse = STAC_COL_FOLD_LSE != 0;
constexpr int kColXBytes = 128 * 32;   // 128 rows x 16 bf16, no swizzle: [16 row groups][2 K chunks][8 rows][16 B]
constexpr int kColCtlRegs = 56, kColExpRegs = 152;
// setmaxnreg only moves registers inside the CTA's allocation, which is fixed at launch to
// (registers per thread the launch bound allows, a multiple of 8) x threads.  A request beyond
// what the control warpgroup released would wait forever.
constexpr int kColLaunchRegs = (65536 / col_threads(kColGroup)) / 8 * 8;
static_assert(128 * kColCtlRegs + 128 * kColGroup * kColExpRegs <= col_threads(kColGroup) * kColLaunchRegs,
              "column-sum kernel: setmaxnreg targets exceed the CTA's register allocation");
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;

struct FwdParams {
  int M, H;
  int T_hot, T_ret;
  float scale_log2;
  const float* bias_ret;
  long long bias_head_stride;
  __nv_bfloat16* out;
  long long out_row_stride;  // elements between query rows
  float* lse;                // [H, M] natural log or nullptr
  float* lse2;               // [H, lse2_stride] log2 domain
  long long lse2_stride;
  int* err;
  // items = (head, 128-row query tile), head-major
  int n_q_tiles, n_items;
  int split;                 // 1: the (item, key tile) units are cut evenly over the grid
  float* part;               // split == 1: two partial-result slots per CTA
  int* part_count;           // split == 1: one arrival counter per cut between CTA c and c + 1 (parts > 1: per item), zero on entry, left zero
  int parts;                 // > 1 (and split == 1): every item is cut in so many parts, a CTA each
  int cluster;               // parts > 1: they are joined through the shared memory of a cluster of `parts` CTAs (1), or the workspace (0)
  // column sums that the column-sum kernel will accumulate with atomic adds: cleared here
  float* zero_colsum;        // [H, zero_stride], entries [0, zero_width) of every head; or nullptr
  long long zero_stride;
  int zero_width;
};

__device__ __forceinline__ uint8_t* align1024(uint8_t* p) {
  return reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(p) + 1023) & ~static_cast<uintptr_t>(1023));
}

#ifdef STAC_TIMESTAMPS
// Debug build only: first start and last end of each kernel on the GPU's nanosecond timer.
__device__ unsigned long long g_ts[8] = {~0ull, 0ull, ~0ull, 0ull, ~0ull, 0ull, ~0ull, 0ull};
__device__ __forceinline__ void ts_mark(int k, bool end) {
  if (threadIdx.x == 0) {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    if (end) atomicMax(&g_ts[2 * k + 1], t);
    else atomicMin(&g_ts[2 * k], t);
  }
}
#define STAC_TS(k, end) ts_mark(k, end)
#else
#define STAC_TS(k, end)
#endif

// ---------------------------------------------------------------------------------------
// Fast forward kernel.  Softmax is invariant to the reference subtracted before the exponent,
// so instead of a running maximum every row uses ONE reference: the exact maximum of its
// first key tile.  Nothing is ever rescaled: P V accumulates in TMEM across all key tiles of
// the row block, the softmax warpgroups (four) take key tiles round-robin and keep only a partial
// row sum each.  The scheme is exact as long as no later score exceeds the reference by more
// than 2^60 (probabilities then stay far inside the bf16 / fp32 range).  A CTA with a row whose sum of
// probabilities leaves that range walks its units a second time, every segment twice: once for the exact row maxima,
// once for the probabilities relative to them; a part of an item that would be joined waits for that.
// (A kernel behind this one that recomputed flagged calls, and returned at once otherwise, cost every call a launch
// and the completion of one more grid: M 1041, N 2082, 16 heads 34.7 -> 32.4 us per call, M 4164, 2 heads 98.5 -> 96.0.
// Calls that all CTAs walk twice: M 1041, N 10410 213 -> 201 us, M 4164, N 17697 1314 -> 1112.)
//
// Shared memory carries only the operands TMA brings in.  Key tiles are 112 keys wide so that
// FOUR score buffers fit beside the output accumulator in the 512 TMEM columns (4 x 112 + 64):
// with four softmax warpgroups each has a buffer of its own and the other three keep the
// exponential unit busy while one waits for its buffer to go through P V and the next Q K^T.
// The probabilities go back into the columns their scores came from (bf16, two per column) and feed
// the P V MMA as its A operand straight from tensor memory.
//
// The scores of tile c + kFastWgs overwrite the probabilities of tile c, which P V reads.  tcgen05.mma instructions
// are only ordered among themselves where they have the accumulator and the shape in common, and these two have neither, so
// the warp that issues Q K^T waits for the commit of that P V: a warp each for the two streams, because a single warp that
// waits between them leaves the tensor pipe idle (M = 1041, N = 2082 38.1 against 37.1 us per call, M = 2000, N = 900 58.4
// against 55.8).  The warps that issue and load share their schedulers with the softmax warps, so their loops hold little
// beside the waits.  (One warp that issues both without a wait in between gave the same bits and took 0.4 to
// 1.5 % less of this kernel's time at 9369 keys and more, 2 % with a bias on every key, but relied on an order that is
// observed and not documented.  Measured and not taken: three softmax warpgroups with
// probabilities in columns of their own, 96-key tiles, 10 % slower; larger FMA shares of the exponentials, no less time.)
//
// Work = items (head, 128-row query tile) x key tiles.  With enough items the kernel runs one
// CTA per SM and cuts that unit sequence into equal contiguous ranges (no partly filled last
// wave); a CTA walks its range segment by segment, a segment being a run of key tiles of one
// item.  An item on a cut is computed in two parts by two CTAs, each with its own row
// references; the CTA that arrives first at a cut leaves its part (unnormalised accumulator, row sums, references) in a
// workspace, and the one that arrives second joins it with its own, which stays in registers (plain
// split-softmax algebra, operands in a fixed order: same bits whichever CTA does it).  Cuts cost a call about 3 us
// (6 when both parts went through memory, rows of 256 bytes per thread).  With at
// most half as many items as SMs every item is cut in equal parts instead, a CTA each, which are joined behind the walk: by a cluster through
// its shared memory, or through the workspace by the CTA whose part comes last (see fwd_parts).  Barrier
// phases, the stages and the score buffers run on across segments; the query tile, the row references and the
// partial row sums are double buffered by segment parity, and so are the barriers that several warpgroups
// arrive on per segment: a warpgroup without a tile in a short first or last segment runs one segment ahead,
// never two (a CTA's middle segments are whole items of at least kFastMinSplitTiles tiles: the scores of a
// warpgroup's last tile there wait for a P V of that segment, whose first one waits until the
// accumulator of the segment before has been read out).
// ---------------------------------------------------------------------------------------
constexpr int kFastWgs = 4;                     // softmax warpgroups; key tile c goes to warpgroup and score buffer c % kFastWgs
constexpr int kFastThreads = 128 + 128 * kFastWgs;   // warpgroup 0 control (warps 0 and 3 TMA, warps 1 and 2 MMA issue), then softmax
constexpr int kFT = 112;                        // keys per tile: three chunks of 32 and one of 16
static_assert(kFT % 32 == 16 && kFT <= kBN && kFastWgs * kFT + kD <= 512, "tensor memory");
constexpr int kFastTileBytes = kFT * 128;       // kFT rows x 64 bf16
constexpr float kFastRowSumLimit = 1.152921504606846976e18f;  // 2^60
constexpr int kPartFloats = kBM * kD + 2 * kBM; // one partial result: O[128][64], row sums, row references
constexpr int kFastMaxCtas = 160;               // partial-result slots are provided for this many CTAs
// shorter key ranges run one CTA per item; every warpgroup has a tile at least kFastWgs tiles into a
// middle segment, i.e. one whose score buffer was last used inside the same segment
constexpr int kFastMinSplitTiles = 2 * kFastWgs;
constexpr int kFastMaxCluster = 8;              // the portable size
static_assert(kPartFloats * 4 <= kFastWgs * kFastTileBytes, "a part that a cluster joins lies where the key tiles were");
constexpr float kFastTileUs = 0.52f, kFastPartUs = 0.42f, kFastClusterUs = 2.2f, kFastWorkspaceUs = 3.2f;
#ifndef STAC_FAST_PAIR_MASK
#define STAC_FAST_PAIR_MASK 0x8080u
#endif
constexpr unsigned kFastPairMask = STAC_FAST_PAIR_MASK;   // which of 16 consecutive PAIRS of exponentials run on the FMA pipes
// setmaxnreg targets; must fit the launch allocation
constexpr int kFastCtlRegs = 64, kFastSoftmaxRegs = 104;
static_assert(128 * kFastCtlRegs + 128 * kFastWgs * kFastSoftmaxRegs <= kFastThreads * ((65536 / kFastThreads) / 8 * 8),
              "fast forward kernel: setmaxnreg targets exceed the CTA's register allocation");

struct FastSmem {
  uint8_t q[2][kTileBytes];                     // query tile of the segment (parity)
  uint8_t k[kFastWgs][kFastTileBytes];
  uint8_t v[kFastWgs][kFastTileBytes];
  float bias2[kFastWgs][kBN];
  float m_ref[2][kBM];                          // row references of the segment (parity)
  float lpart[2][kFastWgs][kBM];                // row sums of the warpgroups (segment parity)
  int live[2][kFastWgs];                        // did a warpgroup see a key that is not masked (segment parity)
  uint64_t q_full[2];
  uint64_t q_empty[2];
  uint64_t k_full[kFastWgs];
  uint64_t v_full[kFastWgs];
  uint64_t s_full[kFastWgs];     // scores of a tile are in TMEM; the place of its keys is free again
  uint64_t p_full[kFastWgs];     // its probabilities are in TMEM
  uint64_t pv_done[kFastWgs];    // the P V MMAs that read them are done: scores may overwrite them, values theirs
  uint64_t ref_ready[2];
  uint64_t l_ready[2];           // the other warpgroups have published their row sums of the segment (parity)
  uint64_t o_done;               // all P V MMAs of the segment are complete
  uint64_t o_free;               // the segment's accumulator has been read out of TMEM
  uint32_t tmem_base;
  int join_all;                  // parts > 1, through the workspace: this CTA's part was the last one of its item
  int join_flag[kFastWgs];       // arrival count seen at a cut (1: the other part is complete), of the warpgroup that closes a segment
  int again;                     // a row's reference did not do: the CTA walks its segments again with exact ones
  int part_again[2];             // the part that this CTA would leave in slot 0 / 1 waits for that
};

// The (item, key tile) units of one CTA, walked segment by segment: a segment is a run of key
// tiles [t0, t1) of one item.  With `split` the units of the whole launch are cut into equal
// contiguous ranges, one per CTA: an item on a cut is then finished by two CTAs, or, with parts > 1 and parts * n_items CTAs,
// every item by `parts` CTAs.  A cut total * c / (parts * n_items) = nt * c / parts falls on an item's end wherever c is a multiple of
// `parts`, so that each of those CTAs has one segment, of one tile at least (parts <= nt): its part may lie in one place, and is
// joined behind the walk.  Without `split` CTA i owns item i.  Every role of the CTA walks the same sequence.
struct FwdWalk {
  int item, t0, left, nt;     // next item, its first tile, tiles of the CTA that are left, tiles per item
  __device__ FwdWalk(const FwdParams& p, int n_tiles) {
    nt = n_tiles;
    if (p.split) {
      const long long total = static_cast<long long>(p.n_items) * nt;
      const long long u = total * blockIdx.x / gridDim.x;
      left = static_cast<int>(total * (blockIdx.x + 1) / gridDim.x - u);
      item = static_cast<int>(u / nt);
      t0 = static_cast<int>(u - static_cast<long long>(item) * nt);
    } else {
      left = nt;
      item = blockIdx.x;
      t0 = 0;
    }
  }
  __device__ bool next(int& item_, int& t0_, int& t1_) {
    if (left <= 0) return false;
    item_ = item;
    t0_ = t0;
    t1_ = min(nt, t0 + left);
    left -= t1_ - t0_;
    ++item;
    t0 = 0;
    return true;
  }
};

// kN scores -> kN probabilities relative to the row reference, packed as bf16 pairs.  Scores
// are handled two at a time with the packed fp32 instructions (scale-and-subtract, row sums).
// The pairs whose bit is set in kFastPairMask take their exponentials on the FMA pipes (cubic,
// 8.6e-5 relative, far below the bf16 rounding of P) to relieve the exponential unit.
// Their arguments go into a running maximum: 2^128 and more, which the exponential unit turns into infinities that the
// row sum shows, would wrap there, and NaN would be a probability of zero.
template <int kJ>
__device__ __forceinline__ uint64_t fast_exp_pair(uint64_t x2, float& top) {
  float x0, x1;
  unpack_f32x2(x2, x0, x1);
  if constexpr ((kFastPairMask >> (kJ & 15)) & 1u) {
    top = fmax3_nan(top, x0, x1);
    return poly_exp2_x2(x2);
  }
  return pack_f32x2(fast_exp2(x0), fast_exp2(x1));
}
template <bool kBias, int kN, int kI = 0>
__device__ __forceinline__ void fast_exp_chunk(const uint32_t (&s)[32], uint32_t (&pk)[16], const float* bias2,
                                               uint64_t c2c2, uint64_t negm2, uint64_t& l0, uint64_t& l1, float& top) {
  if constexpr (kI < kN) {
    uint64_t x0 = pack_f32x2(__uint_as_float(s[kI + 0]), __uint_as_float(s[kI + 1]));
    uint64_t x1 = pack_f32x2(__uint_as_float(s[kI + 2]), __uint_as_float(s[kI + 3]));
    if (kBias) {
      const float4 b = *reinterpret_cast<const float4*>(bias2 + kI);
      x0 = add_f32x2(fma_f32x2(x0, c2c2, pack_f32x2(b.x, b.y)), negm2);
      x1 = add_f32x2(fma_f32x2(x1, c2c2, pack_f32x2(b.z, b.w)), negm2);
    } else {
      x0 = fma_f32x2(x0, c2c2, negm2);
      x1 = fma_f32x2(x1, c2c2, negm2);
    }
    const uint64_t e0 = fast_exp_pair<kI / 2>(x0, top), e1 = fast_exp_pair<kI / 2 + 1>(x1, top);
    l0 = add_f32x2(l0, e0);
    l1 = add_f32x2(l1, e1);
    float a0, a1, a2, a3;
    unpack_f32x2(e0, a0, a1);
    unpack_f32x2(e1, a2, a3);
    pk[kI / 2] = pack_bf16x2(a0, a1);
    pk[kI / 2 + 1] = pack_bf16x2(a2, a3);
    fast_exp_chunk<kBias, kN, kI + 4>(s, pk, bias2, c2c2, negm2, l0, l1, top);
  }
}

// The CTA's warps meet behind their walk: is there a second one?
__device__ __forceinline__ bool fwd_again(const FastSmem& sm) {
  named_bar_sync(6, kFastThreads);
  return sm.again != 0;
}

template <int kN>
__device__ __forceinline__ float fast_max_chunk(const uint32_t (&s)[32], const float* bias2, bool need_bias, float c2,
                                                float mx) {
  if (need_bias) {
#pragma unroll
    for (int i = 0; i < kN; ++i) mx = fmaxf(mx, fmaf(__uint_as_float(s[i]), c2, bias2[i]));
  } else {
#pragma unroll
    for (int i = 0; i < kN; i += 2) mx = fmax3(mx, __uint_as_float(s[i]) * c2, __uint_as_float(s[i + 1]) * c2);
  }
  return mx;
}

__global__ void __launch_bounds__(kFastThreads, 1)
attn_fwd_fast_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k_hot,
                     const __grid_constant__ CUtensorMap tm_v_hot, const __grid_constant__ CUtensorMap tm_k_ret,
                     const __grid_constant__ CUtensorMap tm_v_ret, const FwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  FastSmem& sm = *reinterpret_cast<FastSmem*>(align1024(smem_raw));
  STAC_TS(0, false);
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int n_hot = (p.T_hot + kFT - 1) / kFT;
  const int n_tiles = n_hot + (p.T_ret + kFT - 1) / kFT;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&sm.q_full[i], 1);
      mbar_init(&sm.q_empty[i], 1);
      mbar_init(&sm.ref_ready[i], 128);
      mbar_init(&sm.l_ready[i], 128 * (kFastWgs - 1));
    }
    mbar_init(&sm.o_done, 1);
    for (int b = 0; b < kFastWgs; ++b) {
      mbar_init(&sm.k_full[b], 1);
      mbar_init(&sm.v_full[b], 1);
      mbar_init(&sm.s_full[b], 1);
      mbar_init(&sm.p_full[b], 128);
      mbar_init(&sm.pv_done[b], 1);
    }
    mbar_init(&sm.o_free, 128);
    mbar_fence_init();
    sm.again = sm.part_again[0] = sm.part_again[1] = sm.join_all = 0;
  }
  if (warp == 1) {
    tmem_alloc(&sm.tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sm.tmem_base;
  const uint32_t o_tmem = tmem + kFastWgs * kFT;   // 64 columns behind the score buffers
  // Launched with programmatic serialization behind whatever wrote the queries and the cache: barriers
  // and tensor memory are set up while that drains, nothing in global memory is touched before this.
  grid_dep_wait();
  // The kernel behind this one may be scheduled as soon as an SM has room for it (that is,
  // when this CTA has left); it waits for this grid's completion before it reads the row log-sum-exps.
  grid_dep_launch();

  if (p.zero_colsum != nullptr) {
    // a slice of the column-sum output per CTA (the next kernel adds partial sums onto zeros; negative ones, so that the
    // first of two additions to a key can be told from the second, see there)
    const long long total = static_cast<long long>(p.H) * p.zero_width;
    const long long lo = total * blockIdx.x / gridDim.x, hi = total * (blockIdx.x + 1) / gridDim.x;
    for (long long e = lo + threadIdx.x; e < hi; e += kFastThreads) {
      const long long hh = e / p.zero_width;
      p.zero_colsum[hh * p.zero_stride + (e - hh * p.zero_width)] = -0.f;
    }
  }

  if (warp < 4) {
    setmaxnreg_dec<kFastCtlRegs>();
    if (warp == 0) {
      // ---------------------------------------------------------------- TMA producer: Q and K
      int b = 0, par = 1;          // stage of the tile, phase of its previous use
      bool reused = false;
      int seg = 0;
      for (int pass = 0; pass < 2; ++pass) {
        if (pass == 1 && !fwd_again(sm)) break;
        if (lane == 0) {
          tma_prefetch_desc(&tm_q);
          tma_prefetch_desc(&tm_k_hot);
          FwdWalk walk(p, n_tiles);
          int item, t0, t1;
          while (walk.next(item, t0, t1)) {
            const int h = item / p.n_q_tiles, m_tile = item - h * p.n_q_tiles;
            for (int rep = 0; rep <= pass; ++rep, ++seg) {
              const int qb = seg & 1;
              if (seg >= 2) mbar_wait(&sm.q_empty[qb], ((seg >> 1) - 1) & 1, p.err, DEV_TIMEOUT_CONSUMER);
              mbar_arrive_expect_tx(&sm.q_full[qb], kTileBytes);
              tma_load_3d(sm.q[qb], &tm_q, &sm.q_full[qb], 0, h, m_tile * kBM);
              for (int j = t0; j < t1; ++j) {
                const bool hot = j < n_hot;
                if (reused) mbar_wait(&sm.s_full[b], par, p.err, DEV_TIMEOUT_CONSUMER);
                mbar_arrive_expect_tx(&sm.k_full[b], kFastTileBytes);
                tma_load_3d(sm.k[b], hot ? &tm_k_hot : &tm_k_ret, &sm.k_full[b], 0, (hot ? j : j - n_hot) * kFT, h);
                if (++b == kFastWgs) { b = 0; par ^= 1; reused = true; }
              }
            }
          }
        }
        __syncwarp();
      }
    } else if (warp == 3) {
      // ---------------------------------------------------------------- TMA producer: V
      // Its own thread: a stage's values are released several tiles later than its keys.  The first four value tiles
      // are on their way before the first scores exist.  (Loaded with the keys four tiles later, which are requested
      // when the first scores are done: short calls that find keys and values in DRAM waited for DRAM once more, 200 rows, 4
      // tiles 10.6 against 9.2 us in this kernel, 1041 rows, 19 tiles 20.5 against 19.4.)
      int b = 0, par = 1;
      bool reused = false;
      for (int pass = 0; pass < 2; ++pass) {
        if (pass == 1 && !fwd_again(sm)) break;
        if (lane == 0) {
          tma_prefetch_desc(&tm_v_hot);
          FwdWalk walk(p, n_tiles);
          int item, t0, t1;
          while (walk.next(item, t0, t1)) {
            const int h = item / p.n_q_tiles;
            for (int rep = 0; rep <= pass; ++rep) {
              for (int j = t0; j < t1; ++j) {
                const bool hot = j < n_hot;
                if (reused) mbar_wait(&sm.pv_done[b], par, p.err, DEV_TIMEOUT_CONSUMER);
                mbar_arrive_expect_tx(&sm.v_full[b], kFastTileBytes);
                tma_load_3d(sm.v[b], hot ? &tm_v_hot : &tm_v_ret, &sm.v_full[b], 0, (hot ? j : j - n_hot) * kFT, h);
                if (++b == kFastWgs) { b = 0; par ^= 1; reused = true; }
              }
            }
          }
        }
        __syncwarp();
      }
    } else if (warp == 1) {
      // ---------------------------------------------------------------- MMA issuer: S = Q K^T
      // (all lanes run the loop, one elected lane issues)
      constexpr uint32_t idesc_s = umma_idesc_bf16(kBM, kFT, 0);
      const uint64_t q_desc0 = smem_desc_sw128(smem_u32(sm.q[0]));
      const uint64_t k_desc0 = smem_desc_sw128(smem_u32(sm.k[0]));
      uint32_t b = 0, par = 1;     // stage and buffer of the tile, phase of their previous use
      bool reused = false;         // a buffer's first scores overwrite nothing
      int seg = 0;
      auto segment = [&](int t0, int t1) {
        const int qb = seg & 1;
        const uint64_t q_desc = q_desc0 + static_cast<uint64_t>(qb * (kTileBytes >> 4));
        mbar_wait(&sm.q_full[qb], (seg >> 1) & 1, p.err, DEV_TIMEOUT_TMA);
#pragma unroll 1
        for (int j = t0; j < t1; ++j) {
          const uint64_t k_desc = k_desc0 + static_cast<uint64_t>(b * (kFastTileBytes >> 4));
          const uint32_t d = tmem + b * kFT;
          mbar_wait(&sm.k_full[b], par ^ 1, p.err, DEV_TIMEOUT_TMA);
          if (reused) mbar_wait(&sm.pv_done[b], par, p.err, DEV_TIMEOUT_CONSUMER);
          tc_fence_after();
          if (elect_one()) {
            umma_ss(d, q_desc, k_desc, idesc_s, 0u);
            umma_ss(d, q_desc + 2, k_desc + 2, idesc_s, 1u);
            umma_ss(d, q_desc + 4, k_desc + 4, idesc_s, 1u);
            umma_ss(d, q_desc + 6, k_desc + 6, idesc_s, 1u);
            umma_commit(&sm.s_full[b]);
          }
          __syncwarp();
          if (++b == kFastWgs) { b = 0; par ^= 1; reused = true; }
        }
        if (elect_one()) umma_commit(&sm.q_empty[qb]);
        __syncwarp();
        ++seg;
      };
      for (int pass = 0; pass < 2; ++pass) {
        if (pass == 1 && !fwd_again(sm)) break;
        FwdWalk walk(p, n_tiles);
        int item, t0, t1;
        while (walk.next(item, t0, t1))
#pragma unroll 1
          for (int rep = 0; rep <= pass; ++rep) segment(t0, t1);
      }
    } else if (warp == 2) {
      // ---------------------------------------------------------------- MMA issuer: O += P V
      constexpr uint32_t idesc_o = umma_idesc_bf16(kBM, kD, 1);
      const uint64_t v_desc0 = smem_desc_sw128(smem_u32(sm.v[0]));
      uint32_t b = 0, par = 0;     // stage and buffer of the tile, their phase
      int seg = 0;
      // maxima: there are no probabilities.  (A kind of its own for the compiler: as a run-time flag it cost the call with a bias on
      // every key 1.2 us, M 2603, N 6247, 12 heads 94.9 against 93.7.)
      auto segment = [&](int t0, int t1, auto maxima) {
        uint32_t acc = 0u;
#pragma unroll 1
        for (int j = t0; j < t1; ++j) {
          // A: 16 keys = 8 columns of packed probabilities; B: V advances 16 rows = 2048 bytes
          const uint32_t pa = tmem + b * kFT;
          const uint64_t v_desc = v_desc0 + static_cast<uint64_t>(b * (kFastTileBytes >> 4));
          mbar_wait(&sm.v_full[b], par, p.err, DEV_TIMEOUT_TMA);
          mbar_wait(&sm.p_full[b], par, p.err, DEV_TIMEOUT_CONSUMER);
          // a new segment overwrites the accumulator: the previous one must have been read out
          if (acc == 0u && seg > 0) mbar_wait(&sm.o_free, (seg - 1) & 1, p.err, DEV_TIMEOUT_CONSUMER);
          tc_fence_after();
          if (elect_one()) {
            if constexpr (!decltype(maxima)::value) {
              umma_ts(o_tmem, pa, v_desc, idesc_o, acc);
#pragma unroll
              for (int kk = 1; kk < kFT / 16; ++kk)
                umma_ts(o_tmem, pa + kk * 8, v_desc + static_cast<uint64_t>(kk * (2048 >> 4)), idesc_o, 1u);
            }
            umma_commit(&sm.pv_done[b]);
          }
          __syncwarp();
          acc = 1u;
          if (++b == kFastWgs) { b = 0; par ^= 1; }
        }
        if (elect_one()) umma_commit(&sm.o_done);
        __syncwarp();
        ++seg;
      };
      for (int pass = 0; pass < 2; ++pass) {
        if (pass == 1 && !fwd_again(sm)) break;
        FwdWalk walk(p, n_tiles);
        int item, t0, t1;
        while (walk.next(item, t0, t1)) {
          if (pass == 1) segment(t0, t1, std::true_type{});
          segment(t0, t1, std::false_type{});
        }
      }
    }
    if (p.cluster) {      // with the softmax warps, which join the parts in between
      cluster_sync();
      cluster_sync();
    }
  } else {
    // ------------------------------------------------------------------ softmax warpgroups
    setmaxnreg_inc<kFastSoftmaxRegs>();
    const int g = (warp - 4) >> 2;
    const int wq = warp & 3;
    const int row = wq * 32 + lane;
    const uint32_t lane_base = static_cast<uint32_t>(wq * 32) << 16;
    const float c2 = p.scale_log2;
    const uint64_t c2c2 = pack_f32x2(c2, c2);
    const float* bias2 = sm.bias2[g];
    uint32_t ra[32], rb[32], pk[16];   // rb: the read-out of O
    const uint32_t s_addr = tmem + lane_base + g * kFT;
    float top = 0.f;          // largest exponent (relative to the row reference) that the FMA pipes were given
    // Reads a segment's accumulator out of tensor memory and writes the rows, or leaves or joins a part.  `l`: row sum, `m_ref`: its
    // reference, `bad`: they cannot stand for the row, which is done again (`redo`: it has been).
    auto close = [&](int item, int t0, int t1, int seg, float l, float m_ref, bool seg_live, bool bad, bool redo) {
      const int h = item / p.n_q_tiles, m_tile = item - h * p.n_q_tiles;
      mbar_wait(&sm.o_done, seg & 1, p.err, DEV_TIMEOUT_MMA);
      tc_fence_after();
      tmem_ld32(o_tmem + lane_base, ra);
      tmem_ld32(o_tmem + lane_base + 32, rb);
      tmem_ld_wait();
      tc_fence_before();
      mbar_arrive(&sm.o_free);
      const int mrow = m_tile * kBM + row;
      if (bad) sm.again = 1;
      if (t0 == 0 && t1 == n_tiles) {
        // the whole item was done here: normalise and write the output rows
        const float inv = l > 0.f ? 1.f / l : 0.f;
        if (mrow < p.M) {
          __nv_bfloat16* dst = p.out + static_cast<long long>(mrow) * p.out_row_stride + h * kD;
#pragma unroll
          for (int q8 = 0; q8 < 4; ++q8) {
            uint4 val;
            val.x = pack_bf16x2(__uint_as_float(ra[q8 * 8 + 0]) * inv, __uint_as_float(ra[q8 * 8 + 1]) * inv);
            val.y = pack_bf16x2(__uint_as_float(ra[q8 * 8 + 2]) * inv, __uint_as_float(ra[q8 * 8 + 3]) * inv);
            val.z = pack_bf16x2(__uint_as_float(ra[q8 * 8 + 4]) * inv, __uint_as_float(ra[q8 * 8 + 5]) * inv);
            val.w = pack_bf16x2(__uint_as_float(ra[q8 * 8 + 6]) * inv, __uint_as_float(ra[q8 * 8 + 7]) * inv);
            *reinterpret_cast<uint4*>(dst + q8 * 8) = val;
          }
#pragma unroll
          for (int q8 = 0; q8 < 4; ++q8) {
            uint4 val;
            val.x = pack_bf16x2(__uint_as_float(rb[q8 * 8 + 0]) * inv, __uint_as_float(rb[q8 * 8 + 1]) * inv);
            val.y = pack_bf16x2(__uint_as_float(rb[q8 * 8 + 2]) * inv, __uint_as_float(rb[q8 * 8 + 3]) * inv);
            val.z = pack_bf16x2(__uint_as_float(rb[q8 * 8 + 4]) * inv, __uint_as_float(rb[q8 * 8 + 5]) * inv);
            val.w = pack_bf16x2(__uint_as_float(rb[q8 * 8 + 6]) * inv, __uint_as_float(rb[q8 * 8 + 7]) * inv);
            *reinterpret_cast<uint4*>(dst + 32 + q8 * 8) = val;
          }
          const float l2 = m_ref + log2f(l);
          if (p.lse != nullptr) p.lse[static_cast<long long>(h) * p.M + mrow] = l2 * kLn2;
          p.lse2[static_cast<long long>(h) * p.lse2_stride + mrow] = l2;
        }
      } else {
        // Part of an item: whichever of the two CTAs gets there second joins the parts.  The first one leaves its
        // unnormalised accumulator, row sums and references in its slot (slot 1: the item starts here and ends in the
        // next CTA; slot 0: it began in the previous CTA) and counts its arrival.  The parts lie with a row's 16-byte pieces
        // kBM rows apart, so that a warp writes and reads whole lines.
        const bool first_part = t0 == 0;
        const int cut = first_part ? blockIdx.x : blockIdx.x - 1;   // between CTA cut and cut + 1
        const float m_pub = seg_live ? m_ref : -INFINITY;
        const int slot_at = first_part ? 1 : 0;
        if (redo && sm.part_again[slot_at] == 0) return;      // the first walk has left it
        if (named_bar_or(1 + g, 128, bad)) {     // (and nobody reads the word of the segment before any more)
          if (row == 0) sm.part_again[slot_at] = 1;           // not to be joined with: the second walk leaves it
          return;
        }
        auto leave = [&](float* slot) {
          float4* orow = reinterpret_cast<float4*>(slot) + row;
#pragma unroll
          for (int q4 = 0; q4 < 8; ++q4)
            orow[q4 * kBM] = make_float4(__uint_as_float(ra[q4 * 4 + 0]), __uint_as_float(ra[q4 * 4 + 1]),
                                         __uint_as_float(ra[q4 * 4 + 2]), __uint_as_float(ra[q4 * 4 + 3]));
#pragma unroll
          for (int q4 = 0; q4 < 8; ++q4)
            orow[(8 + q4) * kBM] = make_float4(__uint_as_float(rb[q4 * 4 + 0]), __uint_as_float(rb[q4 * 4 + 1]),
                                               __uint_as_float(rb[q4 * 4 + 2]), __uint_as_float(rb[q4 * 4 + 3]));
          slot[kBM * kD + row] = l;
          slot[kBM * kD + kBM + row] = m_pub;
        };
        if (p.parts > 1) {      // this CTA's only segment, joined behind the walk
          if (p.cluster) {
            leave(reinterpret_cast<float*>(sm.k));     // the key tiles are not needed any more
          } else {
            leave(p.part + static_cast<size_t>(2 * blockIdx.x) * kPartFloats);
            __threadfence();
            named_bar_sync(1 + g, 128);
            if (row == 0) sm.join_all = atomicAdd(p.part_count + item, 1) == p.parts - 1 ? 1 : 0;
          }
          return;
        }
        if (row == 0) sm.join_flag[g] = ld_acquire(p.part_count + cut);
        named_bar_sync(1 + g, 128);
        bool second = sm.join_flag[g] == 1;          // usually: the item's other CTA began with it, or ended with it long ago
        if (!second) {
          leave(p.part + static_cast<size_t>(2 * blockIdx.x + slot_at) * kPartFloats);
          __threadfence();                           // this thread's part is visible device-wide ...
          named_bar_sync(1 + g, 128);                // ... and so is every other row's
          if (row == 0) sm.join_flag[g] = atomicAdd(p.part_count + cut, 1);
          named_bar_sync(1 + g, 128);
          second = sm.join_flag[g] == 1;
        }
        if (second) {
          // the other CTA's part was complete before its counter increment, which came first
          __threadfence();
          if (row == 0) p.part_count[cut] = 0;       // both have arrived: ready for the next call
          const float* other = p.part + static_cast<size_t>(first_part ? 2 * (cut + 1) : 2 * cut + 1) * kPartFloats;
          const float lo_ = __ldcg(other + kBM * kD + row), mo_ = __ldcg(other + kBM * kD + kBM + row);
          // a = the part with the item's first tiles, b = the part with its last ones
          const float la = first_part ? l : lo_, ma = first_part ? m_pub : mo_;
          const float lb = first_part ? lo_ : l, mb = first_part ? mo_ : m_pub;
          const float mm = fmaxf(ma, mb);
          const float m = (mm == -INFINITY) ? 0.f : mm;     // both parts fully masked: zeros, lse = -inf
          const float wa = exp2f(ma - m), wb = exp2f(mb - m);   // a masked part (-inf) weighs nothing
          // explicit operation order: the same bits whichever of the two CTAs computes the join
          const float lsum2 = __fmaf_rn(la, wa, __fmul_rn(lb, wb));
          const float inv = lsum2 > 0.f ? 1.f / lsum2 : 0.f;
          if (mrow < p.M) {
            const float4* orow_o = reinterpret_cast<const float4*>(other) + row;
            __nv_bfloat16* dst = p.out + static_cast<long long>(mrow) * p.out_row_stride + h * kD;
            auto join = [&](uint32_t own, float oth) {
              const float x = __uint_as_float(own);
              const float va = first_part ? x : oth, vb = first_part ? oth : x;
              return __fmul_rn(__fmaf_rn(va, wa, __fmul_rn(vb, wb)), inv);
            };
#pragma unroll
            for (int q8 = 0; q8 < 8; ++q8) {
              const float4 o0 = __ldcg(orow_o + 2 * q8 * kBM), o1 = __ldcg(orow_o + (2 * q8 + 1) * kBM);
              const uint32_t* r8 = q8 < 4 ? &ra[q8 * 8] : &rb[(q8 - 4) * 8];
              uint4 val;
              val.x = pack_bf16x2(join(r8[0], o0.x), join(r8[1], o0.y));
              val.y = pack_bf16x2(join(r8[2], o0.z), join(r8[3], o0.w));
              val.z = pack_bf16x2(join(r8[4], o1.x), join(r8[5], o1.y));
              val.w = pack_bf16x2(join(r8[6], o1.z), join(r8[7], o1.w));
              *reinterpret_cast<uint4*>(dst + q8 * 8) = val;
            }
            const float l2 = m + log2f(lsum2);
            if (p.lse != nullptr) p.lse[static_cast<long long>(h) * p.M + mrow] = l2 * kLn2;
            p.lse2[static_cast<long long>(h) * p.lse2_stride + mrow] = l2;
          }
        }
      }
    };
    FwdWalk walk(p, n_tiles);
    int seg = 0, item, t0, t1;
    int c_base = 0;   // key tiles of earlier segments
    int round = 0;    // tiles that this warpgroup has behind it
    for (; walk.next(item, t0, t1); ++seg) {
      const int h = item / p.n_q_tiles;
      const int len = t1 - t0;
      const int sb = seg & 1;
      float m_ref = 0.f;
      uint64_t l0 = 0ull, l1 = 0ull;    // four partial row sums, two per register pair
      uint64_t negm2 = 0ull;            // (-m_ref, -m_ref)
      bool have_ref = false;
      bool any_live = false;  // some key tile of this warpgroup in this segment had a key that is not masked
      int x = (g - c_base) & (kFastWgs - 1);
      // The reference of the segment, at the first tile of this warpgroup.
      auto reference = [&](bool need_bias) {
        mbar_wait(&sm.s_full[g], round & 1, p.err, DEV_TIMEOUT_MMA);
        tc_fence_after();
        if (x == 0) {
          // exact row maximum of the segment's first tile = the row's reference for the segment
          float mx = -INFINITY;
          tmem_ld32(s_addr, ra);
#pragma unroll
          for (int ch = 0; ch < kFT / 32; ++ch) {
            tmem_ld_wait();
            mx = fast_max_chunk<32>(ra, bias2 + 32 * ch, need_bias, c2, mx);
            if (ch + 1 < kFT / 32) tmem_ld32(s_addr + 32 * (ch + 1), ra);
            else tmem_ld16(s_addr + 32 * (ch + 1), ra);
          }
          tmem_ld_wait();
          mx = fast_max_chunk<16>(ra, bias2 + kFT - 16, need_bias, c2, mx);
          m_ref = (mx == -INFINITY) ? 0.f : mx;
          sm.m_ref[sb][row] = m_ref;
          mbar_arrive(&sm.ref_ready[sb]);
        } else {
          mbar_wait(&sm.ref_ready[sb], (seg >> 1) & 1, p.err, DEV_TIMEOUT_CONSUMER);
          m_ref = sm.m_ref[sb][row];
        }
        negm2 = pack_f32x2(-m_ref, -m_ref);
        have_ref = true;
      };
      // Scores -> probabilities in place, chunk by chunk: load, wait, convert, store.
      auto convert = [&](auto bias_tag) {
        constexpr bool kBias = decltype(bias_tag)::value;
#pragma unroll
        for (int ch = 0; ch < kFT / 32; ++ch) {
          tmem_ld_wait();
          fast_exp_chunk<kBias, 32>(ra, pk, bias2 + 32 * ch, c2c2, negm2, l0, l1, top);
          if (ch + 1 < kFT / 32) tmem_ld32(s_addr + 32 * (ch + 1), ra);
          else tmem_ld16(s_addr + 32 * (ch + 1), ra);
          tmem_st16(s_addr + 16 * ch, pk);
        }
        tmem_ld_wait();
        fast_exp_chunk<kBias, 16>(ra, pk, bias2 + kFT - 16, c2c2, negm2, l0, l1, top);
        tmem_st8(s_addr + (kFT - 16) / 2, pk);
        tmem_st_wait();
        tc_fence_before();
        mbar_arrive(&sm.p_full[g]);
      };
      // whole tiles of the hot cache: no bias, nothing masked
      const int n_plain = min(len, p.T_hot / kFT - t0);
      any_live = x < n_plain;
      if (x < n_plain) reference(false);
#pragma unroll 1
      for (; x < n_plain; x += kFastWgs, ++round) {
        mbar_wait(&sm.s_full[g], round & 1, p.err, DEV_TIMEOUT_MMA);
        tc_fence_after();
        tmem_ld32(s_addr, ra);
        convert(std::false_type{});
      }
      // the ragged last tile of the hot cache, the retrieved pivots
#pragma unroll 1
      for (; x < len; x += kFastWgs, ++round) {
        const int j = t0 + x;
        const bool is_ret = j >= n_hot;
        const int n0 = (is_ret ? j - n_hot : j) * kFT;
        const int valid = min(kFT, (is_ret ? p.T_ret : p.T_hot) - n0);
        float bv = -INFINITY;
        if (row < valid) bv = is_ret ? p.bias_ret[h * p.bias_head_stride + n0 + row] * kLog2e : 0.f;
        named_bar_sync(1 + g, 128);   // the bias is on its way while the warpgroup meets
        if (row < kFT) sm.bias2[g][row] = bv;
        // false: every key of the tile is masked (padding behind the valid pivots)
        const bool tile_live = named_bar_or(1 + g, 128, bv != -INFINITY);
        any_live = any_live || tile_live;
        const bool first = !have_ref;
        if (first) reference(true);
        mbar_wait(&sm.s_full[g], round & 1, p.err, DEV_TIMEOUT_MMA);
        tc_fence_after();
        if (!tile_live && !first) {
          // nothing to exponentiate: all probabilities of this tile are zero
#pragma unroll
          for (int i = 0; i < 16; ++i) pk[i] = 0u;
#pragma unroll
          for (int ch = 0; ch < kFT / 32; ++ch) tmem_st16(s_addr + 16 * ch, pk);
          tmem_st8(s_addr + (kFT - 16) / 2, pk);
          tmem_st_wait();
          tc_fence_before();
          mbar_arrive(&sm.p_full[g]);
          continue;
        }
        tmem_ld32(s_addr, ra);
        convert(std::true_type{});
      }
      // ---- end of the segment
      float la, lb, lc, ld;
      unpack_f32x2(l0, la, lb);
      unpack_f32x2(l1, lc, ld);
      const float lsum = (la + lb) + (lc + ld);
      // a sum or an exponent out of range (or NaN): whoever closes the segment sees a NaN
      sm.lpart[sb][g][row] = lsum <= kFastRowSumLimit && top < 128.f ? lsum : NAN;
      if (row == 0) sm.live[sb][g] = any_live ? 1 : 0;
      if (g != ((c_base + len - 1) & (kFastWgs - 1))) {
        mbar_arrive(&sm.l_ready[sb]);
      } else {
        // The warpgroup of the last tile closes the segment: its next tile is three tiles into the next segment, where the
        // others are working meanwhile.  (Every segment of a CTA behind its first adds 1.0 us to this kernel; 2.5 when
        // warpgroup 0 closed them all, whose next tile was often the first of the next segment.)
        mbar_wait(&sm.l_ready[sb], (seg >> 1) & 1, p.err, DEV_TIMEOUT_CONSUMER);
        const float l = ((sm.lpart[sb][0][row] + sm.lpart[sb][1][row]) + sm.lpart[sb][2][row]) + sm.lpart[sb][3][row];
        // A segment whose keys are all masked has no reference (m_ref is a placeholder): it must not
        // take part in a join.  A segment with live keys whose probabilities all underflowed (its
        // first tile was masked, so the placeholder was used, and the live scores lie far below
        // it) needs another reference.
        bool seg_live = any_live;
#pragma unroll
        for (int w = 0; w < kFastWgs; ++w) seg_live = seg_live || (w != g && sm.live[sb][w] != 0);
        close(item, t0, t1, seg, l, m_ref, seg_live, !(l >= 0.f) || (seg_live && !(l > 0.f)), false);
      }
      c_base += len;
    }
    if (fwd_again(sm)) {
      // The second walk: exact row maxima of a segment, then its probabilities relative to them, on the exponential unit alone.
      // (Both named barriers are crossed once per walk of a segment by all softmax warps, so nobody runs ahead.)
      auto tile_bias = [&](int h, int j) {       // the bias of a tile into shared memory; false: none of its keys has one
        const bool is_ret = j >= n_hot;
        const int n0 = (is_ret ? j - n_hot : j) * kFT;
        const int valid = min(kFT, (is_ret ? p.T_ret : p.T_hot) - n0);
        if (!is_ret && valid == kFT) return false;
        float bv = -INFINITY;
        if (row < valid) bv = is_ret ? p.bias_ret[h * p.bias_head_stride + n0 + row] * kLog2e : 0.f;
        named_bar_sync(1 + g, 128);
        if (row < kFT) sm.bias2[g][row] = bv;
        named_bar_sync(1 + g, 128);
        return true;
      };
      FwdWalk again(p, n_tiles);
      while (again.next(item, t0, t1)) {
        const int h = item / p.n_q_tiles, len = t1 - t0;
        float mx = -INFINITY;
#pragma unroll 1
        for (int x = (g - c_base) & (kFastWgs - 1); x < len; x += kFastWgs, ++round) {
          const bool biased = tile_bias(h, t0 + x);
          mbar_wait(&sm.s_full[g], round & 1, p.err, DEV_TIMEOUT_MMA);
          tc_fence_after();
#pragma unroll 1
          for (int ch = 0; ch < kFT / 16; ++ch) {
            tmem_ld16(s_addr + 16 * ch, ra);
            tmem_ld_wait();
            mx = fast_max_chunk<16>(ra, bias2 + 16 * ch, biased, c2, mx);
          }
          tc_fence_before();
          mbar_arrive(&sm.p_full[g]);
        }
        sm.lpart[0][g][row] = mx;
        named_bar_sync(5, kFastThreads - 128);
        mx = fmaxf(fmaxf(sm.lpart[0][0][row], sm.lpart[0][1][row]), fmaxf(sm.lpart[0][2][row], sm.lpart[0][3][row]));
        const bool seg_live = mx != -INFINITY;
        const float m_ref = seg_live ? mx : 0.f;
        if (g == ((c_base + len - 1) & (kFastWgs - 1))) {
          mbar_wait(&sm.o_done, seg & 1, p.err, DEV_TIMEOUT_MMA);
          mbar_arrive(&sm.o_free);
        }
        c_base += len;
        ++seg;
        float l = 0.f;
#pragma unroll 1
        for (int x = (g - c_base) & (kFastWgs - 1); x < len; x += kFastWgs, ++round) {
          const bool biased = tile_bias(h, t0 + x);
          mbar_wait(&sm.s_full[g], round & 1, p.err, DEV_TIMEOUT_MMA);
          tc_fence_after();
#pragma unroll 1
          for (int ch = 0; ch < kFT / 16; ++ch) {
            tmem_ld16(s_addr + 16 * ch, ra);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; i += 2) {
              const float s0 = __uint_as_float(ra[i]), s1 = __uint_as_float(ra[i + 1]);
              float x0, x1;
              if (biased) {
                x0 = fmaf(s0, c2, bias2[16 * ch + i]) - m_ref;
                x1 = fmaf(s1, c2, bias2[16 * ch + i + 1]) - m_ref;
              } else {
                x0 = fmaf(s0, c2, -m_ref);
                x1 = fmaf(s1, c2, -m_ref);
              }
              const float p0 = fast_exp2(x0), p1 = fast_exp2(x1);
              l += p0 + p1;
              pk[i / 2] = pack_bf16x2(p0, p1);
            }
            tmem_st8(s_addr + 8 * ch, pk);
          }
          tmem_st_wait();
          tc_fence_before();
          mbar_arrive(&sm.p_full[g]);
        }
        sm.lpart[1][g][row] = l;
        named_bar_sync(5, kFastThreads - 128);
        if (g == ((c_base + len - 1) & (kFastWgs - 1)))
          close(item, t0, t1, seg, ((sm.lpart[1][0][row] + sm.lpart[1][1][row]) + sm.lpart[1][2][row]) + sm.lpart[1][3][row],
                m_ref, seg_live, false, true);
        c_base += len;
        ++seg;
      }
    }
    if (p.parts > 1) {
      // kCols columns of row r of the item, from 8 c8 on: its parts from the last to the first (two parts that are joined from registers
      // are added in that order, too).  load4(c, i), load1(c, i): the i-th 16 or 4 bytes of part c.
      const int k = p.parts, it = blockIdx.x / k;
      auto join = [&](auto cols, int c8, int r, auto load4, auto load1) {
        constexpr int kCols = decltype(cols)::value;
        const int h = it / p.n_q_tiles, mrow = (it - h * p.n_q_tiles) * kBM + r;
        float mm = -INFINITY;
#pragma unroll 4
        for (int c = 0; c < k; ++c) mm = fmaxf(mm, load1(c, kBM * kD + kBM + r));
        const float m = (mm == -INFINITY) ? 0.f : mm;     // all parts fully masked: zeros, lse = -inf
        float l = 0.f, acc[kCols];
#pragma unroll
        for (int i = 0; i < kCols; ++i) acc[i] = 0.f;
#pragma unroll 2
        for (int c = k - 1; c >= 0; --c) {
          float4 o[kCols / 4];
#pragma unroll
          for (int q4 = 0; q4 < kCols / 4; ++q4) o[q4] = load4(c, (2 * c8 + q4) * kBM + r);
          const float w = exp2f(load1(c, kBM * kD + kBM + r) - m);     // a masked part (-inf) weighs nothing
          l = __fmaf_rn(load1(c, kBM * kD + r), w, l);
#pragma unroll
          for (int q4 = 0; q4 < kCols / 4; ++q4) {
            acc[4 * q4] = __fmaf_rn(o[q4].x, w, acc[4 * q4]);
            acc[4 * q4 + 1] = __fmaf_rn(o[q4].y, w, acc[4 * q4 + 1]);
            acc[4 * q4 + 2] = __fmaf_rn(o[q4].z, w, acc[4 * q4 + 2]);
            acc[4 * q4 + 3] = __fmaf_rn(o[q4].w, w, acc[4 * q4 + 3]);
          }
        }
        if (mrow >= p.M) return;
        const float inv = l > 0.f ? 1.f / l : 0.f;
        __nv_bfloat16* dst = p.out + static_cast<long long>(mrow) * p.out_row_stride + h * kD + 8 * c8;
#pragma unroll
        for (int q8 = 0; q8 < kCols / 8; ++q8) {
          uint4 val;
          val.x = pack_bf16x2(__fmul_rn(acc[8 * q8], inv), __fmul_rn(acc[8 * q8 + 1], inv));
          val.y = pack_bf16x2(__fmul_rn(acc[8 * q8 + 2], inv), __fmul_rn(acc[8 * q8 + 3], inv));
          val.z = pack_bf16x2(__fmul_rn(acc[8 * q8 + 4], inv), __fmul_rn(acc[8 * q8 + 5], inv));
          val.w = pack_bf16x2(__fmul_rn(acc[8 * q8 + 6], inv), __fmul_rn(acc[8 * q8 + 7], inv));
          *reinterpret_cast<uint4*>(dst + 8 * q8) = val;
        }
        if (c8 == 0) {
          const float l2 = m + log2f(l);
          if (p.lse != nullptr) p.lse[static_cast<long long>(h) * p.M + mrow] = l2 * kLn2;
          p.lse2[static_cast<long long>(h) * p.lse2_stride + mrow] = l2;
        }
      };
      constexpr int kUnits = kBM * kD / 8;                // of eight columns
      static_assert(kUnits == 2 * (kFastThreads - 128), "two units per softmax thread");
      if (p.cluster) {
        cluster_sync();                                   // each CTA joins an equal share of the units
        const int share = (kUnits + k - 1) / k, rank = blockIdx.x - it * k, x = rank * share + threadIdx.x - 128;
        const uint32_t mine = smem_u32(sm.k);
        if (x < min((rank + 1) * share, kUnits))
          join(std::integral_constant<int, 8>{}, x / kBM, x % kBM, [&](int c, int i) { return ld_cluster4(cluster_addr(mine, c) + i * 16); },
               [&](int c, int i) { return ld_cluster(cluster_addr(mine, c) + i * 4); });
        cluster_sync();                                   // nobody leaves while its part is read
      } else {
        named_bar_sync(5, kFastThreads - 128);
        if (sm.join_all != 0) {                           // the CTA whose part came last joins them all
          __threadfence();                                // the other parts were complete before their counts
          if (threadIdx.x == 128) p.part_count[it] = 0;
          const float* first = p.part + static_cast<size_t>(2 * it * k) * kPartFloats;
          join(std::integral_constant<int, 16>{}, 2 * g, row,
               [&](int c, int i) { return __ldcg(reinterpret_cast<const float4*>(first + static_cast<size_t>(2 * c) * kPartFloats) + i); },
               [&](int c, int i) { return __ldcg(first + static_cast<size_t>(2 * c) * kPartFloats + i); });
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
  STAC_TS(0, true);
}

// ---------------------------------------------------------------------------------------
// Column sums.  An item = (head, group of kGroup 128-key tiles: kColGroup, or two or one in short calls), head-major; its units are the
// 128-row query tiles.  All units of the launch form one sequence that is cut into equal
// contiguous ranges, one per persistent CTA, so every SM gets the same amount of work; an item
// that straddles a cut is finished by two CTAs, each adding its partial sums to the zeroed
// output with one atomic add per key (two addends onto zero give the same bits in either
// order).  A query tile is scored in two halves of 64 rows: for each half the MMA warp
// computes S^T = K Q^T for the key tiles of the group against the same query rows in shared memory
// (N = 64, two 64-column TMEM buffers per key tile); warpgroup w owns key tile w, one key
// (TMEM lane) per thread, so a thread's column sum never leaves its registers.  Three exponent
// warps per scheduler keep the exp2 unit busier than two did (85 % against 75 % of the active
// cycles); a fourth (104 registers per thread) measured the same as three.
// The last query tile is ragged unless M_sub is a multiple of 128 (one frame of 1041 tokens fills 17
// of its rows): its second half is not scored when no row lies in it, and of the half that holds
// the last row only the 16-row pieces up to that row are exponentiated.
// (M = 1041, 16 heads: N = 33312 338.7 -> 331.3 us per call with the forward pass, N = 2082 38.5 -> 37.5 us;
// M = 4164 has its last row in the second half: 0.2 %.)
// lse2 holds the row log-sum-exp in the log2 domain; rows past M_sub read as +inf so that
// padded query columns contribute exp2(-inf) = 0.
// ---------------------------------------------------------------------------------------
constexpr int kColHalf = 64;           // query rows per score buffer

template <int kGroup>
struct ColSmem {
  uint8_t k[2][kGroup][kTileBytes];     // [item parity][key tile of the group]
  uint8_t q[kColStages][kTileBytes];
  uint64_t k_full[2];
  uint64_t k_empty[2];
  uint64_t q_full[kColStages];
  uint64_t q_empty[kColStages];
  uint64_t s_full[2];
  uint64_t s_free[2];
  uint64_t x_full[kColStages];            // the row-term operand of a query stage is written
  uint32_t tmem_base;
  int join_flag;                          // arrival count seen at a shared item
  alignas(16) uint8_t ax[kColXBytes];     // ones in K columns 0..2, same for every key
  alignas(16) uint8_t bx[kColStages][kColXBytes];   // per query row: -lse2 / c2 as hi, mid, lo bf16
  alignas(16) float lse2[4];  // (without the fold) flexible: n_q_tiles * 128 floats follow (negated, one head)
};

struct ColParams {
  int M_sub, H;
  int row_stride;  // query row sub-sampling stride
  int T_hot, T_ret;
  int n_hot_tiles, n_tiles;
  int n_groups, n_items;
  int n_q_tiles;
  int split;       // 1: units are cut evenly over the grid (items may be shared by two CTAs)
  float scale_log2;
  float correction;
  const float* bias_ret;
  long long bias_head_stride;
  const float* lse2;
  long long lse2_stride;
  float* colsum;  // [H, colsum_stride], hot keys first then retrieved
  long long colsum_stride;
  // Fewer items than CTAs: an item may be shared by three or more CTAs.  Each writes its partial
  // sums to a slot of its own (two per CTA: [0] an item that began in an earlier CTA, [1] an
  // item that goes on in the next one), counts its arrival at the item, and the CTA that arrives
  // last adds the parts in CTA order and stores the result: same bits whoever does it.  nullptr:
  // an item has at most two parts, added onto the zeroed output with one atomic each.
  float* parts;       // [2 * gridDim.x][kColGroup * kBN]
  int* part_count;    // [n_items], zero on entry, left zero
  // Running scores that the column sums of the hot keys go into (stac/h2o.py:177-216), or nullptr:
  // s = colsum * T_hot / Tq; an old key's score decays, score * temperature + s (two roundings, as mul_ then
  // add_), a new one's is s; counts += 1.
  float* scores;      // [H, score_stride]
  float* counts;
  long long score_stride;
  int old_T;
  float tq, temperature;
  int* err;
};

// The range of units of one CTA, walked item by item (same sequence in every role).
struct ColWalk {
  long long u, u_end;
  int nq;
  __device__ ColWalk(const ColParams& p) {
    nq = p.n_q_tiles;
    if (p.split) {
      const long long total = static_cast<long long>(p.n_items) * nq;
      u = total * blockIdx.x / gridDim.x;
      u_end = total * (blockIdx.x + 1) / gridDim.x;
    } else {
      u = static_cast<long long>(blockIdx.x) * nq;
      u_end = u + nq;
    }
  }
  __device__ bool next(int& item, int& i0, int& i1) {
    if (u >= u_end) return false;
    item = static_cast<int>(u / nq);
    i0 = static_cast<int>(u - static_cast<long long>(item) * nq);
    const long long e = static_cast<long long>(item + 1) * nq;
    i1 = static_cast<int>((e < u_end ? e : u_end) - static_cast<long long>(item) * nq);
    u = static_cast<long long>(item) * nq + i1;
    return true;
  }
};

// 16 scores of one key against 16 query rows: sum of exp2(score * c2 - lse2[row]), two rows at
// a time with the packed fp32 instructions.  The pairs whose bit is set in kColPairMask take
// their exponentials on the FMA pipes (cubic, 8.6e-5 relative): the exponential unit is the
// bottleneck of this kernel.
template <int kJ>
__device__ __forceinline__ uint64_t col_exp_pair(uint64_t s2, uint64_t c2c2, float n0, float n1) {
  const uint64_t x2 = kColFoldLse ? mul_f32x2(s2, c2c2) : fma_f32x2(s2, c2c2, pack_f32x2(n0, n1));
  if ((kColPairMask >> kJ) & 1u) return poly_exp2_x2(x2);
  float x0, x1;
  unpack_f32x2(x2, x0, x1);
  return pack_f32x2(fast_exp2(x0), fast_exp2(x1));
}
__device__ __forceinline__ void col_exp_chunk16(const uint32_t (&s)[32], const float4* nl4, uint64_t c2c2, uint64_t& a01,
                                                uint64_t& a23) {
  float4 n0, n1, n2, n3;
  if (kColFoldLse) {
    n0 = n1 = n2 = n3 = make_float4(0.f, 0.f, 0.f, 0.f);
  } else {
    n0 = nl4[0]; n1 = nl4[1]; n2 = nl4[2]; n3 = nl4[3];
  }
  auto sp = [&](int i) { return pack_f32x2(__uint_as_float(s[i]), __uint_as_float(s[i + 1])); };
  a01 = add_f32x2(a01, col_exp_pair<0>(sp(0), c2c2, n0.x, n0.y));
  a23 = add_f32x2(a23, col_exp_pair<1>(sp(2), c2c2, n0.z, n0.w));
  a01 = add_f32x2(a01, col_exp_pair<2>(sp(4), c2c2, n1.x, n1.y));
  a23 = add_f32x2(a23, col_exp_pair<3>(sp(6), c2c2, n1.z, n1.w));
  a01 = add_f32x2(a01, col_exp_pair<4>(sp(8), c2c2, n2.x, n2.y));
  a23 = add_f32x2(a23, col_exp_pair<5>(sp(10), c2c2, n2.z, n2.w));
  a01 = add_f32x2(a01, col_exp_pair<6>(sp(12), c2c2, n3.x, n3.y));
  a23 = add_f32x2(a23, col_exp_pair<7>(sp(14), c2c2, n3.z, n3.w));
}

// All half tiles of one item for one key (thread): returns the sum over the item's query rows.
// kFast: the key's bias was taken out of the exponent (every lane of the warp agrees).
// A 64-row half is read from TMEM in four pieces of 16 rows, the next piece always in flight
// (the first piece of the next half included: its buffer does not depend on this warpgroup
// finishing the current one).  `tail` > 0: the last half has only that many pieces with rows (1 to 3).
template <bool kFast, class Smem>
__device__ __forceinline__ float col_item_sum(Smem& sm, const ColParams& p, uint32_t t_base, const float* nl_item,
                                              int n_half, int tail, int& ui, float c2, float b2_in) {
  uint32_t ra[32], rb[32];   // 16 registers of each are used
  float a0 = 0.f;
  uint64_t a01 = 0ull, a23 = 0ull;
  const uint64_t c2c2 = pack_f32x2(c2, c2);
  auto consume = [&](const uint32_t (&r)[32], const float* nl) {
    if (kFast) {
      col_exp_chunk16(r, reinterpret_cast<const float4*>(nl), c2c2, a01, a23);
    } else {
#pragma unroll
      for (int q = 0; q < 16; ++q) a0 += fast_exp2(fmaf(__uint_as_float(r[q]), c2, kColFoldLse ? b2_in : b2_in + nl[q]));
    }
  };
  // first half tile of the item: nothing is in flight yet
  {
    const int g = ui & 1, it = ui >> 1;
    mbar_wait(&sm.s_full[g], it & 1, p.err, DEV_TIMEOUT_MMA);
    tc_fence_after();
    tmem_ld16(t_base + g * kColHalf, ra);
  }
  const int n_whole = tail > 0 ? n_half - 1 : n_half;
  for (int hu = 0; hu < n_whole; ++hu, ++ui) {
    const int g = ui & 1;
    const uint32_t s_addr = t_base + g * kColHalf;
    const float* nl = nl_item + hu * kColHalf;
    tmem_ld_wait();
    tmem_ld16(s_addr + 16, rb);
    consume(ra, nl);
    tmem_ld_wait();
    tmem_ld16(s_addr + 32, ra);
    consume(rb, nl + 16);
    tmem_ld_wait();
    tmem_ld16(s_addr + 48, rb);
    consume(ra, nl + 32);
    tmem_ld_wait();
    if (hu + 1 < n_half) {
      const int g2 = (ui + 1) & 1, it2 = (ui + 1) >> 1;
      mbar_wait(&sm.s_full[g2], it2 & 1, p.err, DEV_TIMEOUT_MMA);
      tc_fence_after();
      tmem_ld16(t_base + g2 * kColHalf, ra);
    }
    consume(rb, nl + 48);
    tc_fence_before();
    mbar_arrive(&sm.s_free[g]);
  }
  if (tail > 0) {
    const int g = ui & 1;
    const uint32_t s_addr = t_base + g * kColHalf;
    const float* nl = nl_item + n_whole * kColHalf;
    tmem_ld_wait();
#pragma unroll 1
    for (int piece = 0;;) {
      consume(ra, nl + piece * 16);
      if (++piece == tail) break;
      tmem_ld16(s_addr + piece * 16, ra);
      tmem_ld_wait();
    }
    tc_fence_before();
    mbar_arrive(&sm.s_free[g]);
    ++ui;
  }
  float b0, b1, b2, b3;
  unpack_f32x2(a01, b0, b1);
  unpack_f32x2(a23, b2, b3);
  return a0 + ((b0 + b1) + (b2 + b3));
}

template <int kGroup>
__global__ void __launch_bounds__(col_threads(kGroup), 1)
attn_colsum_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k_hot,
                   const __grid_constant__ CUtensorMap tm_k_ret, const ColParams p) {
  extern __shared__ uint8_t smem_raw[];
  using Smem = ColSmem<kGroup>;
  Smem& sm = *reinterpret_cast<Smem*>(align1024(smem_raw));
  constexpr int kExpThreads = kGroup * 128;
  STAC_TS(2, false);
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int nq = p.n_q_tiles;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&sm.k_full[i], 1);
      mbar_init(&sm.k_empty[i], 1);
      mbar_init(&sm.s_full[i], 1);
      mbar_init(&sm.s_free[i], kExpThreads);
    }
    for (int s = 0; s < kColStages; ++s) {
      mbar_init(&sm.q_full[s], 1);
      mbar_init(&sm.q_empty[s], 1);
      mbar_init(&sm.x_full[s], 1);
    }
    mbar_fence_init();
  }
  if (kColFoldLse && threadIdx.x >= 128 && threadIdx.x < 256) {
    // the constant operand: row r = (1, 1, 1, 0, ..., 0) in bf16
    const int r = threadIdx.x - 128;
    uint8_t* dst = sm.ax + (r >> 3) * 256 + (r & 7) * 16;
    *reinterpret_cast<uint4*>(dst) = make_uint4(0x3F803F80u, 0x00003F80u, 0u, 0u);
    *reinterpret_cast<uint4*>(dst + 128) = make_uint4(0u, 0u, 0u, 0u);
    fence_proxy_async_smem();
  }
  if (warp == 1) {
    tmem_alloc(&sm.tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sm.tmem_base;
  // Launched with programmatic serialization behind the forward kernel: barriers and tensor memory are set up while that drains, and
  // nothing in global memory is touched before this, neither the row log-sum-exps and the zeroed output, which that kernel writes, nor keys and
  // queries, which one before it may have written: a thread sees those only behind a wait of its own.  (Keys and queries loaded ahead of it gave
  // the same bits and took 0.3 to 1.0 us less of a call.)
  grid_dep_wait();

  if (warp < 4) {
    if constexpr (kGroup == kColGroup) setmaxnreg_dec<kColCtlRegs>();   // (smaller CTAs have registers enough)
    if (warp == 0 && lane == 0) {
      // ------------------------------------------------------------------ TMA producer
      tma_prefetch_desc(&tm_q);
      ColWalk walk(p);
      int n = 0, item, i0, i1;
      int s = 0, s_round = 0;   // stage and round of the query ring
      for (; walk.next(item, i0, i1); ++n) {
        const int h = item / p.n_groups, grp = item - h * p.n_groups;   // head-major item order
        const int kb = n & 1;
        if (n >= 2) mbar_wait(&sm.k_empty[kb], ((n >> 1) - 1) & 1, p.err, DEV_TIMEOUT_CONSUMER);
        mbar_arrive_expect_tx(&sm.k_full[kb], kGroup * kTileBytes);
#pragma unroll
        for (int t = 0; t < kGroup; ++t) {
          const int j = min(kGroup * grp + t, p.n_tiles - 1);
          if (j < p.n_hot_tiles) tma_load_3d(sm.k[kb][t], &tm_k_hot, &sm.k_full[kb], 0, j * kBN, h);
          else tma_load_3d(sm.k[kb][t], &tm_k_ret, &sm.k_full[kb], 0, (j - p.n_hot_tiles) * kBN, h);
        }
        for (int i = i0; i < i1; ++i) {
          if (s_round > 0) mbar_wait(&sm.q_empty[s], (s_round - 1) & 1, p.err, DEV_TIMEOUT_CONSUMER);
          mbar_arrive_expect_tx(&sm.q_full[s], kTileBytes);
          tma_load_3d(sm.q[s], &tm_q, &sm.q_full[s], 0, h, i * kBM);
          if (++s == kColStages) { s = 0; ++s_round; }
        }
      }
    } else if (kColFoldLse && warp == 2) {
      // ------------------------------------------------------------------ row-term producer
      // For every query tile: x[m] = -lse2[m] / c2 split into three bf16 (24 bits together), so
      // that ones . (hi, mid, lo) added to the scores by the tensor core makes
      // (s + x) * c2 = s * c2 - lse2.  Rows past M_sub get a huge negative term: their
      // exponentials are exactly zero.
      ColWalk walk(p);
      const float inv_c2 = 1.f / p.scale_log2;
      int item, i0, i1;
      int s = 0, s_round = 0;
      while (walk.next(item, i0, i1)) {
        const int h = item / p.n_groups;
        for (int i = i0; i < i1; ++i) {
          if (s_round > 0) mbar_wait(&sm.q_empty[s], (s_round - 1) & 1, p.err, DEV_TIMEOUT_CONSUMER);
#pragma unroll
          for (int rr = 0; rr < 4; ++rr) {
            const int row = lane * 4 + rr;
            const int m = i * kBM + row;
            float x = -1e30f;
            if (m < p.M_sub)
              x = -p.lse2[static_cast<long long>(h) * p.lse2_stride + static_cast<long long>(m) * p.row_stride] * inv_c2;
            if (!(fabsf(x) < 1e30f)) x = -1e30f;   // lse2 = -inf (a row without live keys) or NaN: contributes nothing
            const __nv_bfloat16 hi = __float2bfloat16_rn(x);
            const float r1 = x - __bfloat162float(hi);
            const __nv_bfloat16 mid = __float2bfloat16_rn(r1);
            const __nv_bfloat16 lo = __float2bfloat16_rn(r1 - __bfloat162float(mid));
            uint8_t* dst = sm.bx[s] + (row >> 3) * 256 + (row & 7) * 16;
            const uint32_t w0 = static_cast<uint32_t>(__bfloat16_as_ushort(hi)) |
                                (static_cast<uint32_t>(__bfloat16_as_ushort(mid)) << 16);
            *reinterpret_cast<uint4*>(dst) = make_uint4(w0, static_cast<uint32_t>(__bfloat16_as_ushort(lo)), 0u, 0u);
            *reinterpret_cast<uint4*>(dst + 128) = make_uint4(0u, 0u, 0u, 0u);
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive(&sm.x_full[s]);
          if (++s == kColStages) { s = 0; ++s_round; }
        }
      }
    } else if (warp == 1) {
      // ------------------------------------------------------------------ MMA issuer
      // (all lanes run the loop so that descriptors are warp-uniform; one elected lane issues)
      constexpr uint32_t idesc = umma_idesc_bf16(kBN, kColHalf, 0);
      const uint64_t ax_desc = smem_desc_nosw(smem_u32(sm.ax), 128, 256);
      const uint64_t bx_desc0 = smem_desc_nosw(smem_u32(sm.bx[0]), 128, 256);
      ColWalk walk(p);
      const uint64_t k_desc0 = smem_desc_sw128(smem_u32(sm.k[0][0]));
      const uint64_t q_desc0 = smem_desc_sw128(smem_u32(sm.q[0]));
      int ui = 0, n = 0, item, i0, i1;   // ui: running count of half tiles
      int s = 0, s_round = 0;
      for (; walk.next(item, i0, i1); ++n) {
        const int kb = n & 1;
        mbar_wait(&sm.k_full[kb], (n >> 1) & 1, p.err, DEV_TIMEOUT_TMA);
        const uint64_t k_desc = k_desc0 + static_cast<uint64_t>(kb * kGroup * (kTileBytes >> 4));
        for (int i = i0; i < i1; ++i) {
          mbar_wait(&sm.q_full[s], s_round & 1, p.err, DEV_TIMEOUT_TMA);
          if (kColFoldLse) mbar_wait(&sm.x_full[s], s_round & 1, p.err, DEV_TIMEOUT_CONSUMER);
          const int last_half = i * kBM + kColHalf < p.M_sub ? 1 : 0;   // no row in the second half: not scored
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            if (half > last_half) break;
            const int g = ui & 1, it = ui >> 1;
            // query rows 64*half.. of the tile: 8192 bytes further in the K-major tile
            const uint64_t q_desc = q_desc0 + static_cast<uint64_t>(s * (kTileBytes >> 4) + half * (8192 >> 4));
            const uint32_t d = tmem + g * kColHalf;
            if (it > 0) mbar_wait(&sm.s_free[g], (it - 1) & 1, p.err, DEV_TIMEOUT_CONSUMER);
            tc_fence_after();
            if (elect_one()) {
#pragma unroll
              for (int t = 0; t < kGroup; ++t) {
                const uint64_t kd = k_desc + static_cast<uint64_t>(t * (kTileBytes >> 4));
                umma_ss(d + t * 128, kd, q_desc, idesc, 0u);
                umma_ss(d + t * 128, kd + 2, q_desc + 2, idesc, 1u);
                umma_ss(d + t * 128, kd + 4, q_desc + 4, idesc, 1u);
                umma_ss(d + t * 128, kd + 6, q_desc + 6, idesc, 1u);
                // the 64 rows of this half: eight row groups of 256 bytes further in the operand
                if (kColFoldLse)
                  umma_ss(d + t * 128, ax_desc, bx_desc0 + static_cast<uint64_t>((s * kColXBytes + half * 2048) >> 4),
                          idesc, 1u);
              }
              umma_commit(&sm.s_full[g]);
              if (half == last_half) {
                umma_commit(&sm.q_empty[s]);
                if (i == i1 - 1) umma_commit(&sm.k_empty[kb]);
              }
            }
            __syncwarp();
            ++ui;
          }
          if (++s == kColStages) { s = 0; ++s_round; }
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ exponent warpgroups
    if constexpr (kGroup == kColGroup) setmaxnreg_inc<kColExpRegs>();
    const int w = (warp - 4) >> 2;   // which key tile of the group
    const int wq = warp & 3;
    const int key = wq * 32 + lane;  // key inside the tile = TMEM lane
    const int tid = threadIdx.x - 128;  // 0..kExpThreads - 1
    const uint32_t t_base = tmem + (static_cast<uint32_t>(wq * 32) << 16) + w * 128;
    const float c2 = p.scale_log2;
    ColWalk walk(p);
    int ui = 0, n = 0, item, i0, i1;
    int cur_h = -1;
    for (; walk.next(item, i0, i1); ++n) {
      const int h = item / p.n_groups, grp = item - h * p.n_groups;   // head-major item order
      // negated row log-sum-exps of the head's query rows, reloaded only when the head changes
      // (a CTA's items are consecutive, so that is once or twice per launch)
      float* nl_s = sm.lse2;
      if (!kColFoldLse && h != cur_h) {
        cur_h = h;
        named_bar_sync(1, kExpThreads);   // everyone is done with the previous head's values
        for (int r = tid; r < nq * kBM; r += kExpThreads) {
          float v = -INFINITY;
          if (r < p.M_sub)
            v = -p.lse2[static_cast<long long>(h) * p.lse2_stride + static_cast<long long>(r) * p.row_stride];
          nl_s[r] = v;
        }
        named_bar_sync(1, kExpThreads);
      }
      const int j = kGroup * grp + w;
      const bool exists = j < p.n_tiles;
      const bool is_ret = j >= p.n_hot_tiles;
      const int n0 = (is_ret ? j - p.n_hot_tiles : j) * kBN;
      const int valid = exists ? min(kBN, (is_ret ? p.T_ret : p.T_hot) - n0) : 0;
      // the key's bias multiplies its whole column: exp2(s c2 + b2 - lse2) = 2^b2 exp2(s c2 - lse2);
      // taken out of the exponent while it is small, else kept inside (rare, slower path)
      float b2 = 0.f;
      if (key < valid && is_ret) b2 = p.bias_ret[h * p.bias_head_stride + n0 + key] * kLog2e;
      // a bias of -inf (padding behind the valid pivots) masks the key: its column sum is 0
      const bool masked = b2 == -INFINITY;
      if (masked) b2 = 0.f;
      const bool b2_small = fabsf(b2) <= 32.f;
      const float b2_in = b2_small ? 0.f : b2;
      const bool warp_fast = __all_sync(0xffffffffu, b2_small);
      // halves with rows, and the 16-row pieces with rows of the last one when it is not full
      const int rows_here = min(i1 * kBM, p.M_sub) - i0 * kBM;
      const int n_half = (rows_here + kColHalf - 1) / kColHalf;
      const int tail = (((rows_here - 1) % kColHalf) / 16 + 1) & 3;    // 4 pieces: a whole half, 0
      const float* nl_item = nl_s + i0 * kBM;
      // the key's running score, on its way while the rows are summed up
      const long long score_at = static_cast<long long>(h) * p.score_stride + n0 + key;
      float old_score = 0.f, old_count = 0.f;
      if (p.scores != nullptr && !is_ret && key < valid) {
        old_score = p.scores[score_at];
        old_count = p.counts[score_at];
      }
      // (warps whose 32 keys are all masked still run the sums: letting them only follow the
      // score buffers was measured slower in the stream, their polling disturbs the others)
      float sum = warp_fast ? col_item_sum<true>(sm, p, t_base, nl_item, n_half, tail, ui, c2, 0.f)
                            : col_item_sum<false>(sm, p, t_base, nl_item, n_half, tail, ui, c2, b2_in);
      if (key < valid) {
        sum *= p.correction;
        if (b2_small) sum *= exp2f(b2);
        if (masked) sum = 0.f;
      }
      float* dst = p.colsum + static_cast<long long>(h) * p.colsum_stride + (is_ret ? p.T_hot : 0) + n0 + key;
      auto update_score = [&](float total) {
        if (p.scores != nullptr && !is_ret) {
          const float sc = __fdiv_rn(__fmul_rn(total, static_cast<float>(p.T_hot)), p.tq);
          p.scores[score_at] = n0 + key >= p.old_T ? sc : __fadd_rn(__fmul_rn(old_score, p.temperature), sc);
          p.counts[score_at] = __fadd_rn(old_count, 1.0f);
        }
      };
      auto finish = [&](float total) {
        *dst = total;
        update_score(total);
      };
      constexpr int kSlot = kGroup * kBN;
      if (i0 == 0 && i1 == nq) {
        if (key < valid) finish(sum);
      } else if (p.parts == nullptr) {
        if (key < valid) {
          if (p.scores == nullptr || is_ret) {
            atomicAdd(dst, sum);      // nothing to wait for
          } else {
            // Of the two additions onto -0 the first finds the sign bit, the second the other CTA's sum, which is +0 at
            // least: the thread of the second has the total, with the bits that are in memory, and updates the score.
            const float before = atomicAdd(dst, sum);
            if (!signbit(before)) update_score(__fadd_rn(before, sum));
          }
        }
      } else {
        // CTA c owns the units [total * c / G, total * (c + 1) / G): owner(u) = ((u + 1) * G - 1) / total
        const long long total = static_cast<long long>(p.n_items) * nq, G = gridDim.x;
        const int c_first = static_cast<int>(((static_cast<long long>(item) * nq + 1) * G - 1) / total);
        const int c_last = static_cast<int>(((static_cast<long long>(item + 1) * nq) * G - 1) / total);
        float* slot = p.parts + static_cast<size_t>(2 * blockIdx.x + (i0 > 0 ? 0 : 1)) * kSlot;
        slot[w * kBN + key] = key < valid ? sum : 0.f;
        __threadfence();                          // this thread's part is visible device-wide ...
        named_bar_sync(1, kExpThreads);        // ... and so is every other key's
        if (tid == 0) sm.join_flag = atomicAdd(p.part_count + item, 1);
        named_bar_sync(1, kExpThreads);
        if (sm.join_flag == c_last - c_first) {
          // every other part was complete before its counter increment, which came earlier
          __threadfence();
          if (key < valid) {
            float acc = 0.f;
            for (int c = c_first; c <= c_last; ++c)
              acc = __fadd_rn(acc, __ldcg(p.parts + static_cast<size_t>(2 * c + (c == c_first ? 1 : 0)) * kSlot + w * kBN + key));
            finish(acc);
          }
          if (tid == 0) p.part_count[item] = 0;
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
  STAC_TS(2, true);
}

// ---------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (fn == nullptr) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) != cudaSuccess ||
        qres != cudaDriverEntryPointSuccess)
      return nullptr;
    fn = reinterpret_cast<EncodeTiledFn>(ptr);
  }
  return fn;
}

// bf16 tensor seen as [d2][d1][64]; box = 64 x box1 x box2 elements, 128-byte swizzle.
int make_map(CUtensorMap* map, const void* base, uint64_t d1, uint64_t d2, uint64_t stride1_bytes,
             uint64_t stride2_bytes, uint32_t box1, uint32_t box2) {
  EncodeTiledFn enc = get_encode_fn();
  if (enc == nullptr) return STAC_ERR_CUDA;
  cuuint64_t dims[3] = {static_cast<cuuint64_t>(kD), d1, d2};
  cuuint64_t strides[2] = {stride1_bytes, stride2_bytes};
  cuuint32_t box[3] = {static_cast<cuuint32_t>(kD), box1, box2};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? STAC_OK : STAC_ERR_CUDA;
}

// Clusters of `size` CTAs of the forward kernel that can be resident at once on this device, -1: no answer (which is asked for again).
int max_fwd_clusters(int dev, int size, int smem) {
  static PerDeviceValue<int> cache[kFastMaxCluster + 1];     // count + 1
  int n = cache[size].get(dev);
  if (n == 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(size);
    cfg.blockDim = dim3(kFastThreads);
    cfg.dynamicSmemBytes = static_cast<size_t>(smem);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(size);
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int active = 0;
    if (cudaOccupancyMaxActiveClusters(&active, attn_fwd_fast_kernel, &cfg) != cudaSuccess) {
      cudaGetLastError();
      return -1;
    }
    cache[size].set(dev, n = active + 1);
  }
  return n - 1;
}

// In how many parts the forward kernel cuts each of its items where there are SMs for them, and whether a cluster joins them.
// The estimate, in us: a key tile 0.52, a part more 0.42 for those who join them, and 2.2 through the shared memory of a cluster or
// 3.2 through the workspace.  (1041 rows, 10410 keys, 1 head, 93 tiles: 1 part 52.7 us, 2, 4 and 8 32.8, 22.4 and 17.6 through clusters, 4, 8, 12 and 16
// 23.0, 18.3, 17.9 and 18.5 through the workspace.  Clusters of eight and four have room for 15 and 33 items only.)
// Parts have references of their own, so their number decides the last bits of an output: it follows from the call's sizes alone.  What a
// device reports depends on which of its SMs are in use (and the query may fail), so that only says who joins them (see attn_colsum_launch;
// both ways add in one order).
constexpr int kFastClusterRoom[kFastMaxCluster + 1] = {0, 0, 74, 45, 33, 26, 22, 15, 15};      // items, of 148 SMs
void fwd_parts(int items, int tiles, int n_sm, bool workspace, int* parts, int* cluster) {
  *parts = 1;
  *cluster = 0;
  float best = kFastTileUs * tiles;
  for (int k = 2; k * items <= n_sm && k <= tiles; ++k) {
    const float loop = kFastTileUs * ((tiles + k - 1) / k) + kFastPartUs * k;
    if (loop + kFastClusterUs >= best) continue;
    const bool fits = k <= kFastMaxCluster && items <= kFastClusterRoom[k];
    const float us = loop + (fits ? kFastClusterUs : kFastWorkspaceUs);
    if (us < best && (fits || workspace)) {
      best = us;
      *parts = k;
      *cluster = fits ? 1 : 0;
    }
  }
}
int fwd_tiles(int T_hot, int T_ret) { return (T_hot + kFT - 1) / kFT + (T_ret + kFT - 1) / kFT; }
bool fwd_evenly(int items, int tiles, int n_sm, bool workspace) {     // one CTA per SM, with equal shares of all units
  return workspace && n_sm <= kFastMaxCtas && tiles >= kFastMinSplitTiles && items >= n_sm;
}

}  // namespace

int attn_forward_plan(int M, int H, int T_hot, int T_ret, int n_sm, bool workspace, int* parts, int* cluster) {
  const int items = (M + kBM - 1) / kBM * H, tiles = fwd_tiles(T_hot, T_ret);
  fwd_parts(items, tiles, n_sm, workspace && n_sm <= kFastMaxCtas, parts, cluster);
  return fwd_evenly(items, tiles, n_sm, workspace) ? n_sm : *parts * items;
}

void attn_subsample_plan(int M, float ratio, int* m_sub, int* stride, float* correction) {
  // attn-cuda/csrc/bindings.cpp:63-83
  if (ratio >= 0.999999f) {
    *m_sub = M; *stride = 1; *correction = 1.f;
    return;
  }
  int ms = static_cast<int>(M * ratio);
  if (ms < 128) ms = 128;
  ms = (ms / 128) * 128;
  if (ms >= M) {
    *m_sub = M; *stride = 1; *correction = 1.f;
  } else {
    *m_sub = ms;
    *stride = M / ms < 1 ? 1 : M / ms;
    *correction = static_cast<float>(M) / static_cast<float>(ms);
  }
}

// Words that have to be zero when a call begins and are zero again when it ends: one arrival counter per cut of
// the forward kernel and per shared item of the column-sum kernel.  They lie in front of the row log-sum-exps [H, M], at the same place
// whatever M and H are, so that one zeroed workspace serves calls of all sizes.
enum { kCtlFwdCuts = 0, kCtlColItems = kCtlFwdCuts + kFastMaxCtas,
       kCtlUsed = kCtlColItems + kFastMaxCtas };
static_assert(kCtlUsed <= kAttnCtlWords, "control words");
size_t attn_lse2_elems(int M, int H) { return static_cast<size_t>(H) * static_cast<size_t>(M) + kAttnCtlWords; }

// partial results of the split forward kernel (two slots per CTA), then the partial column sums of
// a column-sum launch with fewer items than CTAs (two slots per CTA)
constexpr size_t kFwdPartElems = static_cast<size_t>(2) * kFastMaxCtas * kPartFloats;
constexpr size_t kColPartElems = static_cast<size_t>(2) * kFastMaxCtas * kColGroup * kBN;
size_t attn_part_elems() { return kFwdPartElems + kColPartElems; }

int attn_colsum_launch(const AttnArgs& a, int* ctl, bool ctl_zeroed, float* lse2, float* part, int* err,
                       cudaStream_t stream) {
  if (a.D != kD) return STAC_ERR_BAD_ARG;
  if (a.M <= 0 || a.H <= 0 || a.T_hot < 0 || a.T_ret < 0 || a.T_hot + a.T_ret <= 0) return STAC_ERR_BAD_ARG;
  if (a.T_ret > 0 && (a.k_ret == nullptr || a.v_ret == nullptr || a.bias_ret == nullptr)) return STAC_ERR_BAD_ARG;
  if (a.T_hot > 0 && (a.k_hot == nullptr || a.v_hot == nullptr)) return STAC_ERR_BAD_ARG;
  if (a.scores != nullptr && (part == nullptr || a.colsum == nullptr || a.counts == nullptr || a.old_T < 0 || a.score_Tq <= 0))
    return STAC_ERR_BAD_ARG;
  if ((reinterpret_cast<uintptr_t>(a.q) | reinterpret_cast<uintptr_t>(a.k_hot) | reinterpret_cast<uintptr_t>(a.v_hot) |
       reinterpret_cast<uintptr_t>(a.k_ret) | reinterpret_cast<uintptr_t>(a.v_ret) |
       reinterpret_cast<uintptr_t>(a.out)) & 15)
    return STAC_ERR_BAD_ARG;

  int dev = 0;
  if (current_device(&dev) != STAC_OK) return STAC_ERR_CUDA;
  static PerDeviceFlag attr_done;   // the shared-memory opt-in is made once per device
  int m_sub, stride;
  float corr;
  attn_subsample_plan(a.M, a.subsample_ratio, &m_sub, &stride, &corr);
  const int nq = (m_sub + kBM - 1) / kBM;
  auto col_smem = [&](int group) {
    const size_t fixed = group == 1 ? sizeof(ColSmem<1>) : group == 2 ? sizeof(ColSmem<2>) : sizeof(ColSmem<3>);
    return static_cast<int>(fixed) + (kColFoldLse ? 0 : nq * kBM * 4) + 1024;
  };
  if (col_smem(kColGroup) > 227 * 1024) return STAC_ERR_BAD_ARG;
  const int fast_smem = static_cast<int>(sizeof(FastSmem)) + 1024;
  if (attr_done.needs_setup(dev)) {
    if (cudaFuncSetAttribute(attn_fwd_fast_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, fast_smem) !=
        cudaSuccess)
      return STAC_ERR_CUDA;
    for (auto* kernel : {attn_colsum_kernel<1>, attn_colsum_kernel<2>, attn_colsum_kernel<kColGroup>})
      if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess)
        return STAC_ERR_CUDA;
    attr_done.mark(dev);
  }

  const uint64_t eb = 2;  // bytes per element
  CUtensorMap tm_q, tm_qs, tm_kh, tm_kr;
  CUtensorMap tf_kh, tf_vh, tf_kr, tf_vr;   // keys and values in 112-key boxes (forward kernel)
  int rc;
  // q[m, h, :]: dims {64, H, M}
  rc = make_map(&tm_q, a.q, a.H, a.M, kD * eb, a.q_row_stride * eb, 1, kBM);
  if (rc) return rc;
  rc = make_map(&tm_qs, a.q, a.H, m_sub, kD * eb, a.q_row_stride * eb * stride, 1, kBM);
  if (rc) return rc;
  // placeholders keep the maps valid when a segment is empty
  const void* kh = a.T_hot > 0 ? a.k_hot : a.k_ret;
  const void* vh = a.T_hot > 0 ? a.v_hot : a.v_ret;
  const int th = a.T_hot > 0 ? a.T_hot : a.T_ret;
  const long long sh = a.T_hot > 0 ? a.hot_head_stride : a.ret_head_stride;
  const long long rh = a.T_hot > 0 ? a.hot_row_stride : a.ret_row_stride;
  const void* kr = a.T_ret > 0 ? a.k_ret : a.k_hot;
  const void* vr = a.T_ret > 0 ? a.v_ret : a.v_hot;
  const int tr = a.T_ret > 0 ? a.T_ret : a.T_hot;
  const long long sr = a.T_ret > 0 ? a.ret_head_stride : a.hot_head_stride;
  const long long rr = a.T_ret > 0 ? a.ret_row_stride : a.hot_row_stride;
  rc = make_map(&tm_kh, kh, th, a.H, rh * eb, sh * eb, kBN, 1);
  if (rc) return rc;
  rc = make_map(&tm_kr, kr, tr, a.H, rr * eb, sr * eb, kBN, 1);
  if (rc) return rc;
  rc = make_map(&tf_kh, kh, th, a.H, rh * eb, sh * eb, kFT, 1);
  if (rc) return rc;
  rc = make_map(&tf_vh, vh, th, a.H, rh * eb, sh * eb, kFT, 1);
  if (rc) return rc;
  rc = make_map(&tf_kr, kr, tr, a.H, rr * eb, sr * eb, kFT, 1);
  if (rc) return rc;
  rc = make_map(&tf_vr, vr, tr, a.H, rr * eb, sr * eb, kFT, 1);
  if (rc) return rc;

  const float scale_log2 = a.scale * kLog2e;
  FwdParams fp;
  fp.M = a.M; fp.H = a.H; fp.T_hot = a.T_hot; fp.T_ret = a.T_ret;
  fp.scale_log2 = scale_log2;
  fp.bias_ret = a.bias_ret; fp.bias_head_stride = a.bias_head_stride;
  fp.out = static_cast<__nv_bfloat16*>(a.out); fp.out_row_stride = a.out_row_stride;
  fp.lse = a.lse; fp.lse2 = lse2; fp.lse2_stride = a.M;
  fp.err = err;
  int n_sm = 0;
  if (device_sm_count(dev, &n_sm) != STAC_OK) return STAC_ERR_CUDA;
  // With at least one item per SM (and a workspace for the parts) the units are cut evenly over one CTA per SM and an item is shared by at
  // most two of them; with at most half as many items as SMs (few heads, e.g. a head-sharded stream) every item is cut in equal
  // parts where that pays; else every CTA takes one item.
  fp.n_q_tiles = (a.M + kBM - 1) / kBM;
  fp.n_items = fp.n_q_tiles * a.H;
  const int n_tiles_f = fwd_tiles(a.T_hot, a.T_ret);
  const bool workspace = part != nullptr && n_sm <= kFastMaxCtas;
  int grid_split = fwd_evenly(fp.n_items, n_tiles_f, n_sm, workspace) ? n_sm : 0;
  fwd_parts(fp.n_items, n_tiles_f, n_sm, workspace, &fp.parts, &fp.cluster);
  if (fp.cluster && workspace && max_fwd_clusters(dev, fp.parts, fast_smem) < fp.n_items) fp.cluster = 0;     // (would take turns)
  if (fp.parts > 1) grid_split = fp.parts * fp.n_items;
  fp.split = grid_split > 0 ? 1 : 0;
  fp.part = part;
  fp.part_count = ctl + kCtlFwdCuts;    // only used (and only present in the workspace) when split
  const int grid_fast = fp.split ? grid_split : fp.n_items;
  // Column sums: with at least one item per SM the units are cut evenly over one CTA per SM and an
  // item on a cut gets one atomic add per key from each of its two CTAs (the forward kernel clears
  // the output for that; a join through the workspace took 1 to 2 us more per call).  With fewer items (few heads,
  // short key ranges) and a workspace, the units are still cut evenly; an item may then have three or more parts,
  // which go through the workspace and are added in CTA order by the CTA that finishes last.
  const int col_hot_tiles = (a.T_hot + kBN - 1) / kBN, col_tiles = col_hot_tiles + (a.T_ret + kBN - 1) / kBN;
  auto items_of = [&](int group) { return (col_tiles + group - 1) / group * a.H; };
  const int col_items = items_of(kColGroup);
  const bool col_split = a.colsum != nullptr && col_items >= n_sm;
  // (worth it from about six units per CTA: below that the extra key-tile loads and the join of a
  // CTA that touches two items cost more than the even cut gains; measured at M = 1041, N = 2082)
  const bool col_parts = a.colsum != nullptr && !col_split && part != nullptr && n_sm <= kFastMaxCtas &&
                         static_cast<long long>(col_items) * nq >= 6ll * n_sm;
  // Where a call is one wave of one item per CTA, smaller groups fill more SMs as long as they are still one wave: a CTA's
  // query tiles then take an exponent unit less time each, although fewer warps keep it busy.  us per call with groups of
  // three / two / one (where that is one wave): M 1041, N 2082, 16 heads 37.6 / 34.6; M 1041, N 1041 32.6 / 29.0 / 27.6; M 200,
  // N 300, 2 heads 16.6 / 15.6 / 14.8; M 4164, N 1041, 2 heads 69.9 / 55.6 / 44.7.  Same sums in the same order.
  int col_group = kColGroup;
  if (!col_split && !col_parts)
    while (col_group > 1 && items_of(col_group - 1) <= n_sm) --col_group;
  // Every call leaves the control words as it found them, so a workspace that was zeroed once needs no
  // clearing: one memset less per call, and the forward kernel follows the kernel before it directly
  // (M = 1041, N = 2082, H = 16: 42.5 -> 38.2 us per call).
  if (!ctl_zeroed && (col_parts || (fp.split && !fp.cluster)) &&
      cudaMemsetAsync(ctl, 0, sizeof(int) * (col_parts ? kCtlUsed : kCtlColItems), stream) != cudaSuccess)
    return STAC_ERR_CUDA;
  fp.zero_colsum = col_split ? a.colsum : nullptr;
  fp.zero_stride = a.colsum_head_stride;
  fp.zero_width = a.T_hot + a.T_ret;
  if (launch_clusters_behind(attn_fwd_fast_kernel, dim3(grid_fast), fp.cluster ? fp.parts : 1, dim3(kFastThreads), fast_smem, stream, tm_q,
                             tf_kh, tf_vh, tf_kr, tf_vr, fp) != cudaSuccess)
    return STAC_ERR_CUDA;

  if (a.colsum != nullptr) {
    ColParams cp;
    cp.M_sub = m_sub; cp.H = a.H; cp.row_stride = stride;
    cp.T_hot = a.T_hot; cp.T_ret = a.T_ret;
    cp.n_hot_tiles = col_hot_tiles; cp.n_q_tiles = nq;
    cp.n_tiles = col_tiles;
    cp.n_groups = (cp.n_tiles + col_group - 1) / col_group;
    cp.n_items = cp.n_groups * a.H;
    cp.scale_log2 = scale_log2; cp.correction = corr;
    cp.bias_ret = a.bias_ret; cp.bias_head_stride = a.bias_head_stride;
    cp.lse2 = lse2; cp.lse2_stride = a.M;
    cp.colsum = a.colsum; cp.colsum_stride = a.colsum_head_stride;
    cp.err = err;
    cp.split = (col_split || col_parts) ? 1 : 0;      // col_split: the forward kernel has cleared a.colsum
    cp.parts = col_parts ? part + kFwdPartElems : nullptr;
    // Running scores: updated by the thread that has a key's final sum.  (us per call with a launch behind the kernel instead,
    // 16 heads: 128 rows, 3800 keys 32.4 against 31.0, 1041 rows, 3800 keys 51.1 against 49.6, 5600 keys 66.8 against 65.5.)
    cp.scores = a.scores; cp.counts = a.counts; cp.score_stride = a.score_stride;
    cp.old_T = a.old_T; cp.tq = static_cast<float>(a.score_Tq); cp.temperature = a.temperature;
    cp.part_count = ctl + kCtlColItems;
    const int grid_c = cp.split ? n_sm : cp.n_items;
    auto* const col_kernel = col_group == 1 ? attn_colsum_kernel<1> : col_group == 2 ? attn_colsum_kernel<2>
                                                                                     : attn_colsum_kernel<kColGroup>;
    if (launch_behind(col_kernel, dim3(grid_c), dim3(col_threads(col_group)), col_smem(col_group), stream, tm_qs, tm_kh,
                      tm_kr, cp) != cudaSuccess)
      return STAC_ERR_CUDA;
  }
  return STAC_OK;
}

}  // namespace stac

// ---------------------------------------------------------------------------------------
// Allocation-free variant: the row log-sum-exp scratch lives in a fixed array inside the
// loaded module instead of a caller-provided workspace.
// ---------------------------------------------------------------------------------------
namespace stac {
namespace {

// One float per (head, query row).  Every GPU that loads the library carries these 512 KB
// until the process exits.
static __device__ __align__(256) float g_static_lse2[STAC_ATTN_STATIC_MAX_ROWS + 64];  // control words first

float* g_static_lse2_ptr[kMaxDevices] = {nullptr};

// The array's name is only a host-side handle; the kernels need its device address, which
// differs per GPU.  Resolved once per device, with that device current.
int static_scratch_for_current_device(float** out) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return STAC_ERR_CUDA;
  if (g_static_lse2_ptr[dev] == nullptr) {
    void* ptr = nullptr;
    if (cudaGetSymbolAddress(&ptr, g_static_lse2) != cudaSuccess || ptr == nullptr) return STAC_ERR_CUDA;
    g_static_lse2_ptr[dev] = static_cast<float*>(ptr);
  }
  *out = g_static_lse2_ptr[dev];
  return STAC_OK;
}

}  // namespace
}  // namespace stac

extern "C" int stac_attn_colsum_noalloc(const void* q, int64_t q_row_stride, const void* k_hot, const void* v_hot,
                                        int64_t hot_row_stride, int64_t hot_head_stride, int T_hot,
                                        const void* k_ret, const void* v_ret, int64_t ret_row_stride,
                                        int64_t ret_head_stride, int T_ret, const float* bias_ret,
                                        int64_t bias_head_stride, void* out, int64_t out_row_stride, float* lse,
                                        float* colsum, int64_t colsum_head_stride, int M, int H, int D, float scale,
                                        float subsample_ratio, int* dev_status, stac_stream_t stream) {
  if (q == nullptr || out == nullptr) return STAC_ERR_BAD_ARG;
  if (!(subsample_ratio > 0.f && subsample_ratio <= 1.f)) return STAC_ERR_BAD_ARG;
  if (M <= 0 || H <= 0) return STAC_ERR_BAD_ARG;
  // the fixed scratch holds H * M floats at most
  if (static_cast<long long>(M) * H > STAC_ATTN_STATIC_MAX_ROWS) return STAC_ERR_CAPACITY;
  if ((q_row_stride % 8) || (out_row_stride % 8) || (hot_head_stride % 8) || (ret_head_stride % 8) ||
      (hot_row_stride % 8) || (ret_row_stride % 8))
    return STAC_ERR_BAD_ARG;
  float* scratch = nullptr;
  const int rc = stac::static_scratch_for_current_device(&scratch);
  if (rc != STAC_OK) return rc;
  stac::AttnArgs a;
  a.q = q; a.q_row_stride = q_row_stride;
  a.k_hot = k_hot; a.v_hot = v_hot; a.hot_row_stride = hot_row_stride; a.hot_head_stride = hot_head_stride;
  a.T_hot = T_hot;
  a.k_ret = k_ret; a.v_ret = v_ret; a.ret_row_stride = ret_row_stride; a.ret_head_stride = ret_head_stride;
  a.T_ret = T_ret;
  a.bias_ret = bias_ret; a.bias_head_stride = bias_head_stride;
  a.out = out; a.out_row_stride = out_row_stride;
  a.lse = lse; a.colsum = colsum; a.colsum_head_stride = colsum_head_stride;
  a.M = M; a.H = H; a.D = D; a.scale = scale; a.subsample_ratio = subsample_ratio;
  // Every entry of the scratch that the column-sum pass reads (rows < M of each head) is
  // written by the forward pass of this same call, so nothing has to be cleared first.
  return stac::attn_colsum_launch(a, reinterpret_cast<int*>(scratch), false, scratch + 64, nullptr, dev_status,
                                  reinterpret_cast<cudaStream_t>(stream));
}

#ifdef STAC_TIMESTAMPS
extern "C" int stac_debug_stamps(unsigned long long* out, int reset) {
  if (out != nullptr && cudaMemcpyFromSymbol(out, stac::g_ts, sizeof(unsigned long long) * 8) != cudaSuccess) return 1;
  if (reset) {
    const unsigned long long init[8] = {~0ull, 0ull, ~0ull, 0ull, ~0ull, 0ull, ~0ull, 0ull};
    if (cudaMemcpyToSymbol(stac::g_ts, init, sizeof(init)) != cudaSuccess) return 1;
  }
  return 0;
}
#endif
