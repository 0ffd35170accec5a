// H2O heavy-hitter bookkeeping on the hot cache: score update, keep-set selection and the
// gather-compaction of the cache.
//
// Replaces stac/h2o.py:177-216 (_update_scores), stac/h2o.py:244-354 (_parallel_prune_kv:
// index_select + torch.topk + cat + torch.sort over [L*H, T]) and stac/h2o.py:356-436 with
// stac/stac_voxel.py:409-419 (six torch.gather compactions with full-size temporaries).
#include "common.cuh"
#include "stac_internal.h"

namespace stac {
namespace {

// score = colsum * T_live / Tq; new tail is written, the old prefix decays:
// score = score * temperature + s (two roundings, as mul_ then add_), count += 1.
__global__ void scores_update_kernel(const float* __restrict__ colsum, long long colsum_stride,
                                     float* __restrict__ scores, float* __restrict__ counts, long long row_stride,
                                     int H, int T_live, int old_T, float t_live_f, float tq_f, float temperature) {
  grid_dep_wait();   // launched with programmatic serialization behind the column-sum kernel
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int h = blockIdx.y;
  if (t >= T_live) return;
  const float s = __fdiv_rn(__fmul_rn(colsum[h * colsum_stride + t], t_live_f), tq_f);
  const long long o = h * row_stride + t;
  if (t >= old_T) {
    scores[o] = s;
  } else {
    scores[o] = __fadd_rn(__fmul_rn(scores[o], temperature), s);
  }
  counts[o] = __fadd_rn(counts[o], 1.0f);
}

__device__ __forceinline__ unsigned int float_key(float f) {
  const unsigned int u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// One CTA per (layer, head) row.  Positions flagged in `is_base` (pinned and recent tokens)
// are always kept; of the others the `k` highest scores are kept (ties: lower position
// first).  Emits the kept positions and the dropped positions, both ascending.
// Bound by the instructions per key and by a chain of latencies and barriers, so every pass over the keys is kept short: counters
// are bumped by plain shared-memory increments (the unit adds up the lanes of one address; counting the lanes of one digit by a
// ballot first took 3 to 12 % longer, also with one score for all), the first digit is counted while the keys are loaded, the
// search ends when few keys share the prefix that is known, and the positions are written by warps that need no barrier
// between them.  (Cold, 384 rows of 8328, 11451, 15615 tokens 39, 46, 61 -> 26, 28, 35 us, with four passes of eight bits and block scans per
// 4 kThreads positions before; 48 rows of 11451 24 -> 16, 384 of 30000 147 -> 73.)
// 1024 threads, two CTAs per SM, as long as that is one wave of rows, else 512 where three of them or four share an SM.
// (384 rows, 1024 against 512 threads: 8328 tokens 29.7, 25.6 us, 15615 tokens 38.3, 34.8, 18600 tokens 43.0, 41.5.)  A row's
// keys lie in shared memory: from 18881 tokens only two fit an SM, from 28 thousand only one, and the larger CTAs have twice
// the warps there (19500 tokens 43.9, 52.2, 33000 tokens 79, 111).
constexpr int kSelectStaticSmem = 1280;      // counters and such of a CTA of 512 threads, rounded up
static_assert(kSelectStaticSmem >= (256 + 2 * 512 / 32 + 4) * 4, "static shared memory of the selection kernel");
// Keys that share a prefix and are ranked against one another, which takes the square of their number: they fit the counters' memory.  (Up to 256
// of them: rows of 300 equal scores 9.7 against 5.6 us, 384 rows, and 7.0 with four passes before there was a ranking; 600 and 1041 small whole numbers 10.6, 11.2
// against 7.0, 7.2; 4164 scores over many decades 17.3 against 11.2.  Up to 64 or 32: no better.)
constexpr int kSelectFew = 128;
template <int kThreads>
__global__ void __launch_bounds__(kThreads, 2048 / kThreads)
h2o_select_kernel(const float* __restrict__ scores, long long row_stride, const unsigned char* __restrict__ is_base,
                  int T, int n_keep, int* __restrict__ keep_idx, int* __restrict__ drop_idx) {
  grid_dep_wait();   // launched with programmatic serialization behind the previous kernel in the stream
  extern __shared__ unsigned int keys[];
  __shared__ int hist[256];
  __shared__ int warp_gt[kThreads / 32], warp_eq[kThreads / 32];
  __shared__ unsigned int sh_prefix;
  __shared__ int sh_remaining, sh_ties, sh_count;
  const int row = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float* srow = scores + row * row_stride;
  if (threadIdx.x < 256) hist[threadIdx.x] = 0;
  if (threadIdx.x == 0) {
    sh_prefix = 0;
    sh_remaining = n_keep;
    sh_count = 0;
  }
  __syncthreads();
  // four independent loads per thread in flight; the first digit is counted on the way
  for (int base = 0; base < T; base += 4 * kThreads) {
    float sc[4];
    unsigned char bs[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int t = base + j * kThreads + static_cast<int>(threadIdx.x);
      sc[j] = t < T ? srow[t] : 0.f;
      bs[j] = t < T ? is_base[t] : static_cast<unsigned char>(0);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int t = base + j * kThreads + static_cast<int>(threadIdx.x);
      if (t < T) {
        const unsigned int k = bs[j] ? 0xFFFFFFFFu : float_key(sc[j]);
        keys[t] = k;
        atomicAdd(&hist[k >> 24], 1);
      }
    }
  }
  // radix select: find the n_keep-th largest key, 8 bits at a time from the top, until few keys share what is known of it
  unsigned int tau = 0;      // the n_keep-th largest key
  int need_eq = 0;           // how many keys equal to tau are kept
  for (int shift = 24;; shift -= 8) {
    __syncthreads();
    if (warp == 0) {
      // the digit at which the count from the top reaches what remains: lane 0 holds the eight highest
      // counters (one thread walking all 256, four times per row, was a third of the kernel's time: 24 layers
      // of 16 heads, eight frames of 1041 tokens 65 -> 42 us; two layers of 4 heads, 560 tokens 18 -> 6 us)
      const int remaining = sh_remaining;
      const unsigned int prefix = sh_prefix;
      int c[8], sum = 0;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        c[e] = hist[(31 - lane) * 8 + 7 - e];
        sum += c[e];
      }
      int incl = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
      }
      int above = incl - sum;
      __syncwarp();
      if (above < remaining && incl >= remaining) {       // exactly one lane
        int d = 0, ties = 0;
        bool found = false;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          if (!found) {
            if (above + c[e] >= remaining) {
              found = true;
              d = (31 - lane) * 8 + 7 - e;
              ties = c[e];
            } else {
              above += c[e];
            }
          }
        }
        sh_prefix = prefix | (static_cast<unsigned int>(d) << shift);
        sh_remaining = remaining - above;
        sh_ties = ties;
      }
    }
    __syncthreads();
    const unsigned int prefix = sh_prefix;
    const int remaining = sh_remaining, ties = sh_ties;
    tau = prefix;
    need_eq = remaining;
    if (shift == 0) break;
    const unsigned int known = 0xFFFFFFFFu << shift;
    if (ties <= kSelectFew) {
      // they are collected (the counters are done with: their memory) and each is ranked against the others
      for (int t = threadIdx.x; t < T; t += kThreads) {
        const unsigned int k = keys[t];
        if ((k & known) == prefix) hist[atomicAdd(&sh_count, 1)] = static_cast<int>(k);
      }
      __syncthreads();
      if (threadIdx.x < static_cast<unsigned>(ties)) {
        const unsigned int k = static_cast<unsigned int>(hist[threadIdx.x]);
        int gt = 0, eq = 0;
        for (int i = 0; i < ties; ++i) {
          const unsigned int o = static_cast<unsigned int>(hist[i]);
          gt += o > k;
          eq += o == k;
        }
        if (gt < remaining && gt + eq >= remaining) {     // the threads of one key, with the same values
          sh_prefix = k;
          sh_remaining = remaining - gt;
        }
      }
      __syncthreads();
      tau = sh_prefix;
      need_eq = sh_remaining;
      break;
    }
    if (threadIdx.x < 256) hist[threadIdx.x] = 0;
    __syncthreads();
    for (int t = threadIdx.x; t < T; t += kThreads) {
      const unsigned int k = keys[t];
      if ((k & known) == prefix) atomicAdd(&hist[(k >> (shift - 8)) & 255u], 1);
    }
  }
  // Emission: a warp has a run of positions.  It counts its keys above and at tau; with the counts of the warps before it,
  // 32 positions at a time find their places by ballots, without a barrier.
  int* krow = keep_idx + static_cast<long long>(row) * n_keep;
  int* drow = drop_idx + static_cast<long long>(row) * (T - n_keep);
  const int run = ((T + kThreads - 1) / kThreads) * 32;
  const int first = min(T, warp * run), end = min(T, first + run);
  int gt = 0, eq = 0;
  for (int t = first + lane; t < end; t += 32) {
    const unsigned int k = keys[t];
    gt += k > tau;
    eq += k == tau;
  }
  gt = __reduce_add_sync(0xffffffffu, gt);
  eq = __reduce_add_sync(0xffffffffu, eq);
  if (lane == 0) {
    warp_gt[warp] = gt;
    warp_eq[warp] = eq;
  }
  __syncthreads();
  gt = __reduce_add_sync(0xffffffffu, lane < warp ? warp_gt[lane] : 0);
  eq = __reduce_add_sync(0xffffffffu, lane < warp ? warp_eq[lane] : 0);
  int kept = gt + min(eq, need_eq);
  const unsigned int below = (1u << lane) - 1u;
#pragma unroll 2
  for (int base = first; base < end; base += 32) {
    const int t = base + lane;
    const bool in = t < end;
    const unsigned int k = in ? keys[t] : 0u;
    const unsigned int at = __ballot_sync(0xffffffffu, in && k == tau);
    const bool keep = in && (k > tau || (k == tau && eq + __popc(at & below) < need_eq));
    const unsigned int kept_here = __ballot_sync(0xffffffffu, keep);
    const int place = kept + __popc(kept_here & below);       // kept positions of the row before this one
    if (keep) krow[place] = t;
    else if (in) drow[t - place] = t;
    eq += __popc(at);
    kept += __popc(kept_here);
  }
}

// Gather-compaction into a second set of buffers: dst[row, j] = src[row, keep[row, j]].
// K and V move as 16-byte vectors, eight threads per 128-byte (bf16) or sixteen per 256-byte
// (fp32) row.  `keep_stride` is 0 where all rows keep the same positions.
__global__ void compact_kv_kernel(const int* __restrict__ keep_idx, long long keep_stride, int n_keep,
                                  const uint4* __restrict__ k_src,
                                  const uint4* __restrict__ v_src, uint4* __restrict__ k_dst,
                                  uint4* __restrict__ v_dst, long long row_stride_vec, int vec_per_token) {
  grid_dep_wait();   // launched with programmatic serialization behind the previous kernel in the stream
  const long long gid = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int row = blockIdx.y;
  const long long tok = gid / vec_per_token;
  const int part = static_cast<int>(gid % vec_per_token);
  if (tok >= n_keep) return;
  const int src = keep_idx[row * keep_stride + tok];
  const long long so = row * row_stride_vec + static_cast<long long>(src) * vec_per_token + part;
  const long long dof = row * row_stride_vec + tok * vec_per_token + part;
  k_dst[dof] = k_src[so];
  v_dst[dof] = v_src[so];
}

// kScores: the cache has score and count arrays.  (A template and not a test of the pointer: the loads of a
// token are then requested together.  24 layers of 16 heads, rows of 11 frames of 1041 tokens: 53.4 -> 47.4 us.)
template <bool kScores>
__global__ void compact_meta_kernel(const int* __restrict__ keep_idx, long long keep_stride, int n_keep, int T_buf,
                                    const long long* __restrict__ ti_src, long long* __restrict__ ti_dst,
                                    const float* __restrict__ s_src, float* __restrict__ s_dst,
                                    const float* __restrict__ c_src, float* __restrict__ c_dst,
                                    const int* __restrict__ vx_src, int* __restrict__ vx_dst) {
  grid_dep_wait();   // launched with programmatic serialization behind the previous kernel in the stream
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  const int row = blockIdx.y;
  if (j >= T_buf) return;
  const long long o = static_cast<long long>(row) * T_buf + j;
  if (j < n_keep) {
    const long long s = static_cast<long long>(row) * T_buf + keep_idx[row * keep_stride + j];
    ti_dst[o] = ti_src[s];
    if constexpr (kScores) {
      s_dst[o] = s_src[s];
      c_dst[o] = c_src[s];
    }
    if (vx_src != nullptr) vx_dst[o] = vx_src[s];
  } else {
    ti_dst[o] = -1;
    if constexpr (kScores) {
      s_dst[o] = 0.f;
      c_dst[o] = 0.f;
    }
    if (vx_dst != nullptr) vx_dst[o] = -1;
  }
}

// New K/V rows of one layer into the tail of the hot cache plus their global token ids, one
// launch instead of three strided copies (stac/kv_manager.py:285-305).
__global__ void append_kv_kernel(const uint4* __restrict__ k, const uint4* __restrict__ v, long long k_head_stride_vec,
                                 long long k_row_stride_vec, long long v_head_stride_vec, long long v_row_stride_vec,
                                 uint4* __restrict__ k_cache, uint4* __restrict__ v_cache,
                                 long long cache_head_stride_vec, long long* __restrict__ token_idx,
                                 long long idx_head_stride, int T_new, int old_T, long long first_id,
                                 int vec_per_token) {
  grid_dep_wait();   // launched with programmatic serialization: whatever produced k and v is complete now
  const int h = blockIdx.y;
  const long long total = static_cast<long long>(T_new) * vec_per_token;
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
  const long long g0 = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  // four 16-byte vectors of K and of V per thread, all loads before the stores
  uint4 kv[4], vv[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const long long gid = g0 + j * stride;
    if (gid < total) {
      const long long t = gid / vec_per_token;
      const int part = static_cast<int>(gid - t * vec_per_token);
      kv[j] = k[h * k_head_stride_vec + t * k_row_stride_vec + part];
      vv[j] = v[h * v_head_stride_vec + t * v_row_stride_vec + part];
    }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const long long gid = g0 + j * stride;
    if (gid < total) {
      const long long t = gid / vec_per_token;
      const int part = static_cast<int>(gid - t * vec_per_token);
      const long long dst = h * cache_head_stride_vec + (old_T + t) * vec_per_token + part;
      k_cache[dst] = kv[j];
      v_cache[dst] = vv[j];
      if (part == 0) token_idx[h * idx_head_stride + old_T + t] = first_id + t;
    }
  }
}

// The epilogue of the attention layer's QKV projection fused with append_kv
// (causalvggt/layers/attention.py:119-128 and :141): the three 64-value rows q, k, v of every
// (token, head) of the projection output; LayerNorm over the head dimension for q and k (fp32: mean,
// biased variance, eps, affine), the 2-D rotary embedding (dims 0..31 turn with the token's y
// position, dims 32..63 with its x position; 16 frequencies each, rotate-half form, cos / sin
// read from the caller's tables), rounded to bf16, q written to the query tensor and k, v straight into
// the cache tail together with the token id.
//
// Eight lanes per (token, head), eight neighbouring dims each, so that every row moves in 16-byte
// vectors: lane s holds dims 8 s ... 8 s + 7, dim d + 32 lies in lane s ^ 4 and the rotation partner d ^ 16
// in lane s ^ 2.  (One warp per (token, head) with two 2-byte values per lane was bound by its
// instructions, not by memory: 2082 tokens and 16 heads 15.5 -> 10.7 us.  The table rows are read where
// they lie; copies of them took 4.3 us per layer.)

// Total of z(x[d], x[d + 32]) over d = 0..31 for a row held by eight lanes: dims 32 apart first, then 16
// and 8 (across lanes), then 4, 2 and 1.  Values are handed over so that each lane carries on with
// half of its sums; every lane gets the total.
template <typename Z>
__device__ __forceinline__ float row64_sum(const float (&x)[8], int sub, unsigned gmask, Z z) {
  float y4[4], y2[2];
  const bool h4 = sub & 4, h2 = sub & 2, h1 = sub & 1;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float own = h4 ? x[j + 4] : x[j];
    const float oth = __shfl_xor_sync(gmask, h4 ? x[j] : x[j + 4], 4);
    y4[j] = z(h4 ? oth : own, h4 ? own : oth);
  }
#pragma unroll
  for (int j = 0; j < 2; ++j)
    y2[j] = (h2 ? y4[j + 2] : y4[j]) + __shfl_xor_sync(gmask, h2 ? y4[j] : y4[j + 2], 2);
  float t = (h1 ? y2[1] : y2[0]) + __shfl_xor_sync(gmask, h1 ? y2[0] : y2[1], 1);
  t += __shfl_xor_sync(gmask, t, 4);
  t += __shfl_xor_sync(gmask, t, 2);
  t += __shfl_xor_sync(gmask, t, 1);
  return t;
}

template <bool kVec>   // the rows of qkv, q_out and the cache are 16-byte aligned
__global__ void __launch_bounds__(256) qkv_epilogue_kernel(
    const __nv_bfloat16* __restrict__ qkv, long long token_stride, int H, const float* __restrict__ q_w,
    const float* __restrict__ q_b, const float* __restrict__ k_w, const float* __restrict__ k_b, float eps,
    const long long* __restrict__ pos, const float* __restrict__ cos_tab, const float* __restrict__ sin_tab,
    long long tab_stride, int n_pos, __nv_bfloat16* __restrict__ q_out, long long q_row_stride,
    __nv_bfloat16* __restrict__ k_cache, __nv_bfloat16* __restrict__ v_cache, long long cache_head_stride,
    long long* __restrict__ token_idx, long long idx_head_stride, int T_new, int old_T, long long first_id) {
  grid_dep_wait();   // launched with programmatic serialization: the projection that wrote qkv is complete now
  const int sub = threadIdx.x & 7;
  const unsigned gmask = 0xffu << (threadIdx.x & 24);
  const long long w = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 3;
  if (w >= static_cast<long long>(T_new) * H) return;
  const int t = static_cast<int>(w / H), h = static_cast<int>(w - static_cast<long long>(t) * H);
  auto load = [&](const __nv_bfloat16* row) {
    if constexpr (kVec) {
      return reinterpret_cast<const uint4*>(row)[sub];
    } else {
      unsigned v[4];
#pragma unroll
      for (int j = 0; j < 4; ++j)
        v[j] = static_cast<unsigned>(__bfloat16_as_ushort(row[8 * sub + 2 * j])) |
               (static_cast<unsigned>(__bfloat16_as_ushort(row[8 * sub + 2 * j + 1])) << 16);
      return make_uint4(v[0], v[1], v[2], v[3]);
    }
  };
  auto store = [&](__nv_bfloat16* row, uint4 u) {
    if (kVec) {
      reinterpret_cast<uint4*>(row)[sub] = u;
    } else {
      const unsigned v[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        row[8 * sub + 2 * j] = __ushort_as_bfloat16(static_cast<unsigned short>(v[j] & 0xffffu));
        row[8 * sub + 2 * j + 1] = __ushort_as_bfloat16(static_cast<unsigned short>(v[j] >> 16));
      }
    }
  };
  const __nv_bfloat16* src = qkv + t * token_stride + h * 64;
  const uint4 uq = load(src), uk = load(src + H * 64), uv = load(src + 2 * H * 64);
  float c[8], s[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    c[e] = 1.f;
    s[e] = 0.f;
  }
  if (cos_tab != nullptr) {
    long long at = pos[2 * t + (sub >> 2)];          // lanes 0-3 turn with y, 4-7 with x
    at = at < 0 ? 0 : (at >= n_pos ? n_pos - 1 : at);
    const long long o = at * tab_stride + (sub & 1) * 8;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      c[e] = cos_tab[o + e];
      s[e] = sin_tab[o + e];
    }
  }
  const float sign = (sub & 2) ? 1.f : -1.f;     // rotate-half: (-x2, x1)
  auto norm_rope = [&](uint4 u, const float* wgt, const float* bia) {
    float x[8];
    x[0] = __uint_as_float(u.x << 16); x[1] = __uint_as_float(u.x & 0xffff0000u);
    x[2] = __uint_as_float(u.y << 16); x[3] = __uint_as_float(u.y & 0xffff0000u);
    x[4] = __uint_as_float(u.z << 16); x[5] = __uint_as_float(u.z & 0xffff0000u);
    x[6] = __uint_as_float(u.w << 16); x[7] = __uint_as_float(u.w & 0xffff0000u);
    if (wgt != nullptr) {
      const float sum = row64_sum(x, sub, gmask, [](float a, float b) { return a + b; });
      const float mean = sum * (1.f / 64.f);
#pragma unroll
      for (int e = 0; e < 8; ++e) x[e] = x[e] - mean;
      const float sq = row64_sum(x, sub, gmask, [](float a, float b) { return a * a + b * b; });
      const float rstd = rsqrtf(sq * (1.f / 64.f) + eps);
#pragma unroll
      for (int e = 0; e < 8; ++e) x[e] = x[e] * rstd * wgt[8 * sub + e] + bia[8 * sub + e];
    }
    if (cos_tab != nullptr) {
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float px = __shfl_xor_sync(gmask, x[e], 2);
        x[e] = x[e] * c[e] + sign * px * s[e];
      }
    }
    return make_uint4(pack_bf16x2(x[0], x[1]), pack_bf16x2(x[2], x[3]), pack_bf16x2(x[4], x[5]), pack_bf16x2(x[6], x[7]));
  };
  store(q_out + t * q_row_stride + h * 64, norm_rope(uq, q_w, q_b));
  const long long dst = h * cache_head_stride + static_cast<long long>(old_T + t) * 64;
  store(k_cache + dst, norm_rope(uk, k_w, k_b));
  store(v_cache + dst, uv);
  if (sub == 0) token_idx[h * idx_head_stride + old_T + t] = first_id + t;
}

}  // namespace
}  // namespace stac

extern "C" {

int stac_qkv_epilogue_append_tables(const void* qkv, int64_t qkv_token_stride, const float* q_norm_w,
                                    const float* q_norm_b, const float* k_norm_w, const float* k_norm_b, float eps,
                                    const int64_t* pos, const float* cos_table, const float* sin_table,
                                    int64_t table_row_stride, int n_pos, void* q_out, int64_t q_out_row_stride,
                                    void* k_cache, void* v_cache, int64_t cache_head_stride, int64_t* token_idx,
                                    int64_t idx_head_stride, int H, int T_new, int old_T, int64_t first_token_id,
                                    stac_stream_t stream) {
  if (qkv == nullptr || q_out == nullptr || k_cache == nullptr || v_cache == nullptr || token_idx == nullptr ||
      H <= 0 || T_new < 0 || old_T < 0)
    return STAC_ERR_BAD_ARG;
  if ((q_norm_w == nullptr) != (q_norm_b == nullptr) || (k_norm_w == nullptr) != (k_norm_b == nullptr))
    return STAC_ERR_BAD_ARG;
  if (cos_table != nullptr && (sin_table == nullptr || pos == nullptr || n_pos <= 0 || table_row_stride < 16))
    return STAC_ERR_BAD_ARG;
  if (T_new == 0) return STAC_OK;
  const long long lanes = static_cast<long long>(T_new) * H * 8;
  const unsigned blocks = static_cast<unsigned>((lanes + 255) / 256);
  // whole rows move as 16-byte vectors where every row starts on a 16-byte boundary
  const bool vec = ((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(q_out) |
                     reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache)) & 15) == 0 &&
                   qkv_token_stride % 8 == 0 && q_out_row_stride % 8 == 0 && cache_head_stride % 8 == 0;
  if (stac::launch_behind(vec ? stac::qkv_epilogue_kernel<true> : stac::qkv_epilogue_kernel<false>, dim3(blocks),
      dim3(256), 0, reinterpret_cast<cudaStream_t>(stream),
      static_cast<const __nv_bfloat16*>(qkv), qkv_token_stride, H, q_norm_w, q_norm_b, k_norm_w, k_norm_b, eps,
      reinterpret_cast<const long long*>(pos), cos_table, sin_table, table_row_stride, n_pos,
      static_cast<__nv_bfloat16*>(q_out), q_out_row_stride, static_cast<__nv_bfloat16*>(k_cache),
      static_cast<__nv_bfloat16*>(v_cache), cache_head_stride, reinterpret_cast<long long*>(token_idx), idx_head_stride,
      T_new, old_T, first_token_id) != cudaSuccess)
    return STAC_ERR_CUDA;
  return STAC_OK;
}

int stac_qkv_epilogue_append(const void* qkv, int64_t qkv_token_stride, const float* q_norm_w, const float* q_norm_b,
                             const float* k_norm_w, const float* k_norm_b, float eps, const int64_t* pos,
                             const float* cos_table, const float* sin_table, int n_pos, void* q_out,
                             int64_t q_out_row_stride, void* k_cache, void* v_cache, int64_t cache_head_stride,
                             int64_t* token_idx, int64_t idx_head_stride, int H, int T_new, int old_T,
                             int64_t first_token_id, stac_stream_t stream) {
  return stac_qkv_epilogue_append_tables(qkv, qkv_token_stride, q_norm_w, q_norm_b, k_norm_w, k_norm_b, eps, pos,
                                         cos_table, sin_table, 16, n_pos, q_out, q_out_row_stride, k_cache, v_cache,
                                         cache_head_stride, token_idx, idx_head_stride, H, T_new, old_T,
                                         first_token_id, stream);
}

int stac_append_kv(const void* k, const void* v, int64_t k_head_stride, int64_t k_row_stride, int64_t v_head_stride,
                   int64_t v_row_stride, void* k_cache, void* v_cache, int64_t cache_head_stride, int64_t* token_idx,
                   int64_t idx_head_stride, int H, int T_new, int old_T, int64_t first_token_id, int head_dim,
                   int elem_bytes, stac_stream_t stream) {
  if (k == nullptr || v == nullptr || k_cache == nullptr || v_cache == nullptr || token_idx == nullptr || H <= 0 ||
      T_new < 0 || old_T < 0)
    return STAC_ERR_BAD_ARG;
  const int token_bytes = head_dim * elem_bytes;
  if (token_bytes % 16 != 0) return STAC_ERR_BAD_ARG;
  const int epv = 16 / elem_bytes;  // elements per 16-byte vector
  if ((k_head_stride % epv) || (k_row_stride % epv) || (v_head_stride % epv) || (v_row_stride % epv) ||
      (cache_head_stride % epv))
    return STAC_ERR_BAD_ARG;
  if ((reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) | reinterpret_cast<uintptr_t>(k_cache) |
       reinterpret_cast<uintptr_t>(v_cache)) & 15)
    return STAC_ERR_BAD_ARG;
  if (T_new == 0) return STAC_OK;
  const int vpt = token_bytes / 16;
  const long long total = static_cast<long long>(T_new) * vpt;
  dim3 grid(static_cast<unsigned>((total + 4 * 256 - 1) / (4 * 256)), H);   // four vectors per thread
  if (stac::launch_behind(stac::append_kv_kernel, grid, dim3(256), 0, reinterpret_cast<cudaStream_t>(stream),
      static_cast<const uint4*>(k), static_cast<const uint4*>(v), k_head_stride / epv, k_row_stride / epv,
      v_head_stride / epv, v_row_stride / epv, static_cast<uint4*>(k_cache), static_cast<uint4*>(v_cache),
      cache_head_stride / epv, reinterpret_cast<long long*>(token_idx), idx_head_stride, T_new, old_T, first_token_id,
      vpt) != cudaSuccess)
    return STAC_ERR_CUDA;
  return STAC_OK;
}

int stac_scores_update(const float* colsum, int64_t colsum_head_stride, float* scores, float* counts,
                       int64_t row_stride, int H, int T_live, int old_T, int Tq, float temperature,
                       stac_stream_t stream) {
  if (colsum == nullptr || scores == nullptr || counts == nullptr || H <= 0 || T_live < 0 || old_T < 0 || Tq <= 0)
    return STAC_ERR_BAD_ARG;
  if (T_live == 0) return STAC_OK;
  dim3 grid((T_live + 255) / 256, H);
  if (stac::launch_behind(stac::scores_update_kernel, grid, dim3(256), 0, reinterpret_cast<cudaStream_t>(stream),
                          colsum, colsum_head_stride, scores, counts, row_stride, H, T_live, old_T,
                          static_cast<float>(T_live), static_cast<float>(Tq), temperature) != cudaSuccess)
    return STAC_ERR_CUDA;
  return STAC_OK;
}

int stac_h2o_select(const float* scores, int64_t row_stride, int n_rows, const uint8_t* is_base, int T, int n_keep,
                    int* keep_idx, int* drop_idx, stac_stream_t stream) {
  if (scores == nullptr || is_base == nullptr || keep_idx == nullptr || (drop_idx == nullptr && n_keep < T) ||
      n_rows <= 0 || T <= 0 || n_keep <= 0 || n_keep > T)
    return STAC_ERR_BAD_ARG;
  const int smem = T * 4;
  if (smem > 200 * 1024) return STAC_ERR_CAPACITY;
  int dev = 0, n_sm = 0;
  if (stac::current_device(&dev) != STAC_OK || stac::device_sm_count(dev, &n_sm) != STAC_OK) return STAC_ERR_CUDA;
  static stac::PerDeviceFlag attr_done;   // the shared-memory opt-in is made once per device
  if (attr_done.needs_setup(dev)) {
    for (auto* kernel : {stac::h2o_select_kernel<1024>, stac::h2o_select_kernel<512>})
      if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) != cudaSuccess)
        return STAC_ERR_CUDA;
    attr_done.mark(dev);
  }
  // (228 KB per SM, 1 KB of it per CTA for the system)
  const bool three_per_sm = 3 * (smem + stac::kSelectStaticSmem + 1024) <= 228 * 1024;
  const bool small = n_rows > 2 * n_sm && three_per_sm;
  if (stac::launch_behind(small ? stac::h2o_select_kernel<512> : stac::h2o_select_kernel<1024>, dim3(n_rows),
                          dim3(small ? 512 : 1024), smem, reinterpret_cast<cudaStream_t>(stream),
                          scores, row_stride, is_base, T, n_keep, keep_idx, drop_idx) != cudaSuccess)
    return STAC_ERR_CUDA;
  return cudaGetLastError() == cudaSuccess ? STAC_OK : STAC_ERR_CUDA;
}

}  // extern "C"

namespace {

int compact_launch(const int* keep_idx, long long keep_stride, int n_rows, int n_keep, int T_buf, int head_dim, int elem_bytes,
                 const void* k_src, const void* v_src, void* k_dst, void* v_dst, const int64_t* ti_src,
                 int64_t* ti_dst, const float* s_src, float* s_dst, const float* c_src, float* c_dst,
                 const int* vx_src, int* vx_dst, stac_stream_t stream) {
  if ((vx_src == nullptr) != (vx_dst == nullptr)) return STAC_ERR_BAD_ARG;
  const int token_bytes = head_dim * elem_bytes;
  if (token_bytes % 16 != 0 || (elem_bytes != 2 && elem_bytes != 4)) return STAC_ERR_BAD_ARG;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int vpt = token_bytes / 16;
  if (n_keep > 0) {
    const long long total = static_cast<long long>(n_keep) * vpt;
    dim3 grid(static_cast<unsigned>((total + 255) / 256), n_rows);
    if (stac::launch_behind(stac::compact_kv_kernel, grid, dim3(256), 0, st, keep_idx, keep_stride, n_keep,
                            static_cast<const uint4*>(k_src), static_cast<const uint4*>(v_src),
                            static_cast<uint4*>(k_dst), static_cast<uint4*>(v_dst),
                            static_cast<long long>(T_buf) * vpt, vpt) != cudaSuccess)
      return STAC_ERR_CUDA;
  }
  dim3 grid_m((T_buf + 255) / 256, n_rows);
  auto* const meta_kernel = s_src != nullptr ? stac::compact_meta_kernel<true> : stac::compact_meta_kernel<false>;
  if (stac::launch_behind(meta_kernel, grid_m, dim3(256), 0, st, keep_idx, keep_stride, n_keep, T_buf,
                          reinterpret_cast<const long long*>(ti_src), reinterpret_cast<long long*>(ti_dst), s_src,
                          s_dst, c_src, c_dst, vx_src, vx_dst) != cudaSuccess)
    return STAC_ERR_CUDA;
  return cudaGetLastError() == cudaSuccess ? STAC_OK : STAC_ERR_CUDA;
}

}  // namespace

extern "C" {

int stac_compact(const int* keep_idx, int n_rows, int n_keep, int T_buf, int head_dim, int elem_bytes,
                 const void* k_src, const void* v_src, void* k_dst, void* v_dst, const int64_t* ti_src,
                 int64_t* ti_dst, const float* s_src, float* s_dst, const float* c_src, float* c_dst,
                 const int* vx_src, int* vx_dst, stac_stream_t stream) {
  if (keep_idx == nullptr || k_src == nullptr || v_src == nullptr || k_dst == nullptr || v_dst == nullptr ||
      ti_src == nullptr || ti_dst == nullptr || s_src == nullptr || s_dst == nullptr || c_src == nullptr ||
      c_dst == nullptr || n_rows <= 0 || n_keep < 0 || n_keep > T_buf)
    return STAC_ERR_BAD_ARG;
  return compact_launch(keep_idx, n_keep, n_rows, n_keep, T_buf, head_dim, elem_bytes, k_src, v_src, k_dst, v_dst, ti_src,
                        ti_dst, s_src, s_dst, c_src, c_dst, vx_src, vx_dst, stream);
}

int stac_compact_window(const int* keep_idx, int n_rows, int n_keep, int T_buf, int head_dim, int elem_bytes,
                        const void* k_src, const void* v_src, void* k_dst, void* v_dst, const int64_t* ti_src,
                        int64_t* ti_dst, stac_stream_t stream) {
  if (keep_idx == nullptr || k_src == nullptr || v_src == nullptr || k_dst == nullptr || v_dst == nullptr ||
      ti_src == nullptr || ti_dst == nullptr || n_rows <= 0 || n_keep < 0 || n_keep > T_buf)
    return STAC_ERR_BAD_ARG;
  return compact_launch(keep_idx, 0, n_rows, n_keep, T_buf, head_dim, elem_bytes, k_src, v_src, k_dst, v_dst, ti_src,
                        ti_dst, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, stream);
}

}  // extern "C"
