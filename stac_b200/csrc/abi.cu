// extern "C" entry points of libstac_b200.so: argument checks and dispatch only.
#include "common.cuh"
#include "stac_internal.h"

namespace stac {
namespace {

__global__ void bounded_wait_selftest_kernel(int max_polls, int* err) {
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    mbar_fence_init();
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    // Nothing ever arrives on this barrier: the poll loop must run out and report.
    bool done = false;
    for (int it = 0; it < max_polls && !done; ++it) done = mbar_try_wait(&bar, 0);
    if (!done) report_error(err, DEV_TEST_TIMEOUT);
  }
}

}  // namespace

int current_device(int* dev) {
  int d = -1;
  if (cudaGetDevice(&d) != cudaSuccess || !device_index_ok(d)) return STAC_ERR_CUDA;
  *dev = d;
  return STAC_OK;
}

int device_sm_count(int dev, int* n_sm) {
  static PerDeviceValue<int> cache;
  int n = cache.get(dev);
  if (n == 0) {
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return STAC_ERR_CUDA;
    cache.set(dev, n);
  }
  *n_sm = n;
  return STAC_OK;
}

}  // namespace stac

extern "C" {

const char* stac_status_string(int status) {
  switch (status) {
    case STAC_OK: return "ok";
    case STAC_ERR_BAD_ARG: return "bad argument";
    case STAC_ERR_CUDA: return "CUDA call failed";
    case STAC_ERR_CAPACITY: return "capacity too small";
    default: return "unknown status";
  }
}

int stac_abi_version(void) { return 2; }

uint64_t stac_kernel_launches(void) { return stac::g_kernel_launches.load(std::memory_order_relaxed); }

int stac_event_create(void** event) {
  if (event == nullptr) return STAC_ERR_BAD_ARG;
  cudaEvent_t e;
  if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) return STAC_ERR_CUDA;
  *event = e;
  return STAC_OK;
}

int stac_event_destroy(void* event) {
  if (event == nullptr) return STAC_ERR_BAD_ARG;
  return cudaEventDestroy(static_cast<cudaEvent_t>(event)) == cudaSuccess ? STAC_OK : STAC_ERR_CUDA;
}

int stac_event_wait(void* event) {
  if (event == nullptr) return STAC_ERR_BAD_ARG;
  return cudaEventSynchronize(static_cast<cudaEvent_t>(event)) == cudaSuccess ? STAC_OK : STAC_ERR_CUDA;
}

int stac_event_done(void* event, int* done) {
  if (event == nullptr || done == nullptr) return STAC_ERR_BAD_ARG;
  const cudaError_t rc = cudaEventQuery(static_cast<cudaEvent_t>(event));
  *done = rc == cudaSuccess ? 1 : 0;
  if (rc != cudaSuccess) cudaGetLastError();      // (an answer, no error that a later call is to find)
  return rc == cudaSuccess || rc == cudaErrorNotReady ? STAC_OK : STAC_ERR_CUDA;
}

int stac_ints_to_host(int* host, const int* a, int na, const int* b, int nb, void* event, stac_stream_t stream) {
  if (host == nullptr || event == nullptr || na < 0 || (na > 0 && a == nullptr) || nb < 0 || (nb > 0 && b == nullptr)) return STAC_ERR_BAD_ARG;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (na > 0 && cudaMemcpyAsync(host, a, sizeof(int) * na, cudaMemcpyDeviceToHost, st) != cudaSuccess) return STAC_ERR_CUDA;
  if (nb > 0 && cudaMemcpyAsync(host + na, b, sizeof(int) * nb, cudaMemcpyDeviceToHost, st) != cudaSuccess) return STAC_ERR_CUDA;
  return cudaEventRecord(static_cast<cudaEvent_t>(event), st) == cudaSuccess ? STAC_OK : STAC_ERR_CUDA;
}

size_t stac_attn_workspace_bytes(int M, int H) {
  if (M <= 0 || H <= 0) return 0;
  // control words and row log-sum-exps (rounded up to 256 bytes), then the partial results
  const size_t lse_bytes = (stac::attn_lse2_elems(M, H) * sizeof(float) + 255) & ~static_cast<size_t>(255);
  return lse_bytes + stac::attn_part_elems() * sizeof(float);
}

int stac_attn_forward_plan(int M, int H, int T_hot, int T_ret, int n_sm, int workspace, int* parts, int* cluster) {
  if (M <= 0 || H <= 0 || T_hot < 0 || T_ret < 0 || T_hot + T_ret <= 0 || n_sm <= 0 || parts == nullptr || cluster == nullptr) return 0;
  return stac::attn_forward_plan(M, H, T_hot, T_ret, n_sm, workspace != 0, parts, cluster);
}

}  // extern "C"

namespace {

int attn_colsum_in_workspace(bool zeroed, const void* q, int64_t q_row_stride, const void* k_hot, const void* v_hot,
                     int64_t hot_row_stride, int64_t hot_head_stride, int T_hot, const void* k_ret, const void* v_ret,
                     int64_t ret_row_stride, int64_t ret_head_stride, int T_ret, const float* bias_ret, int64_t bias_head_stride, void* out,
                     int64_t out_row_stride, float* lse, float* colsum, int64_t colsum_head_stride, int M, int H,
                     int D, float scale, float subsample_ratio, void* workspace, size_t workspace_bytes,
                     int* dev_status, stac_stream_t stream, float* scores = nullptr, float* counts = nullptr,
                     int64_t score_stride = 0, int old_T = 0, int Tq = 0, float temperature = 0.f) {
  if (q == nullptr || out == nullptr || workspace == nullptr) return STAC_ERR_BAD_ARG;
  if (!(subsample_ratio > 0.f && subsample_ratio <= 1.f)) return STAC_ERR_BAD_ARG;
  if (workspace_bytes < stac_attn_workspace_bytes(M, H)) return STAC_ERR_CAPACITY;
  if (reinterpret_cast<uintptr_t>(workspace) & 255) return STAC_ERR_BAD_ARG;
  if ((q_row_stride % 8) || (out_row_stride % 8) || (hot_head_stride % 8) || (ret_head_stride % 8) ||
      (hot_row_stride % 8) || (ret_row_stride % 8))
    return STAC_ERR_BAD_ARG;
  stac::AttnArgs a;
  a.q = q; a.q_row_stride = q_row_stride;
  a.k_hot = k_hot; a.v_hot = v_hot; a.hot_row_stride = hot_row_stride; a.hot_head_stride = hot_head_stride; a.T_hot = T_hot;
  a.k_ret = k_ret; a.v_ret = v_ret; a.ret_row_stride = ret_row_stride; a.ret_head_stride = ret_head_stride; a.T_ret = T_ret;
  a.bias_ret = bias_ret; a.bias_head_stride = bias_head_stride;
  a.out = out; a.out_row_stride = out_row_stride;
  a.lse = lse; a.colsum = colsum; a.colsum_head_stride = colsum_head_stride;
  a.M = M; a.H = H; a.D = D; a.scale = scale; a.subsample_ratio = subsample_ratio;
  a.scores = scores; a.counts = counts; a.score_stride = score_stride;
  a.old_T = old_T; a.score_Tq = Tq; a.temperature = temperature;
  const size_t lse_bytes = (stac::attn_lse2_elems(M, H) * sizeof(float) + 255) & ~static_cast<size_t>(255);
  float* part = reinterpret_cast<float*>(static_cast<char*>(workspace) + lse_bytes);
  return stac::attn_colsum_launch(a, static_cast<int*>(workspace), zeroed,
                                  static_cast<float*>(workspace) + stac::kAttnCtlWords, part, dev_status,
                                  reinterpret_cast<cudaStream_t>(stream));
}

}  // namespace

extern "C" {

int stac_attn_colsum(const void* q, int64_t q_row_stride, const void* k_hot, const void* v_hot,
                     int64_t hot_row_stride, int64_t hot_head_stride, int T_hot, const void* k_ret, const void* v_ret,
                     int64_t ret_row_stride, int64_t ret_head_stride, int T_ret, const float* bias_ret, int64_t bias_head_stride, void* out,
                     int64_t out_row_stride, float* lse, float* colsum, int64_t colsum_head_stride, int M, int H,
                     int D, float scale, float subsample_ratio, void* workspace, size_t workspace_bytes,
                     int* dev_status, stac_stream_t stream) {
  return attn_colsum_in_workspace(false, q, q_row_stride, k_hot, v_hot, hot_row_stride, hot_head_stride, T_hot, k_ret, v_ret,
      ret_row_stride, ret_head_stride, T_ret, bias_ret, bias_head_stride, out, out_row_stride,
      lse, colsum, colsum_head_stride, M, H, D, scale, subsample_ratio, workspace,
      workspace_bytes, dev_status, stream);
}

int stac_attn_colsum_kept(const void* q, int64_t q_row_stride, const void* k_hot, const void* v_hot,
                     int64_t hot_row_stride, int64_t hot_head_stride, int T_hot, const void* k_ret, const void* v_ret,
                     int64_t ret_row_stride, int64_t ret_head_stride, int T_ret, const float* bias_ret, int64_t bias_head_stride, void* out,
                     int64_t out_row_stride, float* lse, float* colsum, int64_t colsum_head_stride, int M, int H,
                     int D, float scale, float subsample_ratio, void* workspace, size_t workspace_bytes,
                     int* dev_status, stac_stream_t stream) {
  return attn_colsum_in_workspace(true, q, q_row_stride, k_hot, v_hot, hot_row_stride, hot_head_stride, T_hot, k_ret, v_ret,
      ret_row_stride, ret_head_stride, T_ret, bias_ret, bias_head_stride, out, out_row_stride,
      lse, colsum, colsum_head_stride, M, H, D, scale, subsample_ratio, workspace,
      workspace_bytes, dev_status, stream);
}

int stac_selftest_bounded_wait(int max_polls, int* dev_status, stac_stream_t stream) {
  if (max_polls <= 0 || dev_status == nullptr) return STAC_ERR_BAD_ARG;
  stac::bounded_wait_selftest_kernel<<<1, 32, 0, reinterpret_cast<cudaStream_t>(stream)>>>(max_polls, dev_status);
  return stac::count_launch(cudaGetLastError()) == cudaSuccess ? STAC_OK : STAC_ERR_CUDA;
}

int stac_attn_colsum_scored(const void* q, int64_t q_row_stride, const void* k_hot, const void* v_hot,
                            int64_t hot_row_stride, int64_t hot_head_stride, int T_hot, const void* k_ret, const void* v_ret,
                            int64_t ret_row_stride, int64_t ret_head_stride, int T_ret, const float* bias_ret,
                            int64_t bias_head_stride, void* out, int64_t out_row_stride, float* lse, float* colsum,
                            int64_t colsum_head_stride, int M, int H, int D, float scale, float subsample_ratio,
                            float* scores, float* counts, int64_t score_row_stride, int old_T, int Tq, float temperature,
                            void* workspace, size_t workspace_bytes, int* dev_status, stac_stream_t stream) {
  if (colsum == nullptr || scores == nullptr || counts == nullptr || old_T < 0 || Tq <= 0) return STAC_ERR_BAD_ARG;
  // rows of different heads that overlap would be written by several CTAs at once
  if (H > 1 && score_row_stride < T_hot) return STAC_ERR_BAD_ARG;
  return attn_colsum_in_workspace(true, q, q_row_stride, k_hot, v_hot, hot_row_stride, hot_head_stride, T_hot, k_ret, v_ret,
                                  ret_row_stride, ret_head_stride, T_ret, bias_ret, bias_head_stride, out, out_row_stride,
                                  lse, colsum, colsum_head_stride, M, H, D, scale, subsample_ratio, workspace,
                                  workspace_bytes, dev_status, stream, scores, counts, score_row_stride, old_T, Tq, temperature);
}

}  // extern "C"
