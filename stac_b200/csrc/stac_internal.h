// Internal declarations shared by the translation units of libstac_b200.so.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <atomic>

#include "../../include/stac_b200.h"
#include "per_device.h"

namespace stac {

struct AttnArgs {
  const void* q;            // bf16 [M, H, 64] with row stride q_row_stride elements
  long long q_row_stride;
  const void* k_hot;        // bf16; key n, head h at n*hot_row_stride + h*hot_head_stride
  const void* v_hot;
  long long hot_row_stride;
  long long hot_head_stride;
  int T_hot;
  const void* k_ret;        // bf16 [H, >=T_ret, 64]
  const void* v_ret;
  long long ret_row_stride;
  long long ret_head_stride;
  int T_ret;
  const float* bias_ret;    // [H, >=T_ret]
  long long bias_head_stride;
  void* out;                // bf16, same layout as q
  long long out_row_stride;
  float* lse;               // [H, M] or nullptr
  float* colsum;            // [H, colsum_head_stride] or nullptr
  long long colsum_head_stride;
  int M, H, D;
  float scale;
  float subsample_ratio;
  // running scores that the column sums of the hot keys go into, or nullptr (needs `colsum` and `part`)
  float* scores = nullptr;  // [H, score_stride]
  float* counts = nullptr;
  long long score_stride = 0;
  int old_T = 0, score_Tq = 0;
  float temperature = 0.f;
};

// Ordinal of the current device (checked against kMaxDevices) / its SM count, cached per device.
int current_device(int* dev);
int device_sm_count(int dev, int* n_sm);

void attn_subsample_plan(int M, float ratio, int* m_sub, int* stride, float* correction);
int attn_forward_plan(int M, int H, int T_hot, int T_ret, int n_sm, bool workspace, int* parts, int* cluster);
constexpr int kAttnCtlWords = 512;   // control words in front of the row log-sum-exps of a workspace
size_t attn_lse2_elems(int M, int H);
size_t attn_part_elems();
// `part`: attn_part_elems() floats for the split forward kernel, or nullptr (one CTA per item then)
// `ctl`: the control words; ctl_zeroed: they are zero (else the call clears the ones it uses)
int attn_colsum_launch(const AttnArgs& a, int* ctl, bool ctl_zeroed, float* lse2, float* part, int* err,
                       cudaStream_t stream);

// Kernels that this library has launched in this process (stac_kernel_launches): `launched` is the
// result of a launch, counted where it succeeded and handed on.
inline std::atomic<uint64_t> g_kernel_launches{0};
inline cudaError_t count_launch(cudaError_t launched) {
  if (launched == cudaSuccess) g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
  return launched;
}

// Launch with programmatic stream serialization: the kernel may become resident while the
// kernel before it in the stream drains; it calls grid_dep_wait() before it touches anything
// that kernel wrote.  STAC_PDL=0 builds fall back to plain stream order.
#ifndef STAC_PDL
#define STAC_PDL 1
#endif
template <typename... KArgs, typename... Args>
cudaError_t launch_clusters_behind(void (*kernel)(KArgs...), dim3 grid, int cluster, dim3 block, int smem, cudaStream_t stream,
                                   const Args&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = static_cast<size_t>(smem);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = STAC_PDL;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = static_cast<unsigned>(cluster);
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  return count_launch(cudaLaunchKernelEx(&cfg, kernel, args...));
}
template <typename... KArgs, typename... Args>
cudaError_t launch_behind(void (*kernel)(KArgs...), dim3 grid, dim3 block, int smem, cudaStream_t stream,
                          const Args&... args) {
  return launch_clusters_behind(kernel, grid, 1, block, smem, stream, args...);
}

}  // namespace stac
