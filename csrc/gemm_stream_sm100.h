// Host API of the streamed GEMM (csrc/gemm_stream_sm100.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "stream_gemm_plan.h"

namespace penny {
namespace sm100 {

enum StreamEpilogue : int {
  STREAM_EPI_PLAIN = 0,     // out[r][n] = acc
  STREAM_EPI_SILU = 1,      // out[r][f] = silu(gate) * up
  STREAM_EPI_RESIDUAL = 2,  // z = acc + residual; residual = z; out = z * norm_w; sumsq_out = sum z^2 per 128 columns
};

// out = x * W^T for at most 256 rows of x per group, bf16, fp32 accumulation.
struct StreamGemm {
  const void* x;  // [rows, K], leading dimension ldx
  const void* w;  // [groups * w_rows, K], leading dimension ldw
  void* out;      // leading dimension ldo
  int rows;       // rows of x in the largest group (one group: all of them)
  int x_rows;     // rows of the x matrix (>= every group's end)
  int w_rows, K;  // weight rows per group
  int ldx, ldw, ldo;
  int epi;
  // SILU: distance from a gate row to the up row of the same feature: 64 (rows come in blocks of 64
  // gate rows followed by their 64 up rows) or w_rows / 2 (all gate rows, then all up rows)
  int up_offset;
  // groups > 0: rows ranges[s g] .. ranges[s g + 1] of x (device memory, s = range_stride) meet weight rows
  // g * w_rows ..; 0: all rows, one weight
  int groups;
  const int* ranges;
  int range_stride;  // 2: (start, end) pairs; 1: group g ends where g + 1 starts
  // null, or per-row sums of squares [scale_parts][rows]: every output is multiplied by
  // rsqrt(sum / scale_width + eps), which finishes an RMSNorm whose weight x already carries
  const float* scale_sumsq;
  int scale_parts, scale_width;
  float eps;
  // RESIDUAL epilogue
  void* residual;      // [rows, w_rows], ldo
  const void* norm_w;  // [w_rows]; null: only the residual add
  float* sumsq_out;    // [w_rows / 128][rows]
  void* workspace;     // stream_workspace_bytes(rows, 74 or more pairs), zeroed once
  size_t workspace_bytes;
  bool pdl;            // programmatic dependent launch; W must not be written by the kernel before
  int cluster;         // pairs that split the K steps of a tile inside a cluster: 0 choose, 1 flat split, 2-4
  int smem_kb;         // shared memory the ring may grow to; 0: by size
};

cudaError_t launch_gemm_stream(const StreamGemm& g, uint32_t* error_word, cudaStream_t stream);
// Most CTA pairs a launch uses on the current device (for stream_workspace_bytes).
int stream_max_pairs();

}  // namespace sm100
}  // namespace penny
