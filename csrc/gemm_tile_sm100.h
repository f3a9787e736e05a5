// Host API of the tiled GEMM with fused epilogues (csrc/gemm_tile_sm100.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace penny {
namespace sm100 {

enum TileEpilogue : int {
  TILE_EPI_PLAIN = 0,     // out[m][n] = acc
  TILE_EPI_SILU = 1,      // out[m][f] = silu(acc of gate row f) * (acc of up row f): b's rows are gate, then up
  TILE_EPI_RESIDUAL = 2,  // z = acc + residual; residual = z; out = z * norm_w; sumsq_out = sum z^2 per 128 columns
};

// out = a * b^T (bf16, fp32 accumulation), a [M, K], b [groups * b_rows, K].
struct TileGemm {
  const void* a;
  const void* b;
  void* out;
  int M, b_rows, K;
  int lda, ldb, ldo;
  int epi;
  // groups > 0: rows ranges[s g] .. ranges[s g + 1] of a and out (device memory, s = range_stride) meet b rows
  // g * b_rows ..  (what lies outside [0, M) is left out)
  int groups;
  const int* ranges;
  int range_stride;  // 2: (start, end) pairs; 1: group g ends where g + 1 starts
  // null, or [scale_parts][M] sums of squares of the rows of a before their norm weight: every output is
  // multiplied by rsqrt(sum / K + eps)
  const float* scale_sumsq;
  int scale_parts;
  float eps;
  void* residual;       // [M, b_rows], ldo
  const void* norm_w;   // [b_rows]; null: only the residual add (out unused)
  float* sumsq_out;     // [b_rows / 128][M]
  int block_n;          // 0: choose; 128 / 192 / 256: single CTAs; 512: CTA pairs, 256 x 256
  int cluster;          // pairs (block_n 512) or CTAs that split the K steps of a tile, up to 4; 0, 1: none.  With
                        // groups only for M <= the tile's rows
  bool pdl;             // may start, and without groups load b, while the kernel before it on the stream still runs:
                        // that kernel must not write b
};

cudaError_t launch_gemm_tile(const TileGemm& g, uint32_t* error_word, cudaStream_t stream);

}  // namespace sm100
}  // namespace penny
