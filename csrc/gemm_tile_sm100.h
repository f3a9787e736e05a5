// Host API of the tiled GEMM with fused epilogues (csrc/gemm_tile_sm100.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace penny {
namespace sm100 {

enum TileEpilogue : int {
  TILE_EPI_PLAIN = 0,     // out[m][n] = acc
  TILE_EPI_SILU = 1,      // out[m][f] = silu(acc of gate row f) * (acc of up row f): b's rows are gate, then up (or silu_pairs)
  TILE_EPI_RESIDUAL = 2,  // z = acc + residual; residual = z; out = z * norm_w; sumsq_out = sums of z^2
};

// out = a * b^T (bf16, fp32 accumulation), a [M, K], b [groups * b_rows, K].
struct TileGemm {
  const void* a;
  const void* b;
  void* out;
  int M, b_rows, K;
  int lda, ldb, ldo;
  int epi;
  bool silu_pairs;  // TILE_EPI_SILU, without groups: b's rows are blocks of 64 gate rows and the 64 up rows of the same features
  // TILE_EPI_SILU, not with pair = 2: the quotient gate / (1 + exp(-gate)) is that of a division, as the decode GEMM's is;
  // else it is off by up to 2 units of fp32 and zero for gates below -87.3 (their 1 + exp(-gate) is above 2^126)
  bool exact_silu;
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
  void* residual;       // [M, b_rows], ldo; bf16, or with residual_fp32 fp32
  bool residual_fp32;   // (the models of this package pass bf16)
  void* stream_out;     // residual_fp32: null, or [M, b_rows], ldo: the sum once more in bf16
  const void* norm_w;   // [b_rows]; null: only the residual add (out unused)
  float* sumsq_out;     // [b_rows / 128][M]: a sum for every 128 columns (which wants tiles of whole 128s; kept for callers
                        // of that form), or with sumsq_cap > 0 [sumsq_cap][M]
  int sumsq_cap;        // above 0: the first rows of sumsq_out take one sum per tile, or CTA of a cluster, of its columns
                        // (launch_gemm_tile says how many rows): any width of tile will do, and a cluster shares out a
                        // tile's columns evenly
  int block_n;          // 0: choose; else the columns of a tile: a multiple of 16 up to 256, or of 32 up to 512 (two
                        // accumulators).  pair = 0: 512 stands for CTA pairs, 256 x 256
  int pair;             // 0: by block_n, or choose with it; 1: CTA pairs, tiles of 256 rows; -1: single CTAs; 2: pairs
                        // with 256 rows of the weight on the M side and tiles of up to block_n rows of a (a multiple of
                        // 16 up to 256, 0: 256), plain or silu, no cluster
  int cluster;          // pairs or CTAs that split the K steps of a tile, up to 4; 1: none; 0: none, or with block_n = 0
                        // choose.  (block_n = 0: where some width can be shared so.)  With groups only for M <= the tile's rows
  bool pdl;             // may start, and without groups load b, while the kernel before it on the stream still runs:
                        // that kernel must not write b
};

// block_n, pair and cluster that a launch with block_n = 0 takes on the current device (block_n 0: none).
TileGemm gemm_tile_choice(const TileGemm& g);

// sumsq_rows: null, or the rows of sumsq_out that the launch writes.
cudaError_t launch_gemm_tile(const TileGemm& g, uint32_t* error_word, cudaStream_t stream, int* sumsq_rows = nullptr);

}  // namespace sm100
}  // namespace penny
