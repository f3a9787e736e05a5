// Work split of the streamed GEMM (gemm_stream_sm100.cu): plain C++, used by the
// kernel, its launcher and (through the host simulator library) the CPU tests.
//
// The weight matrix is cut into pair tiles of 256 rows and K steps of 64
// elements; the K steps of all tiles (tile major) form one line of `units`, and
// pair p of `pairs` CTA pairs works on the contiguous range
//     [units * p / pairs, units * (p + 1) / pairs)
// so every pair streams the same number of bytes to within one step.  A range
// crosses tile borders where it falls; a tile worked on by several pairs is
// summed from their fp32 partials in pair order.
#pragma once
#include <stddef.h>
#include <stdint.h>

#if defined(__CUDACC__)
#define PENNY_STREAM_HD __host__ __device__ inline
#else
#define PENNY_STREAM_HD inline
#endif

namespace penny {
namespace sm100 {

constexpr int kStreamMaxRows = 256;        // rows of x per group: the N side of one tcgen05.mma
constexpr int kStreamMaxGroups = 256;
constexpr int kStreamCounters = 1 << 15;   // arrival counters at the head of the workspace, four per pair tile
// A range shorter than this many K steps costs more in the sum over its tile's
// ranges than it saves in streaming: fewer pairs are used then.
constexpr int kStreamMinUnits = 6;

PENNY_STREAM_HD int stream_round_rows(int rows) { return (rows + 31) / 32 * 32; }

PENNY_STREAM_HD int stream_pairs(int units, int max_pairs) {
  const int p = units / kStreamMinUnits;
  return p < 1 ? 1 : (p < max_pairs ? p : max_pairs);
}
// Pairs per cluster.  With fewer tiles than pairs every tile is shared, and pairs of one cluster add their
// parts through each other's shared memory instead of the workspace: the most (up to 4) that are resident
// together (clusters[c]: how many clusters of c pairs the GPU holds) with at least four K steps each.
// 1: the flat split.
PENNY_STREAM_HD int stream_cluster(int tiles, int num_kb, const int* clusters) {
  int cl = 1;
  for (int c = 2; c <= 4; ++c)
    if (tiles <= clusters[c] && num_kb / c >= 4) cl = c;
  return cl;
}
// units * pairs fits 32 bits (the launcher checks)
PENNY_STREAM_HD int stream_begin(int units, int pairs, int p) { return units * p / pairs; }
// The pair whose range holds unit u.
PENNY_STREAM_HD int stream_pair_of(int units, int pairs, int u) {
  int p = (int)((float)u * (float)pairs / (float)units);
  while (p + 1 < pairs && stream_begin(units, pairs, p + 1) <= u) ++p;
  while (p > 0 && (p >= pairs || stream_begin(units, pairs, p) > u)) --p;
  return p;
}
// A pair owns two partial slots: 0 for the tile its range starts in, 1 for the
// tile its range ends in (whole tiles in between need none).
PENNY_STREAM_HD int stream_slot(int units, int pairs, int p, int num_kb, int tile) {
  return 2 * p + (stream_begin(units, pairs, p) / num_kb == tile ? 0 : 1);
}
// Bytes of the caller's workspace for up to `rows` rows per group: the counters
// (zeroed once, they reset themselves), then [pairs][2 slots][2 CTAs] partials
// of [rows][128] fp32.
PENNY_STREAM_HD size_t stream_workspace_bytes(int rows, int max_pairs) {
  return (size_t)kStreamCounters * 4 + (size_t)max_pairs * 4 * (size_t)stream_round_rows(rows) * 128 * 4;
}

}  // namespace sm100
}  // namespace penny
