// Work split of the decode GEMM (gemm_decode_sm100.cu): plain C++, used by the
// kernel, by its launcher and (through the host simulator library) by the CPU
// tests.
//
//   out[B, N] = x[B, K] W[N, K]^T for a decode batch (one slab of B <= 128 rows; larger batches run
//   their slabs side by side in the same launch, so the slabs of a weight tile read it from L2 together).
//   * one CTA per (weight tile of 128 rows, K range); the `splits` CTAs of a tile
//     form one thread-block cluster and reduce their fp32 partials through
//     distributed shared memory: no global workspace, no counters, no fix-up pass;
//   * the K steps (64 elements each) are dealt out as `splits` contiguous ranges
//     whose sizes differ by at most one;
//   * after its MMAs a CTA keeps the accumulator columns (= batch rows) of its
//     own slice and sends every other slice to the CTA that owns it: CTA r owns
//     columns [r * slice, min(rows, (r + 1) * slice)) of the rows that the slab has
//     (the last slab of a larger batch may have fewer than its tile is wide).
#pragma once
#include <stddef.h>
#include <stdint.h>

#if defined(__CUDACC__)
#define PENNY_PLAN_HD __host__ __device__ inline
#else
#define PENNY_PLAN_HD inline
#endif

namespace penny {
namespace sm100 {

constexpr int kDecodeMaxSplits = 8;  // portable cluster size
constexpr int kDecodeMaxBatch = 1024;  // rows of x per launch

// (num_kb < 2^25 and r <= 8: no 64-bit division in the kernel's prologue)
PENNY_PLAN_HD int decode_kb_begin(int num_kb, int splits, int r) { return num_kb * r / splits; }
// columns owned by one CTA of the cluster, of `bt` that there are
PENNY_PLAN_HD int decode_slice(int bt, int splits) { return (bt + splits - 1) / splits; }
// slot of source CTA `src` in the receive area of CTA `dst` (src != dst): sources in rank order, dst left out
PENNY_PLAN_HD int decode_recv_slot(int src, int dst) { return src - (src > dst ? 1 : 0); }
// fp32 words of the receive area: [splits - 1][slice][128 rows]
PENNY_PLAN_HD size_t decode_recv_floats(int bt, int splits) {
  if (splits <= 1) return 0;
  return (size_t)(splits - 1) * (size_t)decode_slice(bt, splits) * 128;
}

// The cluster size (K ranges per weight tile), from measurements on B200 at batch 64
// (cluster sizes 1-8 timed on every shard shape of a Llama-3-8B layer at TP 1, 2, 4, 8):
//   * what a decode GEMM needs is enough CTAs streaming at once - about two per SM,
//     each with three or four 16 KB weight stages in flight;
//   * all CTAs must be resident together: `capacity[s]` is the number of CTAs the
//     GPU holds at once when they come in clusters of s (the launcher asks the
//     occupancy API; clusters must fit a GPC, so it is a little below 2 x SMs).  A
//     second wave costs far more than a smaller cluster;
//   * a K range shorter than 6 steps (384 elements) is not worth a cluster: the
//     reduction then costs more than the shorter stream saves.
// So: the largest s <= 8 with tiles * s <= capacity[s] and num_kb / s >= 6; 1 when
// nothing larger qualifies (narrow K, or more tiles than fit at once).
PENNY_PLAN_HD int decode_choose_splits(int tiles, int num_kb, const int* capacity) {
  int best = 1;
  for (int s = 2; s <= kDecodeMaxSplits; ++s) {
    if (num_kb / s < 6) break;
    if ((long long)tiles * s <= (long long)capacity[s]) best = s;
  }
  return best;
}

// The same for a linear between the folded norms of one rank's step, whose clusters were timed in its chain of launches:
// either rule is enough, the device's answer or up to five CTAs on three SMs.
//   * The stream runs at 32 GB/s per CTA, so at 31 to 35 tiles a seventh range pays although the occupancy query, which
//     wants whole clusters per GPC, has room for 210 CTAs in sevens (a layer's linears at hidden 4096, o and down of 32
//     tiles in six / seven, 1 row: 78.8 / 77.9 us, 40 rows 87.0 / 85.7; 34 tiles level); 288 CTAs no longer run side by
//     side (q / k / v 11.0 us in five, 16.1 in six).
//   * Five on three alone keeps clusters small that the device has room for: 64 tiles, K 4096, gate/up and down in three /
//     four 25.0 / 23.7 us, 128 tiles in one / two 39.8 / 38.7, a layer of hidden 5376 123.3 / 121.4.
//   * Its room filled to the last cluster is too much for a chain, where CTAs of the launch before are still at work (44
//     tiles in six, 264 of 264 CTAs: 153.3 us a layer, in five 150.6; 90 in three, 270 of 270: 31.4, in two 30.3).
// Batch tiles of 128 rows hold one CTA per SM and keep to the rule above.
PENNY_PLAN_HD int decode_choose_splits_chain(int tiles, int num_kb, int sms, const int* capacity) {
  int best = 1;
  for (int s = 2; s <= kDecodeMaxSplits; ++s) {
    if (num_kb / s < 6) break;
    const long long ctas = (long long)tiles * s;
    if (ctas < (long long)capacity[s] || ctas * 3 <= (long long)sms * 5) best = s;
  }
  return best;
}

// capacity[] stand-in for a GPU of `sms` SMs in GPCs of `gpc_sms`, two CTAs per SM,
// whole clusters per GPC (used by the CPU tests; the launcher uses the real figure).
PENNY_PLAN_HD void decode_model_capacity(int sms, int gpc_sms, int* capacity) {
  capacity[0] = 0;
  for (int s = 1; s <= kDecodeMaxSplits; ++s) {
    const int gpcs = sms / gpc_sms, rest = sms - gpcs * gpc_sms;
    capacity[s] = (gpcs * ((2 * gpc_sms) / s) + (2 * rest) / s) * s;
  }
}

}  // namespace sm100
}  // namespace penny
