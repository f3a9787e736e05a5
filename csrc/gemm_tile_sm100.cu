// Launchers of the tiled GEMM (kernel: gemm_tile_sm100.cuh).
#include "gemm_tile_sm100.cuh"

#include <algorithm>

#include "gemm_sm100.h"
#include "kernel_setup.h"

namespace penny {
namespace sm100 {

namespace {

template <bool PAIR, int BN, int EPI>
cudaError_t launch_tile(const TileGemm& g, TileArgs a, int sms, uint32_t* error_word, cudaStream_t stream) {
  using Cfg = TileCfg<PAIR, BN>;
  constexpr bool kSilu = EPI == TILE_EPI_SILU;
  a.cl = 1;
  a.tiles_n = (a.n_out + (kSilu ? BN / 2 : BN) - 1) / (kSilu ? BN / 2 : BN);
  a.band = std::max(1, 2048 / Cfg::kRows);
  CUtensorMap ma, mb;
  cudaError_t rc = make_tile_map(&ma, g.a, (uint64_t)g.M, (uint64_t)g.K, (uint64_t)g.lda, kBlockM);
  if (rc != cudaSuccess) return rc;
  rc = make_tile_map(&mb, g.b, (uint64_t)std::max(1, g.groups) * g.b_rows, (uint64_t)g.K, (uint64_t)g.ldb,
                     (uint32_t)(PAIR || kSilu ? BN / 2 : BN));
  if (rc != cudaSuccess) return rc;
  const void* fn = nullptr;
  if constexpr (PAIR) fn = reinterpret_cast<const void*>(gemm_tile_pair<BN, EPI>);
  else fn = reinterpret_cast<const void*>(gemm_tile_single<BN, EPI>);
  const KernelSetup ks = kernel_setup(fn, Cfg::kSmemBytes, PAIR ? kTileThreads : 0);
  if (ks.rc != cudaSuccess) return ks.rc;
  // grouped: the tile count is only known on the device
  const long long tiles = (long long)((g.M + Cfg::kRows - 1) / Cfg::kRows) * a.tiles_n;
  const int slots = PAIR ? ks.pairs : sms;
  a.cl = std::max(1, std::min({g.cluster, kTileMaxCluster, a.num_kb}));
  // A cluster works on one tile, so with groups (whose tiles the device counts) no group may have two row tiles.
  if (a.cl > 1 && g.groups > 0 && g.M > Cfg::kRows) return cudaErrorInvalidValue;
  const int workers = a.cl > 1 ? (g.groups > 0 ? g.groups * a.tiles_n : (int)tiles) : (g.groups > 0 ? slots : (int)std::min<long long>(slots, tiles));
  if constexpr (PAIR)
    return launch_kernel_ex(gemm_tile_pair<BN, EPI>, dim3((unsigned)(2 * workers * a.cl)), dim3(kTileThreads),
                            Cfg::kSmemBytes, stream, g.pdl, 2 * a.cl, ma, mb, a, error_word);
  else
    return launch_kernel_ex(gemm_tile_single<BN, EPI>, dim3((unsigned)(workers * a.cl)), dim3(kTileThreads),
                            Cfg::kSmemBytes, stream, g.pdl, a.cl, ma, mb, a, error_word);
}

// Tile and cluster by rounds times the time of a K step.  Steps measured on B200, one 4096-long K (us per
// step, all operands through the 64 B / clk that an SM takes in): 128 x 128 0.32, 128 x 192 0.36, 128 x 256
// 0.40, 256 x 256 on a pair 0.36.  The exchange of a cluster's sums takes about as long as 13 steps of single
// CTAs (q / k / v of 128 tokens: 23.2 us whole, 17.5 in two; down 72.5 whole, 31.6 in four, 40.5 on pairs in
// three) and 18 of a pair.
void choose_tile(TileGemm& g, int sms, int pairs) {
  const long long m128 = (g.M + 127) / 128, m256 = (g.M + 255) / 256;
  const int num_kb = (g.K + kBlockK - 1) / kBlockK;
  double best = 0;
  auto offer = [&](int block_n, int cluster, long long tiles, int slots, double steps) {
    const double cost = (double)((tiles + slots - 1) / slots) * steps;
    if (g.block_n == 0 || cost < best) best = cost, g.block_n = block_n, g.cluster = cluster;
  };
  auto clusters = [&](bool pair, int c) {
    if (pair)
      return max_clusters(reinterpret_cast<const void*>(gemm_tile_pair<256, TILE_EPI_PLAIN>), 2 * c, kTileThreads,
                          TileCfg<true, 256>::kSmemBytes);
    const void* fn = reinterpret_cast<const void*>(gemm_tile_single<128, TILE_EPI_PLAIN>);
    if (kernel_setup(fn, TileCfg<false, 128>::kSmemBytes).rc != cudaSuccess) return 0;
    return max_clusters(fn, c, kTileThreads, TileCfg<false, 128>::kSmemBytes);
  };
  auto cols = [&](int bn) { return (long long)((g.b_rows + bn - 1) / bn); };
  offer(128, 1, m128 * cols(128), sms, 0.32 * num_kb);
  if (g.epi == TILE_EPI_PLAIN) offer(192, 1, m128 * cols(192), sms, 0.36 * num_kb);
  offer(256, 1, m128 * cols(256), sms, 0.40 * num_kb);
  for (int c = 2; c <= kTileMaxCluster && g.groups == 0; ++c)
    if (m128 * cols(128) <= clusters(false, c) && num_kb >= 4 * c)
      offer(128, c, m128 * cols(128), sms, 0.32 * ((num_kb + c - 1) / c + 13));
  if (pairs > 0 && pair_kernel_enabled()) {
    const long long tiles = m256 * cols(256);
    offer(512, 1, tiles, pairs, 0.36 * num_kb);
    for (int c = 2; c <= kTileMaxCluster && g.groups == 0; ++c)
      if (tiles <= clusters(true, c) && num_kb >= 4 * c) offer(512, c, tiles, pairs, 0.36 * ((num_kb + c - 1) / c + 18));
  }
}

template <int EPI>
cudaError_t launch_tile_n(const TileGemm& g, const TileArgs& a, int block_n, int sms, uint32_t* error_word,
                          cudaStream_t stream) {
  switch (block_n) {
    case 128: return launch_tile<false, 128, EPI>(g, a, sms, error_word, stream);
    case 192:
      if constexpr (EPI == TILE_EPI_PLAIN) return launch_tile<false, 192, EPI>(g, a, sms, error_word, stream);
      return cudaErrorInvalidValue;
    case 256: return launch_tile<false, 256, EPI>(g, a, sms, error_word, stream);
    case 512: return launch_tile<true, 256, EPI>(g, a, sms, error_word, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace

cudaError_t launch_gemm_tile(const TileGemm& g, uint32_t* error_word, cudaStream_t stream) {
  if (g.M <= 0 || g.b_rows <= 0 || g.K <= 0 || g.K % 8 != 0 || g.lda % 8 != 0 || g.ldb % 8 != 0 || g.groups < 0 ||
      g.groups > kTileMaxGroups || (g.groups > 0 && (g.ranges == nullptr || g.scale_sumsq != nullptr)))
    return cudaErrorInvalidValue;
  if (g.epi == TILE_EPI_SILU && g.b_rows % 2 != 0) return cudaErrorInvalidValue;
  if (g.epi == TILE_EPI_RESIDUAL &&
      (g.groups > 0 || g.b_rows % 128 != 0 || g.ldo % 8 != 0 || g.residual == nullptr ||
       (g.norm_w != nullptr && (g.out == nullptr || g.sumsq_out == nullptr)) ||
       ((reinterpret_cast<uintptr_t>(g.out) | reinterpret_cast<uintptr_t>(g.residual) | reinterpret_cast<uintptr_t>(g.norm_w)) & 15u) != 0))
    return cudaErrorInvalidValue;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  TileArgs a = {};
  a.out = reinterpret_cast<__nv_bfloat16*>(g.out);
  a.ldo = g.ldo;
  a.M = g.M;
  a.n_out = g.epi == TILE_EPI_SILU ? g.b_rows / 2 : g.b_rows;
  a.num_kb = (g.K + kBlockK - 1) / kBlockK;
  a.groups = g.groups;
  a.b_rows = g.b_rows;
  a.ranges = g.ranges;
  a.range_stride = g.range_stride;
  a.scale_sumsq = g.scale_sumsq;
  a.scale_parts = g.scale_parts;
  a.inv_width = 1.f / (float)g.K;
  a.eps = g.eps;
  a.residual = reinterpret_cast<__nv_bfloat16*>(g.residual);
  a.norm_w = reinterpret_cast<const __nv_bfloat16*>(g.norm_w);
  a.sumsq_out = g.sumsq_out;
  TileGemm c = g;
  if (g.block_n == 0) {
    const KernelSetup ks = kernel_setup(reinterpret_cast<const void*>(gemm_tile_pair<256, TILE_EPI_PLAIN>),
                                        TileCfg<true, 256>::kSmemBytes, kTileThreads);
    choose_tile(c, sms, ks.rc == cudaSuccess ? ks.pairs : 0);
  }
  switch (g.epi) {
    case TILE_EPI_PLAIN: return launch_tile_n<TILE_EPI_PLAIN>(c, a, c.block_n, sms, error_word, stream);
    case TILE_EPI_SILU: return launch_tile_n<TILE_EPI_SILU>(c, a, c.block_n, sms, error_word, stream);
    case TILE_EPI_RESIDUAL: return launch_tile_n<TILE_EPI_RESIDUAL>(c, a, c.block_n, sms, error_word, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace sm100
}  // namespace penny
