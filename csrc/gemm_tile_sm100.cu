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
  const int workers = g.groups > 0 ? slots : (int)std::min<long long>(slots, tiles);
  if constexpr (PAIR)
    return launch_kernel_ex(gemm_tile_pair<BN, EPI>, dim3((unsigned)(2 * workers)), dim3(kTileThreads), Cfg::kSmemBytes,
                            stream, g.pdl, 1, ma, mb, a, error_word);
  else
    return launch_kernel_ex(gemm_tile_single<BN, EPI>, dim3((unsigned)workers), dim3(kTileThreads), Cfg::kSmemBytes,
                            stream, g.pdl, 1, ma, mb, a, error_word);
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
  int block_n = g.block_n;
  if (block_n == 0) {
    const KernelSetup ks = kernel_setup(reinterpret_cast<const void*>(gemm_tile_pair<256, TILE_EPI_PLAIN>),
                                        TileCfg<true, 256>::kSmemBytes, kTileThreads);
    block_n = choose_block_n(g.M, g.b_rows, g.K, sms, ks.rc == cudaSuccess ? ks.pairs : 0);
    if (block_n == 192 && g.epi != TILE_EPI_PLAIN) block_n = 256;
  }
  switch (g.epi) {
    case TILE_EPI_PLAIN: return launch_tile_n<TILE_EPI_PLAIN>(g, a, block_n, sms, error_word, stream);
    case TILE_EPI_SILU: return launch_tile_n<TILE_EPI_SILU>(g, a, block_n, sms, error_word, stream);
    case TILE_EPI_RESIDUAL: return launch_tile_n<TILE_EPI_RESIDUAL>(g, a, block_n, sms, error_word, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace sm100
}  // namespace penny
