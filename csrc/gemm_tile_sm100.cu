// Launchers of the tiled GEMM (kernel: gemm_tile_sm100.cuh).
#include "gemm_swap_sm100.cuh"

#include <algorithm>
#include <array>
#include <map>
#include <mutex>

#include "gemm_sm100.h"
#include "kernel_setup.h"

namespace penny {
namespace sm100 {

namespace {

constexpr int kTileSmem = 224 << 10;  // ring and staging of the one CTA of an SM
constexpr int kTileEpiBytes = 16 << 10;
static_assert(TileEpi<TILE_EPI_PLAIN, false>::kBytes <= kTileEpiBytes && TileEpi<TILE_EPI_SILU, false>::kBytes <= kTileEpiBytes &&
              TileEpi<TILE_EPI_RESIDUAL, false>::kBytes <= kTileEpiBytes, "staging of the epilogues");

// Gate and up rows in blocks: the tiles of `nsub` accumulators of `sub_out` features each, and log2 of the rows that an
// accumulator takes of a block (the most, 8 to 64, that leave the fewest tiles).  -1 where no such strip fits.
int strip_tiles(int n_out, int sub_out, int nsub, int* tiles_n) {
  int best = -1;
  for (int shift = 6; shift >= 3; --shift) {
    if (sub_out % (1 << shift) != 0) continue;
    const int per = kPairRows >> shift, blocks = nsub * (sub_out >> shift);
    const int tiles = (n_out / kPairRows + blocks - 1) / blocks * per;
    if (best < 0 || tiles < *tiles_n) best = shift, *tiles_n = tiles;
  }
  return best;
}

template <bool PAIR, int EPI, bool SPLIT, int NSUB>
cudaError_t launch_tile(const TileGemm& g, TileArgs a, TileShape t, int sms, uint32_t* error_word, cudaStream_t stream) {
  constexpr bool kSilu = EPI == TILE_EPI_SILU || EPI == kTileEpiSiluExact;
  const int sub_out = kSilu ? t.sub / 2 : t.sub;
  a.sub = t.sub;
  a.tiles_n = (a.n_out + t.nsub * sub_out - 1) / (t.nsub * sub_out);
  a.strip_shift = -1;
  if (kSilu && g.silu_pairs) {
    a.strip_shift = strip_tiles(a.n_out, sub_out, t.nsub, &a.tiles_n);
    if (a.strip_shift < 0) return cudaErrorInvalidValue;
  }
  a.band = std::max(1, 2048 / t.rows());
  CUtensorMap ma, mb;
  cudaError_t rc = make_tile_map(&ma, g.a, (uint64_t)g.M, (uint64_t)g.K, (uint64_t)g.lda, kBlockM);
  if (rc != cudaSuccess) return rc;
  if (kSilu) {
    const int shift = a.strip_shift;
    rc = shift < 0 ? make_gate_up_map(&mb, g.b, (uint64_t)std::max(1, g.groups), (uint64_t)g.b_rows / 2, (uint64_t)g.K, (uint64_t)g.ldb,
                                      1, (uint32_t)sub_out)
                   : make_gate_up_map(&mb, g.b, (uint64_t)a.n_out / kPairRows, kPairRows, (uint64_t)g.K, (uint64_t)g.ldb,
                                      (uint32_t)(sub_out >> shift), 1u << shift);
  } else {
    rc = make_tile_map(&mb, g.b, (uint64_t)std::max(1, g.groups) * g.b_rows, (uint64_t)g.K, (uint64_t)g.ldb,
                       (uint32_t)(PAIR ? t.sub / 2 : t.sub));
  }
  if (rc != cudaSuccess) return rc;
  const auto kernel = gemm_tile_kernel<PAIR, EPI, SPLIT, NSUB>;
  const KernelSetup ks = kernel_setup(reinterpret_cast<const void*>(kernel), kTileSmem, PAIR ? kTileThreads : 0);
  if (ks.rc != cudaSuccess) return ks.rc;
  // grouped: the tile count is only known on the device
  const long long tiles = (long long)((g.M + t.rows() - 1) / t.rows()) * a.tiles_n;
  const int slots = PAIR ? ks.pairs : sms;
  // A cluster works on one tile, so with groups (whose tiles the device counts) no group may have two row tiles.
  if (SPLIT && g.groups > 0 && g.M > t.rows()) return cudaErrorInvalidValue;
  const long long workers = SPLIT ? (g.groups > 0 ? (long long)g.groups * a.tiles_n : tiles)
                                  : (g.groups > 0 ? slots : std::min<long long>(slots, tiles));
  const int epi_bytes = TileEpi<EPI, SPLIT>::kBytes;
  const int kb_per = (a.num_kb + a.cl - 1) / a.cl;
  a.stages = std::min({kTileMaxStages, kb_per, (kTileSmem - epi_bytes - 1024) / t.stage_bytes()});
  if (SPLIT) {  // the ring takes the peers' sums
    const int own = (sub_out / 16 + a.cl - 1) / a.cl * 16;
    const int recv = (a.cl - 1) * std::max(own, a.ss_cols) * (kSilu ? 2 : 1) * kBlockM * 4;
    a.stages = std::max(a.stages, (recv + t.stage_bytes() - 1) / t.stage_bytes());
  }
  a.stages = std::max(a.stages, 2);
  const int smem = a.stages * t.stage_bytes() + epi_bytes + 1024;
  if (smem > kTileSmem) return cudaErrorInvalidValue;
  const int cols = t.nsub * t.sub;
  a.accs = 2 * cols <= 512 && (g.groups > 0 ? !SPLIT : tiles > workers) ? 2 : 1;
  a.tmem_cols = 32;
  while (a.tmem_cols < a.accs * cols) a.tmem_cols *= 2;
  return launch_kernel_ex(kernel, dim3((unsigned)((PAIR ? 2 : 1) * workers * a.cl)), dim3(kTileThreads), (size_t)smem, stream, g.pdl,
                          (PAIR ? 2 : 1) * a.cl, ma, mb, a, error_word);
}

// Width of the tiles, CTAs or pairs, and cluster, by a time model fitted to launches on B200 in chains with weights from HBM.
// Against every width, pair and cluster of 272 shapes (65 to 3072 rows, the linears of layers of hidden 1024 to 8192, ffn 3.5
// times that) its choice takes 1.6 % longer than the best on average; the worst are K of 1024 and 2048, 27 to 33 % longer at
// 1152 to 2048 rows, where the epilogue counts more than below.  In cycles at 1.8 GHz and us:
//   * a K step takes the MMAs' time (2 cycles a column) or that of filling its stage: 71 bytes a cycle and 64 cycles on
//     pairs, 83 and 19 on single CTAs.  A ring of two stages (single CTAs from 448 columns on) does not keep up: 1.04 us a step of
//     512 columns instead of 0.6 (640 x 12288 x 8192 137 us against 103 of 256 columns), so three are wanted;
//   * a round that is partly empty costs three quarters of a whole one (the rest comes back as clock or as memory
//     bandwidth for the others);
//   * the last epilogue, and each one where a single set of accumulators has to be drained first (above 256 columns), 0.6 us
//     and 0.04 a column; handing the sums of a cluster over 3.2 and 0.03 a column of the share that is sent.
void choose_tile(TileGemm& g, int sms, int pairs) {
  const int num_kb = (g.K + kBlockK - 1) / kBlockK;
  const bool silu = g.epi == TILE_EPI_SILU, blocks = g.epi == TILE_EPI_RESIDUAL && g.norm_w != nullptr && g.sumsq_cap <= 0;
  auto clusters = [&](bool pair, int c) {
    const void* fn = pair ? reinterpret_cast<const void*>(gemm_tile_kernel<true, TILE_EPI_PLAIN, true, 1>)
                          : reinterpret_cast<const void*>(gemm_tile_kernel<false, TILE_EPI_PLAIN, true, 1>);
    if (kernel_setup(fn, kTileSmem).rc != cudaSuccess) return 0;
    return max_clusters(fn, (pair ? 2 : 1) * c, kTileThreads, kTileSmem);
  };
  // what the caller has settled: CTA pairs or single CTAs (pair), and how many of them share a tile (cluster)
  const int want_pair = g.pair, want_cl = std::min({g.cluster, kTileMaxCluster, num_kb});
  double best = 0;
  g.block_n = 0;
  for (int pair = 0; pair <= 1; ++pair) {
    if (pair != 0 && (pairs <= 0 || (want_pair == 0 && !pair_kernel_enabled()))) continue;
    if (want_pair != 0 && (want_pair > 0) != (pair != 0)) continue;
    const int slots = pair ? pairs : sms, rows = pair ? 2 * kBlockM : kBlockM;
    const double fill = pair ? 71. : 83., step0 = pair ? 64. : 19.;
    for (int c = 1; c <= kTileMaxCluster; ++c) {
      if (want_cl > 0 ? c != want_cl : c > 1 && (g.groups > 0 || num_kb < 4 * c)) continue;
      if (c > 1 && g.groups > 0 && g.M > rows) continue;
      const int room = c > 1 ? clusters(pair != 0, c) : 0;
      if (c > 1 && room <= 0) continue;
      for (int bn = blocks ? 128 : 64; bn <= (c > 1 ? 256 : 512); bn += blocks ? 128 : (bn < 256 ? 16 : 32)) {
        const TileShape t{pair != 0, bn > 256 ? bn / 2 : bn, bn > 256 ? 2 : 1};
        if (blocks && t.sub % 128 != 0) continue;
        if (3 * t.stage_bytes() > kTileSmem - kTileEpiBytes - 1024) continue;
        const int sub_out = silu ? t.sub / 2 : t.sub, out = t.nsub * sub_out;
        if (c > 1 && (sub_out % 16 != 0 || sub_out < 16 * c)) continue;
        const int n_out = silu ? g.b_rows / 2 : g.b_rows;
        int tiles_n = (n_out + out - 1) / out;
        if (silu && g.silu_pairs && strip_tiles(n_out, sub_out, t.nsub, &tiles_n) < 0) continue;
        if (g.sumsq_cap > 0 && tiles_n * c > g.sumsq_cap) continue;
        const long long tiles = (long long)((g.M + rows - 1) / rows) * tiles_n;
        if (want_cl <= 0 && c > 1 && tiles > room) continue;
        const double share = (double)tiles * c / slots;
        const double rounds = 0.75 * (double)((tiles * c + slots - 1) / slots) + 0.25 * std::max(1., share);
        const double step = std::max(2.1 * bn, t.stage_bytes() / fill + step0) / 1800.;
        const double drain = 0.6 + 0.04 * (silu ? 0.7 * bn : bn);
        double cost = rounds * ((num_kb + c - 1) / c) * step + (pair ? 0.6 : 0.);
        if (c > 1) cost += 3.2 + 0.03 * bn * (c - 1) / c + 0.04 * bn / c;
        else cost += drain * (2 * bn > 512 ? (double)((tiles + slots - 1) / slots) : 1.);
        if (g.block_n == 0 || cost < best) best = cost, g.block_n = bn, g.pair = pair ? 1 : -1, g.cluster = c;
      }
    }
  }
  if (g.block_n == 0 && want_cl > 1) {  // no width that so many could share
    g.cluster = 0;
    choose_tile(g, sms, pairs);
  }
}

// The choice depends on the shape and the device alone and takes some 10 us: kept per shape, up to a bound.
void choose_tile_once(TileGemm& g, int dev, int sms, int pairs) {
  struct Choice {
    int block_n, pair, cluster;
  };
  static std::mutex mu;
  static std::map<std::array<int, 12>, Choice> kept;
  const std::array<int, 12> key = {dev, g.M, g.b_rows, g.K, g.epi, g.groups > 0, g.norm_w != nullptr, g.sumsq_cap,
                                   pair_kernel_enabled(), g.silu_pairs, g.pair, g.cluster};
  {
    std::lock_guard<std::mutex> lock(mu);
    const auto it = kept.find(key);
    if (it != kept.end()) {
      g.block_n = it->second.block_n;
      g.pair = it->second.pair;
      g.cluster = it->second.cluster;
      return;
    }
  }
  choose_tile(g, sms, pairs);
  std::lock_guard<std::mutex> lock(mu);
  if (kept.size() >= 4096) kept.clear();
  kept[key] = Choice{g.block_n, g.pair, g.cluster};
}

template <bool SILU>
cudaError_t launch_swap(const TileGemm& g, const TileArgs& t, uint32_t* error_word, cudaStream_t stream) {
  const int width = g.block_n > 0 ? g.block_n : 256;
  if (width % 16 != 0 || width < 16 || width > 256 || g.cluster > 1) return cudaErrorInvalidValue;
  SwapArgs a = {};
  a.out = t.out;
  a.ldo = t.ldo;
  a.M = t.M;
  a.n_out = t.n_out;
  a.num_kb = t.num_kb;
  const int cols = SILU ? kBlockM : 2 * kBlockM;  // of out that a pair's rows of the weight are
  a.m_tiles = (t.n_out + cols - 1) / cols;
  a.groups = t.groups;
  a.b_rows = t.b_rows;
  a.width = width;
  a.ranges = t.ranges;
  a.range_stride = t.range_stride;
  a.scale_sumsq = t.scale_sumsq;
  a.scale_parts = t.scale_parts;
  a.inv_width = t.inv_width;
  a.eps = t.eps;
  a.stage_bytes = kTileABytes + width / 2 * kBlockK * 2;
  const int rest = 8 * kSwapWarpBytes + kSwapScaleBytes + 1024;
  a.stages = std::min(kTileMaxStages, (kTileSmem - rest) / a.stage_bytes);
  CUtensorMap mw, mx;
  cudaError_t rc = make_tile_map(&mw, g.b, (uint64_t)std::max(1, g.groups) * g.b_rows, (uint64_t)g.K, (uint64_t)g.ldb,
                                 (uint32_t)(SILU ? kBlockM / 2 : kBlockM));
  if (rc != cudaSuccess) return rc;
  rc = make_tile_map(&mx, g.a, (uint64_t)g.M, (uint64_t)g.K, (uint64_t)g.lda, (uint32_t)(width / 2));
  if (rc != cudaSuccess) return rc;
  const KernelSetup ks = kernel_setup(reinterpret_cast<const void*>(gemm_swap_kernel<SILU>), kTileSmem, kTileThreads);
  if (ks.rc != cudaSuccess) return ks.rc;
  const long long tiles = (long long)((g.M + width - 1) / width) * a.m_tiles;  // grouped: counted on the device
  const int workers = (int)(g.groups > 0 ? ks.pairs : std::min<long long>(ks.pairs, tiles));
  return launch_kernel_ex(gemm_swap_kernel<SILU>, dim3((unsigned)(2 * workers)), dim3(kTileThreads),
                          (size_t)(a.stages * a.stage_bytes + rest), stream, g.pdl, 2, mw, mx, a, error_word);
}

template <int EPI>
cudaError_t launch_tile_epi(const TileGemm& g, TileArgs a, int sms, uint32_t* error_word, cudaStream_t stream, int* sumsq_rows) {
  TileShape t;
  t.pair = g.pair > 0 || (g.pair == 0 && g.block_n == 512);
  const int block_n = g.pair == 0 && g.block_n == 512 ? 256 : g.block_n;
  t.nsub = block_n > 256 ? 2 : 1;
  t.sub = block_n / t.nsub;
  if (block_n < 32 || block_n > 512 || block_n % (16 * t.nsub) != 0) return cudaErrorInvalidValue;
  const int sub_out = EPI == TILE_EPI_SILU || EPI == kTileEpiSiluExact ? t.sub / 2 : t.sub;
  a.cl = std::max(1, std::min({g.cluster, kTileMaxCluster, a.num_kb}));
  a.ss_cols = EPI == TILE_EPI_RESIDUAL && g.norm_w != nullptr && g.sumsq_cap <= 0 ? 128 : 0;
  if (a.ss_cols > 0 && t.sub % a.ss_cols != 0) return cudaErrorInvalidValue;
  if (a.cl > 1 && (t.nsub > 1 || sub_out % 16 != 0 || sub_out < 16 * a.cl)) return cudaErrorInvalidValue;
  const int ss_rows = a.ss_cols > 0 ? g.b_rows / a.ss_cols : (g.b_rows + t.nsub * t.sub - 1) / (t.nsub * t.sub) * a.cl;
  if (EPI == TILE_EPI_RESIDUAL && g.norm_w != nullptr && a.ss_cols == 0 && ss_rows > g.sumsq_cap) return cudaErrorInvalidValue;
  if (sumsq_rows != nullptr) *sumsq_rows = EPI == TILE_EPI_RESIDUAL && g.norm_w != nullptr ? ss_rows : 0;
  if (a.cl > 1)
    return t.pair ? launch_tile<true, EPI, true, 1>(g, a, t, sms, error_word, stream)
                  : launch_tile<false, EPI, true, 1>(g, a, t, sms, error_word, stream);
  if (t.nsub > 1)
    return t.pair ? launch_tile<true, EPI, false, 2>(g, a, t, sms, error_word, stream)
                  : launch_tile<false, EPI, false, 2>(g, a, t, sms, error_word, stream);
  return t.pair ? launch_tile<true, EPI, false, 1>(g, a, t, sms, error_word, stream)
                : launch_tile<false, EPI, false, 1>(g, a, t, sms, error_word, stream);
}

}  // namespace

TileGemm gemm_tile_choice(const TileGemm& g) {
  TileGemm c = g;
  if (g.block_n != 0 || g.pair == 2) return c;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const KernelSetup ks = kernel_setup(reinterpret_cast<const void*>(gemm_tile_kernel<true, TILE_EPI_PLAIN, false, 1>), kTileSmem,
                                      kTileThreads);
  choose_tile_once(c, dev, sms, ks.rc == cudaSuccess ? ks.pairs : 0);
  return c;
}

cudaError_t launch_gemm_tile(const TileGemm& g, uint32_t* error_word, cudaStream_t stream, int* sumsq_rows) {
  if (g.pair < -1 || g.pair > 2) return cudaErrorInvalidValue;
  if (g.M <= 0 || g.b_rows <= 0 || g.K <= 0 || g.K % 8 != 0 || g.lda % 8 != 0 || g.ldb % 8 != 0 || g.groups < 0 ||
      g.groups > kTileMaxGroups || (g.groups > 0 && (g.ranges == nullptr || g.scale_sumsq != nullptr)))
    return cudaErrorInvalidValue;
  if (g.silu_pairs && (g.epi != TILE_EPI_SILU || g.groups > 0 || g.pair == 2 || g.b_rows % (2 * kPairRows) != 0))
    return cudaErrorInvalidValue;
  if (g.exact_silu && (g.epi != TILE_EPI_SILU || g.pair == 2)) return cudaErrorInvalidValue;
  if (g.epi == TILE_EPI_SILU && g.b_rows % 2 != 0) return cudaErrorInvalidValue;
  if (g.epi == TILE_EPI_RESIDUAL &&
      (g.groups > 0 || g.b_rows % 128 != 0 || g.ldo % 8 != 0 || g.residual == nullptr ||
       (g.norm_w != nullptr && (g.out == nullptr || g.sumsq_out == nullptr)) ||
       ((reinterpret_cast<uintptr_t>(g.out) | reinterpret_cast<uintptr_t>(g.residual) | reinterpret_cast<uintptr_t>(g.stream_out) |
         reinterpret_cast<uintptr_t>(g.norm_w)) & 15u) != 0))
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
  a.residual = reinterpret_cast<char*>(g.residual);
  a.res_bytes = g.residual_fp32 ? 4 : 2;
  a.stream_out = reinterpret_cast<__nv_bfloat16*>(g.stream_out);
  a.norm_w = reinterpret_cast<const __nv_bfloat16*>(g.norm_w);
  a.sumsq_out = g.sumsq_out;
  if (sumsq_rows != nullptr) *sumsq_rows = 0;
  if (g.pair == 2) {
    if (g.epi == TILE_EPI_PLAIN) return launch_swap<false>(g, a, error_word, stream);
    return g.epi == TILE_EPI_SILU ? launch_swap<true>(g, a, error_word, stream) : cudaErrorInvalidValue;
  }
  const TileGemm c = gemm_tile_choice(g);
  if (c.block_n == 0) return cudaErrorInvalidValue;
  switch (g.epi) {
    case TILE_EPI_PLAIN: return launch_tile_epi<TILE_EPI_PLAIN>(c, a, sms, error_word, stream, sumsq_rows);
    case TILE_EPI_SILU:
      return g.exact_silu ? launch_tile_epi<kTileEpiSiluExact>(c, a, sms, error_word, stream, sumsq_rows)
                          : launch_tile_epi<TILE_EPI_SILU>(c, a, sms, error_word, stream, sumsq_rows);
    case TILE_EPI_RESIDUAL: return launch_tile_epi<TILE_EPI_RESIDUAL>(c, a, sms, error_word, stream, sumsq_rows);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace sm100
}  // namespace penny
