// The persistent tcgen05 GEMM of gemm_tile_sm100.cu:
//     out = a * b^T, a [M, K], b [N, K], bf16, fp32 accumulation
// on 128 x BN tiles of one CTA or 256 x 256 tiles of a CTA pair (cta_group::2), with
// the work that follows a linear in its epilogue.
//
// What bounds it: the tensor pipe for long K (pairs: 94 % of active cycles), the
// L2 -> shared memory fill for the narrower tiles, and the last wave.  Layout:
//   warp 0     TMA producer: [128 x 64] of a and this CTA's share of the b tile per
//              step into a ring (128-byte swizzle, no multicast)
//   warp 1     MMA issuer (the pair's leader): two accumulators in TMEM, so the
//              epilogue of a tile runs under the next tile's MMAs
//   warps 2-9  epilogue: TMEM -> registers (thread = row) -> swizzled staging rows ->
//              128-byte row segments; two warps per lane quarter share the columns
// Few tiles with a long K (the linears of a few hundred tokens): the pairs or CTAs of
// a cluster split the K steps of a tile and hand each other their fp32 sums through
// shared memory, each finishing the rows of its share of the four TMEM quarters.
// SILU: a b tile is BN / 2 gate rows and the BN / 2 up rows of the same features, so
// both halves of a product are columns of one accumulator and only the activation
// is written.  RESIDUAL: the output is added to the residual stream, which is kept
// in the reader's form too (times the next norm's weight) together with the sums
// of squares; the consumer multiplies its accumulator rows by 1 / rms.  The norm
// between two linears then costs no pass of its own.
// Groups (the experts of a MoE layer): the tile list is made on the device from the
// row ranges, so the host needs to know no expert's load.
#pragma once
#include "gemm_kernel_sm100.cuh"
#include "gemm_tile_sm100.h"
#include "pdl.h"

namespace penny {
namespace sm100 {

constexpr int kTileThreads = 320;
constexpr int kTileMaxGroups = 256;
constexpr int kTileMaxCluster = 4;  // pairs or single CTAs: a TMEM quarter each

struct TileArgs {
  __nv_bfloat16* out;
  int ldo, M, n_out;     // n_out: columns of out
  int num_kb, tiles_n, band;
  int groups, b_rows;
  int cl;                // pairs (or CTAs) per cluster; above 1 a cluster splits the K steps of its tile
  const int* ranges;
  int range_stride;
  const float* scale_sumsq;
  int scale_parts;
  float inv_width, eps;
  __nv_bfloat16* residual;
  const __nv_bfloat16* norm_w;
  float* sumsq_out;
};

template <bool PAIR, int BN>
struct TileCfg {
  static constexpr int kRows = PAIR ? 2 * kBlockM : kBlockM;  // rows of a tile
  static constexpr int kBRows = PAIR ? BN / 2 : BN;           // b rows this CTA stages
  static constexpr int kABytes = kBlockM * kBlockK * 2;
  static constexpr int kBBytes = kBRows * kBlockK * 2;
  static constexpr int kStageBytes = kABytes + kBBytes;
  static constexpr int kStages = (192 << 10) / kStageBytes < 8 ? (192 << 10) / kStageBytes : 8;
  static constexpr int kTmemCols = BN == 192 ? 512 : 2 * BN;
  static constexpr int kEpiBytes = 8 * 32 * kStageRowBytes;
  static constexpr int kSmemBytes = kStages * kStageBytes + kEpiBytes + 1024;
};

// Walks the tiles of all groups in order; `tile` only grows.
struct TileCursor {
  int g, first, rows0, rows1, mt;  // current group, its first tile, its rows, its row tiles
};

template <bool PAIR, int BN, int EPI>
__device__ __forceinline__ void gemm_tile_body(const CUtensorMap& map_a, const CUtensorMap& map_b, const TileArgs& a,
                                               uint32_t* error_word) {
  using Cfg = TileCfg<PAIR, BN>;
  constexpr int kStages = Cfg::kStages;
  constexpr bool kSilu = EPI == TILE_EPI_SILU;
  constexpr int kNOut = kSilu ? BN / 2 : BN;  // output columns of a tile
  extern __shared__ unsigned char smem_raw[];
  __shared__ uint64_t s_bars[2 * kStages + 4];
  __shared__ uint64_t s_peer_ready[kTileMaxCluster], s_recv;
  __shared__ short s_group[kTileMaxGroups];
  __shared__ float s_half[2][kBlockM];  // RESIDUAL, 128 columns: sums of squares of the second 64
  __shared__ uint32_t s_tmem;
  __shared__ int s_active, s_tiles;
  __shared__ volatile int s_abort;
  unsigned char* tiles = align_tiles(smem_raw);
  unsigned char* epi_stage = tiles + kStages * Cfg::kStageBytes;
  uint64_t* full = s_bars;
  uint64_t* empty = s_bars + kStages;
  uint64_t* tmem_full = s_bars + 2 * kStages;
  uint64_t* tmem_empty = tmem_full + 2;
  volatile int* abort_flag = &s_abort;

  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t crank = cluster_ctarank(), r = PAIR ? crank & 1u : 0u, lead = PAIR ? crank & ~1u : crank;
  const int cl = a.cl, cs = (int)(PAIR ? crank >> 1 : crank);  // K range in a cluster that shares a tile
  const int worker = (PAIR ? (int)blockIdx.x >> 1 : (int)blockIdx.x) / cl;
  const int workers = (PAIR ? (int)gridDim.x >> 1 : (int)gridDim.x) / cl;
  auto cta_of = [&](int d) { return PAIR ? 2u * (uint32_t)d + r : (uint32_t)d; };  // same rows, K range d
  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tmem_full[i], 1);
      mbar_init(&tmem_empty[i], PAIR ? 16 : 8);  // eight epilogue warps in each CTA
    }
    for (int i = 0; i < kTileMaxCluster; ++i) mbar_init(&s_peer_ready[i], 1);
    mbar_init(&s_recv, 1);
    s_abort = 0;
    s_active = 1;
    s_group[0] = 0;
    s_tiles = (a.M + Cfg::kRows - 1) / Cfg::kRows * a.tiles_n;
    mbar_fence_init();
    tma_prefetch_desc(&map_a);
    tma_prefetch_desc(&map_b);
  }
  __syncwarp();
  if (warp == 1) {
    if (PAIR) tmem_alloc_pair(&s_tmem, Cfg::kTmemCols);
    else tmem_alloc(&s_tmem, Cfg::kTmemCols);
  }
  if (a.groups > 0) pdl_wait();  // the row ranges come from the kernel before this one
  // Only rows that a and out have: a range that leaves them would be stored past out, and in a cluster bring a
  // second tile that nobody waits for.
  auto group_rows = [&](int g, int& r0, int& r1) {
    r0 = min(max(a.ranges[a.range_stride * g], 0), a.M);
    r1 = min(max(a.ranges[a.range_stride * g + 1], r0), a.M);
  };
  if (a.groups > 0 && warp == 0) {
    int n = 0, tot = 0;
    for (int g0 = 0; g0 < a.groups; g0 += 32) {
      const int g = g0 + lane;
      int r0 = 0, r1 = 0;
      if (g < a.groups) group_rows(g, r0, r1);
      const int rows = r1 - r0;
      const unsigned m = __ballot_sync(0xffffffffu, rows > 0);
      if (rows > 0) s_group[n + __popc(m & ((1u << lane) - 1u))] = (short)g;
      n += __popc(m);
      int mt = (rows + Cfg::kRows - 1) / Cfg::kRows;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) mt += __shfl_xor_sync(0xffffffffu, mt, o);
      tot += mt;
    }
    if (lane == 0) {
      s_active = n;
      s_tiles = tot * a.tiles_n;
    }
  }
  tc_fence_before_sync();
  __syncwarp();
  if (PAIR || cl > 1) cluster_sync_all();
  else __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = s_tmem;
  const int num_tiles = s_tiles, active = s_active;

  const int kb0 = a.num_kb * cs / cl, kb1 = a.num_kb * (cs + 1) / cl;
  auto fail = [&](uint32_t code) {
    s_abort = 1;
    for (uint32_t c = 0; c < (PAIR ? 2u : 1u) * (uint32_t)cl; ++c)
      if (c != crank) st_cluster_u32(map_to_cta(smem_u32(const_cast<int*>(&s_abort)), c), 1u);
    atomicCAS(error_word, 0u, code);
  };
  auto open_group = [&](TileCursor& c) {
    if (a.groups > 0) {
      group_rows(s_group[c.g], c.rows0, c.rows1);
    } else {
      c.rows0 = 0;
      c.rows1 = a.M;
    }
    c.mt = (c.rows1 - c.rows0 + Cfg::kRows - 1) / Cfg::kRows;
  };
  auto start = [&](TileCursor& c) {
    c.g = 0;
    c.first = 0;
    if (active > 0) open_group(c);
  };
  // first row of this CTA's share of the tile, column block
  auto locate = [&](TileCursor& c, int tile, int& row, int& n_blk) {
    while (tile - c.first >= c.mt * a.tiles_n) {
      c.first += c.mt * a.tiles_n;
      ++c.g;
      open_group(c);
    }
    // bands of `band` row tiles, rows fastest inside a band
    const int t = tile - c.first, per_band = a.band * a.tiles_n;
    const int bnd = t / per_band, in = t - bnd * per_band, m0 = bnd * a.band;
    const int h = min(c.mt - m0, a.band);
    n_blk = in / h;
    row = c.rows0 + (m0 + in - n_blk * h) * Cfg::kRows + (int)r * kBlockM;
  };

  if (warp == 0) {
    if (lane == 0) {
      // ------------------------------------------------------------ TMA producer
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      // b (weights) does not depend on the predecessor: its share of the first ring is requested before the
      // wait, the rows of a after it
      int ahead = 0;
      TileCursor cur;
      start(cur);
      auto b_row = [&](int n_blk) {
        const int b0 = s_group[cur.g] * a.b_rows + n_blk * kNOut;
        if (!PAIR) return b0;
        return kSilu ? b0 + (int)r * (a.b_rows / 2) : b0 + (int)r * (BN / 2);
      };
      auto load_b = [&](int stage, int kb, int by) {
        unsigned char* sb = tiles + stage * Cfg::kStageBytes + Cfg::kABytes;
        if (PAIR) {
          if (r == 0) mbar_expect_tx(&full[stage], 2u * Cfg::kStageBytes);
          tma_load_2d_pair(sb, &map_b, map_to_cta(smem_u32(&full[stage]), lead), kb * kBlockK, by);
        } else {
          mbar_expect_tx(&full[stage], Cfg::kStageBytes);
          tma_load_2d(sb, &map_b, &full[stage], kb * kBlockK, by);
          if (kSilu) tma_load_2d(sb + Cfg::kBBytes / 2, &map_b, &full[stage], kb * kBlockK, by + a.b_rows / 2);
        }
      };
      if (a.groups == 0 && worker < num_tiles) {
        int row, n_blk;
        locate(cur, worker, row, n_blk);
        ahead = min(kStages, kb1 - kb0);
        for (int i = 0; i < ahead; ++i) load_b(i, kb0 + i, b_row(n_blk));
      }
      pdl_wait();
      for (int tile = worker; ok && tile < num_tiles && !s_abort; tile += workers) {
        int row, n_blk;
        locate(cur, tile, row, n_blk);
        const int by = b_row(n_blk);
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait_abortable(&empty[stage], phase ^ 1u, abort_flag)) {
            ok = false;
            break;
          }
          unsigned char* sa = tiles + stage * Cfg::kStageBytes;
          if (ahead > 0) --ahead;
          else load_b(stage, kb, by);
          if (PAIR) tma_load_2d_pair(sa, &map_a, map_to_cta(smem_u32(&full[stage]), lead), kb * kBlockK, row);
          else tma_load_2d(sa, &map_a, &full[stage], kb * kBlockK, row);
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (!ok) fail(GEMM_ERR_PRODUCER_WAIT);
      }
      // every commit aimed at this CTA's slot barriers has arrived before it may leave
      for (int i = 0; PAIR && ok && i < kStages && !s_abort; ++i) {
        if (!mbar_wait_abortable(&empty[stage], phase ^ 1u, abort_flag)) break;
        if (++stage == kStages) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && r == 0) {
      // -------------------------------------------------------------- MMA issuer
      constexpr uint32_t idesc = make_idesc_bf16(Cfg::kRows, BN);
      int stage = 0;
      uint32_t phase = 0;
      int it = 0;
      for (int tile = worker; tile < num_tiles && !s_abort; tile += workers, ++it) {
        const int ab = it & 1;
        bool ok = mbar_wait_abortable(&tmem_empty[ab], (((uint32_t)it >> 1) & 1u) ^ 1u, abort_flag);
        tc_fence_after_sync();
        const uint32_t d = tmem_base + (uint32_t)(ab * BN);
        for (int kb = kb0; ok && kb < kb1; ++kb) {
          if (!mbar_wait_abortable(&full[stage], phase, abort_flag)) {
            ok = false;
            break;
          }
          tc_fence_after_sync();
          const uint32_t sa = smem_u32(tiles + stage * Cfg::kStageBytes);
          const uint64_t da = make_smem_desc(sa), db = make_smem_desc(sa + Cfg::kABytes);
#pragma unroll
          for (int k = 0; k < kBlockK / kUmmaK; ++k) {
            if (PAIR) umma_bf16_pair(d, advance_desc_k(da, k), advance_desc_k(db, k), idesc, kb != kb0 || k != 0);
            else umma_bf16(d, advance_desc_k(da, k), advance_desc_k(db, k), idesc, kb != kb0 || k != 0);
          }
          if (PAIR) umma_commit_pair(&empty[stage], (uint16_t)(3u << lead));
          else umma_commit(&empty[stage]);
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (!ok) {
          fail(GEMM_ERR_MMA_WAIT);
          break;
        }
        if (PAIR) umma_commit_pair(&tmem_full[ab], (uint16_t)(3u << lead));
        else umma_commit(&tmem_full[ab]);
      }
    }
  } else {
    // ---------------------------------------------- epilogue (this CTA's 128 rows)
    const int q = warp & 3, h = (warp - 2) >> 2;  // TMEM lane quarter; which of the two warps of it
    unsigned char* stg = epi_stage + (warp - 2) * (32 * kStageRowBytes);
    // 64-column passes of this warp.  (RESIDUAL writes a sum of squares per 128 columns: both passes of them, or
    // with 128 columns in all the two warps of a quarter add theirs.)
    constexpr int kPasses = kNOut / 64;
    constexpr bool kHalves = EPI == TILE_EPI_RESIDUAL && kPasses == 2;
    constexpr int kGrain = EPI == TILE_EPI_RESIDUAL && !kHalves ? 2 : 1;
    constexpr int kHalf = (kPasses / kGrain + 1) / 2 * kGrain;
    const int c_begin = h * kHalf, c_end = min(kPasses, c_begin + kHalf);
    // in a cluster the quarters [q0, q1) of the rows are finished here
    const int q0 = (4 * cs + cl - 1) / cl, q1 = (4 * (cs + 1) + cl - 1) / cl, owner = q * cl / 4;
    // The two warps of a quarter that meet at a barrier below leave this loop together: a bounded wait that ran
    // out in one of them, or an abort that only one has seen, ends it for both.
    auto agree = [&](bool ok) {
      ok = __all_sync(0xffffffffu, ok);
      return kHalves ? named_bar_all(1 + q, 64, ok) : ok;
    };
    TileCursor cur;
    start(cur);
    pdl_wait();
    int it = 0;
    for (int tile = worker; tile < num_tiles; tile += workers, ++it) {
      int row, n_blk;
      locate(cur, tile, row, n_blk);
      row += q * 32;
      const int row_end = cur.rows1;
      const int ab = it & 1;
      float scale = 1.f;
      if (a.scale_sumsq != nullptr) {
        float s = 0.f;
        const int rr = min(row + lane, a.M - 1);
#pragma unroll 8
        for (int p = 0; p < a.scale_parts; ++p) s += __ldcg(a.scale_sumsq + (size_t)p * a.M + rr);
        scale = rsqrtf(s * a.inv_width + a.eps);
      }
      // RESIDUAL (the launcher wants whole, aligned rows of 64 columns here): the stream and the norm's weight
      // travel while the product is finished, a pass ahead (behind it they were 3 us of the tail)
      uint4 res[8], nw = make_uint4(0, 0, 0, 0);
      auto load_residual = [&](int c) {
        const int col = n_blk * kNOut + c * 64 + (lane & 7) * 8;
        const __nv_bfloat16* rp = a.residual + (size_t)(row + (lane >> 3)) * a.ldo + col;
#pragma unroll
        for (int i = 0; i < 8; ++i)
          if (row + i * 4 + (lane >> 3) < row_end && col < a.n_out) res[i] = *reinterpret_cast<const uint4*>(rp + (size_t)(i * 4) * a.ldo);
        if (a.norm_w != nullptr && col < a.n_out) nw = __ldg(reinterpret_cast<const uint4*>(a.norm_w + col));
      };
      if (EPI == TILE_EPI_RESIDUAL && owner == cs && c_begin < c_end) load_residual(c_begin);
      bool ok = !s_abort && mbar_wait_abortable(&tmem_full[ab], ((uint32_t)it >> 1) & 1u, abort_flag);
      if (!ok && lane == 0) fail(GEMM_ERR_EPILOGUE_WAIT);
      if (!agree(ok)) break;
      tc_fence_after_sync();
      const uint32_t tacc = tmem_base + (uint32_t)(ab * BN) + ((uint32_t)(q * 32) << 16);
      // Cluster: a quarter's sums go to its owner, as [sender][accumulator column / 4][its rows] float4 in the
      // ring of a CTA that has said that its MMAs are complete (a cluster works on one tile).
      auto slot = [&](int from, int to, int rows, int q_first) {  // of this thread's row
        return ((from - (from > to ? 1 : 0)) * (BN / 4)) * rows + (q - q_first) * 32 + lane;
      };
      const int own_rows = (q1 - q0) * 32;
      const float4* s_in = reinterpret_cast<const float4*>(tiles);
      if (cl > 1) {
        if (threadIdx.x == 64) mbar_expect_tx(&s_recv, (uint32_t)(own_rows * BN * 4 * (cl - 1)));
        if (warp == 2 && lane < cl && lane != cs) mbar_arrive_cluster(map_to_cta(smem_u32(&s_peer_ready[cs]), cta_of(lane)));
        if (owner != cs) {
          const int d0 = (4 * owner + cl - 1) / cl, rows = ((4 * (owner + 1) + cl - 1) / cl - d0) * 32;
          ok = mbar_wait_cluster(&s_peer_ready[owner], 0u, abort_flag);
          if (!ok && lane == 0) fail(GEMM_ERR_EPILOGUE_WAIT);
          if (!__all_sync(0xffffffffu, ok)) break;  // (this branch leaves the loop before the barrier anyway)
          const uint32_t bar = map_to_cta(smem_u32(&s_recv), cta_of(owner));
          const uint32_t remote = map_to_cta(smem_u32(tiles), cta_of(owner)) + (uint32_t)slot(cs, owner, rows, d0) * 16;
#pragma unroll 1
          for (int k = h * (BN / 2); k < (h + 1) * (BN / 2); k += 32) {
            uint32_t x[32];
            tmem_ld_32x32(tacc + k, x);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 8; ++j)
              st_async_v4(remote + (uint32_t)((k / 4 + j) * rows * 16), bar, x[4 * j], x[4 * j + 1], x[4 * j + 2], x[4 * j + 3]);
          }
          break;
        }
        ok = mbar_wait_cluster(&s_recv, 0u, abort_flag);
        if (!ok && lane == 0) fail(GEMM_ERR_EPILOGUE_WAIT);
        if (!agree(ok)) break;
      }
      // 32 accumulator columns of pass c of the finished tile: k in [0, kAcc)
      auto load32 = [&](int c, int k, uint32_t (&x)[32]) {
        const int col = k < 64 ? c * 64 + k : BN / 2 + c * 64 + k - 64;
        tmem_ld_32x32(tacc + col, x);
        tmem_ld_wait();
        if (cl == 1) return;
        float v[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = 0.f;
        for (int p = 0; p < cl; ++p) {  // in K order, this CTA's own part in its place
          if (p == cs) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] += __uint_as_float(x[j]);
          } else {
            const float4* src = s_in + slot(p, cs, own_rows, q0) + col / 4 * own_rows;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const float4 y = src[j * own_rows];
              v[4 * j] += y.x;
              v[4 * j + 1] += y.y;
              v[4 * j + 2] += y.z;
              v[4 * j + 3] += y.w;
            }
          }
        }
#pragma unroll
        for (int j = 0; j < 32; ++j) x[j] = __float_as_uint(v[j]);
      };
      float ss[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) ss[i] = 0.f;
#pragma unroll 1
      for (int c = c_begin; c < c_end; ++c) {
        // 64 output columns of this warp's 32 rows
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          uint32_t x[32];
          load32(c, hf * 32, x);
          if (kSilu) {
            uint32_t up[32];
            load32(c, 64 + hf * 32, up);
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              const float gv = __uint_as_float(x[j]) * scale, uv = __uint_as_float(up[j]) * scale;
              x[j] = __float_as_uint(__fdividef(gv, 1.f + __expf(-gv)) * uv);
            }
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) x[j] = __float_as_uint(__uint_as_float(x[j]) * scale);
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            uint4 v;
            v.x = pack_bf16x2(x[8 * j], x[8 * j + 1]);
            v.y = pack_bf16x2(x[8 * j + 2], x[8 * j + 3]);
            v.z = pack_bf16x2(x[8 * j + 4], x[8 * j + 5]);
            v.w = pack_bf16x2(x[8 * j + 6], x[8 * j + 7]);
            *reinterpret_cast<uint4*>(stg + lane * kStageRowBytes + (((hf * 4 + j) ^ (lane & 7)) << 4)) = v;
          }
        }
        __syncwarp();
        const int col = n_blk * kNOut + c * 64 + (lane & 7) * 8;
        if (EPI == TILE_EPI_RESIDUAL) {
          const uint32_t ww[4] = {nw.x, nw.y, nw.z, nw.w};
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int rr = i * 4 + (lane >> 3);
            const uint4 p = *reinterpret_cast<const uint4*>(stg + rr * kStageRowBytes + (((lane & 7) ^ (rr & 7)) << 4));
            if (row + rr >= row_end || col >= a.n_out) continue;
            const uint32_t pw[4] = {p.x, p.y, p.z, p.w}, rw[4] = {res[i].x, res[i].y, res[i].z, res[i].w};
            uint32_t zo[4], wo[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const float z0 = __uint_as_float(pw[k] << 16) + __uint_as_float(rw[k] << 16);
              const float z1 = __uint_as_float(pw[k] & 0xffff0000u) + __uint_as_float(rw[k] & 0xffff0000u);
              ss[i] += z0 * z0 + z1 * z1;
              zo[k] = pack_bf16x2(__float_as_uint(z0), __float_as_uint(z1));
              wo[k] = pack_bf16x2(__float_as_uint(z0 * __uint_as_float(ww[k] << 16)),
                                  __float_as_uint(z1 * __uint_as_float(ww[k] & 0xffff0000u)));
            }
            const size_t off = (size_t)(row + rr) * a.ldo + col;
            *reinterpret_cast<uint4*>(a.residual + off) = make_uint4(zo[0], zo[1], zo[2], zo[3]);
            if (a.norm_w != nullptr) *reinterpret_cast<uint4*>(a.out + off) = make_uint4(wo[0], wo[1], wo[2], wo[3]);
          }
          if (c + 1 < c_end) load_residual(c + 1);
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int rr = i * 4 + (lane >> 3);
            const uint4 p = *reinterpret_cast<const uint4*>(stg + rr * kStageRowBytes + (((lane & 7) ^ (rr & 7)) << 4));
            store16_local(a.out, a.ldo, row + rr, col, p, row_end, a.n_out);
          }
        }
        __syncwarp();
        if (EPI == TILE_EPI_RESIDUAL && a.norm_w != nullptr && (kHalves || (c & 1))) {
          // 128 columns done: sum over the eight lanes of a row
          if (kHalves && h == 0) named_bar_sync(1 + q, 64);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            float s = ss[i];
            s += __shfl_xor_sync(0xffffffffu, s, 4);
            s += __shfl_xor_sync(0xffffffffu, s, 2);
            s += __shfl_xor_sync(0xffffffffu, s, 1);
            const int rr = row + i * 4 + (lane >> 3);
            float* other = &s_half[it & 1][q * 32 + i * 4 + (lane >> 3)];
            if (kHalves && h == 1) {
              if ((lane & 7) == 0) *other = s;
            } else if ((lane & 7) == 0 && rr < row_end && col < a.n_out) {
              if (kHalves) s += *other;
              a.sumsq_out[(size_t)(n_blk * (BN / 128) + (c >> 1)) * a.M + rr] = s;
            }
            ss[i] = 0.f;
          }
          if (kHalves && h == 1) named_bar_sync(1 + q, 64);
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) {
        if (PAIR) mbar_arrive_cluster(map_to_cta(smem_u32(&tmem_empty[ab]), lead));
        else mbar_arrive(&tmem_empty[ab]);
      }
    }
  }
  // ------------------------------------------------------------------- teardown
  tc_fence_before_sync();
  __syncwarp();
  pdl_wait();  // no thread leaves before the predecessor has finished
  if (PAIR || cl > 1) cluster_sync_all();
  else __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    if (PAIR) tmem_dealloc_pair(tmem_base, Cfg::kTmemCols);
    else tmem_dealloc(tmem_base, Cfg::kTmemCols);
  }
}

template <int BN, int EPI>
__global__ void __launch_bounds__(kTileThreads, 1)
gemm_tile_pair(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const TileArgs a,
               uint32_t* error_word) {
  gemm_tile_body<true, BN, EPI>(map_a, map_b, a, error_word);
}
template <int BN, int EPI>
__global__ void __launch_bounds__(kTileThreads, 1)
gemm_tile_single(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const TileArgs a,
                 uint32_t* error_word) {
  gemm_tile_body<false, BN, EPI>(map_a, map_b, a, error_word);
}

}  // namespace sm100
}  // namespace penny
