// The tiled GEMM with the weight on the M side (gemm_tile_sm100.cu): out = a * b^T for row counts that are no multiples
// of 256, and for groups of rows (the experts of a MoE layer), plain or with silu(gate) * up.
//
// A CTA pair's MMA has 256 rows whatever the data: with the rows of a there, eight experts of 1000 rows are paid as eight
// of 1024 to 1280, and the surplus rows are other experts' data, which cost power too.  Here 256 rows of the weight, whose
// sizes are multiples of that, meet up to 256 rows of a on the N side, where the width of an MMA is any multiple of 16: a
// group's rows are cut into equal tiles and each is paid to the next 16 rows.  Bound by the tensor pipe at the clock that
// the power limit leaves, by HBM for few rows (the ring then holds little else than weights).  The roles and the fill per
// step are those of gemm_tile_sm100.cuh: a step of 256 x 256 takes 530 cycles.  8 experts, hidden 4096, ffn 14336, gate/up
// and down of 1000 rows 389 -> 370 and 262 -> 205 us against tiles of 128 rows, of 2000 rows 571 -> 515 and 376 -> 295.
//   TMEM lane = row of the weight = column of out, TMEM column = row of a.  A warp takes 32 lanes x 16 columns at a time
//   and turns them in shared memory.
//   SILU: each CTA has 64 gate rows (lanes 0-63) and the 64 up rows of the same features (lanes 64-127); the warps of
//   quarters q and q + 2 hand each other half of their columns, so that each finishes eight rows of a.
#pragma once
#include "gemm_tile_sm100.cuh"

namespace penny {
namespace sm100 {

struct SwapArgs {
  __nv_bfloat16* out;
  int ldo, M, n_out;
  int num_kb, m_tiles;  // tiles of the weight
  int groups, b_rows;
  int width;            // rows of a per tile at most: a multiple of 16, up to 256
  int stages, stage_bytes;
  const int* ranges;
  int range_stride;
  const float* scale_sumsq;
  int scale_parts;
  float inv_width, eps;
};

constexpr int kSwapWarpBytes = 2 * 1024 + 1024;  // exchange (two buffers of 8 x 32 fp32), 16 x 32 bf16
constexpr int kSwapScaleBytes = 2 * 256 * 4;
constexpr int kSwapBand = 8;                     // row tiles that meet a weight tile one after another

template <bool SILU>
__global__ void __launch_bounds__(kTileThreads, 1)
gemm_swap_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const SwapArgs a,
                 uint32_t* error_word) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ uint64_t s_bars[2 * kTileMaxStages + 4];
  __shared__ short s_group[kTileMaxGroups];
  __shared__ uint32_t s_tmem;
  __shared__ int s_active, s_tiles;
  __shared__ volatile int s_abort;
  constexpr int kFeat = SILU ? 64 : kBlockM;  // columns of out that a CTA's rows of the weight are
  const int stages = a.stages, stage_bytes = a.stage_bytes;  // a stage: 128 rows of the weight, half of a tile's of a
  unsigned char* tiles = align_tiles(smem_raw);
  unsigned char* warp_area = tiles + stages * stage_bytes;
  float* s_scale = reinterpret_cast<float*>(warp_area + 8 * kSwapWarpBytes);  // [accumulator][row of the tile]
  uint64_t* full = s_bars;
  uint64_t* empty = s_bars + kTileMaxStages;
  uint64_t* tmem_full = s_bars + 2 * kTileMaxStages;
  uint64_t* tmem_empty = tmem_full + 2;
  volatile int* abort_flag = &s_abort;

  pdl_launch_dependents();
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t r = cluster_ctarank();
  const int worker = (int)blockIdx.x >> 1, workers = (int)gridDim.x >> 1;
  if (threadIdx.x == 0) {
    for (int i = 0; i < stages; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tmem_full[i], 1);
      mbar_init(&tmem_empty[i], 16);  // eight epilogue warps in each CTA
    }
    s_abort = 0;
    s_active = 1;
    s_group[0] = 0;
    s_tiles = (a.M + a.width - 1) / a.width * a.m_tiles;
    mbar_fence_init();
    tma_prefetch_desc(&map_w);
    tma_prefetch_desc(&map_x);
  }
  __syncwarp();
  if (warp == 1) tmem_alloc_pair(&s_tmem, 512);
  if (a.groups > 0) pdl_wait();  // the row ranges come from the kernel before this one
  auto group_rows = [&](int g, int& r0, int& r1) {  // only rows that a and out have
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
      int nt = (rows + a.width - 1) / a.width;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) nt += __shfl_xor_sync(0xffffffffu, nt, o);
      tot += nt;
    }
    if (lane == 0) {
      s_active = n;
      s_tiles = tot * a.m_tiles;
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_after_init();
  tc_fence_after_sync();
  const uint32_t tmem_base = s_tmem;
  const int num_tiles = s_tiles, active = s_active;

  auto fail = [&](uint32_t code) {
    s_abort = 1;
    st_cluster_u32(map_to_cta(smem_u32(const_cast<int*>(&s_abort)), r ^ 1u), 1u);
    atomicCAS(error_word, 0u, code);
  };
  // Walks the tiles of all groups in order; `tile` only grows.
  struct Cursor {
    int g, first, rows0, rows1, nt, step;  // group, its first tile, its rows, how many row tiles of how many rows
  };
  auto open_group = [&](Cursor& c) {
    if (a.groups > 0) {
      group_rows(s_group[c.g], c.rows0, c.rows1);
    } else {
      c.rows0 = 0;
      c.rows1 = a.M;
    }
    const int rows = c.rows1 - c.rows0;
    c.nt = (rows + a.width - 1) / a.width;
    c.step = ((rows + c.nt - 1) / c.nt + 15) & ~15;  // equal tiles, none empty: (nt - 1) * step <= (nt - 1) * width < rows
  };
  auto start = [&](Cursor& c) {
    c.g = 0;
    c.first = 0;
    if (active > 0) open_group(c);
  };
  // rows [row, row + rows) of a, tile m of the weight
  auto locate = [&](Cursor& c, int tile, int& row, int& rows, int& m) {
    while (tile - c.first >= c.nt * a.m_tiles) {
      c.first += c.nt * a.m_tiles;
      ++c.g;
      open_group(c);
    }
    const int t = tile - c.first, per_band = kSwapBand * a.m_tiles;
    const int band = t / per_band, in = t - band * per_band, n0 = band * kSwapBand;
    const int w = min(c.nt - n0, kSwapBand);
    m = in / w;
    row = c.rows0 + (n0 + in - m * w) * c.step;
    rows = min(c.rows1 - row, c.step);
  };
  auto mma_cols = [](int rows) { return (rows + 15) & ~15; };

  if (warp == 0) {
    // -------------------------------------------------------------- TMA producer
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    int ahead = 0;
    Cursor cur;
    start(cur);
    auto load_w = [&](int stage, int kb, int m) {
      unsigned char* sw = tiles + stage * stage_bytes;
      if (r == 0) mbar_expect_tx(&full[stage], 2u * (uint32_t)stage_bytes);
      const uint32_t bar = map_to_cta(smem_u32(&full[stage]), 0u);
      const int y = s_group[cur.g] * a.b_rows + m * 2 * kFeat + (int)r * kFeat;
      tma_load_2d_pair(sw, &map_w, bar, kb * kBlockK, y);
      if (SILU) tma_load_2d_pair(sw + kTileABytes / 2, &map_w, bar, kb * kBlockK, y + a.b_rows / 2);
    };
    if (a.groups == 0 && worker < num_tiles) {  // the weight does not depend on the predecessor
      int row, rows, m;
      locate(cur, worker, row, rows, m);
      ahead = min(stages, a.num_kb);
      for (int i = 0; i < ahead; ++i) {
        if (elect_one()) load_w(i, i, m);
        __syncwarp();
      }
    }
    pdl_wait();
    for (int tile = worker; ok && tile < num_tiles; tile += workers) {
      int row, rows, m;
      locate(cur, tile, row, rows, m);
      const int y = row + (int)r * (mma_cols(rows) / 2);  // the half of the MMA's columns that this CTA stages
      for (int kb = 0; kb < a.num_kb; ++kb) {
        ok = __all_sync(0xffffffffu, mbar_wait_abortable(&empty[stage], phase ^ 1u, abort_flag));
        if (!ok) break;
        if (elect_one()) {
          if (ahead <= 0) load_w(stage, kb, m);
          tma_load_2d_pair(tiles + stage * stage_bytes + kTileABytes, &map_x, map_to_cta(smem_u32(&full[stage]), 0u),
                           kb * kBlockK, y);
        }
        __syncwarp();
        --ahead;
        if (++stage == stages) {
          stage = 0;
          phase ^= 1u;
        }
      }
      if (!ok && lane == 0) fail(GEMM_ERR_PRODUCER_WAIT);
    }
    // every commit aimed at this CTA's slot barriers has arrived before it may leave
    for (int i = 0; ok && i < stages; ++i) {
      ok = __all_sync(0xffffffffu, mbar_wait_abortable(&empty[stage], phase ^ 1u, abort_flag));
      if (++stage == stages) {
        stage = 0;
        phase ^= 1u;
      }
    }
  } else if (warp == 1) {
    if (r == 0) {
      // ---------------------------------------------------------------- MMA issuer
      const uint64_t desc0 = make_smem_desc(smem_u32(tiles));
      const uint32_t desc_hi = (uint32_t)(desc0 >> 32);
      int stage = 0;
      uint32_t phase = 0;
      int it = 0;
      Cursor cur;
      start(cur);
      for (int tile = worker; tile < num_tiles; tile += workers, ++it) {
        int row, rows, m;
        locate(cur, tile, row, rows, m);
        const uint32_t idesc = make_idesc_bf16(2 * kBlockM, mma_cols(rows));
        const int ab = it & 1;
        bool ok = __all_sync(0xffffffffu, mbar_wait_abortable(&tmem_empty[ab], (((uint32_t)it >> 1) & 1u) ^ 1u, abort_flag));
        tc_fence_after_sync();
        const uint32_t d = tmem_base + (uint32_t)(ab * 256);
        for (int kb = 0; ok && kb < a.num_kb; ++kb) {
          ok = __all_sync(0xffffffffu, mbar_wait_abortable(&full[stage], phase, abort_flag));
          if (!ok) break;
          tc_fence_after_sync();
          const uint32_t lw = (uint32_t)desc0 + (uint32_t)(stage * (stage_bytes >> 4)), lx = lw + (kTileABytes >> 4);
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < kBlockK / kUmmaK; ++k)
              umma_bf16_pair(d, make_desc(desc_hi, lw + 2 * k), make_desc(desc_hi, lx + 2 * k), idesc, kb != 0 || k != 0);
            umma_commit_pair(&empty[stage], (uint16_t)3u);
          }
          __syncwarp();
          if (++stage == stages) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (!ok) {
          if (lane == 0) fail(GEMM_ERR_MMA_WAIT);
          break;
        }
        if (elect_one()) umma_commit_pair(&tmem_full[ab], (uint16_t)3u);
        __syncwarp();
      }
    }
  } else {
    // ------------------------------------- epilogue (this CTA's 128 rows of the weight)
    const int q = warp & 3, h = (warp - 2) >> 2;  // TMEM lane quarter; which of the two warps of it
    unsigned char* mine = warp_area + (warp - 2) * kSwapWarpBytes;
    const int other = h * 4 + ((q ^ 2) + 2) % 4;  // epilogue warp of the quarter with the other half of the products
    const float* theirs = reinterpret_cast<const float*>(warp_area + other * kSwapWarpBytes);
    float* xchg = reinterpret_cast<float*>(mine);
    unsigned char* stg = mine + 2048;
    // SILU: the two warps that meet at a barrier below leave the loop together
    const int pair_bar = 1 + (q & 1) + 2 * h;
    auto agree = [&](bool ok) {
      ok = __all_sync(0xffffffffu, ok);
      return SILU ? named_bar_all(pair_bar, 64, ok) : ok;
    };
    Cursor cur;
    start(cur);
    pdl_wait();
    int it = 0, turn = 0;
    for (int tile = worker; tile < num_tiles; tile += workers, ++it) {
      int row, rows, m;
      locate(cur, tile, row, rows, m);
      const int ab = it & 1;
      float* scale = s_scale + ab * 256;
      if (a.scale_sumsq != nullptr) {
        // 1 / rms of the tile's rows, a row per thread, under the product.  (All warps have left the tile before the one
        // that used this half last: the barriers of the tile between them.)
        const int i = (int)threadIdx.x - 64;
        float s = 0.f;
        if (i < rows) {
#pragma unroll 8
          for (int p = 0; p < a.scale_parts; ++p) s += __ldcg(a.scale_sumsq + (size_t)p * a.M + row + i);
        }
        scale[i] = rsqrtf(s * a.inv_width + a.eps);
        named_bar_sync(5, 256);
      }
      bool ok = !s_abort && mbar_wait_abortable(&tmem_full[ab], ((uint32_t)it >> 1) & 1u, abort_flag);
      if (!ok && lane == 0) fail(GEMM_ERR_EPILOGUE_WAIT);
      ok = agree(ok);
      if (a.scale_sumsq != nullptr) ok = named_bar_all(5, 256, ok);  // (that barrier has all eight warps)
      if (!ok) break;
      tc_fence_after_sync();
      const uint32_t tacc = tmem_base + (uint32_t)(ab * 256) + ((uint32_t)(q * 32) << 16);
      const int chunks = (rows + 15) / 16;
#pragma unroll 1
      for (int c = h; c < chunks; c += 2, ++turn) {
        uint32_t x[16];
        tmem_ld_32x16(tacc + c * 16, x);
        tmem_ld_wait();
        if (a.scale_sumsq != nullptr) {
#pragma unroll
          for (int j = 0; j < 16; ++j) x[j] = __float_as_uint(__uint_as_float(x[j]) * scale[c * 16 + j]);
        }
        __nv_bfloat16* line = reinterpret_cast<__nv_bfloat16*>(stg) + lane;  // [row][32 columns]
        if (SILU) {
          // gate (q < 2) finishes rows 0-7 of the chunk, up rows 8-15
          float* to = xchg + (turn & 1) * 256;
#pragma unroll
          for (int j = 0; j < 8; ++j) to[j * 32 + lane] = __uint_as_float(q < 2 ? x[8 + j] : x[j]);
          named_bar_sync(pair_bar, 64);  // (one per turn: two buffers)
          const float* from = theirs + (turn & 1) * 256;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float got = from[j * 32 + lane], kept = __uint_as_float(q < 2 ? x[j] : x[8 + j]);
            const float gv = q < 2 ? kept : got, uv = q < 2 ? got : kept;
            line[j * 32] = __float2bfloat16_rn(__fdividef(gv, 1.f + __expf(-gv)) * uv);
          }
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j) line[j * 32] = __float2bfloat16_rn(__uint_as_float(x[j]));
        }
        __syncwarp();
        const int col0 = (m * 2 + (int)r) * kFeat + (q & (SILU ? 1 : 3)) * 32 + (lane & 3) * 8;
        const int row0 = row + c * 16 + (SILU && q >= 2 ? 8 : 0);
#pragma unroll
        for (int j = 0; j < (SILU ? 1 : 2); ++j) {
          const int rr = j * 8 + (lane >> 2);
          const uint4 p = *reinterpret_cast<const uint4*>(stg + rr * 64 + (lane & 3) * 16);
          store16_local(a.out, a.ldo, row0 + rr, col0, p, row + rows, a.n_out);
        }
        __syncwarp();
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(map_to_cta(smem_u32(&tmem_empty[ab]), 0u));
    }
  }
  // ------------------------------------------------------------------- teardown
  tc_fence_before_sync();
  __syncwarp();
  pdl_wait();  // no thread leaves before the predecessor has finished
  cluster_sync_all();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

}  // namespace sm100
}  // namespace penny
