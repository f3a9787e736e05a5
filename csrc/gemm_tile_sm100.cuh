// The persistent tcgen05 GEMM of gemm_tile_sm100.cu:
//     out = a * b^T, a [M, K], b [N, K], bf16, fp32 accumulation
// on tiles of 128 rows (one CTA) or 256 rows (a CTA pair, cta_group::2) and of as many columns as the
// launcher asks for, with the work that follows a linear in its epilogue.
//
// What bounds it: the tensor pipe for long K, the L2 -> shared memory fill for the narrower tiles, and the last
// round of tiles.  That is why the tile's width is a run-time number: `nsub` (1 or 2) accumulators of `sub` columns
// (a multiple of 16, up to 256 each: one MMA each per K step) share the staged rows of a, and the launcher picks
// the width with which the tiles fill the SMs.  Layout:
//   warp 0     TMA producer: [128 x 64] of a and this CTA's share of the b tile per
//              step into a ring (128-byte swizzle, no multicast)
//   warp 1     MMA issuer (the pair's leader): up to 256 columns there are two sets of accumulators in TMEM, so
//              the epilogue of a tile runs under the next tile's MMAs
//   warps 2-9  epilogue: TMEM -> registers (thread = row) -> swizzled staging rows ->
//              row segments; two warps per lane quarter share the columns
// Few tiles with a long K (the linears of a few hundred tokens): the pairs or CTAs of
// a cluster split the K steps of a tile (SPLIT) and hand each other their fp32 sums through
// shared memory, each finishing all rows of its share of the columns.
// SILU: an accumulator is sub / 2 gate columns and the sub / 2 up columns of the same features, so
// both halves of a product are in one thread and only the activation
// is written.  The weight holds all gate rows before all up rows, or both in turn in blocks of 64 (what the decode GEMM
// reads): an accumulator then takes a strip of the same 2^k rows of each of several blocks, which is one box of a tensor
// map of four dimensions, so the features of a tile may still be any multiple of 8 (whole blocks alone would leave 112 tiles
// to 148 SMs where 14336 features of up to 128 rows have 144).  RESIDUAL: the output is added to the residual stream, which is kept
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
constexpr int kTileMaxCluster = 4;  // pairs or single CTAs
constexpr int kTileMaxStages = 8;
constexpr int kTileABytes = kBlockM * kBlockK * 2;
constexpr int kPairRows = 64;  // gate rows, and up rows, of a block of a weight that holds them in turn

constexpr int kTileEpiSiluExact = 3;  // TILE_EPI_SILU with exact_silu: kernels of their own

struct TileArgs {
  __nv_bfloat16* out;
  int ldo, M, n_out;     // n_out: columns of out
  int num_kb, tiles_n, band;
  int groups, b_rows;
  int sub;               // columns of an accumulator (NSUB of them are a tile)
  int strip_shift;       // SILU: -1, or (blocks of gate and up rows) log2 of the rows of a block in an accumulator
  int stages, accs;      // ring; sets of accumulators
  int tmem_cols;
  int cl;                // pairs (or CTAs) per cluster; above 1 a cluster splits the K steps of its tile
  const int* ranges;
  int range_stride;
  const float* scale_sumsq;
  int scale_parts;
  float inv_width, eps;
  char* residual;
  int res_bytes;         // of an element of the residual: 2 (bf16) or 4 (fp32)
  __nv_bfloat16* stream_out;
  const __nv_bfloat16* norm_w;
  float* sumsq_out;
  int ss_cols;           // columns behind an entry of sumsq_out: 128, or 0: all that a CTA finishes of a tile
};

// What a launch chooses, and what follows from it.
struct TileShape {
  bool pair;
  int sub, nsub;
  __host__ __device__ int rows() const { return pair ? 2 * kBlockM : kBlockM; }
  __host__ __device__ int b_bytes() const { return (pair ? sub / 2 : sub) * kBlockK * 2; }  // of one accumulator, staged by this CTA
  __host__ __device__ int stage_bytes() const { return kTileABytes + nsub * b_bytes(); }
};
// Epilogue staging of a warp: 32 rows of 32 bf16, or (SPLIT) 16 bf16 or (RESIDUAL) 16 fp32
template <int EPI, bool SPLIT>
struct TileEpi {
  static constexpr int kChunk = SPLIT || EPI == TILE_EPI_RESIDUAL ? 16 : 32;  // output columns of a pass
  static constexpr int kRowBytes = kChunk * (EPI == TILE_EPI_RESIDUAL ? 4 : 2);
  static constexpr int kBytes = 8 * 32 * kRowBytes;
};

// silu(g) = g / (1 + exp(-g)) for |g| up to kNearGate by long division: an approximate quotient, and the remainder that it
// leaves, which an fma gives exactly, divided once more.  (The divisor stays far below 2^126, where the fast division gives
// up.)  Against the same quotient in 64 bits, all fp32 gates of 2^-40 to 40 on either side: 0.500000 units of fp32 at most, the
// compiler's division 0.499999; two of 759 million differ between them.
constexpr float kNearGate = 40.f;
__device__ __forceinline__ float silu_near(float g) {
  const float d = 1.f + __expf(-g), r = __fdividef(1.f, d), q = g * r;
  return fmaf(fmaf(-q, d, g), r, q);
}

// Walks the tiles of all groups in order; `tile` only grows.
struct TileCursor {
  int g, first, rows0, rows1, mt;  // current group, its first tile, its rows, its row tiles
};

// (NSUB is a template parameter: with a run-time branch around the second accumulator's MMAs a K step of 256 x 256
// tiles took 0.50 us instead of 0.38.)
template <bool PAIR, int EPI, bool SPLIT, int NSUB>
__device__ __forceinline__ void gemm_tile_body(const CUtensorMap& map_a, const CUtensorMap& map_b, const TileArgs& a,
                                               uint32_t* error_word) {
  using Epi = TileEpi<EPI, SPLIT>;
  constexpr bool kExact = EPI == kTileEpiSiluExact, kSilu = EPI == TILE_EPI_SILU || kExact, kRes = EPI == TILE_EPI_RESIDUAL;
  constexpr int kRows = PAIR ? 2 * kBlockM : kBlockM;
  constexpr int kChunk = Epi::kChunk, kRowBytes = Epi::kRowBytes;
  extern __shared__ unsigned char smem_raw[];
  __shared__ uint64_t s_bars[2 * kTileMaxStages + 4];
  __shared__ uint64_t s_peer_ready[kTileMaxCluster], s_recv;
  __shared__ short s_group[kTileMaxGroups];
  __shared__ float s_half[2][kBlockM];  // RESIDUAL: sums of squares of the second warp of a quarter
  __shared__ uint32_t s_tmem;
  __shared__ int s_active, s_tiles;
  __shared__ volatile int s_abort;
  constexpr int nsub = NSUB;
  const int stages = a.stages, sub = a.sub;
  const int b_bytes = (PAIR ? sub / 2 : sub) * kBlockK * 2, stage_bytes = kTileABytes + nsub * b_bytes;
  const int sub_out = kSilu ? sub / 2 : sub;  // output columns of an accumulator
  unsigned char* tiles = align_tiles(smem_raw);
  unsigned char* epi_stage = tiles + stages * stage_bytes;
  uint64_t* full = s_bars;
  uint64_t* empty = s_bars + kTileMaxStages;
  uint64_t* tmem_full = s_bars + 2 * kTileMaxStages;
  uint64_t* tmem_empty = tmem_full + 2;
  volatile int* abort_flag = &s_abort;

  pdl_launch_dependents();
  // (read from lane 0, so that the compiler knows it to be the same in all lanes)
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t crank = PAIR || SPLIT ? cluster_ctarank() : 0u, r = PAIR ? crank & 1u : 0u, lead = PAIR ? crank & ~1u : crank;
  const int cl = SPLIT ? a.cl : 1, cs = SPLIT ? (int)(PAIR ? crank >> 1 : crank) : 0;  // K range in a cluster that shares a tile
  const int worker = (PAIR ? (int)blockIdx.x >> 1 : (int)blockIdx.x) / cl;
  const int workers = (PAIR ? (int)gridDim.x >> 1 : (int)gridDim.x) / cl;
  auto cta_of = [&](int d) { return PAIR ? 2u * (uint32_t)d + r : (uint32_t)d; };  // same rows, K range d
  if (threadIdx.x == 0) {
    for (int i = 0; i < stages; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tmem_full[i], 1);
      mbar_init(&tmem_empty[i], PAIR ? 16 : 8);  // eight epilogue warps in each CTA
    }
    for (int i = 0; SPLIT && i < kTileMaxCluster; ++i) mbar_init(&s_peer_ready[i], 1);
    if (SPLIT) mbar_init(&s_recv, 1);
    s_abort = 0;
    s_active = 1;
    s_group[0] = 0;
    s_tiles = (a.M + kRows - 1) / kRows * a.tiles_n;
    mbar_fence_init();
    tma_prefetch_desc(&map_a);
    tma_prefetch_desc(&map_b);
  }
  __syncwarp();
  if (warp == 1) {
    if (PAIR) tmem_alloc_pair(&s_tmem, (uint32_t)a.tmem_cols);
    else tmem_alloc(&s_tmem, (uint32_t)a.tmem_cols);
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
      int mt = (rows + kRows - 1) / kRows;
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
  __syncthreads();  // (orders the other threads' shared memory behind thread 0's initialisation and fence)
  if (PAIR || SPLIT) cluster_sync_after_init();
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
    c.mt = (c.rows1 - c.rows0 + kRows - 1) / kRows;
  };
  auto start = [&](TileCursor& c) {
    c.g = 0;
    c.first = 0;
    if (active > 0) open_group(c);
  };
  // SILU: where the first accumulator's features begin, row in the block and block (without strips: feature, group), and
  // what a further accumulator adds to either
  const bool strips = kSilu && a.strip_shift >= 0;
  const int next_row = strips ? 0 : sub_out, next_block = strips ? sub_out >> a.strip_shift : 0;
  auto features = [&](int n_blk, int group, int& row, int& block) {
    row = n_blk * nsub * sub_out;
    block = group;
    if (strips) {
      const int per = kPairRows >> a.strip_shift, g = n_blk / per;  // (the strips of a block are neighbours)
      row = (n_blk - g * per) << a.strip_shift;
      block = g * nsub * next_block;
    }
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
    row = c.rows0 + (m0 + in - n_blk * h) * kRows + (int)r * kBlockM;
  };

  // Producer and issuer run as whole warps and elect a lane only for the instructions themselves: operands that are
  // the same in all lanes then stay in uniform registers.  In a branch of one lane every TMA and MMA fetched its operands
  // one by one, and a K step took 600 cycles on pairs (540 on single CTAs) however narrow the tile; now 300 at 64
  // columns, 335 at 128, 470 at 192, 562 at 256 (single 64: 346, 128: 433), where the fill of shared memory at 60 to 75
  // bytes a cycle bounds it.
  if (warp == 0) {
    // -------------------------------------------------------------- TMA producer
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    // b (weights) does not depend on the predecessor: its share of the first ring is requested before the
    // wait, the rows of a after it
    int ahead = 0;
    TileCursor cur;
    start(cur);
    // rows of b of the tile's first accumulator (the second one's lie sub_out behind), SILU: as `features`
    auto b_rows_at = [&](int n_blk, int& by, int& bz) {
      if (kSilu) features(n_blk, s_group[cur.g], by, bz);
      else by = s_group[cur.g] * a.b_rows + n_blk * nsub * sub_out + (PAIR ? (int)r * (sub / 2) : 0), bz = 0;
    };
    auto load_b = [&](int stage, int kb, int by, int bz) {
      unsigned char* sb = tiles + stage * stage_bytes + kTileABytes;
      const int x = kb * kBlockK;
      if (PAIR) {
        if (r == 0) mbar_expect_tx(&full[stage], 2u * (uint32_t)stage_bytes);
        const uint32_t bar = map_to_cta(smem_u32(&full[stage]), lead);
        if (kSilu) {  // one CTA has the gate rows, the other the up rows
          tma_load_4d_pair(sb, &map_b, bar, x, by, (int)r, bz);
          if (nsub > 1) tma_load_4d_pair(sb + b_bytes, &map_b, bar, x, by + next_row, (int)r, bz + next_block);
        } else {
          tma_load_2d_pair(sb, &map_b, bar, x, by);
          if (nsub > 1) tma_load_2d_pair(sb + b_bytes, &map_b, bar, x, by + sub_out);
        }
      } else {
        mbar_expect_tx(&full[stage], (uint32_t)stage_bytes);
#pragma unroll
        for (int s = 0; s < nsub; ++s) {
          if (kSilu) {
            tma_load_4d(sb, &map_b, &full[stage], x, by + s * next_row, 0, bz + s * next_block);
            tma_load_4d(sb + b_bytes / 2, &map_b, &full[stage], x, by + s * next_row, 1, bz + s * next_block);
          } else {
            tma_load_2d(sb, &map_b, &full[stage], x, by + s * sub_out);
          }
          sb += b_bytes;
        }
      }
    };
    if (a.groups == 0 && worker < num_tiles) {
      int row, n_blk;
      locate(cur, worker, row, n_blk);
      ahead = min(stages, kb1 - kb0);
      int by, bz;
      b_rows_at(n_blk, by, bz);
      for (int i = 0; i < ahead; ++i) {
        if (elect_one()) load_b(i, kb0 + i, by, bz);
        __syncwarp();
      }
    }
    pdl_wait();
    for (int tile = worker; ok && tile < num_tiles; tile += workers) {
      int row, n_blk;
      locate(cur, tile, row, n_blk);
      int by, bz;
      b_rows_at(n_blk, by, bz);
      for (int kb = kb0; kb < kb1; ++kb) {
        ok = __all_sync(0xffffffffu, mbar_wait_abortable(&empty[stage], phase ^ 1u, abort_flag));
        if (!ok) break;
        unsigned char* sa = tiles + stage * stage_bytes;
        if (elect_one()) {
          if (ahead <= 0) load_b(stage, kb, by, bz);
          if (PAIR) tma_load_2d_pair(sa, &map_a, map_to_cta(smem_u32(&full[stage]), lead), kb * kBlockK, row);
          else tma_load_2d(sa, &map_a, &full[stage], kb * kBlockK, row);
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
    for (int i = 0; PAIR && ok && i < stages; ++i) {
      ok = __all_sync(0xffffffffu, mbar_wait_abortable(&empty[stage], phase ^ 1u, abort_flag));
      if (++stage == stages) {
        stage = 0;
        phase ^= 1u;
      }
    }
  } else if (warp == 1) {
    if (r == 0) {
      // ---------------------------------------------------------------- MMA issuer
      const uint32_t idesc = make_idesc_bf16(kRows, sub);
      const uint64_t desc0 = make_smem_desc(smem_u32(tiles));
      const uint32_t desc_hi = (uint32_t)(desc0 >> 32);
      int stage = 0;
      uint32_t phase = 0;
      int it = 0;
      for (int tile = worker; tile < num_tiles; tile += workers, ++it) {
        const int ab = a.accs > 1 ? it & 1 : 0;
        const uint32_t use = (uint32_t)(a.accs > 1 ? it >> 1 : it);
        bool ok = __all_sync(0xffffffffu, mbar_wait_abortable(&tmem_empty[ab], (use & 1u) ^ 1u, abort_flag));
        tc_fence_after_sync();
        const uint32_t d = tmem_base + (uint32_t)(ab * nsub * sub);
        for (int kb = kb0; ok && kb < kb1; ++kb) {
          ok = __all_sync(0xffffffffu, mbar_wait_abortable(&full[stage], phase, abort_flag));
          if (!ok) break;
          tc_fence_after_sync();
          const uint32_t la = (uint32_t)desc0 + (uint32_t)(stage * (stage_bytes >> 4));  // addresses in 16-byte units
          const uint32_t lb = la + (kTileABytes >> 4), lb2 = lb + (uint32_t)(b_bytes >> 4);
          const bool first = kb == kb0;
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < kBlockK / kUmmaK; ++k) {
              const uint64_t da = make_desc(desc_hi, la + 2 * k), db = make_desc(desc_hi, lb + 2 * k);
              if (PAIR) umma_bf16_pair(d, da, db, idesc, !first || k != 0);
              else umma_bf16(d, da, db, idesc, !first || k != 0);
              if (nsub > 1) {
                const uint64_t db2 = make_desc(desc_hi, lb2 + 2 * k);
                if (PAIR) umma_bf16_pair(d + (uint32_t)sub, da, db2, idesc, !first || k != 0);
                else umma_bf16(d + (uint32_t)sub, da, db2, idesc, !first || k != 0);
              }
            }
            if (PAIR) umma_commit_pair(&empty[stage], (uint16_t)(3u << lead));
            else umma_commit(&empty[stage]);
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
        if (elect_one()) {
          if (PAIR) umma_commit_pair(&tmem_full[ab], (uint16_t)(3u << lead));
          else umma_commit(&tmem_full[ab]);
        }
        __syncwarp();
      }
    }
  } else {
    // ---------------------------------------------- epilogue (this CTA's 128 rows)
    const int q = warp & 3, h = (warp - 2) >> 2;  // TMEM lane quarter; which of the two warps of it
    unsigned char* stg = epi_stage + (warp - 2) * (32 * kRowBytes);
    // Passes of kChunk output columns; the two warps of a quarter take them in turn.  RESIDUAL: an entry of sumsq_out
    // is the sum over a block of passes, to which both warps add theirs.
    const int per_sub = (sub_out + kChunk - 1) / kChunk;
    // SPLIT: the columns that range d finishes, in units of 16 (or of the 128 behind an entry of sumsq_out)
    const int unit = kRes && a.ss_cols > 0 ? a.ss_cols : 16, units = sub_out / unit;
    auto first_col = [&](int d) { return units * d / cl * unit; };
    const int own0 = SPLIT ? first_col(cs) : 0, own1 = SPLIT ? first_col(cs + 1) : 0;
    const int owner = SPLIT && own0 == own1 ? -1 : cs;
    const int passes = SPLIT ? (own1 - own0) / kChunk : nsub * per_sub;
    const int per_block = kRes && a.ss_cols > 0 ? a.ss_cols / kChunk : passes;
    // The two warps of a quarter that meet at a barrier below leave this loop together: a bounded wait that ran
    // out in one of them, or an abort that only one has seen, ends it for both.
    auto agree = [&](bool ok) {
      ok = __all_sync(0xffffffffu, ok);
      return kRes ? named_bar_all(1 + q, 64, ok) : ok;
    };
    TileCursor cur;
    start(cur);
    pdl_wait();
    int it = 0, blk = 0;
    for (int tile = worker; tile < num_tiles; tile += workers, ++it) {
      int row, n_blk;
      locate(cur, tile, row, n_blk);
      row += q * 32;
      const int row_end = cur.rows1;
      const int ab = a.accs > 1 ? it & 1 : 0;
      float scale = 1.f;
      if (a.scale_sumsq != nullptr) {
        float s = 0.f;
        const int rr = min(row + lane, a.M - 1);
#pragma unroll 8
        for (int p = 0; p < a.scale_parts; ++p) s += __ldcg(a.scale_sumsq + (size_t)p * a.M + rr);
        scale = rsqrtf(s * a.inv_width + a.eps);
      }
      // pass i: its accumulator, the columns in it, the first column of out
      auto sub_of = [&](int i) { return SPLIT || nsub == 1 || i < per_sub ? 0 : 1; };
      auto in_sub = [&](int i) { return SPLIT ? own0 + i * kChunk : (i - sub_of(i) * per_sub) * kChunk; };
      int f_row = 0, f_block = 0;
      if (strips) features(n_blk, 0, f_row, f_block);
      // strips: column of out of column `c` of accumulator s (eight columns, 16 bytes, never cross a strip)
      auto strip_col = [&](int s, int c) {
        const int in = c & ((1 << a.strip_shift) - 1);
        return (f_block + s * next_block + (c >> a.strip_shift)) * kPairRows + f_row + in;
      };
      auto out_col = [&](int i) {
        return strips ? strip_col(sub_of(i), in_sub(i)) : (n_blk * nsub + sub_of(i)) * sub_out + in_sub(i);
      };
      // RESIDUAL (the launcher wants whole, aligned rows of 16 columns here): the stream and the norm's weight
      // travel two passes ahead, the first ones while the product is finished: 16 columns take a warp less time than their
      // loads (one pass ahead: 1152 x 4096 in one round of tiles 36.4 us instead of 32).  A thread has kResRows rows of
      // eight columns.
      constexpr int kVecs = kChunk / 8, kResRows = kVecs;  // (32 rows x kVecs vectors over 32 lanes)
      struct Ahead {
        uint4 res[kResRows][2], nw;
      } next, after;
      auto load_residual = [&](int i, Ahead& to) {
        const int col = out_col(i) + lane % kVecs * 8;
        if (i >= passes || col >= a.n_out) return;
#pragma unroll
        for (int j = 0; j < kResRows; ++j) {
          const int rr = row + j * (32 / kVecs) + lane / kVecs;
          if (rr >= row_end) continue;
          const uint4* rp = reinterpret_cast<const uint4*>(a.residual + ((size_t)rr * a.ldo + col) * a.res_bytes);
          to.res[j][0] = rp[0];
          if (a.res_bytes == 4) to.res[j][1] = rp[1];
        }
        if (a.norm_w != nullptr) to.nw = __ldg(reinterpret_cast<const uint4*>(a.norm_w + col));
      };
      if (kRes && owner == cs) {
        load_residual(h, next);
        load_residual(h + 2, after);
      }
      const uint32_t use = (uint32_t)(a.accs > 1 ? it >> 1 : it);
      bool ok = !s_abort && mbar_wait_abortable(&tmem_full[ab], use & 1u, abort_flag);
      if (!ok && lane == 0) fail(GEMM_ERR_EPILOGUE_WAIT);
      if (!agree(ok)) break;
      tc_fence_after_sync();
      const uint32_t tacc = tmem_base + (uint32_t)(ab * nsub * sub) + ((uint32_t)(q * 32) << 16);
      // Cluster: the sums of the columns that another CTA finishes go there, as [sender][column / 4][128 rows] float4
      // in the ring of a CTA that has said that its MMAs are complete (a cluster works on one tile).  SILU: the gate
      // columns, then the up columns.
      constexpr int kKinds = kSilu ? 2 : 1;
      auto slot = [&](int from, int to) { return from - (from > to ? 1 : 0); };
      const float4* s_in = reinterpret_cast<const float4*>(tiles);
      const int own4 = (own1 - own0) / 4 * kKinds;  // float4 columns that every peer sends here
      if (SPLIT) {
        if (threadIdx.x == 64 && owner == cs) mbar_expect_tx(&s_recv, (uint32_t)(own4 * kBlockM * 16 * (cl - 1)));
        if (warp == 2 && lane < cl && lane != cs) mbar_arrive_cluster(map_to_cta(smem_u32(&s_peer_ready[cs]), cta_of(lane)));
        for (int i = 1; ok && i < cl; ++i) {
          const int d = cs + i < cl ? cs + i : cs + i - cl, d0 = first_col(d), w = first_col(d + 1) - d0;
          if (w == 0) continue;
          ok = mbar_wait_cluster(&s_peer_ready[d], 0u, abort_flag);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok && lane == 0) fail(GEMM_ERR_EPILOGUE_WAIT);
          if (!ok) continue;
          const uint32_t bar = map_to_cta(smem_u32(&s_recv), cta_of(d));
          const uint32_t remote = map_to_cta(smem_u32(tiles), cta_of(d)) +
                                  (uint32_t)((slot(cs, d) * (w / 4 * kKinds) * kBlockM + q * 32 + lane) * 16);
          const int n = w / 16 * kKinds;
#pragma unroll 1
          for (int k = h; k < n; k += 2) {
            const int c = k * 16;  // of the columns sent: gate, then up
            uint32_t x[16];
            tmem_ld_32x16(tacc + (c < w ? d0 + c : sub_out + d0 + c - w), x);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 4; ++j)
              st_async_v4(remote + (uint32_t)((k * 4 + j) * kBlockM * 16), bar, x[4 * j], x[4 * j + 1], x[4 * j + 2], x[4 * j + 3]);
          }
        }
        if (owner != cs) {  // nothing to finish here
          break;
        }
        ok = ok && mbar_wait_cluster(&s_recv, 0u, abort_flag);
        if (!ok && lane == 0) fail(GEMM_ERR_EPILOGUE_WAIT);
        if (!agree(ok)) break;
      }
      // accumulator columns of pass i of the finished tile (kind 1: up)
      auto load_acc = [&](int i, int kind, float (&v)[kChunk]) {
        const int in = in_sub(i), col = sub_of(i) * sub + kind * sub_out + in;
        uint32_t x[16];
        tmem_ld_32x16(tacc + col, x);
        tmem_ld_wait();
        if constexpr (SPLIT) {
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = 0.f;
#pragma unroll 1
          for (int p = 0; p < cl; ++p) {  // in K order, this CTA's own part in its place
            if (p == cs) {
#pragma unroll
              for (int j = 0; j < 16; ++j) v[j] += __uint_as_float(x[j]);
            } else {
              const float4* src = s_in + (slot(p, cs) * own4 + (kind * (own1 - own0) + in - own0) / 4) * kBlockM + q * 32 + lane;
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const float4 y = src[j * kBlockM];
                v[4 * j] += y.x;
                v[4 * j + 1] += y.y;
                v[4 * j + 2] += y.z;
                v[4 * j + 3] += y.w;
              }
            }
          }
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(x[j]);
          if constexpr (kChunk > 16) {
            if (in + 16 < sub_out) {  // (the columns of an accumulator may end in the middle of a pass)
              tmem_ld_32x16(tacc + col + 16, x);
              tmem_ld_wait();
            }
#pragma unroll
            for (int j = 0; j < 16; ++j) v[16 + j] = __uint_as_float(x[j]);
          }
        }
      };
#pragma unroll 1
      for (int b0 = 0; b0 < passes; b0 += per_block, ++blk) {
        float ss[kResRows] = {};
        const int b1 = min(b0 + per_block, passes);
#pragma unroll 1
        for (int i = b0 + h; i < b1; i += 2) {
          const int col0 = out_col(i);
          if (col0 >= a.n_out) continue;
          const Ahead now = next;
          next = after;
          if (kRes) load_residual(i + 4, after);
          float v[kChunk];
          load_acc(i, 0, v);
          if (kSilu) {
            float up[kChunk];
            load_acc(i, 1, up);
            if constexpr (kExact) {
              // The compiler's division branches for each quotient, and the zeros behind the last row take its slow side (8
              // layers and the head of a decode step, us, without an exact quotient / with a division: 65 rows 1031 / 1137, 128
              // 1197 / 1226, 192 1701 / 1804).  Gates in the ordinary range take silu_near (65 rows 1045 / 1052, 128 1192 / 1194,
              // 192 1710 / 1715); one outside it brings its warp's pass to the division.  (As a run-time branch this cost the
              // launches without it 0.5 to 1 %: gate/up of one expert 52.7 -> 53.2 us.)
              bool near = true;
#pragma unroll
              for (int j = 0; j < kChunk; ++j) near &= fabsf(v[j] * scale) <= kNearGate;
              if (__all_sync(0xffffffffu, near)) {
#pragma unroll
                for (int j = 0; j < kChunk; ++j) v[j] = silu_near(v[j] * scale) * (up[j] * scale);
              } else {
#pragma unroll 1
                for (int j = 0; j < kChunk; ++j) {
                  const float gv = v[0] * scale, uv = up[0] * scale;
#pragma unroll
                  for (int k = 0; k + 1 < kChunk; ++k) v[k] = v[k + 1], up[k] = up[k + 1];
                  v[kChunk - 1] = gv / (1.f + __expf(-gv)) * uv;
                }
              }
            } else {
#pragma unroll
              for (int j = 0; j < kChunk; ++j) {
                const float gv = v[j] * scale, uv = up[j] * scale;
                v[j] = __fdividef(gv, 1.f + __expf(-gv)) * uv;
              }
            }
          } else {
#pragma unroll
            for (int j = 0; j < kChunk; ++j) v[j] *= scale;
          }
          // staging rows: 16-byte pieces, exchanged so that eight lanes meet eight different bank groups
          constexpr int kPieces = kRowBytes / 16, kFlip = 8 / kPieces;
          auto piece = [&](int rr, int j) { return stg + rr * kRowBytes + ((j ^ ((rr / kFlip) & (kPieces - 1))) << 4); };
#pragma unroll
          for (int j = 0; j < kPieces; ++j) {
            uint4 o;
            if (kRes) {
              o = make_uint4(__float_as_uint(v[(4 * j) % kChunk]), __float_as_uint(v[(4 * j + 1) % kChunk]),
                             __float_as_uint(v[(4 * j + 2) % kChunk]), __float_as_uint(v[(4 * j + 3) % kChunk]));
            } else {
              uint32_t w[4];
#pragma unroll
              for (int k = 0; k < 4; ++k)
                w[k] = pack_bf16x2(__float_as_uint(v[(8 * j + 2 * k) % kChunk]), __float_as_uint(v[(8 * j + 2 * k + 1) % kChunk]));
              o = make_uint4(w[0], w[1], w[2], w[3]);
            }
            *reinterpret_cast<uint4*>(piece(lane, j)) = o;
          }
          __syncwarp();
          if (kRes) {
            const int col = col0 + lane % kVecs * 8;
            const uint32_t ww[4] = {now.nw.x, now.nw.y, now.nw.z, now.nw.w};
            const bool wide = a.res_bytes == 4;
#pragma unroll
            for (int j = 0; j < kResRows; ++j) {
              const int rr = j * (32 / kVecs) + lane / kVecs;
              const uint4 p0 = *reinterpret_cast<const uint4*>(piece(rr, lane % kVecs * 2));
              const uint4 p1 = *reinterpret_cast<const uint4*>(piece(rr, lane % kVecs * 2 + 1));
              if (row + rr >= row_end || col >= a.n_out) continue;
              const uint32_t pw[8] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w};
              const uint32_t rw[8] = {now.res[j][0].x, now.res[j][0].y, now.res[j][0].z, now.res[j][0].w,
                                      now.res[j][1].x, now.res[j][1].y, now.res[j][1].z, now.res[j][1].w};
              uint32_t z[8], zo[4], wo[4];
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                const float z0 = __uint_as_float(pw[2 * k]) + __uint_as_float(wide ? rw[2 * k] : rw[k] << 16);
                const float z1 = __uint_as_float(pw[2 * k + 1]) + __uint_as_float(wide ? rw[2 * k + 1] : rw[k] & 0xffff0000u);
                ss[j] += z0 * z0 + z1 * z1;
                z[2 * k] = __float_as_uint(z0);
                z[2 * k + 1] = __float_as_uint(z1);
                zo[k] = pack_bf16x2(z[2 * k], z[2 * k + 1]);
                wo[k] = pack_bf16x2(__float_as_uint(z0 * __uint_as_float(ww[k] << 16)),
                                    __float_as_uint(z1 * __uint_as_float(ww[k] & 0xffff0000u)));
              }
              const size_t off = (size_t)(row + rr) * a.ldo + col;
              uint4* rp = reinterpret_cast<uint4*>(a.residual + off * a.res_bytes);
              const uint4 zb = make_uint4(zo[0], zo[1], zo[2], zo[3]);
              if (wide) {
                rp[0] = make_uint4(z[0], z[1], z[2], z[3]);
                rp[1] = make_uint4(z[4], z[5], z[6], z[7]);
                if (a.stream_out != nullptr) *reinterpret_cast<uint4*>(a.stream_out + off) = zb;
              } else {
                rp[0] = zb;
              }
              if (a.norm_w != nullptr) *reinterpret_cast<uint4*>(a.out + off) = make_uint4(wo[0], wo[1], wo[2], wo[3]);
            }
          } else {
            constexpr int kPer = 32 / kPieces;  // rows of a store instruction
            // column of out of this lane's eight columns, and where they end (beyond the accumulator: nowhere)
            const int pc = lane % kPieces, in = in_sub(i) + pc * 8;
            const int col = strips ? strip_col(sub_of(i), in) : col0 + pc * 8;
            const int col_end = strips ? (in < sub_out ? a.n_out : 0) : min(a.n_out, col0 - in_sub(i) + sub_out);
#pragma unroll
            for (int j = 0; j < kPieces; ++j) {
              const int rr = j * kPer + lane / kPieces;
              const uint4 p = *reinterpret_cast<const uint4*>(piece(rr, pc));
              store16_local(a.out, a.ldo, row + rr, col, p, row_end, col_end);
            }
          }
          __syncwarp();
        }
        if (kRes && a.norm_w != nullptr) {
          if (h == 0) named_bar_sync(1 + q, 64);
#pragma unroll
          for (int j = 0; j < kResRows; ++j) {
            float s = ss[j];
#pragma unroll
            for (int o = kVecs / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            const int rr = j * (32 / kVecs) + lane / kVecs;
            float* other = &s_half[blk & 1][q * 32 + rr];
            if (h == 1) {
              if (lane % kVecs == 0) *other = s;
            } else if (lane % kVecs == 0 && row + rr < row_end) {
              const int part = a.ss_cols > 0 ? (n_blk * nsub * sub_out + own0) / a.ss_cols + b0 / per_block : n_blk * cl + cs;
              if (a.ss_cols == 0 || part * a.ss_cols < a.n_out) a.sumsq_out[(size_t)part * a.M + row + rr] = s + *other;
            }
          }
          if (h == 1) named_bar_sync(1 + q, 64);
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
  if (PAIR || SPLIT) cluster_sync_all();
  else __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    if (PAIR) tmem_dealloc_pair(tmem_base, (uint32_t)a.tmem_cols);
    else tmem_dealloc(tmem_base, (uint32_t)a.tmem_cols);
  }
}

template <bool PAIR, int EPI, bool SPLIT, int NSUB>
__global__ void __launch_bounds__(kTileThreads, 1)
gemm_tile_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const TileArgs a,
                 uint32_t* error_word) {
  gemm_tile_body<PAIR, EPI, SPLIT, NSUB>(map_a, map_b, a, error_word);
}

}  // namespace sm100
}  // namespace penny
