// Streamed GEMM on sm_100a for few rows of activations:
//     out[r, n] = sum_k x[r, k] W[n, k]      bf16, fp32 accumulation, up to 256 rows
// The time is one read of W, so everything is arranged around keeping that read
// going at the rate of the memory:
//
//   * Flat split.  The K steps of all weight tiles form one line and every CTA
//     pair takes an equal contiguous piece (stream_gemm_plan.h).  Measured on B200
//     with the loads alone, 1 GB of weights: 6.7 TB/s from contiguous pieces, 5.1
//     TB/s when the CTAs step through the tiles side by side, 4.4 TB/s with their
//     starting points staggered; six 16 KB stages per SM are enough (13 are
//     slower).
//   * CTA pairs (cta_group::2): M = 256 weight rows, N = the rows of x.  A CTA
//     loads its own 128 weight rows and HALF of the x rows, so the x traffic from
//     L2 is half of what single CTAs need, without multicast.
//   * A tile that several pairs work on is summed from fp32 partials in the
//     caller's workspace (L2): every pair parks its part and counts itself in, the
//     last one adds the parts in pair order (so the sum does not depend on who was
//     last) and runs the epilogue.  Nobody waits for anybody: pairs need not be
//     resident together.
//   * Programmatic dependent launch: barriers, TMEM and the first ring of weights
//     are set up before the wait for the predecessor; with at most 128 rows the
//     ring leaves half of the shared memory to the next kernel of the step, which
//     does the same under this one's tail.
//   * Epilogues that would be kernels of their own: silu(gate) * up; residual add
//     with the next RMSNorm's weight and sums of squares, whose 1 / rms the
//     consumer applies to its accumulator (a row scale commutes with the product).
//   * Groups: the rows of x fall into groups with a weight each (the experts of a
//     MoE layer); their ranges are read on the device and empty groups cost nothing.
//
// 320 threads: warp 0 TMA, warp 1 MMA (leader CTA), warps 2-9 epilogue, two per
// TMEM lane quarter, each with half of the columns.  Every wait is bounded.
#include "gemm_stream_sm100.h"

#include <cuda.h>

#include <algorithm>

#include "gemm_kernel_sm100.cuh"
#include "gemm_sm100.h"
#include "kernel_setup.h"
#include "pdl.h"

namespace penny {
namespace sm100 {

namespace {

constexpr int kStThreads = 320;
constexpr int kStMaxStages = 8;
constexpr int kStMaxCluster = 4;  // pairs
constexpr int kStWBytes = kBlockM * kBlockK * 2;  // this CTA's 128 weight rows of one K step
constexpr int kStChunk = 16;                      // columns per epilogue pass and half
constexpr int kStEpiBytes = 2 * kStChunk * kBlockM * 4;

struct StreamArgs {
  __nv_bfloat16* out;
  int ldo, rows, n_out;  // n_out: columns of out
  int num_kb, tiles, groups, w_rows;
  int half_rows, y_step, up_offset;  // weight rows of CTA block b: b * y_step .. +64 and up_offset further .. +64
  int bt;                            // columns reserved per accumulator (rows rounded up to 32)
  int xbox;                          // rows of one x load
  int stages;
  int own_recv;                      // cluster: the peers' sums have an area behind the staging rows
  int cl;                            // pairs per cluster; above 1 a cluster splits the K steps of one tile
  const int* ranges;
  int range_stride;
  const float* scale_sumsq;
  int scale_parts;
  float inv_width, eps;
  __nv_bfloat16* residual;
  const __nv_bfloat16* norm_w;
  float* sumsq_out;
  unsigned* counters;
  float* parts;
};

__device__ __forceinline__ void tmem_ld_32x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
// Weight tile load of a CTA of the pair; the weights are read once, so their lines
// leave L2 first (the partials and activations stay).
__device__ __forceinline__ void tma_load_2d_pair_once(void* smem_dst, const CUtensorMap* m, uint32_t bar_cluster_addr,
                                                      int x, int y, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint "
      "[%0], [%1, {%3, %4}], [%2], %5;" ::"r"(smem_u32(smem_dst)),
      "l"(m), "r"(bar_cluster_addr), "r"(x), "r"(y), "l"(policy)
      : "memory");
}
__device__ __forceinline__ float bf16_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }
__device__ __forceinline__ uint4 pack8(const float (&v)[8]) {
  uint4 o;
  o.x = pack_bf16x2(__float_as_uint(v[0]), __float_as_uint(v[1]));
  o.y = pack_bf16x2(__float_as_uint(v[2]), __float_as_uint(v[3]));
  o.z = pack_bf16x2(__float_as_uint(v[4]), __float_as_uint(v[5]));
  o.w = pack_bf16x2(__float_as_uint(v[6]), __float_as_uint(v[7]));
  return o;
}

template <int EPI>
__global__ void __launch_bounds__(kStThreads, 2)
gemm_stream_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                   const StreamArgs a, uint32_t* error_word) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ float s_scale[kStreamMaxRows];
  __shared__ short s_group[kStreamMaxGroups];
  __shared__ uint64_t s_bars[2 * kStMaxStages + 4];
  __shared__ uint64_t s_peer_ready[kStMaxCluster], s_recv;
  __shared__ uint32_t s_tmem;
  __shared__ int s_active;
  __shared__ volatile int s_abort;
  __shared__ volatile int s_last[2];
  unsigned char* tiles = align_tiles(smem_raw);
  const int stages = a.stages;
  const int stage_bytes = kStWBytes + a.bt / 2 * (kBlockK * 2);
  float* s_epi = reinterpret_cast<float*>(tiles + (size_t)stages * stage_bytes);
  uint64_t* full = s_bars;                      // used in the leader only
  uint64_t* empty = s_bars + kStMaxStages;      // one in each CTA
  uint64_t* tmem_full = s_bars + 2 * kStMaxStages;
  uint64_t* tmem_empty = tmem_full + 2;         // used in the leader only
  volatile int* abort_flag = &s_abort;

  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t crank = cluster_ctarank(), r = crank & 1u, lead = crank & ~1u;
  const int cs = (int)crank >> 1, cl = a.cl;  // this pair's K range in a cluster that shares a tile
  const int pair = (int)blockIdx.x >> 1, npairs = (int)gridDim.x >> 1;
  const int tmem_cols = a.bt <= 16 ? 32 : (a.bt <= 32 ? 64 : (a.bt <= 64 ? 128 : (a.bt <= 128 ? 256 : 512)));
  const int acc_cols = tmem_cols / 2;
  if (threadIdx.x == 0) {
    for (int i = 0; i < stages; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tmem_full[i], 1);
      mbar_init(&tmem_empty[i], 16);  // eight epilogue warps in each CTA
    }
    for (int i = 0; i < kStMaxCluster; ++i) mbar_init(&s_peer_ready[i], 1);
    mbar_init(&s_recv, 1);
    s_abort = 0;
    s_active = 1;
    s_group[0] = 0;
    mbar_fence_init();
    tma_prefetch_desc(&map_w);
    tma_prefetch_desc(&map_x);
  }
  __syncwarp();
  if (warp == 1) tmem_alloc_pair(&s_tmem, (uint32_t)tmem_cols);
  if (a.groups > 0) {
    // the row ranges come from the kernel before this one
    pdl_wait();
    if (warp == 0) {
      int n = 0;
      for (int g0 = 0; g0 < a.groups; g0 += 32) {
        const int g = g0 + lane;
        const bool live = g < a.groups && a.ranges[a.range_stride * g + 1] > a.ranges[a.range_stride * g];
        const unsigned m = __ballot_sync(0xffffffffu, live);
        if (live) s_group[n + __popc(m & ((1u << lane) - 1u))] = (short)g;
        n += __popc(m);
      }
      if (lane == 0) s_active = n;
    }
  }
  tc_fence_before_sync();
  __syncwarp();
  cluster_sync_all();
  tc_fence_after_sync();
  const uint32_t tmem_base = s_tmem;
  const int units = s_active * a.tiles * a.num_kb;
  // (a launch is sized for all groups being live; the pairs a smaller line does not need have no units)
  const int pairs = a.groups > 0 ? stream_pairs(units, npairs) : npairs;
  int u0 = pair < pairs ? stream_begin(units, pairs, pair) : 0;
  int u1 = pair < pairs ? stream_begin(units, pairs, pair + 1) : 0;
  if (cl > 1) {
    u0 = pair / cl * a.num_kb + stream_begin(a.num_kb, cl, cs);
    u1 = pair / cl * a.num_kb + stream_begin(a.num_kb, cl, cs + 1);
  }

  auto fail = [&](uint32_t code) {
    s_abort = 1;
    for (uint32_t c = 0; c < 2u * (uint32_t)cl; ++c)
      if (c != crank) st_cluster_u32(map_to_cta(smem_u32(const_cast<int*>(&s_abort)), c), 1u);
    atomicCAS(error_word, 0u, code);
  };
  // rows of group slot `gs`: first row of x, count
  auto group_rows = [&](int gs, int& row0, int& n) {
    if (a.groups == 0) {
      row0 = 0;
      n = a.rows;
    } else {
      const int g = s_group[gs];
      row0 = a.ranges[a.range_stride * g];
      n = min(a.rows, a.ranges[a.range_stride * g + 1] - row0);
    }
  };

  if (warp == 0) {
    if (lane == 0) {
      // ---------------------------------------------- TMA producer (in each CTA)
      uint64_t policy;
      asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
      const uint32_t full0 = map_to_cta(smem_u32(&full[0]), lead);
      auto load_w = [&](int stage, int gs, int t, int kb) {
        unsigned char* sw = tiles + (size_t)stage * stage_bytes;
        const uint32_t bar = full0 + (uint32_t)stage * 8u;
        const int y = s_group[gs] * a.w_rows + (2 * t + (int)r) * a.y_step;
        tma_load_2d_pair_once(sw, &map_w, bar, kb * kBlockK, y, policy);
        if (a.up_offset != kBlockM / 2)  // gate and up rows are not neighbours: boxes of 64 rows
          tma_load_2d_pair_once(sw + kStWBytes / 2, &map_w, bar, kb * kBlockK, y + a.up_offset, policy);
      };
      auto load_x = [&](int stage, int row0, int n_half, int kb) {
        unsigned char* sx = tiles + (size_t)stage * stage_bytes + kStWBytes;
        const uint32_t bar = full0 + (uint32_t)stage * 8u;
        for (int i = 0; i < n_half; i += a.xbox)
          tma_load_2d_pair(sx + i * (kBlockK * 2), &map_x, bar, kb * kBlockK, row0 + (int)r * n_half + i);
      };
      const int pre = a.groups == 0 ? min(stages, u1 - u0) : 0;
      // one group: the first ring of weights does not depend on the predecessor
      int tile = u0 / a.num_kb, kb = u0 - tile * a.num_kb;
      for (int i = 0; i < pre; ++i) {
        if (r == 0) mbar_expect_tx(&full[i], 2u * kStWBytes + (uint32_t)a.bt * (kBlockK * 2));
        load_w(i, 0, tile, kb);
        if (++kb == a.num_kb) {
          kb = 0;
          ++tile;
        }
      }
      pdl_wait();
      for (int i = 0; i < pre; ++i) load_x(i, 0, a.bt / 2, (u0 + i) % a.num_kb);
      int stage = pre == stages ? 0 : pre;
      uint32_t phase = pre == stages ? 1u : 0u;
      bool ok = true;
      int gs = -1, t = 0, row0 = 0, n = 0, n_half = 0;
      for (int u = u0 + pre; u < u1; ++u) {
        if (gs < 0 || kb == 0) {  // another tile
          gs = tile / a.tiles;
          t = tile - gs * a.tiles;
          group_rows(gs, row0, n);
          n_half = stream_round_rows(n) / 2;
        }
        if (!mbar_wait_abortable(&empty[stage], phase ^ 1u, abort_flag)) {
          ok = false;
          break;
        }
        if (r == 0) mbar_expect_tx(&full[stage], 2u * kStWBytes + 2u * (uint32_t)n_half * (kBlockK * 2));
        load_w(stage, gs, t, kb);
        load_x(stage, row0, n_half, kb);
        if (++stage == stages) {
          stage = 0;
          phase ^= 1u;
        }
        if (++kb == a.num_kb) {
          kb = 0;
          ++tile;
        }
      }
      if (!ok) fail(GEMM_ERR_PRODUCER_WAIT);
      // every commit aimed at this CTA's slot barriers has arrived before it may leave
      for (int i = 0; ok && i < stages && !s_abort; ++i) {
        if (!mbar_wait_abortable(&empty[stage], phase ^ 1u, abort_flag)) break;
        if (++stage == stages) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && r == 0) {
      // ------------------------------------------- MMA issuer (leader CTA only)
      int stage = 0;
      uint32_t phase = 0;
      int it = 0;
      for (int u = u0; u < u1 && !s_abort; ++it) {
        const int tile = u / a.num_kb;
        const int end = min(u1, (tile + 1) * a.num_kb);
        int row0, n;
        group_rows(tile / a.tiles, row0, n);
        const uint32_t idesc = make_idesc_bf16(2 * kBlockM, stream_round_rows(n));
        const int ab = it & 1;
        bool ok = mbar_wait_abortable(&tmem_empty[ab], (((uint32_t)it >> 1) & 1u) ^ 1u, abort_flag);
        tc_fence_after_sync();
        const uint32_t d = tmem_base + (uint32_t)(ab * acc_cols);
        for (bool first = true; ok && u < end; ++u, first = false) {
          if (!mbar_wait_abortable(&full[stage], phase, abort_flag)) {
            ok = false;
            break;
          }
          tc_fence_after_sync();
          const uint32_t sw = smem_u32(tiles + (size_t)stage * stage_bytes);
          const uint64_t dw = make_smem_desc(sw), dx = make_smem_desc(sw + kStWBytes);
#pragma unroll
          for (int k = 0; k < kBlockK / kUmmaK; ++k)
            umma_bf16_pair(d, advance_desc_k(dw, k), advance_desc_k(dx, k), idesc, !first || k != 0);
          umma_commit_pair(&empty[stage], (uint16_t)(3u << lead));
          if (++stage == stages) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (!ok) {
          fail(GEMM_ERR_MMA_WAIT);
          break;
        }
        umma_commit_pair(&tmem_full[ab], (uint16_t)(3u << lead));
      }
    }
  } else {
    // ------------------------------- epilogue (own 128 weight rows, in each CTA)
    const int q = warp & 3, h = (warp - 2) >> 2;
    const int tid = (int)threadIdx.x - 64 - h * 128;  // thread of this column half
    const int row = q * 32 + lane;                    // weight row inside the CTA's block
    float* stg = s_epi + h * (kStChunk * kBlockM);    // [16 columns][128 rows]
    pdl_wait();  // stores and the partials' slots: after everything the predecessor did
    if (a.scale_sumsq != nullptr) {
      for (int t = (int)threadIdx.x - 64; t < a.rows; t += 256) {
        float s = 0.f;
#pragma unroll 8
        for (int p = 0; p < a.scale_parts; ++p) s += __ldcg(a.scale_sumsq + (size_t)p * a.rows + t);
        s_scale[t] = rsqrtf(s * a.inv_width + a.eps);
      }
      named_bar_sync(3, 256);
    }
    int it = 0;
    for (int u = u0; u < u1; ++it) {
      const int tile = u / a.num_kb;
      const int gs = tile / a.tiles, t = tile - gs * a.tiles;
      u = min(u1, (tile + 1) * a.num_kb);
      int row0, n;
      group_rows(gs, row0, n);
      const int ncol = stream_round_rows(n) / 2, col0 = h * ncol;  // this half's columns
      const int p0 = cl > 1 ? 0 : stream_pair_of(units, pairs, tile * a.num_kb);
      const int p1 = cl > 1 ? 0 : stream_pair_of(units, pairs, (tile + 1) * a.num_kb - 1);
      const int ab = it & 1;
      const bool ok = !s_abort && mbar_wait_abortable(&tmem_full[ab], ((uint32_t)it >> 1) & 1u, abort_flag);
      if (!ok && lane == 0) fail(GEMM_ERR_EPILOGUE_WAIT);
      if (!named_bar_all(1 + h, 128, ok)) break;
      tc_fence_after_sync();
      const uint32_t trow = tmem_base + (uint32_t)(ab * acc_cols) + ((uint32_t)(q * 32) << 16);
      const uint32_t tacc = trow + (uint32_t)col0;
      // Cluster: CTA cs finishes the 16-column blocks [cs * per, + per) of its 128 rows.  Its peers put their
      // sums, [peer][4 per][128 rows] float4, into an area of their own or, when that would cost the ring
      // too much, into the ring of a CTA that has said that its MMAs are complete.
      const int blocks = ncol / (kStChunk / 2), per = (blocks + cl - 1) / cl;
      float* s_in = reinterpret_cast<float*>(a.own_recv ? tiles + (size_t)stages * stage_bytes + kStEpiBytes : tiles);
      if (cl > 1) {
        if (threadIdx.x == 64)
          mbar_expect_tx(&s_recv, (uint32_t)(max(0, min(per, blocks - cs * per)) * (cl - 1) * kStChunk * kBlockM * 4));
        if (!a.own_recv && warp == 2 && lane < cl && lane != cs)
          mbar_arrive_cluster(map_to_cta(smem_u32(&s_peer_ready[cs]), 2u * (uint32_t)lane + r));
        for (int d = 1; d < cl; ++d) {
          const int dst = (cs + d) % cl;  // everybody starts with another peer
          if (!a.own_recv && !mbar_wait_cluster(&s_peer_ready[dst], 0u, abort_flag)) fail(GEMM_ERR_EPILOGUE_WAIT);
          const uint32_t remote = map_to_cta(smem_u32(s_in), 2u * (uint32_t)dst + r) +
                                  (uint32_t)((cs - (cs > dst ? 1 : 0)) * per * kStChunk * kBlockM * 4 + row * 16);
          const uint32_t bar = map_to_cta(smem_u32(&s_recv), 2u * (uint32_t)dst + r);
          for (int b = h; b < per && dst * per + b < blocks; b += 2) {
            uint32_t v[16];
            tmem_ld_32x16(trow + (uint32_t)((dst * per + b) * kStChunk), v);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 4; ++j)
              st_async_v4(remote + (uint32_t)((b * 4 + j) * kBlockM * 16), bar, v[4 * j], v[4 * j + 1], v[4 * j + 2],
                          v[4 * j + 3]);
          }
        }
        const bool got = mbar_wait_cluster(&s_recv, 0u, abort_flag);
        if (!got) fail(GEMM_ERR_EPILOGUE_WAIT);
        if (!named_bar_all(1 + h, 128, got)) break;
      }
      // partial of pair p for this tile, this CTA's rows: [columns / 4][128 rows] float4
      auto part = [&](int p) {
        const size_t slot = (size_t)stream_slot(units, pairs, p, a.num_kb, tile) * 2 + r;
        return reinterpret_cast<float4*>(a.parts + slot * ((size_t)a.bt * kBlockM)) + (size_t)(col0 / 4) * kBlockM + row;
      };
      bool last = true;
      if (p0 != p1) {
        // where the other pairs have all been here already (a tile that ends one pair's range and began
        // another's) nobody needs this part: no write, no fence
        if (tid == 0) {
          unsigned* cnt = a.counters + (tile * 4 + (int)r * 2 + h);
          const int only_me = (int)*reinterpret_cast<volatile unsigned*>(cnt) == p1 - p0;
          if (only_me) *cnt = 0u;
          s_last[h] = only_me;
        }
        named_bar_sync(1 + h, 128);
        last = s_last[h] != 0;
        if (last) __threadfence();
      }
      if (!last) {
        named_bar_sync(1 + h, 128);  // s_last has been read
        float4* dst = part(pair);
#pragma unroll 1
        for (int c = 0; c < ncol; c += kStChunk) {
          uint32_t v[16];
          tmem_ld_32x16(tacc + c, v);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 4; ++j)
            dst[(size_t)(c / 4 + j) * kBlockM] = make_float4(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]),
                                                             __uint_as_float(v[4 * j + 2]), __uint_as_float(v[4 * j + 3]));
        }
        __threadfence();
        named_bar_sync(1 + h, 128);
        if (tid == 0) {
          unsigned* cnt = a.counters + (tile * 4 + (int)r * 2 + h);
          const int mine = (int)atomicAdd(cnt, 1u) == p1 - p0;
          if (mine) *cnt = 0u;  // every part has arrived: ready for the next launch
          s_last[h] = mine;
        }
        named_bar_sync(1 + h, 128);
        last = s_last[h] != 0;
        if (last) __threadfence();
      }
      if (last) {
        const int blk = 2 * t + (int)r;
        // 16-column blocks of this half: every one of its columns, or every other one of the cluster share
        const int b_end = cl > 1 ? min(per, blocks - cs * per) : ncol / kStChunk;
#pragma unroll 1
        for (int b = cl > 1 ? h : 0; b < b_end; b += cl > 1 ? 2 : 1) {
          const int c = cl > 1 ? (cs * per + b) * kStChunk - col0 : b * kStChunk;  // columns from col0
          float v[16];
          {
            uint32_t own[16];
            tmem_ld_32x16(tacc + c, own);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(own[j]);
          }
          if (cl > 1) {
            // peers in K order, this CTA's own part in its place
            float own[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              own[j] = v[j];
              v[j] = 0.f;
            }
            for (int p = 0; p < cl; ++p) {
              if (p == cs) {
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] += own[j];
              } else {
                const float4* src =
                    reinterpret_cast<const float4*>(s_in) + ((p - (p > cs ? 1 : 0)) * per + b) * (4 * kBlockM) + row;
                float4 x[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) x[j] = src[j * kBlockM];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  v[4 * j] += x[j].x;
                  v[4 * j + 1] += x[j].y;
                  v[4 * j + 2] += x[j].z;
                  v[4 * j + 3] += x[j].w;
                }
              }
            }
          }
          if (p0 != p1) {
            // parts in pair order, two in flight at a time
            float4 own[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              own[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
              v[4 * j] = v[4 * j + 1] = v[4 * j + 2] = v[4 * j + 3] = 0.f;
            }
            for (int p = p0; p <= p1; p += 2) {
              float4 b[2][4];
#pragma unroll
              for (int i = 0; i < 2; ++i) {
                if (p + i <= p1 && p + i != pair) {
                  const float4* src = part(p + i) + (size_t)(c / 4) * kBlockM;
#pragma unroll
                  for (int j = 0; j < 4; ++j) b[i][j] = __ldcg(src + (size_t)j * kBlockM);
                }
              }
#pragma unroll
              for (int i = 0; i < 2; ++i) {
                if (p + i <= p1) {
#pragma unroll
                  for (int j = 0; j < 4; ++j) {
                    const float4 x = p + i == pair ? own[j] : b[i][j];
                    v[4 * j] += x.x;
                    v[4 * j + 1] += x.y;
                    v[4 * j + 2] += x.z;
                    v[4 * j + 3] += x.w;
                  }
                }
              }
            }
          }
#pragma unroll
          for (int j = 0; j < 16; ++j) stg[j * kBlockM + row] = v[j];
          named_bar_sync(1 + h, 128);
          // eight consecutive output columns of one row of x per item
          constexpr int kGroups = EPI == STREAM_EPI_SILU ? 8 : 16;
#pragma unroll
          for (int i = 0; i < kStChunk * kGroups / 128; ++i) {
            const int idx = tid + i * 128;
            const int j = idx / kGroups, g = idx % kGroups;
            const int xr = col0 + c + j;  // row of x inside the group
            const bool live = xr < n;
            const float4* s4 = reinterpret_cast<const float4*>(stg + j * kBlockM + g * 8);
            float o[8];
            {
              const float4 y0 = s4[0], y1 = s4[1];
              o[0] = y0.x; o[1] = y0.y; o[2] = y0.z; o[3] = y0.w;
              o[4] = y1.x; o[5] = y1.y; o[6] = y1.z; o[7] = y1.w;
            }
            if (a.scale_sumsq != nullptr) {
              const float s = live ? s_scale[xr] : 0.f;
#pragma unroll
              for (int k = 0; k < 8; ++k) o[k] *= s;
            }
            if (EPI == STREAM_EPI_SILU) {
              const float4 y0 = s4[16], y1 = s4[17];  // the up rows, 64 further
              float up[8] = {y0.x, y0.y, y0.z, y0.w, y1.x, y1.y, y1.z, y1.w};
              const float s = a.scale_sumsq != nullptr && live ? s_scale[xr] : 1.f;
#pragma unroll
              for (int k = 0; k < 8; ++k) o[k] = o[k] / (1.f + __expf(-o[k])) * (up[k] * s);
            }
            const int col = blk * (kGroups * 8) + g * 8;
            const size_t off = (size_t)(row0 + xr) * a.ldo + col;
            if (EPI == STREAM_EPI_RESIDUAL) {
              float ss = 0.f;
              if (live && col < a.n_out) {
                const uint4 res = *reinterpret_cast<const uint4*>(a.residual + off);
                const uint4 nw = a.norm_w != nullptr ? __ldg(reinterpret_cast<const uint4*>(a.norm_w + col)) : uint4{};
                const uint32_t rw[4] = {res.x, res.y, res.z, res.w}, ww[4] = {nw.x, nw.y, nw.z, nw.w};
                float zw[8];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                  o[2 * k] += bf16_lo(rw[k]);
                  o[2 * k + 1] += bf16_hi(rw[k]);
                  ss += o[2 * k] * o[2 * k] + o[2 * k + 1] * o[2 * k + 1];
                  zw[2 * k] = o[2 * k] * bf16_lo(ww[k]);
                  zw[2 * k + 1] = o[2 * k + 1] * bf16_hi(ww[k]);
                }
                *reinterpret_cast<uint4*>(a.residual + off) = pack8(o);
                if (a.norm_w != nullptr) *reinterpret_cast<uint4*>(a.out + off) = pack8(zw);
              }
              // the 16 lanes of a row of x
#pragma unroll
              for (int d = 8; d > 0; d >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, d);
              if (g == 0 && live && a.norm_w != nullptr) a.sumsq_out[(size_t)blk * a.rows + xr] = ss;
            } else if (live) {
              __nv_bfloat16* dst = a.out + off;
              if (col + 8 <= a.n_out && (reinterpret_cast<uintptr_t>(dst) & 15u) == 0) {
                *reinterpret_cast<uint4*>(dst) = pack8(o);
              } else {
#pragma unroll
                for (int k = 0; k < 8; ++k)
                  if (col + k < a.n_out) dst[k] = __float2bfloat16_rn(o[k]);
              }
            }
          }
          named_bar_sync(1 + h, 128);
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(map_to_cta(smem_u32(&tmem_empty[ab]), lead));
    }
  }
  // ------------------------------------------------------------------- teardown
  tc_fence_before_sync();
  __syncwarp();
  pdl_wait();  // no thread leaves before the predecessor has finished
  cluster_sync_all();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc_pair(tmem_base, (uint32_t)tmem_cols);
  }
}

template <int EPI>
cudaError_t launch_epi(const CUtensorMap& mw, const CUtensorMap& mx, const StreamArgs& a, int grid, size_t smem, bool pdl,
                       uint32_t* error_word, cudaStream_t stream) {
  const cudaError_t rc = kernel_setup(reinterpret_cast<const void*>(gemm_stream_kernel<EPI>), 220 << 10).rc;
  if (rc != cudaSuccess) return rc;
  return launch_kernel_ex(gemm_stream_kernel<EPI>, dim3((unsigned)grid), dim3(kStThreads), smem, stream, pdl, 2 * a.cl, mw, mx, a,
                          error_word);
}

}  // namespace

int stream_max_pairs() {
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  (void)cudaGetLastError();
  return std::max(1, sms / 2);
}

cudaError_t launch_gemm_stream(const StreamGemm& g, uint32_t* error_word, cudaStream_t stream) {
  if (g.rows < 1 || g.rows > kStreamMaxRows || g.w_rows < 1 || g.K < 1 || g.K % 8 != 0 || g.ldx % 8 != 0 ||
      g.ldw % 8 != 0 || g.groups < 0 || g.groups > kStreamMaxGroups)
    return cudaErrorInvalidValue;
  const bool silu = g.epi == STREAM_EPI_SILU;
  if (silu && (g.w_rows % 128 != 0 || (g.up_offset != 64 && g.up_offset != g.w_rows / 2))) return cudaErrorInvalidValue;
  const int groups = std::max(1, g.groups);
  StreamArgs a = {};
  a.out = reinterpret_cast<__nv_bfloat16*>(g.out);
  a.ldo = g.ldo;
  a.rows = g.rows;
  a.n_out = silu ? g.w_rows / 2 : g.w_rows;
  a.num_kb = (g.K + kBlockK - 1) / kBlockK;
  a.tiles = (g.w_rows + 2 * kBlockM - 1) / (2 * kBlockM);
  a.groups = g.groups;
  a.w_rows = g.w_rows;
  a.y_step = silu && g.up_offset != 64 ? kBlockM / 2 : kBlockM;
  a.up_offset = silu ? g.up_offset : kBlockM / 2;
  a.bt = stream_round_rows(g.rows);
  a.xbox = g.groups > 0 ? 16 : a.bt / 2;
  a.ranges = g.ranges;
  a.range_stride = g.range_stride;
  a.scale_sumsq = g.scale_sumsq;
  a.scale_parts = g.scale_parts;
  a.inv_width = g.scale_width > 0 ? 1.f / (float)g.scale_width : 0.f;
  a.eps = g.eps;
  a.residual = reinterpret_cast<__nv_bfloat16*>(g.residual);
  a.norm_w = reinterpret_cast<const __nv_bfloat16*>(g.norm_w);
  a.sumsq_out = g.sumsq_out;
  if ((long long)groups * a.tiles * 4 > kStreamCounters) return cudaErrorInvalidValue;
  if (g.epi == STREAM_EPI_RESIDUAL &&
      (g.groups > 0 || g.w_rows % 128 != 0 || g.ldo % 8 != 0 || g.residual == nullptr ||
       (g.norm_w != nullptr && g.sumsq_out == nullptr) ||
       ((reinterpret_cast<uintptr_t>(g.out) | reinterpret_cast<uintptr_t>(g.residual) | reinterpret_cast<uintptr_t>(g.norm_w)) & 15u) != 0))
    return cudaErrorInvalidValue;
  if (g.groups > 0 && (g.ranges == nullptr || g.scale_sumsq != nullptr)) return cudaErrorInvalidValue;
  const int max_pairs = stream_max_pairs();
  const long long units = (long long)groups * a.tiles * a.num_kb;
  if (units * max_pairs > 0x7fffffffll) return cudaErrorInvalidValue;
  const int pairs = stream_pairs((int)units, max_pairs);
  if (g.workspace == nullptr || (reinterpret_cast<uintptr_t>(g.workspace) & 15u) != 0 ||
      g.workspace_bytes < stream_workspace_bytes(g.rows, pairs))
    return cudaErrorInvalidValue;
  // Ring: up to 128 rows it stays within half of the shared memory, so that the next kernel of a chain
  // sets up and fills its own ring beside this one; above that one kernel has the SM.
  const int stage_bytes = kStWBytes + a.bt / 2 * (kBlockK * 2);
  const size_t budget = (size_t)(g.smem_kb > 0 ? std::min(g.smem_kb, 216) : (a.bt <= 128 ? 108 : 200)) << 10;
  // Without an area of its own the ring has to hold what the peers of a cluster send.
  auto plan_ring = [&](int cl) {
    const int peer_bytes = (cl - 1) * ((a.bt / kStChunk + cl - 1) / cl) * kStChunk * kBlockM * 4;
    a.own_recv = peer_bytes <= 24 << 10;
    const size_t fixed = kStEpiBytes + 1024 + (a.own_recv ? peer_bytes : 0);
    a.stages = 2;
    while (!a.own_recv && a.stages * stage_bytes < peer_bytes) ++a.stages;
    while (a.stages < kStMaxStages && fixed + (size_t)(a.stages + 1) * stage_bytes <= budget) ++a.stages;
    return fixed + (size_t)a.stages * stage_bytes;
  };
  a.cl = g.cluster;
  if (g.cluster == 0) {
    int held[kStMaxCluster + 1] = {};
    const void* fn = reinterpret_cast<const void*>(gemm_stream_kernel<STREAM_EPI_PLAIN>);
    if (kernel_setup(fn, 220 << 10).rc == cudaSuccess)
      for (int c = 2; c <= kStMaxCluster && g.groups == 0; ++c) {
        const size_t bytes = plan_ring(c);
        // (the query counts one CTA per SM; where two fit, twice as many clusters run together)
        held[c] = max_clusters(fn, 2 * c, kStThreads, bytes) * (bytes + 3072 <= ((size_t)228 << 10) / 2 ? 2 : 1);
      }
    a.cl = stream_cluster(a.tiles, a.num_kb, held);
  }
  if (a.cl < 1 || a.cl > kStMaxCluster || (a.cl > 1 && (g.groups > 0 || a.num_kb < a.cl))) return cudaErrorInvalidValue;
  const size_t smem = plan_ring(a.cl);
  const int grid = 2 * (a.cl > 1 ? a.tiles * a.cl : pairs);
  a.counters = reinterpret_cast<unsigned*>(g.workspace);
  a.parts = reinterpret_cast<float*>(a.counters + kStreamCounters);
  CUtensorMap mw, mx;
  cudaError_t rc = make_tile_map(&mw, g.w, (uint64_t)groups * g.w_rows, (uint64_t)g.K, (uint64_t)g.ldw,
                                 a.up_offset != kBlockM / 2 ? kBlockM / 2 : kBlockM);
  if (rc != cudaSuccess) return rc;
  rc = make_tile_map(&mx, g.x, (uint64_t)g.x_rows, (uint64_t)g.K, (uint64_t)g.ldx, (uint32_t)a.xbox);
  if (rc != cudaSuccess) return rc;
  switch (g.epi) {
    case STREAM_EPI_PLAIN: return launch_epi<STREAM_EPI_PLAIN>(mw, mx, a, grid, smem, g.pdl, error_word, stream);
    case STREAM_EPI_SILU: return launch_epi<STREAM_EPI_SILU>(mw, mx, a, grid, smem, g.pdl, error_word, stream);
    case STREAM_EPI_RESIDUAL: return launch_epi<STREAM_EPI_RESIDUAL>(mw, mx, a, grid, smem, g.pdl, error_word, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace sm100
}  // namespace penny
