// Decode-batch linear on sm_100a:
//     out[B, N] = x[B, K] * W[N, K]^T        bf16, fp32 accumulate, B <= 128
// With a handful of activation rows the operation is one read of W; at
// tensor-parallel shard sizes that read lasts 1-5 us, so what decides the time
// of a decode step is how early every SM starts streaming and how little
// happens after the last byte has arrived.
//
//   * Operands are swapped with respect to a large GEMM: the 128 rows of a W tile
//     are the M side of tcgen05.mma (K-major as stored), the batch rows of x are
//     the N side (16, 32, 48, 64 or 128 wide).  TMEM lane = output column n, TMEM column =
//     batch row.
//   * One CTA per (W tile, K range).  The K ranges of a tile belong to the CTAs
//     of one thread-block cluster (1-8 CTAs), which add their fp32 partials
//     through distributed shared memory: every CTA owns a slice of the batch
//     columns, receives that slice from its peers (st.async, the bytes counted
//     on its mbarrier), adds in rank order and stores bf16.  No global
//     workspace, no atomics, no second pass, deterministic.  The cluster size is
//     chosen per shape from a small time model (decode_gemm_plan.h).
//   * Programmatic dependent launch: the kernel may start while its predecessor
//     is still running.  Barrier set-up, TMEM allocation, the cluster handshake,
//     the TMA loads of the first W stages and an L2 prefetch of the rest of this
//     CTA's W range (bounded by a byte budget) all happen BEFORE the dependency
//     wait; only the x tiles wait for the predecessor.  W must therefore not be
//     written by the kernel launched just before (weights never are).
//   * TMA ring of 18-24 KB stages (B <= 64): three or four at 64 rows, five or six up to 16, in at most
//     112 KB of shared memory, so two of these kernels (or one and the decode attention) are resident per
//     SM: that is what lets the next kernel's prologue overlap this one.
//   * warp 0: TMA producer, warp 1: MMA issuer, warps 2-9: epilogue.  Every wait
//     is bounded; TMEM is always freed.
//
// Epilogues: plain store; silu(gate) * up for a gate/up weight whose rows are
// interleaved in blocks of 64 (tile = 64 gate rows + the 64 up rows of the same
// features; out is [B, N / 2]); residual add with what the next norm needs
// (DecodeFold).
//
// The reference has no GEMM of any kind (it is a collectives library used
// inside vLLM / SGLang, README.md:20-33); this kernel is what lets the TP-decode
// benchmark run without a vendor GEMM between the collectives.
#include "gemm_decode_sm100.h"

#include <cuda.h>

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <map>
#include <mutex>
#include <type_traits>

#include "all_reduce_oneshot.cuh"
#include "decode_gemm_plan.h"
#include "gemm_kernel_sm100.cuh"
#include "gemm_sm100.h"
#include "kernel_setup.h"
#include "pdl.h"

namespace penny {

namespace {
std::atomic<int> g_pdl{-1};
}
void set_pdl_enabled(int on) { g_pdl.store(on < 0 ? -1 : (on != 0)); }
bool pdl_enabled() {
  const int v = g_pdl.load();
  if (v >= 0) return v != 0;
  static const bool on = []() {
    const char* e = getenv("PENNY_PDL");
    return !(e != nullptr && e[0] == '0');
  }();
  return on;
}

namespace sm100 {

namespace {

constexpr int kDecEpiThreads = 256;  // eight epilogue warps
constexpr int kDecThreads = 64 + kDecEpiThreads;
constexpr int kMaxStages = 8;

// Diagnostics: with PENNY_DEC_STAMPS=1 the first 512 CTAs of a launch record
// %globaltimer at eight points (see gemm_decode_stamps in the header).
constexpr int kStampCtas = 512, kStampPoints = 8;
__device__ unsigned long long g_dec_stamps[kStampCtas * kStampPoints];

struct DecodeArgs {
  __nv_bfloat16* out;
  int ldo;
  int B, N, K;
  int num_kb;       // K steps of 64 elements
  int splits;       // CTAs per cluster = K ranges per tile
  int stages;       // depth of the TMA ring
  int l2_prefetch;  // K steps beyond the ring that the producer prefetches into L2 before the dependency wait
  int l2_ahead;     // steady state: W of step i + l2_ahead is prefetched into L2 when step i is loaded
  int k_stagger;    // 1: tiles start their K range at different offsets
  int stamps;       // 1: record timestamps
  int epi;          // DECODE_EPI_*
  int slabs;        // batch slabs of BT rows (1 unless B > 128)
  DecodePush push;  // world == 0: plain store
  const float* scale_sumsq;
  int scale_parts;
  float inv_width, eps;
  char* residual;
  int res_bytes;  // of an element of the residual: 2 (bf16) or 4 (fp32)
  __nv_bfloat16* stream_out;
  const __nv_bfloat16* norm_w;
  float* sumsq_out;
};

template <int BT>
struct DecodeCfg {
  static constexpr int kWBytes = kBlockM * kBlockK * 2;  // 16 KB of weights per stage
  static constexpr int kXBytes = BT * kBlockK * 2;
  static constexpr int kStageBytes = kWBytes + kXBytes;
  static constexpr int kTmemCols = BT <= 32 ? 32 : (BT <= 64 ? 64 : 128);
  static constexpr int kHalf = (BT / 2 + 15) / 16 * 16;  // columns of the first of a quarter's two epilogue warps
  static constexpr int kBarBytes = 256;
  // the peers' partials of this CTA's column slice: [splits - 1][slice][128 rows] fp32, for the rows that a slab has
  __host__ __device__ static size_t recv_floats(int splits, int B) { return decode_recv_floats(B < BT ? B : BT, splits); }
  // The ring doubles as the [BT][128] fp32 staging area of the epilogue, so it is never smaller than that.
  __host__ __device__ static int min_stages() { return (BT * kBlockM * 4 + kStageBytes - 1) / kStageBytes; }
  static size_t smem_bytes(int stages, int splits, int B = BT) {
    return (size_t)stages * kStageBytes + recv_floats(splits, B) * 4 + 1024 /*alignment*/ + kBarBytes + BT * 4 /*s_scale*/;
  }
};

// One [128 x 64] box of W into L2 only (no shared memory, no barrier).
__device__ __forceinline__ void tma_prefetch_l2_2d(const CUtensorMap* m, int x, int y) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];" ::"l"(m), "r"(x), "r"(y) : "memory");
}

template <int BT>
__global__ void __launch_bounds__(kDecThreads)
gemm_decode_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                   const DecodeArgs a, uint32_t* error_word) {
  using Cfg = DecodeCfg<BT>;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* tiles = align_tiles(smem_raw);
  const int S = a.splits, stages = a.stages;
  float* aux = reinterpret_cast<float*>(tiles + (size_t)stages * Cfg::kStageBytes);
  float* s_recv = aux;  // [S - 1][slice][128]
  uint64_t* bars = reinterpret_cast<uint64_t*>(aux + Cfg::recv_floats(S, a.B));
  uint64_t* full = bars;
  uint64_t* empty = bars + kMaxStages;
  uint64_t* tmem_full = bars + 2 * kMaxStages;
  uint64_t* recv_bar = bars + 2 * kMaxStages + 1;  // the peers' partials of my columns, counted in bytes
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(bars + 2 * kMaxStages + 2);
  volatile int* s_abort = reinterpret_cast<volatile int*>(tmem_holder + 1);
  float* s_scale = reinterpret_cast<float*>(bars + Cfg::kBarBytes / 8);  // [BT] 1 / rms of this CTA's columns

  pdl_launch_dependents();
  const int cta_lin = (int)(blockIdx.y * gridDim.x + blockIdx.x);
  auto stamp = [&](int point) {
    if (a.stamps && cta_lin < kStampCtas) g_dec_stamps[cta_lin * kStampPoints + point] = gtime_ns();
  };
  if (threadIdx.x == 0) stamp(0);  // CTA start

  // (read from lane 0, so that the compiler knows it to be the same in all lanes)
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t crank = S > 1 ? cluster_ctarank() : 0u;
  // batches above BT rows: grid y = tile * slabs + slab, so the slabs of a weight tile are dispatched
  // next to each other and read the tile from DRAM once
  int tile = (int)blockIdx.y, row0 = 0;
  if (a.slabs > 1) {
    row0 = tile % a.slabs * BT;
    tile /= a.slabs;
  }
  const int kb0 = decode_kb_begin(a.num_kb, S, (int)crank), kb1 = decode_kb_begin(a.num_kb, S, (int)crank + 1);
  const int nkb = kb1 - kb0;
  // the batch rows of this slab are dealt out over the cluster: columns [lo, hi) are finished here
  const int nB = min(BT, a.B - row0);
  const int sl = decode_slice(nB, S);
  const int lo = (int)crank * sl, hi = min(nB, lo + sl);
  // Tiles walk their K range from different starting points (and wrap around), so that at any
  // moment the CTAs of a wave read different column ranges of W rather than the same few
  // hundred bytes of every row.
  const int kshift = a.k_stagger ? (int)(((unsigned)tile * 2654435761u >> 8) % (unsigned)nkb) : 0;
  auto kb_at = [&](int i) {
    int k = i + kshift;
    if (k >= nkb) k -= nkb;
    return kb0 + k;
  };

  const int pre = min(stages, nkb);
  if (threadIdx.x == 0) {
    for (int i = 0; i < stages; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    mbar_init(tmem_full, 1);
    mbar_init(recv_bar, 1);
    *s_abort = 0;
    mbar_fence_init();
    if (S > 1 && lo < hi) mbar_expect_tx(recv_bar, (uint32_t)((S - 1) * (hi - lo) * kBlockM * 4));
    // The first ring-full of W tiles is requested before anything else happens in
    // the CTA (TMEM allocation, the block and cluster barriers): its HBM latency
    // runs under the rest of the prologue.  W never depends on the predecessor.
    for (int i = 0; i < pre; ++i) {
      mbar_expect_tx(&full[i], Cfg::kStageBytes);
      tma_load_2d(tiles + (size_t)i * Cfg::kStageBytes, &map_w, &full[i], kb_at(i) * kBlockK, tile * kBlockM);
    }
    tma_prefetch_desc(&map_x);
  }
  if (warp == 1) tmem_alloc(tmem_holder, Cfg::kTmemCols);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  // The peers' receive barriers must exist before anyone arrives on them: every thread
  // arrives on the cluster barrier now and waits for it only where it first needs the
  // peers (epilogue warps: before their first remote store; the others: before they leave),
  // so the cluster-wide rendezvous is off the path to the first load and the first MMA.
  // (Relaxed: the fence behind the barriers' initialisation covers all that the peers will touch.  A release here held
  // every warp for about a microsecond: launches of a chain, 1 row, q/k/v 10.4 -> 9.9 us, down 20.8 -> 20.0; 64 rows 13.5 ->
  // 12.9, 24.3 -> 23.7.)
  if (S > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  const uint32_t tmem_base = *tmem_holder;
  auto fail = [&](uint32_t code) {
    *s_abort = 1;
    atomicCAS(error_word, 0u, code);
  };

  // Producer and issuer run as whole warps and elect a lane only for the instructions themselves: operands that are the
  // same in all lanes then stay in uniform registers.  In a branch of one lane every TMA and MMA fetched its operands one by
  // one, some 60 cycles each.  Launches of a chain, 1 row: q/k/v 9.9 -> 9.5 us, o 8.0 -> 7.3, down 20.0 -> 19.6; 128 rows 16.0 ->
  // 15.1, 13.0 -> 12.1, 28.3 -> 27.5; gate/up (two CTAs per SM, bound by HBM) 37.3 -> 37.1.
  if (warp == 0) {
    // -------------------------------------------------------------- TMA producer
    // W of the next K steps goes to L2 ahead of the ring (the whole range when the
    // matrix fits the L2 budget, else a rolling window), still before the
    // dependency wait; the x tiles come after it.
    int pf_next = min(nkb, pre + a.l2_prefetch);
    for (int i = pre; i < pf_next; ++i) {
      if (elect_one()) tma_prefetch_l2_2d(&map_w, kb_at(i) * kBlockK, tile * kBlockM);
      __syncwarp();
    }
    if (lane == 0) stamp(1);  // prologue done, about to wait for the predecessor
    pdl_wait();
    if (lane == 0) stamp(2);  // predecessor complete
    for (int i = 0; i < pre; ++i) {
      if (elect_one())
        tma_load_2d(tiles + (size_t)i * Cfg::kStageBytes + Cfg::kWBytes, &map_x, &full[i], kb_at(i) * kBlockK, row0);
      __syncwarp();
    }
    int stage = pre == stages ? 0 : pre;
    uint32_t phase = pre == stages ? 1u : 0u;
    bool ok = true;
    for (int i = pre; i < nkb; ++i) {
      ok = __all_sync(0xffffffffu, mbar_wait_abortable(&empty[stage], phase ^ 1u, s_abort));
      if (!ok) break;
      unsigned char* sw = tiles + (size_t)stage * Cfg::kStageBytes;
      const bool pf = pf_next < nkb && pf_next < i + a.l2_ahead;
      if (elect_one()) {
        mbar_expect_tx(&full[stage], Cfg::kStageBytes);
        tma_load_2d(sw, &map_w, &full[stage], kb_at(i) * kBlockK, tile * kBlockM);
        tma_load_2d(sw + Cfg::kWBytes, &map_x, &full[stage], kb_at(i) * kBlockK, row0);
        if (pf) tma_prefetch_l2_2d(&map_w, kb_at(pf_next) * kBlockK, tile * kBlockM);
      }
      __syncwarp();
      if (pf) ++pf_next;
      if (++stage == stages) {
        stage = 0;
        phase ^= 1u;
      }
    }
    if (lane == 0) stamp(3);  // last load issued
    if (!ok && lane == 0) fail(GEMM_ERR_PRODUCER_WAIT);
    __syncwarp();
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issuer
    constexpr uint32_t idesc = make_idesc_bf16(kBlockM, BT);
    const uint64_t desc0 = make_smem_desc(smem_u32(tiles));
    const uint32_t desc_hi = (uint32_t)(desc0 >> 32);
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int i = 0; i < nkb; ++i) {
      ok = __all_sync(0xffffffffu, mbar_wait_abortable(&full[stage], phase, s_abort));
      if (!ok) break;
      tc_fence_after_sync();
      const uint32_t lw = (uint32_t)desc0 + (uint32_t)(stage * (Cfg::kStageBytes >> 4));  // addresses in 16-byte units
      const uint32_t lx = lw + (Cfg::kWBytes >> 4);
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < kBlockK / kUmmaK; ++k)
          umma_bf16(tmem_base, make_desc(desc_hi, lw + 2 * k), make_desc(desc_hi, lx + 2 * k), idesc, (i | k) != 0);
        umma_commit(&empty[stage]);
      }
      __syncwarp();
      if (++stage == stages) {
        stage = 0;
        phase ^= 1u;
      }
    }
    if (lane == 0) stamp(4);  // last MMA issued
    if (ok) {
      if (elect_one()) umma_commit(tmem_full);
    } else if (lane == 0) {
      fail(GEMM_ERR_MMA_WAIT);
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ epilogue
    // Everything after the TMEM read works on shared memory with run-time loops:
    // the code stays small (an unrolled per-column epilogue costs more in
    // instruction-cache misses than the whole GEMM takes).  What is left is a chain of
    // latencies, so eight warps share it, two per TMEM lane quarter.
    const int q = warp & 3, h = (warp - 2) >> 2;
    const int row = q * 32 + lane;  // weight row inside the tile = output column
    const int tid = (int)threadIdx.x - 64;
    const bool silu = a.epi == DECODE_EPI_SILU_PAIRS, resid = a.epi == DECODE_EPI_RESIDUAL;
    pdl_wait();  // this thread's stores (and the loads below) come after everything the predecessor did
    if (a.scale_sumsq != nullptr && lo < hi) {
      // 1 / rms of my columns, under the product: several threads per column where there are few
      const int n = hi - lo;
      int tpc = 32;
      while (n * tpc > kDecEpiThreads) tpc >>= 1;
      const int c = tid / tpc;
      float s = 0.f;
      if (c < n) {
        const float* p = a.scale_sumsq + row0 + lo + c;
#pragma unroll 8
        for (int i = tid % tpc; i < a.scale_parts; i += tpc) s += __ldcg(p + (size_t)i * a.B);
      }
      for (int o = tpc >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (c < n && tid % tpc == 0) s_scale[c] = rsqrtf(s * a.inv_width + a.eps);
    }
    // A work item is 8 consecutive rows (output columns) of one batch column; a thread's items are of one row group.
    const int groups = silu ? 8 : 16;
    const int g = tid % groups, n0 = tile * (silu ? kBlockM / 2 : kBlockM) + g * 8;
    // RESIDUAL: the stream's rows travel an item ahead, the first ones and the norm's weight under the product
    uint4 r_next[2], nw = make_uint4(0, 0, 0, 0);
    r_next[0] = r_next[1] = nw;
    auto load_residual = [&](int j) {
      if (j >= hi) return;
      const uint4* p = reinterpret_cast<const uint4*>(a.residual + ((size_t)(row0 + j) * a.ldo + n0) * a.res_bytes);
      r_next[0] = p[0];
      if (a.res_bytes == 4) r_next[1] = p[1];
    };
    if (resid) {
      if (a.norm_w != nullptr) nw = __ldg(reinterpret_cast<const uint4*>(a.norm_w + n0));
      load_residual(lo + tid / groups);
    }
    bool ok = mbar_wait_abortable(tmem_full, 0u, s_abort);
    if (!ok && lane == 0) fail(GEMM_ERR_EPILOGUE_WAIT);
    ok = __all_sync(0xffffffffu, ok);
    if (tid == 0) stamp(5);  // accumulator complete
    tc_fence_after_sync();
    // accumulator -> shared memory, column-major [BT columns][128 rows] fp32, in the
    // pipeline stages (every MMA that read them has completed)
    float* s_acc = reinterpret_cast<float*>(tiles);
    const float4* s_acc4 = reinterpret_cast<const float4*>(s_acc);
    const int c_begin = h * Cfg::kHalf, c_end = h == 0 ? min(nB, Cfg::kHalf) : nB;
    if (ok) {
      const uint32_t tacc = tmem_base + ((uint32_t)(q * 32) << 16);
#pragma unroll 1
      for (int c = c_begin; c < c_end; c += 16) {
        uint32_t r[16];
        tmem_ld_32x16(tacc + c, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j) s_acc[(c + j) * kBlockM + row] = __uint_as_float(r[j]);
      }
    }
    __syncwarp();
    if (S > 1) {
      asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");  // the peers' barriers exist
      if (ok) {
        // ---- hand every other CTA the columns of its slice that this warp has: a store instruction
        // covers 4 columns x 128 bytes and counts its bytes on the owner's barrier, so nothing waits
        // for the stores (an arrival behind them was 1.5-2 us of a split GEMM's 3 us exchange) ----
        const uint32_t recv_local = smem_u32(s_recv), bar_local = smem_u32(recv_bar);
        const int rv = q * 8 + (lane & 7);  // float4 of my quarter
        const uint32_t per = (65536u + (uint32_t)sl - 1u) / (uint32_t)sl;
        for (int c = c_begin + (lane >> 3); c < c_end; c += 4) {
          const int d = (int)(((uint32_t)c * per) >> 16);  // owner: c / sl
          if (d == (int)crank) continue;
          const float4 v = s_acc4[c * (kBlockM / 4) + rv];
          st_async_v4(map_to_cta(recv_local, (uint32_t)d) +
                          (uint32_t)(((decode_recv_slot((int)crank, d) * sl + c - d * sl) * (kBlockM / 4) + rv) * 16),
                      map_to_cta(bar_local, (uint32_t)d), __float_as_uint(v.x), __float_as_uint(v.y), __float_as_uint(v.z),
                      __float_as_uint(v.w));
        }
      }
    }
    named_bar_sync(1, kDecEpiThreads);  // all rows and columns staged, s_scale written
    if (ok && S > 1 && lo < hi) {
      ok = mbar_wait_cluster(recv_bar, 0u, s_abort);
      if (!ok && lane == 0) fail(GEMM_ERR_EPILOGUE_WAIT);
      ok = __all_sync(0xffffffffu, ok);
    }
    if (tid == 0) stamp(6);  // peers' partials received
    if (ok) {
      // ---- my slice: add the peers' partials in rank order, apply the epilogue, store ----
      const int n_out = silu ? a.N / 2 : a.N;
      const bool vec_ok = (a.ldo % 8 == 0) && ((reinterpret_cast<uintptr_t>(a.out) & 15u) == 0);
      // push mode: the call number of the all-reduce that follows (final: the predecessor has
      // finished) selects the scratch half and stamps the lines
      unsigned long long push_seq = 0;
      size_t push_base = 0;
      if (a.push.world > 0) {
        push_seq = *reinterpret_cast<const volatile unsigned long long*>(a.push.call_seq);
        push_base = scratch_half(a.push.scratch_off, a.push.scratch_bytes, push_seq);
      }
      for (int j = lo + tid / groups; j < hi; j += kDecEpiThreads / groups) {
        // sum over the cluster of rows r0 .. r0 + 7 of column j
        auto sum8 = [&](int r0, float (&acc)[8]) {
#pragma unroll
          for (int k = 0; k < 8; ++k) acc[k] = 0.f;
          for (int src = 0; src < S; ++src) {
            const float4* p = src == (int)crank
                                  ? s_acc4 + (j * kBlockM + r0) / 4
                                  : reinterpret_cast<const float4*>(s_recv) +
                                        ((decode_recv_slot(src, (int)crank) * sl + (j - lo)) * kBlockM + r0) / 4;
            const float4 v0 = p[0], v1 = p[1];
            acc[0] += v0.x; acc[1] += v0.y; acc[2] += v0.z; acc[3] += v0.w;
            acc[4] += v1.x; acc[5] += v1.y; acc[6] += v1.z; acc[7] += v1.w;
          }
        };
        float v[8];
        sum8(g * 8, v);
        const float sc = a.scale_sumsq != nullptr ? s_scale[j - lo] : 1.f;
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] *= sc;
        if (resid) {
          const uint32_t rw[8] = {r_next[0].x, r_next[0].y, r_next[0].z, r_next[0].w, r_next[1].x, r_next[1].y, r_next[1].z, r_next[1].w};
          const uint32_t ww[4] = {nw.x, nw.y, nw.z, nw.w};
          const bool wide = a.res_bytes == 4;
          load_residual(j + kDecEpiThreads / groups);
          uint32_t zo[4], ho[4];
          float ss = 0.f;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float z0 = v[2 * k] + __uint_as_float(wide ? rw[2 * k] : rw[k] << 16);
            const float z1 = v[2 * k + 1] + __uint_as_float(wide ? rw[2 * k + 1] : rw[k] & 0xffff0000u);
            v[2 * k] = z0;
            v[2 * k + 1] = z1;
            ss += z0 * z0 + z1 * z1;
            zo[k] = pack_bf16x2(__float_as_uint(z0), __float_as_uint(z1));
            ho[k] = pack_bf16x2(__float_as_uint(z0 * __uint_as_float(ww[k] << 16)),
                                __float_as_uint(z1 * __uint_as_float(ww[k] & 0xffff0000u)));
          }
          const size_t off = (size_t)(row0 + j) * a.ldo + n0;
          uint4* rp = reinterpret_cast<uint4*>(a.residual + off * a.res_bytes);
          const uint4 zb = make_uint4(zo[0], zo[1], zo[2], zo[3]);
          if (wide) {
            rp[0] = make_uint4(__float_as_uint(v[0]), __float_as_uint(v[1]), __float_as_uint(v[2]), __float_as_uint(v[3]));
            rp[1] = make_uint4(__float_as_uint(v[4]), __float_as_uint(v[5]), __float_as_uint(v[6]), __float_as_uint(v[7]));
            if (a.stream_out != nullptr) *reinterpret_cast<uint4*>(a.stream_out + off) = zb;
          } else {
            rp[0] = zb;
          }
          if (a.norm_w == nullptr) continue;
          *reinterpret_cast<uint4*>(a.out + off) = make_uint4(ho[0], ho[1], ho[2], ho[3]);
          const unsigned half = 0xffffu << (lane & 16);  // the sixteen row groups of this column
#pragma unroll
          for (int o = 8; o > 0; o >>= 1) ss += __shfl_xor_sync(half, ss, o);
          if (g == 0) a.sumsq_out[(size_t)tile * a.B + row0 + j] = ss;
          continue;
        }
        if (silu) {
          // rows 0-63 of the tile are gate, rows 64-127 the matching up rows
          float u[8];
          sum8(64 + g * 8, u);
#pragma unroll
          for (int k = 0; k < 8; ++k) v[k] = v[k] / (1.f + __expf(-v[k])) * (u[k] * sc);
        }
        __nv_bfloat16* dst = a.out + (size_t)(row0 + j) * a.ldo + n0;
        if (vec_ok && n0 + 8 <= n_out) {
          uint4 o;
          o.x = pack_bf16x2(__float_as_uint(v[0]), __float_as_uint(v[1]));
          o.y = pack_bf16x2(__float_as_uint(v[2]), __float_as_uint(v[3]));
          o.z = pack_bf16x2(__float_as_uint(v[4]), __float_as_uint(v[5]));
          o.w = pack_bf16x2(__float_as_uint(v[6]), __float_as_uint(v[7]));
          const int owner = a.push.world > 0 ? j / a.push.per : -1;
          if (owner >= 0 && owner != a.push.rank) {
            // a row another rank reduces: straight into that rank's receive lines of the coming
            // all-reduce (flag-in-data: two 16-byte lines carry the 16 bytes and the call's stamp)
            const uint32_t e = ll_flag(push_seq);
            V16 l0, l1;
            l0.w[0] = o.x; l0.w[1] = e; l0.w[2] = o.y; l0.w[3] = e;
            l1.w[0] = o.z; l1.w[1] = e; l1.w[2] = o.w; l1.w[3] = e;
            char* line = a.push.heap[owner] + push_base +
                         (((size_t)a.push.rank * a.push.per + (j - owner * a.push.per)) * a.push.hv + n0 / 8) * 32;
            st16_volatile(line, l0);
            st16_volatile(line + 16, l1);
          } else {
            *reinterpret_cast<uint4*>(dst) = o;
          }
        } else {
          for (int k = 0; k < 8; ++k)
            if (n0 + k < n_out) dst[k] = __float2bfloat16_rn(v[k]);
        }
      }
    }
  }
  // ------------------------------------------------------------------- teardown
  if (S > 1 && warp < 2) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  tc_fence_before_sync();
  __syncthreads();
  if (threadIdx.x == 64) stamp(7);  // done
  pdl_wait();  // no thread leaves before the predecessor has finished
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, Cfg::kTmemCols);
  }
}

// CTAs of this kernel the current device holds at once, by cluster size (asked once per device).
template <int BT>
const int* decode_capacity(int sms) {
  struct Table {
    int cap[kDecodeMaxSplits + 1];
  };
  static std::mutex mu;
  static std::map<int, Table> tables;
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lock(mu);
  auto it = tables.find(dev);
  if (it != tables.end()) return it->second.cap;
  Table t;
  decode_model_capacity(sms, 16, t.cap);  // fallback if a query fails
  const void* fn = reinterpret_cast<const void*>(gemm_decode_kernel<BT>);
  if (kernel_setup(fn, 227 << 10).rc == cudaSuccess) {
    for (int s = 1; s <= kDecodeMaxSplits; ++s) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3((unsigned)s, (unsigned)(2 * sms), 1);
      cfg.blockDim = dim3(kDecThreads, 1, 1);
      cfg.dynamicSmemBytes = DecodeCfg<BT>::smem_bytes(3, s);  // what a split launch typically asks for
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = (unsigned)s;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      int n = 0;
      if (cudaOccupancyMaxActiveClusters(&n, fn, &cfg) == cudaSuccess && n > 0)
        t.cap[s] = n * s;
      else
        (void)cudaGetLastError();
      // The cluster query counts one CTA per SM.  Measured (start stamps of every CTA): with
      // shared memory for two CTAs per SM a second round of clusters becomes resident on
      // the same SMs within 2-3 us, so twice that many CTAs run as ONE wave; beyond it the
      // rest waits for the first CTAs to finish.
      if (cfg.dynamicSmemBytes + 1024 <= ((size_t)228 << 10) / 2) t.cap[s] *= 2;
    }
  }
  tables[dev] = t;
  return tables[dev].cap;
}

template <int BT>
cudaError_t launch_decode_bt(const void* x, const void* w, void* out, int B, int N, int K, int ldx, int ldw, int ldo,
                             int epi, int splits, bool pdl, long long l2_budget, int smem_kb, const DecodePush* push,
                             const DecodeFold* fold, int sms, uint32_t* error_word, cudaStream_t stream) {
  using Cfg = DecodeCfg<BT>;
  CUtensorMap mw, mx;
  cudaError_t rc = make_tile_map(&mw, w, (uint64_t)N, (uint64_t)K, (uint64_t)ldw, kBlockM);
  if (rc != cudaSuccess) return rc;
  rc = make_tile_map(&mx, x, (uint64_t)B, (uint64_t)K, (uint64_t)ldx, BT);
  if (rc != cudaSuccess) return rc;
  DecodeArgs a;
  a.out = reinterpret_cast<__nv_bfloat16*>(out);
  a.ldo = ldo;
  a.B = B;
  a.N = N;
  a.K = K;
  a.num_kb = (K + kBlockK - 1) / kBlockK;
  const int tiles = (N + kBlockM - 1) / kBlockM;
  const int slabs = (B + BT - 1) / BT;  // > 1 only with BT = 128
  if ((long long)tiles * slabs > 65535) return cudaErrorInvalidValue;
  a.slabs = slabs;
  if (splits <= 0 && BT <= 64 && fold != nullptr && (fold->scale_sumsq != nullptr || fold->residual != nullptr))
    splits = decode_choose_splits_chain(tiles * slabs, a.num_kb, sms, decode_capacity<BT>(sms));
  if (splits <= 0) splits = decode_choose_splits(tiles * slabs, a.num_kb, decode_capacity<BT>(sms));
  splits = std::max(1, std::min(splits, std::min(kDecodeMaxSplits, a.num_kb)));
  a.splits = splits;
  a.epi = epi;
  if (push != nullptr)
    a.push = *push;
  else
    a.push.world = 0;
  const DecodeFold f = fold != nullptr ? *fold : DecodeFold{};
  a.scale_sumsq = f.scale_sumsq;
  a.scale_parts = f.scale_parts;
  a.inv_width = 1.f / (float)K;
  a.eps = f.eps;
  a.residual = reinterpret_cast<char*>(f.residual);
  a.res_bytes = f.residual_fp32 ? 4 : 2;
  a.stream_out = reinterpret_cast<__nv_bfloat16*>(f.stream_out);
  a.norm_w = reinterpret_cast<const __nv_bfloat16*>(f.norm_w);
  a.sumsq_out = f.sumsq_out;
  // ring depth: what fits next to the receive area in 106 to 112 KB (two CTAs per SM, of this kernel or the next:
  // one sets up and fills its ring while the other drains).  With a 128-wide batch tile and no more CTAs than
  // SMs one per SM and as deep as the range needs.  A second round of CTAs wants the two as well (the step
  // of 128 sequences, gate/up 62.8 us -> 45, the LM head at one sequence 176 -> 163, at 64 195 -> 181, at 128
  // 232 -> 209).
  const int kb_per = (a.num_kb + splits - 1) / splits;
  // (measured, whole N = 1 decode step: 106 KB 6.08 ms, 75 KB 6.40, 56 KB 6.72, 150 KB 7.40.  112 KB is the most that two CTAs
  // leave room for: with the receive area as large as the batch asks for, a fifth stage for up to 8 rows, 0.5 % of a step)
  const size_t budget = smem_kb > 0 ? (size_t)std::min(smem_kb, 226) << 10 : (BT <= 64 || tiles * slabs * splits > sms ? (size_t)(BT <= 64 ? 112 : 106) << 10 : (size_t)200 << 10);
  int stages = Cfg::min_stages();
  while (stages < kMaxStages && stages < kb_per && Cfg::smem_bytes(stages + 1, splits, B) <= budget) ++stages;
  a.stages = stages;
  const size_t smem = Cfg::smem_bytes(stages, splits, B);
  if (smem > ((size_t)227 << 10)) return cudaErrorInvalidValue;
  // L2 prefetch of the rest of the weight range while the predecessor runs: only when
  // the whole matrix fits the budget (a shard of a tensor-parallel layer does; the
  // full-size matrices of a single GPU would just evict one another)
  const long long w_bytes = (long long)tiles * a.num_kb * Cfg::kWBytes;
  static const int env_ahead = getenv("PENNY_DEC_AHEAD") ? atoi(getenv("PENNY_DEC_AHEAD")) : 0;
  static const int env_stagger = getenv("PENNY_DEC_STAGGER") ? atoi(getenv("PENNY_DEC_STAGGER")) : 1;
  a.l2_ahead = env_ahead > 0 ? stages + env_ahead : 0;
  a.l2_prefetch = (w_bytes <= l2_budget) ? kb_per : env_ahead;
  a.k_stagger = env_stagger;
  static const int env_stamps = getenv("PENNY_DEC_STAMPS") ? atoi(getenv("PENNY_DEC_STAMPS")) : 0;
  a.stamps = env_stamps;
  rc = kernel_setup(reinterpret_cast<const void*>(gemm_decode_kernel<BT>), 227 << 10).rc;
  if (rc != cudaSuccess) return rc;
  return launch_kernel_ex(gemm_decode_kernel<BT>, dim3((unsigned)splits, (unsigned)(tiles * slabs), 1), dim3(kDecThreads), smem,
                          stream, pdl, splits, mw, mx, a, error_word);
}

}  // namespace

cudaError_t launch_gemm_decode(const void* x, const void* w, void* out, int B, int N, int K, int ldx, int ldw,
                               int ldo, int epi, int splits, bool pdl, long long l2_budget_bytes,
                               int smem_kb, const DecodePush* push, const DecodeFold* fold, uint32_t* error_word,
                               cudaStream_t stream) {
  if (B <= 0 || B > kDecodeMaxBatch || N <= 0 || K <= 0 || K % 8 != 0 || ldx % 8 != 0 || ldw % 8 != 0)
    return cudaErrorInvalidValue;
  if (push != nullptr && B > 128) return cudaErrorInvalidValue;  // the owners' receive lines cover one slab
  if (epi < DECODE_EPI_PLAIN || epi > DECODE_EPI_RESIDUAL) return cudaErrorInvalidValue;
  if (epi == DECODE_EPI_RESIDUAL &&
      (N % kBlockM != 0 || ldo % 8 != 0 || push != nullptr || fold == nullptr || fold->residual == nullptr ||
       (fold->norm_w != nullptr && (out == nullptr || fold->sumsq_out == nullptr)) ||
       ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(fold->residual) |
         reinterpret_cast<uintptr_t>(fold->stream_out) | reinterpret_cast<uintptr_t>(fold->norm_w)) & 15u) != 0))
    return cudaErrorInvalidValue;
  if (epi == DECODE_EPI_SILU_PAIRS && N % kBlockM != 0) return cudaErrorInvalidValue;
  if ((N + kBlockM - 1) / kBlockM > 65535) return cudaErrorInvalidValue;
  if (push != nullptr && (push->world < 2 || push->world > 8 || epi != DECODE_EPI_PLAIN || N % 8 != 0 || ldo % 8 != 0 ||
                          push->hv * 8 != N || push->per < 1 || (reinterpret_cast<uintptr_t>(out) & 15u) != 0))
    return cudaErrorInvalidValue;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (l2_budget_bytes < 0) l2_budget_bytes = (long long)32 << 20;
  // Batch tiles in steps of 16 rows where the launch is one of a chain of folded linears: fewer rows of x per K step and a
  // smaller exchange leave a stage more for the weights (a step of 1 / 8 / 37 rows, the latter on 16 and 48 instead of 32 and
  // 64: 792 -> 783, 913 -> 909, 1358 -> 1333 us).  Launches without a fold (several ranks) were not timed on them.
  const bool chain = fold != nullptr && (fold->scale_sumsq != nullptr || fold->residual != nullptr);
  auto go = [&](auto bt) {
    return launch_decode_bt<decltype(bt)::value>(x, w, out, B, N, K, ldx, ldw, ldo, epi, splits, pdl, l2_budget_bytes, smem_kb, push,
                                                 fold, sms, error_word, stream);
  };
  if (chain && B <= 16) return go(std::integral_constant<int, 16>());
  if (B <= 32) return go(std::integral_constant<int, 32>());
  if (chain && B <= 48) return go(std::integral_constant<int, 48>());
  if (B <= 64) return go(std::integral_constant<int, 64>());
  return go(std::integral_constant<int, 128>());
}

int gemm_decode_stamps(unsigned long long* out, int max_ctas) {
  const int n = std::min(max_ctas, kStampCtas);
  if (cudaMemcpyFromSymbol(out, g_dec_stamps, (size_t)n * kStampPoints * sizeof(unsigned long long)) != cudaSuccess) {
    (void)cudaGetLastError();
    return 0;
  }
  return n;
}

namespace {
const int* capacity_of(int B, bool folded, int sms) {
  if (folded && B <= 16) return decode_capacity<16>(sms);
  if (B <= 32) return decode_capacity<32>(sms);
  if (folded && B <= 48) return decode_capacity<48>(sms);
  return B <= 64 ? decode_capacity<64>(sms) : decode_capacity<128>(sms);
}
int current_sms() {
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  (void)cudaGetLastError();
  return sms > 0 ? sms : 148;
}
}  // namespace

int gemm_decode_capacity(int B, int splits) {
  if (splits < 1 || splits > kDecodeMaxSplits) return 0;
  return capacity_of(B, false, current_sms())[splits];
}

int gemm_decode_splits(int B, int N, int K, bool folded) {
  const int sms = current_sms();
  const int num_kb = (K + kBlockK - 1) / kBlockK, tiles = (N + kBlockM - 1) / kBlockM * ((std::max(B, 1) + 127) / 128);
  const int* cap = capacity_of(B, folded, sms);
  return folded && B <= 64 ? decode_choose_splits_chain(tiles, num_kb, sms, cap) : decode_choose_splits(tiles, num_kb, cap);
}

}  // namespace sm100
}  // namespace penny
