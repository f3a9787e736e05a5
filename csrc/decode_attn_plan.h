// How the decode attention cuts the rows of a batch by their lengths (decode_attention_fused.cu): plain C++, used by the
// kernel, by its launcher and (through the host simulator library) by the CPU tests.
//
// The launcher sizes the grid from the cache's length alone, the kernel cuts by the positions it finds on the device.  A
// row with more pieces than the grid has CTAs for would wait for ever for a piece that nobody computes, so both sides
// count with positions inside the cache: one past its end is cut like the last one.
#pragma once

#if defined(__CUDACC__)
#define PENNY_ATTN_HD __host__ __device__ inline
#else
#define PENNY_ATTN_HD inline
#endif

namespace penny {
namespace attn {

// Shortest piece and most pieces of a row: a merge is 2 us.  One row of 2048 positions in 1 / 4 / 8 / 16 pieces: 17.3 /
// 8.0 / 6.9 / 7.7 us, of 16000 in 8 / 16 / 37: 23.6 / 17.7 / 19.5, of 100 in 1 / 8 / 16: 2.7 / 5.1 / 6.5.
constexpr int kMinPiece = 256, kMaxPieces = 16;

PENNY_ATTN_HD int at_least(int a, int b) { return a > b ? a : b; }
PENNY_ATTN_HD int at_most(int a, int b) { return a < b ? a : b; }

// cached rows that a token at `pos` attends to, and what they count as where rows are cut
PENNY_ATTN_HD int cached_rows(int pos, int max_len) { return at_most(at_least(pos, 0), max_len); }
PENNY_ATTN_HD int cut_rows(int pos, int max_len) { return at_least(0, at_most(pos, max_len - 1)); }

// CTAs that a balanced launch counts on; 0, no pieces, where there are four rounds of (row, KV head) pairs anyhow, which
// the GPU deals out as they end.
PENNY_ATTN_HD int balance_slots(int items, int sms) { return items > 8 * sms ? 0 : 2 * sms; }
// Pieces beyond one per (row, KV head) pair: what a cut takes at most, and no more than the cache's length allows (the
// launch behind this one begins when every CTA of this one has begun, so CTAs without a piece keep its weights waiting).
PENNY_ATTN_HD int balance_extra(int items, int slots) { return items * 2 > slots ? 2 * slots : slots; }
PENNY_ATTN_HD int grid_extra(int items, int slots, int max_len) {
  const long long by_len = (long long)items * (at_most(kMaxPieces, at_least(1, (max_len - 1) / kMinPiece)) - 1);
  const int most = slots > 0 ? balance_extra(items, slots) : 0;
  return by_len < most ? (int)by_len : most;
}

// The length of a piece: the batch's positions (their cut_rows: `total`, the longest `top`) over `slots`, over twice as
// many where the rows are of mixed lengths and alone fill half of them.
PENNY_ATTN_HD int piece_len(long long total, int top, int B, int Hkv, int slots) {
  const bool mixed = (long long)top * B * 4 > total * 5 && B * Hkv * 2 > slots;
  const int target = mixed ? 2 * slots : slots;
  return at_least(kMinPiece, (int)((total * Hkv + target - 1) / target));
}
// A row has as many pieces as fit it whole.
PENNY_ATTN_HD int pieces_of(int rows, int len) { return at_most(kMaxPieces, at_least(1, rows / len)); }

}  // namespace attn
}  // namespace penny
