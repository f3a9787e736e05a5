// Torch-facing wrappers of the decode-step kernels.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <pybind11/pybind11.h>
#include <torch/extension.h>

#include "decode_kernels.h"
#include "gemm_tile_sm100.h"
#include "moe_routing.h"

namespace py = pybind11;
using namespace penny;

uint32_t* penny_gemm_error_word();  // gemm_binding.cpp

namespace {
cudaStream_t cur() { return at::cuda::getCurrentCUDAStream().stream(); }
void need(bool ok, const char* msg) { TORCH_CHECK(ok, "penny: ", msg); }
void ck(cudaError_t rc, const char* what) {
  TORCH_CHECK(rc == cudaSuccess, "penny: ", what, ": ", cudaGetErrorString(rc));
}
bool bf16_cuda(const at::Tensor& t) {
  return t.is_cuda() && t.is_contiguous() && t.scalar_type() == at::kBFloat16;
}
// Matrices of one shape that lie back to back in one storage.  Looked at on every call: entries of a caller's list
// may be other tensors by now, or the same ones over other memory (tensor.data = ...).
bool stacked(const std::vector<at::Tensor>& mats) {
  if (mats.empty() || !bf16_cuda(mats[0]) || mats[0].dim() != 2 || ((uintptr_t)mats[0].data_ptr() & 15) != 0) return false;
  const at::Tensor& t0 = mats[0];
  for (size_t i = 1; i < mats.size(); ++i)
    if (!bf16_cuda(mats[i]) || mats[i].sizes() != t0.sizes() ||
        mats[i].storage().unsafeGetStorageImpl() != t0.storage().unsafeGetStorageImpl() ||
        mats[i].storage_offset() != t0.storage_offset() + (int64_t)i * t0.numel())
      return false;
  return true;
}
}  // namespace

void bind_decode(py::module_& m) {
  m.def("rope_append", [](at::Tensor qkv, at::Tensor kcache, at::Tensor vcache, at::Tensor positions,
                          int64_t Hq, int64_t Hkv, int64_t D, double theta) {
    need(bf16_cuda(qkv) && bf16_cuda(kcache) && bf16_cuda(vcache), "rope_append expects contiguous bf16 CUDA tensors");
    need(positions.is_cuda() && positions.scalar_type() == at::kInt && positions.is_contiguous(), "positions must be int32 CUDA");
    need(qkv.dim() == 2 && qkv.size(1) == (Hq + 2 * Hkv) * D, "qkv must be [B, (Hq + 2 Hkv) D]");
    need(kcache.dim() == 4 && kcache.size(0) == qkv.size(0) && kcache.size(1) == Hkv && kcache.size(3) == D &&
             vcache.sizes() == kcache.sizes(), "caches must be [B, Hkv, max_len, D]");
    need(positions.numel() == qkv.size(0), "one position per row");
    const at::cuda::OptionalCUDAGuard guard(qkv.device());
    ck(launch_rope_append(qkv.data_ptr(), kcache.data_ptr(), vcache.data_ptr(), positions.data_ptr<int>(),
                          (int)qkv.size(0), (int)Hq, (int)Hkv, (int)D, (int)kcache.size(2), (float)theta, cur()),
       "rope_append");
  });
  m.def("rope_rows", [](at::Tensor qkv, int64_t Hq, int64_t Hkv, int64_t D, int64_t pos0, double theta) {
    need(bf16_cuda(qkv) && qkv.dim() == 2 && qkv.size(1) == (Hq + 2 * Hkv) * D, "rope_rows expects [T, (Hq + 2 Hkv) D] bf16");
    const at::cuda::OptionalCUDAGuard guard(qkv.device());
    ck(launch_rope_rows(qkv.data_ptr(), (int)qkv.size(0), (int)Hq, (int)Hkv, (int)D, (int)pos0, (float)theta, cur()),
       "rope_rows");
  });
  // residual: bf16 or fp32.  ids [rows] int64: the rows of src (an embedding table) that become the stream; in pinned host memory they are read
  // from there when the kernel runs
  m.def("norm_prep", [](at::Tensor src, at::Tensor norm_w, at::Tensor residual, at::Tensor out, at::Tensor sumsq,
                        c10::optional<at::Tensor> ids) {
    need(bf16_cuda(src) && bf16_cuda(norm_w) && bf16_cuda(out) &&
             (bf16_cuda(residual) || (residual.is_cuda() && residual.scalar_type() == at::kFloat && residual.is_contiguous())) && src.dim() == 2 && residual.dim() == 2,
         "norm_prep expects contiguous bf16 CUDA tensors");
    const int64_t rows = ids.has_value() ? ids->numel() : src.size(0), H = src.size(1);
    if (ids.has_value())
      need((ids->is_cuda() || ids->is_pinned()) && ids->scalar_type() == at::kLong && ids->is_contiguous(),
           "norm_prep: ids must be int64, CUDA or pinned");
    need(residual.size(0) == rows && residual.size(1) == H && out.sizes() == residual.sizes() && norm_w.numel() == H &&
             sumsq.is_cuda() && sumsq.scalar_type() == at::kFloat && sumsq.is_contiguous() && sumsq.numel() == rows,
         "norm_prep shapes");
    for (const at::Tensor* t : {&src, &norm_w, &residual, &out})
      need(((uintptr_t)t->data_ptr() & 15) == 0, "norm_prep: 16-byte aligned tensors");
    const at::cuda::OptionalCUDAGuard guard(src.device());
    ck(launch_norm_prep(src.data_ptr(), ids.has_value() ? (const long long*)ids->data_ptr<int64_t>() : nullptr, src.size(0),
                        norm_w.data_ptr(), residual.data_ptr(), residual.scalar_type() == at::kFloat, out.data_ptr(), sumsq.data_ptr<float>(), (int)rows, (int)H,
                        cur()),
       "norm_prep");
  }, py::arg("src"), py::arg("norm_w"), py::arg("residual"), py::arg("out"), py::arg("sumsq"), py::arg("ids") = py::none());
  m.def("decode_attn_workspace_bytes", [](int64_t B, int64_t Hq, int64_t splits) {
    return (int64_t)decode_attn_workspace_bytes((int)B, (int)Hq, (int)splits);
  });
  m.def("decode_attention", [](at::Tensor qkv, at::Tensor kcache, at::Tensor vcache, at::Tensor positions,
                               at::Tensor out, at::Tensor workspace, int64_t Hq, int64_t Hkv, int64_t splits,
                               double scale) {
    need(bf16_cuda(qkv) && bf16_cuda(kcache) && bf16_cuda(vcache) && bf16_cuda(out), "decode_attention expects contiguous bf16 CUDA tensors");
    need(positions.is_cuda() && positions.scalar_type() == at::kInt, "positions must be int32 CUDA");
    const int64_t B = qkv.size(0), D = kcache.size(3);
    need(qkv.size(1) == (Hq + 2 * Hkv) * D && out.numel() == B * Hq * D, "decode_attention shapes");
    need(workspace.is_cuda() && (int64_t)workspace.nbytes() >= (int64_t)decode_attn_workspace_bytes((int)B, (int)Hq, (int)splits),
         "workspace too small (decode_attn_workspace_bytes)");
    need(((uintptr_t)workspace.data_ptr() & 15) == 0, "workspace must be 16-byte aligned");
    const at::cuda::OptionalCUDAGuard guard(qkv.device());
    ck(launch_decode_attention(qkv.data_ptr(), kcache.data_ptr(), vcache.data_ptr(), positions.data_ptr<int>(),
                               out.data_ptr(), workspace.data_ptr(), (int)B, (int)Hq, (int)Hkv, (int)D,
                               (int)kcache.size(2), (int)splits, (float)scale, cur()),
       "decode_attention");
  });
  m.def("decode_attn_fused_workspace_bytes", [](int64_t B, int64_t Hq, int64_t Hkv, int64_t splits) {
    return (int64_t)decode_attn_fused_workspace_bytes((int)B, (int)Hq, (int)Hkv, (int)splits);
  });
  // rope + KV append + split-KV attention + merge in one launch; qkv is the raw projection of the new token
  m.def("decode_attention_fused", [](at::Tensor qkv, at::Tensor kcache, at::Tensor vcache, at::Tensor positions,
                                     at::Tensor out, at::Tensor workspace, int64_t Hq, int64_t Hkv, int64_t splits,
                                     double scale, double theta, bool pdl, bool balance) {
    need(bf16_cuda(qkv) && bf16_cuda(kcache) && bf16_cuda(vcache) && bf16_cuda(out), "decode_attention_fused expects contiguous bf16 CUDA tensors");
    need(positions.is_cuda() && positions.scalar_type() == at::kInt && positions.is_contiguous(), "positions must be int32 CUDA");
    need(kcache.dim() == 4 && vcache.sizes() == kcache.sizes(), "caches must be [B, Hkv, max_len, D]");
    const int64_t B = qkv.size(0), D = kcache.size(3);
    need(qkv.dim() == 2 && qkv.size(1) == (Hq + 2 * Hkv) * D && out.numel() == B * Hq * D && kcache.size(0) == B &&
             kcache.size(1) == Hkv && positions.numel() == B, "decode_attention_fused shapes");
    need(workspace.is_cuda() && (int64_t)workspace.nbytes() >=
                                    (int64_t)decode_attn_fused_workspace_bytes((int)B, (int)Hq, (int)Hkv, (int)splits),
         "workspace too small (decode_attn_fused_workspace_bytes)");
    need(((uintptr_t)workspace.data_ptr() & 15) == 0, "workspace must be 16-byte aligned");
    const at::cuda::OptionalCUDAGuard guard(qkv.device());
    ck(launch_decode_attention_fused(qkv.data_ptr(), kcache.data_ptr(), vcache.data_ptr(), positions.data_ptr<int>(),
                                     out.data_ptr(), workspace.data_ptr(), (int)B, (int)Hq, (int)Hkv, (int)D,
                                     (int)kcache.size(2), (int)splits, (float)scale, (float)theta, pdl, balance, cur()),
       "decode_attention_fused");
  }, py::arg("qkv"), py::arg("kcache"), py::arg("vcache"), py::arg("positions"), py::arg("out"), py::arg("workspace"),
     py::arg("Hq"), py::arg("Hkv"), py::arg("splits"), py::arg("scale"), py::arg("theta"), py::arg("pdl") = true,
     py::arg("balance") = false);
  m.def("decode_attn_balanced_splits", [](int64_t B, int64_t Hkv) {
    need(B >= 1 && Hkv >= 1, "decode_attn_balanced_splits: rows and KV heads");
    return (int64_t)decode_attn_balanced_splits((int)B, (int)Hkv);
  });
  // pairs: gate and up columns in turn, 64 of each (what a weight in gemm_decode's silu_pairs layout gives)
  m.def("silu_mul", [](at::Tensor gate_up, at::Tensor out, bool pairs) {
    need(bf16_cuda(gate_up) && bf16_cuda(out) && gate_up.dim() == 2, "silu_mul expects [rows, 2F] bf16");
    const int64_t rows = gate_up.size(0), F = gate_up.size(1) / 2;
    need(out.numel() == rows * F, "silu_mul output must be [rows, F]");
    const at::cuda::OptionalCUDAGuard guard(gate_up.device());
    ck(launch_silu_mul(gate_up.data_ptr(), out.data_ptr(), (int)rows, (int)F, cur(), pairs ? 64 : 0), "silu_mul");
  }, py::arg("gate_up"), py::arg("out"), py::arg("pairs") = false);
  // dst (int64 in host memory) = src; returns whether every id lies in [0, rows).  One call from Python for both: a look at
  // the ids by numpy beside the copy was 1.3 us of a step, more on a cold first one.
  m.def("take_ids", [](at::Tensor src, at::Tensor dst, int64_t rows) {
    need(dst.device().is_cpu() && dst.scalar_type() == at::kLong && dst.is_contiguous(), "take_ids: dst int64 on the host");
    dst.copy_(src);
    const int64_t *id = dst.data_ptr<int64_t>(), *end = id + dst.numel();
    bool ok = true;
    for (; id < end; ++id) ok &= *id >= 0 && *id < rows;
    return ok;
  });
  m.def("argmax_workspace_bytes", [](int64_t rows) { return (int64_t)argmax_workspace_bytes((int)rows); });
  m.def("argmax_rows", [](at::Tensor logits, at::Tensor out_val, at::Tensor out_idx, int64_t index_base,
                          c10::optional<at::Tensor> workspace, c10::optional<at::Tensor> pair,
                          c10::optional<at::Tensor> next_tokens, c10::optional<at::Tensor> tokens,
                          c10::optional<at::Tensor> positions, c10::optional<at::Tensor> host_tokens) {
    need(bf16_cuda(logits) && logits.dim() == 2, "argmax_rows expects [rows, cols] bf16");
    const int64_t rows = logits.size(0);
    need(out_val.is_cuda() && out_val.scalar_type() == at::kFloat && out_val.numel() == rows, "out_val [rows] fp32");
    need(out_idx.is_cuda() && out_idx.scalar_type() == at::kLong && out_idx.numel() == rows, "out_idx [rows] int64");
    void* ws = nullptr;
    if (workspace.has_value()) {
      need(workspace->is_cuda() && workspace->is_contiguous() &&
               (int64_t)workspace->nbytes() >= (int64_t)argmax_workspace_bytes((int)rows),
           "workspace too small (argmax_workspace_bytes) or not contiguous; it must be zeroed once");
      ws = workspace->data_ptr();
    }
    float* pp = nullptr;
    if (pair.has_value()) {
      need(pair->is_cuda() && pair->scalar_type() == at::kFloat && pair->is_contiguous() && pair->numel() == 2 * rows,
           "pair [2 * rows] fp32");
      pp = pair->data_ptr<float>();
    }
    GreedyStep step = {};
    need(next_tokens.has_value() || !host_tokens.has_value(), "host_tokens: beside next_tokens");
    if (next_tokens.has_value()) {
      need(tokens.has_value() && positions.has_value() && next_tokens->is_cuda() && tokens->is_cuda() && positions->is_cuda() &&
               next_tokens->scalar_type() == at::kLong && tokens->scalar_type() == at::kLong &&
               positions->scalar_type() == at::kInt && next_tokens->numel() == rows && tokens->numel() == rows &&
               positions->numel() == rows && next_tokens->is_contiguous() && tokens->is_contiguous() && positions->is_contiguous(),
           "next_tokens / tokens [rows] int64, positions [rows] int32, together");
      step = {(long long*)next_tokens->data_ptr<int64_t>(), (long long*)tokens->data_ptr<int64_t>(), positions->data_ptr<int>(), nullptr};
      if (host_tokens.has_value()) {
        need(host_tokens->is_pinned() && host_tokens->scalar_type() == at::kLong && host_tokens->is_contiguous() &&
                 host_tokens->numel() == rows, "host_tokens: pinned [rows] int64");
        step.host_tokens = (long long*)host_tokens->data_ptr<int64_t>();
      }
    }
    const at::cuda::OptionalCUDAGuard guard(logits.device());
    ck(launch_argmax(logits.data_ptr(), (int)rows, (int)logits.size(1), out_val.data_ptr<float>(),
                     (long long*)out_idx.data_ptr<int64_t>(), pp, (long long)index_base, ws, step, cur()),
       "argmax_rows");
  }, py::arg("logits"), py::arg("out_val"), py::arg("out_idx"), py::arg("index_base"),
     py::arg("workspace") = py::none(), py::arg("pair") = py::none(), py::arg("next_tokens") = py::none(),
     py::arg("tokens") = py::none(), py::arg("positions") = py::none(), py::arg("host_tokens") = py::none());
  // Expert-parallel MoE routing on the device (csrc/moe_routing.cu)
  m.def("moe_route", [](at::Tensor logits, int64_t topk) {
    need(bf16_cuda(logits) && logits.dim() == 2, "moe_route expects [tokens, experts] bf16");
    const int64_t T = logits.size(0), E = logits.size(1);
    const at::cuda::OptionalCUDAGuard guard(logits.device());
    at::Tensor ids = at::empty({T, topk}, logits.options().dtype(at::kInt));
    at::Tensor gates = at::empty({T, topk}, logits.options().dtype(at::kFloat));
    ck(launch_moe_topk(logits.data_ptr(), (int)T, (int)E, (int)topk, ids.data_ptr<int>(), gates.data_ptr<float>(), cur()),
       "moe_route");
    return std::make_tuple(ids, gates);
  });
  m.def("moe_tables", [](at::Tensor ids, int64_t experts) {
    need(ids.is_cuda() && ids.scalar_type() == at::kInt && ids.is_contiguous(), "moe_tables expects contiguous int32 ids");
    const int64_t P = ids.numel();
    const at::cuda::OptionalCUDAGuard guard(ids.device());
    auto opt = ids.options();
    at::Tensor order = at::empty({P}, opt), sorted = at::empty({P}, opt), send_off = at::empty({experts + 1}, opt),
               counts = at::empty({experts}, opt);
    ck(launch_moe_tables(ids.data_ptr<int>(), (int)P, (int)experts, order.data_ptr<int>(), sorted.data_ptr<int>(),
                         send_off.data_ptr<int>(), counts.data_ptr<int>(), cur()),
       "moe_tables");
    return std::make_tuple(order, sorted, send_off, counts);
  });
  m.def("moe_placement", [](at::Tensor counts_all) {
    need(counts_all.is_cuda() && counts_all.scalar_type() == at::kInt && counts_all.is_contiguous() &&
             counts_all.dim() == 2,
         "moe_placement expects [world, experts] int32");
    const int64_t W = counts_all.size(0), E = counts_all.size(1);
    const at::cuda::OptionalCUDAGuard guard(counts_all.device());
    auto opt = counts_all.options();
    at::Tensor dst_base = at::empty({W, E}, opt), rows = at::empty({W}, opt), ranges = at::empty({E, 2}, opt);
    ck(launch_moe_placement(counts_all.data_ptr<int>(), (int)W, (int)E, dst_base.data_ptr<int>(), rows.data_ptr<int>(),
                            ranges.data_ptr<int>(), cur()),
       "moe_placement");
    return std::make_tuple(dst_base, rows, ranges);
  });
  // stacked() as one matrix of all rows, or None.
  m.def("stacked_rows", [](const std::vector<at::Tensor>& mats) -> c10::optional<at::Tensor> {
    if (!stacked(mats)) return c10::nullopt;
    const int64_t K = mats[0].size(1);
    return mats[0].detach().as_strided({(int64_t)mats.size() * mats[0].size(0), K}, {K, 1});
  });
  // A MoE layer of one rank: router, rows by expert, expert SwiGLU FFNs, gate-weighted sum.  Nothing comes
  // back to the host, and it is one call: as Python calls the launches took 113 us of host time, of which a
  // layer of a few tokens hid half.  w13: per expert [2 ffn, hidden] (gate rows, then up rows), w2: [hidden, ffn], each
  // list one stack, else None is returned and nothing runs; block_n and down_cluster as in gemm_tile, up_rows and down_rows
  // above 0: gate/up and down with the weight on the M side (gemm_tile's pair 2) and tiles of that many rows.  The router meets
  // the library's GEMM only and may have any strides.
  m.def("moe_layer", [](at::Tensor x, at::Tensor router, const std::vector<at::Tensor>& w13, const std::vector<at::Tensor>& w2,
                        int64_t topk, int64_t block_n, int64_t down_cluster, int64_t up_rows,
                        int64_t down_rows) -> c10::optional<at::Tensor> {
    if (!stacked(w13) || !stacked(w2)) return c10::nullopt;
    need(bf16_cuda(x) && x.dim() == 2 && ((uintptr_t)x.data_ptr() & 15) == 0, "moe_layer: 2-D aligned contiguous bf16 x");
    need(router.is_cuda() && router.scalar_type() == at::kBFloat16 && router.dim() == 2, "moe_layer: 2-D bf16 router");
    const int T = (int)x.size(0), H = (int)x.size(1), E = (int)router.size(0), F = (int)w2[0].size(1), P = T * (int)topk;
    need(router.size(1) == H && (int)w13.size() == E && (int)w2.size() == E && w13[0].size(0) == 2 * (int64_t)F &&
             w13[0].size(1) == H && w2[0].size(0) == H && T > 0, "moe_layer shapes");
    const at::cuda::OptionalCUDAGuard guard(x.device());
    const cudaStream_t stream = cur();
    const at::Tensor logits = at::matmul(x, router.t()).contiguous();
    // [ids | order | expert of sorted | row of pair | borders | counts], then the gates
    const at::Tensor tables = at::empty({4 * (int64_t)P + 2 * E + 1}, x.options().dtype(at::kInt));
    const at::Tensor gates = at::empty({P}, x.options().dtype(at::kFloat));
    const at::Tensor rows = at::empty({P, H}, x.options()), act = at::empty({P, F}, x.options()), out = at::empty_like(x);
    int* ids = tables.data_ptr<int>();
    int *order = ids + P, *sorted = order + P, *row_of_pair = sorted + P, *borders = row_of_pair + P, *counts = borders + E + 1;
    ck(launch_moe_route_tables(logits.data_ptr(), T, E, (int)topk, ids, gates.data_ptr<float>(), order, sorted, borders, counts,
                               stream), "moe_layer: routing");
    ck(launch_moe_gather(x.data_ptr(), order, P, (int)topk, H, rows.data_ptr(), row_of_pair, stream), "moe_layer: rows");
    sm100::TileGemm g = {};
    g.a = rows.data_ptr();
    g.b = w13[0].data_ptr();
    g.out = act.data_ptr();
    g.M = P;
    g.b_rows = 2 * F;
    g.K = g.lda = g.ldb = H;
    g.ldo = F;
    g.epi = sm100::TILE_EPI_SILU;
    g.groups = E;
    g.ranges = borders;
    g.range_stride = 1;
    auto tiles = [&](int64_t rows) {
      g.pair = rows > 0 ? 2 : 0;
      g.block_n = (int)(rows > 0 ? rows : block_n);
    };
    tiles(up_rows);
    g.pdl = true;
    ck(sm100::launch_gemm_tile(g, penny_gemm_error_word(), stream), "moe_layer: gate / up");
    g.a = act.data_ptr();
    g.b = w2[0].data_ptr();
    g.out = rows.data_ptr();  // (their inputs are used up)
    g.b_rows = H;
    g.K = g.lda = g.ldb = F;
    g.ldo = H;
    g.epi = sm100::TILE_EPI_PLAIN;
    tiles(down_rows);
    g.cluster = down_rows > 0 ? 0 : (int)down_cluster;
    ck(sm100::launch_gemm_tile(g, penny_gemm_error_word(), stream), "moe_layer: down");
    ck(launch_moe_sum(rows.data_ptr(), row_of_pair, gates.data_ptr<float>(), T, (int)topk, H, out.data_ptr(), stream), "moe_layer: sum");
    return out;
  }, py::arg("x"), py::arg("router"), py::arg("w13"), py::arg("w2"), py::arg("topk"), py::arg("block_n"), py::arg("down_cluster"),
     py::arg("up_rows") = 0, py::arg("down_rows") = 0);
  m.def("sample_finish", [](at::Tensor pairs, int64_t world, at::Tensor next_tokens, at::Tensor tokens,
                            at::Tensor positions) {
    const int64_t B = next_tokens.numel();
    need(pairs.is_cuda() && pairs.scalar_type() == at::kFloat && pairs.is_contiguous() && pairs.numel() == world * 2 * B,
         "pairs [world, 2, B] fp32");
    need(next_tokens.scalar_type() == at::kLong && tokens.scalar_type() == at::kLong && tokens.numel() == B &&
             positions.scalar_type() == at::kInt && positions.numel() == B && next_tokens.is_cuda() &&
             tokens.is_cuda() && positions.is_cuda(),
         "next_tokens / tokens [B] int64, positions [B] int32");
    const at::cuda::OptionalCUDAGuard guard(pairs.device());
    ck(launch_sample_finish(pairs.data_ptr<float>(), (int)world, (int)B, (long long*)next_tokens.data_ptr<int64_t>(),
                            (long long*)tokens.data_ptr<int64_t>(), positions.data_ptr<int>(), cur()),
       "sample_finish");
  });

}
