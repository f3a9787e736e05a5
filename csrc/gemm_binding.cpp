// Torch-facing functions of the tcgen05 GEMM family (standalone GEMM here; the
// fused GEMM -> reduce-scatter and all-gather -> GEMM are bound next to the
// communicator because they need its heap).
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <pybind11/pybind11.h>
#include <torch/extension.h>

#include "gemm_decode_sm100.h"
#include "gemm_tile_sm100.h"
#include "pdl.h"
#include "gemm_sm100.h"

namespace py = pybind11;

uint32_t* penny_gemm_error_word() {
  uint32_t* word = penny::sm100::gemm_error_word();
  TORCH_CHECK(word != nullptr, "gemm: no error word on this device");
  return word;
}

void bind_gemm(py::module_& m) {
  // out[M, N] = a[M, K] @ b[N, K]^T (the nn.Linear convention: b is the weight)
  m.def("gemm_bf16", [](at::Tensor a, at::Tensor b, at::Tensor out, int64_t block_n) {
    TORCH_CHECK(a.is_cuda() && b.is_cuda() && out.is_cuda(), "gemm_bf16: CUDA tensors");
    TORCH_CHECK(a.scalar_type() == at::kBFloat16 && b.scalar_type() == at::kBFloat16 &&
                    out.scalar_type() == at::kBFloat16, "gemm_bf16: bf16 only");
    TORCH_CHECK(a.dim() == 2 && b.dim() == 2 && out.dim() == 2, "gemm_bf16: 2-D tensors");
    TORCH_CHECK(a.stride(1) == 1 && b.stride(1) == 1 && out.stride(1) == 1, "gemm_bf16: rows must be contiguous");
    const int64_t M = a.size(0), K = a.size(1), N = b.size(0);
    TORCH_CHECK(b.size(1) == K && out.size(0) == M && out.size(1) == N, "gemm_bf16: shape mismatch");
    const at::cuda::OptionalCUDAGuard guard(a.device());
    cudaError_t rc = penny::sm100::launch_gemm_bf16(
        a.data_ptr(), b.data_ptr(), out.data_ptr(), (int)M, (int)N, (int)K, (int)a.stride(0), (int)b.stride(0),
        (int)out.stride(0), (int)block_n, penny_gemm_error_word(), at::cuda::getCurrentCUDAStream().stream());
    TORCH_CHECK(rc == cudaSuccess, "gemm_bf16: ", cudaGetErrorString(rc));
  }, py::arg("a"), py::arg("b"), py::arg("out"), py::arg("block_n") = 0);
  // Decode-batch linear: out[B, N] = x[B, K] @ w[N, K]^T for B <= 1024 (slabs of 128 rows in one launch).  One CTA per (weight tile, K
  // range); the K ranges of a tile are reduced inside a thread-block cluster through distributed shared
  // memory.  pdl: may start (and load w) while the previous kernel on the stream still runs, so w must not
  // be written by that kernel.  silu_pairs: w's rows are blocks of 64 gate + 64 up rows and out is
  // [B, N / 2] = silu(gate) * up.  sumsq, residual, norm_w, sumsq_out: as in gemm_tile below;
  // the residual may be fp32, stream_out then takes the sum in bf16 as well.
  m.def("gemm_decode", [](at::Tensor x, at::Tensor w, at::Tensor out, bool silu_pairs, int64_t splits, bool pdl,
                          int64_t l2_budget, int64_t smem_kb, c10::optional<at::Tensor> push,
                          c10::optional<at::Tensor> sumsq, double eps, c10::optional<at::Tensor> residual,
                          c10::optional<at::Tensor> norm_w, c10::optional<at::Tensor> sumsq_out,
                          c10::optional<at::Tensor> stream_out) {
    TORCH_CHECK(x.is_cuda() && w.is_cuda() && out.is_cuda(), "gemm_decode: CUDA tensors");
    TORCH_CHECK(x.scalar_type() == at::kBFloat16 && w.scalar_type() == at::kBFloat16 &&
                    out.scalar_type() == at::kBFloat16, "gemm_decode: bf16 only");
    TORCH_CHECK(x.dim() == 2 && w.dim() == 2 && out.dim() == 2, "gemm_decode: 2-D tensors");
    TORCH_CHECK(x.stride(1) == 1 && w.stride(1) == 1 && out.stride(1) == 1, "gemm_decode: rows must be contiguous");
    const int64_t B = x.size(0), K = x.size(1), N = w.size(0);
    TORCH_CHECK(B >= 1 && B <= penny::sm100::kDecodeMaxBatch, "gemm_decode: 1 <= rows of x <= 1024 (use gemm_bf16 beyond)");
    TORCH_CHECK(!push.has_value() || B <= 128, "gemm_decode: push needs rows of x <= 128");
    TORCH_CHECK(w.size(1) == K && out.size(0) == B && out.size(1) == (silu_pairs ? N / 2 : N),
                "gemm_decode: shape mismatch");
    TORCH_CHECK(splits >= 0 && splits <= 8, "gemm_decode: 0 <= splits <= 8");
    const at::cuda::OptionalCUDAGuard guard(x.device());
    // push: the bytes of a DecodePush from comm_fused_norm_push_target (rows other ranks own go to them)
    penny::sm100::DecodePush pd;
    const penny::sm100::DecodePush* pp = nullptr;
    if (push.has_value()) {
      TORCH_CHECK(push->device().is_cpu() && push->scalar_type() == at::kByte && push->is_contiguous() &&
                      push->numel() == (int64_t)sizeof(pd), "gemm_decode: push must come from comm_fused_norm_push_target");
      memcpy(&pd, push->data_ptr(), sizeof(pd));
      pp = &pd;
    }
    penny::sm100::DecodeFold fold = {};
    fold.eps = (float)eps;
    if (sumsq.has_value()) {
      TORCH_CHECK(sumsq->is_cuda() && sumsq->scalar_type() == at::kFloat && sumsq->is_contiguous() && sumsq->dim() == 2 &&
                      sumsq->size(1) == B, "gemm_decode: sumsq must be [parts, rows] fp32");
      fold.scale_sumsq = sumsq->data_ptr<float>();
      fold.scale_parts = (int)sumsq->size(0);
    }
    int epi = silu_pairs ? penny::sm100::DECODE_EPI_SILU_PAIRS : penny::sm100::DECODE_EPI_PLAIN;
    TORCH_CHECK(residual.has_value() || !(norm_w.has_value() || sumsq_out.has_value() || stream_out.has_value()),
                "gemm_decode: norm_w, sumsq_out and stream_out beside a residual");
    if (residual.has_value()) {
      auto bf16 = [](const at::Tensor& t) { return t.is_cuda() && t.scalar_type() == at::kBFloat16 && t.stride(-1) == 1; };
      fold.residual_fp32 = residual->scalar_type() == at::kFloat;
      TORCH_CHECK(epi == penny::sm100::DECODE_EPI_PLAIN && N % 128 == 0 && residual->is_cuda() && residual->stride(-1) == 1 &&
                      (fold.residual_fp32 || bf16(*residual)) && residual->sizes() == out.sizes() &&
                      residual->stride(0) == out.stride(0) && norm_w.has_value() == sumsq_out.has_value(),
                  "gemm_decode: residual like out, rows of w a multiple of 128; norm_w and sumsq_out together");
      epi = penny::sm100::DECODE_EPI_RESIDUAL;
      fold.residual = residual->data_ptr();
      if (stream_out.has_value()) {
        TORCH_CHECK(fold.residual_fp32 && bf16(*stream_out) && stream_out->sizes() == out.sizes() &&
                        stream_out->stride(0) == out.stride(0), "gemm_decode: stream_out like out, beside an fp32 residual");
        fold.stream_out = stream_out->data_ptr();
      }
      if (norm_w.has_value()) {
        TORCH_CHECK(bf16(*norm_w) && norm_w->is_contiguous() && norm_w->numel() == N && sumsq_out->is_cuda() &&
                        sumsq_out->scalar_type() == at::kFloat && sumsq_out->is_contiguous() &&
                        sumsq_out->numel() == N / 128 * B,
                    "gemm_decode: contiguous norm_w [rows of w], sumsq_out [rows of w / 128, rows]");
        fold.norm_w = norm_w->data_ptr();
        fold.sumsq_out = sumsq_out->data_ptr<float>();
      }
    }
    cudaError_t rc = penny::sm100::launch_gemm_decode(
        x.data_ptr(), w.data_ptr(), out.data_ptr(), (int)B, (int)N, (int)K, (int)x.stride(0), (int)w.stride(0),
        (int)out.stride(0), epi, (int)splits, pdl, (long long)l2_budget, (int)smem_kb, pp, &fold,
        penny_gemm_error_word(),
        at::cuda::getCurrentCUDAStream().stream());
    TORCH_CHECK(rc == cudaSuccess, "gemm_decode: ", cudaGetErrorString(rc));
  }, py::arg("x"), py::arg("w"), py::arg("out"), py::arg("silu_pairs") = false, py::arg("splits") = 0,
     py::arg("pdl") = true, py::arg("l2_budget") = -1, py::arg("smem_kb") = 0, py::arg("push") = py::none(),
     py::arg("sumsq") = py::none(), py::arg("eps") = 1e-5, py::arg("residual") = py::none(), py::arg("norm_w") = py::none(),
     py::arg("sumsq_out") = py::none(), py::arg("stream_out") = py::none());
  // Tiled GEMM with a fused epilogue (csrc/gemm_tile_sm100.cu).  epi: 0 plain, 1 silu(gate) * up (b's gate
  // rows before its up rows, or with silu_pairs, without ranges, as for gemm_decode; out [M, rows / 2]; exact_silu, not
  // with pair 2: with a division that is no approximation, also for gates below -87.3), 2 residual add.  ranges:
  // [groups, 2] starts and ends or [groups + 1] borders of the rows of a and out that meet each group of b [groups * rows, K].  sumsq
  // [parts, M]: rows of a before their norm weight; every output is scaled by rsqrt(sum / K + eps).  pdl: may start,
  // and without ranges load b, while the kernel before it on the stream still runs, so that kernel must not write
  // b (a weight); everything else is waited for.  The residual may be fp32, stream_out then takes the sum in bf16 as
  // well.  sumsq_out [rows of b / 128, M]: a sum for every 128 columns; [rows of b / 16, M]: as many rows as the call returns
  // hold sums of some columns each, which leaves the width of the tiles free.  block_n: columns of a tile; pair 1 / -1: CTA
  // pairs or single CTAs (0: pairs of 256 x 256 for block_n 512); cluster: CTAs or pairs that share a tile's K.  With block_n
  // 0 what is 0 of the three is chosen, a cluster taken where some width can be shared so.  pair 2: pairs with the weight on
  // the M side and up to block_n rows of a (plain or silu).
  m.def("gemm_tile", [](at::Tensor a, at::Tensor b, at::Tensor out, int64_t epi, c10::optional<at::Tensor> ranges,
                        c10::optional<at::Tensor> sumsq, double eps, c10::optional<at::Tensor> residual,
                        c10::optional<at::Tensor> norm_w, c10::optional<at::Tensor> sumsq_out, int64_t block_n, bool pdl,
                        int64_t cluster, c10::optional<at::Tensor> stream_out, int64_t pair, bool silu_pairs, bool exact_silu) {
    auto bf16 = [](const at::Tensor& t) { return t.is_cuda() && t.scalar_type() == at::kBFloat16 && t.stride(-1) == 1; };
    TORCH_CHECK(bf16(a) && bf16(b) && bf16(out) && a.dim() == 2 && b.dim() == 2 && out.dim() == 2,
                "gemm_tile: 2-D bf16 CUDA tensors with contiguous rows");
    penny::sm100::TileGemm g = {};
    g.a = a.data_ptr();
    g.b = b.data_ptr();
    g.out = out.data_ptr();
    g.M = (int)a.size(0);
    g.K = (int)a.size(1);
    g.b_rows = (int)b.size(0);
    if (ranges.has_value()) {
      // [groups, 2] starts and ends, or [groups + 1] borders
      TORCH_CHECK(ranges->is_cuda() && ranges->scalar_type() == at::kInt && ranges->is_contiguous() &&
                      (ranges->dim() == 1 || (ranges->dim() == 2 && ranges->size(1) == 2)),
                  "gemm_tile: ranges must be [groups, 2] or [groups + 1] int32 CUDA");
      g.groups = (int)(ranges->dim() == 1 ? ranges->size(0) - 1 : ranges->size(0));
      g.range_stride = (int)ranges->dim();
      TORCH_CHECK(g.groups > 0 && b.size(0) % g.groups == 0, "gemm_tile: the weight must be whole groups of rows");
      g.ranges = ranges->data_ptr<int>();
      g.b_rows = (int)(b.size(0) / g.groups);
    }
    TORCH_CHECK(b.size(1) == g.K && out.size(0) == g.M && out.size(1) == (epi == 1 ? g.b_rows / 2 : g.b_rows),
                "gemm_tile: shape mismatch");
    g.lda = (int)a.stride(0);
    g.ldb = (int)b.stride(0);
    g.ldo = (int)out.stride(0);
    g.epi = (int)epi;
    g.eps = (float)eps;
    if (sumsq.has_value()) {
      TORCH_CHECK(sumsq->is_cuda() && sumsq->scalar_type() == at::kFloat && sumsq->is_contiguous() && sumsq->dim() == 2 &&
                      sumsq->size(1) == g.M, "gemm_tile: sumsq must be [parts, rows] fp32");
      g.scale_sumsq = sumsq->data_ptr<float>();
      g.scale_parts = (int)sumsq->size(0);
    }
    if (epi == 2) {
      g.residual_fp32 = residual.has_value() && residual->scalar_type() == at::kFloat;
      TORCH_CHECK(residual.has_value() && residual->is_cuda() && residual->stride(-1) == 1 &&
                      (g.residual_fp32 || bf16(*residual)) && residual->sizes() == out.sizes() &&
                      residual->stride(0) == out.stride(0) && norm_w.has_value() == sumsq_out.has_value(),
                  "gemm_tile: residual like out; norm_w and sumsq_out together");
      g.residual = residual->data_ptr();
      if (stream_out.has_value()) {
        TORCH_CHECK(g.residual_fp32 && bf16(*stream_out) && stream_out->sizes() == out.sizes() &&
                        stream_out->stride(0) == out.stride(0), "gemm_tile: stream_out like out, beside an fp32 residual");
        g.stream_out = stream_out->data_ptr();
      }
      if (norm_w.has_value()) {
        TORCH_CHECK(bf16(*norm_w) && norm_w->is_contiguous() && norm_w->numel() == g.b_rows && sumsq_out->is_cuda() &&
                        sumsq_out->scalar_type() == at::kFloat && sumsq_out->is_contiguous() &&
                        (sumsq_out->numel() == (int64_t)(g.b_rows / 128) * g.M ||
                         sumsq_out->numel() == (int64_t)(g.b_rows / 16) * g.M),
                    "gemm_tile: contiguous norm_w [rows of b], sumsq_out [rows of b / 128 or / 16, rows]");
        g.sumsq_cap = sumsq_out->numel() == (int64_t)(g.b_rows / 128) * g.M ? 0 : g.b_rows / 16;
        g.norm_w = norm_w->data_ptr();
        g.sumsq_out = sumsq_out->data_ptr<float>();
      }
    }
    g.block_n = (int)block_n;
    g.pdl = pdl;
    g.cluster = (int)cluster;
    g.pair = (int)pair;
    g.silu_pairs = silu_pairs;
    g.exact_silu = exact_silu;
    TORCH_CHECK(epi == 2 || !stream_out.has_value(), "gemm_tile: stream_out beside a residual");
    const at::cuda::OptionalCUDAGuard guard(a.device());
    int sumsq_rows = 0;
    const cudaError_t rc = penny::sm100::launch_gemm_tile(g, penny_gemm_error_word(),
                                                          at::cuda::getCurrentCUDAStream().stream(), &sumsq_rows);
    TORCH_CHECK(rc == cudaSuccess, "gemm_tile: ", cudaGetErrorString(rc));
    return sumsq_rows;
  }, py::arg("a"), py::arg("b"), py::arg("out"), py::arg("epi") = 0, py::arg("ranges") = py::none(),
     py::arg("sumsq") = py::none(), py::arg("eps") = 1e-5, py::arg("residual") = py::none(), py::arg("norm_w") = py::none(),
     py::arg("sumsq_out") = py::none(), py::arg("block_n") = 0, py::arg("pdl") = false,
     py::arg("cluster") = 0, py::arg("stream_out") = py::none(), py::arg("pair") = 0,
     py::arg("silu_pairs") = false, py::arg("exact_silu") = false);
  m.def("gemm_tile_choice", [](int64_t M, int64_t N, int64_t K, int64_t epi, int64_t groups, int64_t pair, int64_t cluster,
                               bool silu_pairs) {
    penny::sm100::TileGemm g = {};
    g.M = (int)M;
    g.b_rows = (int)N;
    g.K = (int)K;
    g.epi = (int)epi;
    g.groups = (int)groups;
    g.pair = (int)pair;
    g.cluster = (int)cluster;
    g.silu_pairs = silu_pairs;
    TORCH_CHECK(M > 0 && N > 0 && K > 0 && epi >= 0 && epi <= 2 && pair >= -1 && pair <= 1, "gemm_tile_choice: sizes, epi, pair");
    const penny::sm100::TileGemm c = penny::sm100::gemm_tile_choice(g);
    return std::make_tuple(c.block_n, c.pair, c.cluster);
  }, py::arg("M"), py::arg("N"), py::arg("K"), py::arg("epi") = 0, py::arg("groups") = 0, py::arg("pair") = 0,
     py::arg("cluster") = 0, py::arg("silu_pairs") = false,
     "(block_n, pair, cluster) of gemm_tile(block_n=0) without norm_w; N: rows of b, per group");
  m.def("gemm_decode_splits", [](int64_t B, int64_t N, int64_t K, bool folded) {
    return penny::sm100::gemm_decode_splits((int)B, (int)N, (int)K, folded);
  }, py::arg("B"), py::arg("N"), py::arg("K"), py::arg("folded") = false,
     "cluster size of gemm_decode(splits=0); folded: with sumsq or residual");
  m.def("gemm_decode_capacity", [](int64_t B, int64_t splits) {
    return penny::sm100::gemm_decode_capacity((int)B, (int)splits);
  });
  m.def("gemm_decode_stamps", [](int64_t max_ctas) {
    auto t = torch::zeros({max_ctas, 8}, torch::TensorOptions().dtype(torch::kInt64));
    cudaDeviceSynchronize();
    const int n = penny::sm100::gemm_decode_stamps(reinterpret_cast<unsigned long long*>(t.data_ptr<int64_t>()), (int)max_ctas);
    return t.narrow(0, 0, n);
  }, py::arg("max_ctas") = 512, "timestamps of the last gemm_decode launch (needs PENNY_DEC_STAMPS=1)");
  m.def("set_pdl", [](int64_t on) { penny::set_pdl_enabled((int)on); }, py::arg("on"),
        "1 / 0: launch this library's decode kernels with / without programmatic dependent launch; -1: PENNY_PDL decides");
  m.def("pdl_enabled", []() { return penny::pdl_enabled(); });
  m.def("gemm_set_split_tail", [](int64_t on) { penny::sm100::set_split_tail((int)on); }, py::arg("on"),
        "1 / 0: split (or not) the ragged last wave of the CTA-pair GEMM along K; -1: PENNY_GEMM_SPLIT_TAIL decides");
  m.def("gemm_pair_enabled", []() { return penny::sm100::pair_kernel_enabled(); },
        "False when PENNY_GEMM_PAIR=0 keeps the GEMMs on single-CTA tiles");
  // Synchronises; returns and clears the error code of the GEMM kernels (0 = fine).
  m.def("gemm_error", []() {
    uint32_t* word = penny_gemm_error_word();
    const cudaStream_t stream = at::cuda::getCurrentCUDAStream().stream();
    int v = 0;
    cudaError_t rc = cudaMemcpyAsync(&v, word, sizeof(v), cudaMemcpyDeviceToHost, stream);
    if (rc == cudaSuccess) rc = cudaStreamSynchronize(stream);
    if (rc == cudaSuccess && v != 0) rc = cudaMemsetAsync(word, 0, sizeof(v), stream);
    TORCH_CHECK(rc == cudaSuccess, "gemm_error: ", cudaGetErrorString(rc));
    return v;
  });
  // The word itself as an int32 tensor [1] of the current device, to be looked at without a synchronisation.
  m.def("gemm_error_word", []() {
    int dev = 0;
    cudaGetDevice(&dev);
    return at::from_blob(penny_gemm_error_word(), {1}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, dev));
  });
}
