"""The work this framework is used for on one GPU, as cases that a timing harness can call.

Three public entry points carry a user's program here:

  decode   LlamaTPDecoder.step(): one token for every sequence of a batch, host tokens in, host tokens
           out, the whole step in a CUDA graph.  Small batches are a stream of weights, large ones
           meet the tensor cores, long contexts are a stream of the KV cache.
  prefill  LlamaSPPrefill.forward(): a prompt through transformer layers (column- and row-parallel
           linears with their collectives fused in, RoPE, causal attention, norms).
  moe      MoeEPLayer.forward(): router, dispatch, expert FFNs, combine, from a handful of decode
           tokens to a prefill batch.

The collectives between GPUs need several of them, and their time on one GPU (all ranks emulated in one
launch) says nothing about NVLink; they enter here as the world-of-one form inside prefill and moe.

Shapes are those of benchmarks and tests of this repository: Llama-3-8B-shaped and Mixtral-8x7B-shaped
layers, batch 1 / 8 / 64 / 256, a 2048-token cache, prompts of whole 128-row blocks, bf16 (the type of
all three paths).  Decode and prefill run a stack of 8 and 4 equal layers: the time of a deeper one is
that many times a layer's.
"""
import math

import torch

from penny_b200.models.llama_sp import LlamaSPPrefill
from penny_b200.models.llama_tp import LlamaConfig, LlamaTPDecoder
from penny_b200.models.moe_ep import MoeConfig, MoeEPLayer
from penny_b200.parallel.comm import Communicator

DECODE_LAYERS = 8
PREFILL_LAYERS = 4
MAX_KV_ROWS = 256 * 1024  # batch x context of the largest decode: what a server's KV pool would hold


def listed():
    return [
        # one user, a short chat: all latency and weights
        {"name": "decode_b1_kv100", "kind": "decode", "batch": 1, "kv": 100, "mixed": False},
        # a few users at the context length of the headline benchmark
        {"name": "decode_b8_kv2048", "kind": "decode", "batch": 8, "kv": 2048, "mixed": False},
        # the headline benchmark's batch and context
        {"name": "decode_b64_kv2048", "kind": "decode", "batch": 64, "kv": 2048, "mixed": False},
        # continuous batching: an odd number of sequences, every one at another position
        {"name": "decode_b37_mixed4096", "kind": "decode", "batch": 37, "kv": 4096, "mixed": True},
        # long documents: few sequences, long caches
        {"name": "decode_b3_kv15000", "kind": "decode", "batch": 3, "kv": 15000, "mixed": False},
        # the largest batch of the benchmark series
        {"name": "decode_b256_kv1024", "kind": "decode", "batch": 256, "kv": 1024, "mixed": False},
        # a short prompt (or one chunk of a chunked prefill)
        {"name": "prefill_t128", "kind": "prefill", "tokens": 128},
        # an ordinary prompt, an odd number of row blocks
        {"name": "prefill_t1152", "kind": "prefill", "tokens": 1152},
        # the prefill benchmark's prompt, the longest that the row-parallel linear takes at this width
        {"name": "prefill_t4096", "kind": "prefill", "tokens": 4096},
        # a decode step of a handful of sequences
        {"name": "moe_t5", "kind": "moe", "tokens": 5},
        # a decode step of a busy server, ragged expert loads
        {"name": "moe_t203", "kind": "moe", "tokens": 203},
        # a prefill batch
        {"name": "moe_t4096", "kind": "moe", "tokens": 4096},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "prefill", "moe"])
    if kind == "decode":
        batch = _log_uniform(rng, 1, 256)
        kv = _log_uniform(rng, 16, min(16000, MAX_KV_ROWS // batch))
        return {"kind": "decode", "batch": batch, "kv": kv, "mixed": rng.random() < 0.5}
    if kind == "prefill":
        return {"kind": "prefill", "tokens": 128 * _log_uniform(rng, 1, 32)}
    # (the layer's default receive capacity, twice the balanced load in multiples of 8 rows, needs 2 tokens)
    return {"kind": "moe", "tokens": _log_uniform(rng, 2, 4096)}


def prepare(case, seed):
    return {"decode": _prepare_decode, "prefill": _prepare_prefill, "moe": _prepare_moe}[case["kind"]](case, seed)


def run(state):
    return state["run"](state)


def _prepare_decode(case, seed):
    """A captured decoder with a filled cache, as bench.py makes it, and this step's tokens and positions."""
    cfg = LlamaConfig.llama3_8b()
    cfg.layers = DECODE_LAYERS
    batch, kv = case["batch"], case["kv"]
    model = LlamaTPDecoder(cfg, max_batch=batch, max_len=kv + 64, seed=seed)
    model.fill_synthetic_kv(kv, seed=seed)
    g = torch.Generator().manual_seed(seed)
    positions = torch.full((batch,), kv, dtype=torch.int32)
    if case["mixed"]:
        positions = torch.randint(1, kv + 1, (batch,), generator=g, dtype=torch.int32)
    model.positions.copy_(positions)
    model.capture()
    return {"run": _run_decode, "model": model, "positions": positions.cuda(),
            "tokens": torch.randint(0, cfg.vocab, (batch,), generator=g)}


def _run_decode(state):
    model = state["model"]
    model.positions.copy_(state["positions"])  # the scheduler's view of the batch; step() advances it
    model.step(state["tokens"])
    # The step's results before the last comparison.  The token ids it returns are the arg-max of these
    # logits: with random weights the two largest of 128256 bf16 values are often equal or one rounding
    # apart, so the ids of two correct implementations differ.
    return {"logits": model.logits, "max": model.max_val, "residual": model.residual, "positions": model.positions,
            "k_first": model.kcache[0], "v_first": model.vcache[0], "k_last": model.kcache[-1],
            "v_last": model.vcache[-1]}


def _prepare_prefill(case, seed):
    cfg = LlamaConfig.llama3_8b()
    tokens = case["tokens"]
    comm = Communicator.emulated(1, heap_bytes=max(256 << 20, tokens * (128 << 10)), timeout_ms=5000)
    model = LlamaSPPrefill(cfg, comm=comm, tokens=tokens, layers=PREFILL_LAYERS, seed=seed)
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(tokens, cfg.hidden, device="cuda", generator=g).bfloat16()
    return {"run": _run_prefill, "model": model, "x": x}


def _run_prefill(state):
    return state["model"].forward(state["x"])


def _prepare_moe(case, seed):
    cfg = MoeConfig.mixtral_8x7b()
    tokens = case["tokens"]
    comm = Communicator.emulated(1, heap_bytes=max(64 << 20, tokens * (64 << 10)), timeout_ms=5000)
    layer = MoeEPLayer(cfg, comm, tokens=tokens, seed=seed)
    g = torch.Generator(device="cuda").manual_seed(seed)
    # hidden states share a direction, so the router prefers some experts: their loads differ severalfold
    common = torch.randn(1, cfg.hidden, device="cuda", generator=g)
    x = (torch.randn(tokens, cfg.hidden, device="cuda", generator=g) + 0.5 * common).bfloat16()
    return {"run": _run_moe, "layer": layer, "x": [x]}


def _run_moe(state):
    return state["layer"].forward(state["x"])


def work(case):
    """Each weight and cached row read once, each input and output moved once; multiply-adds count two."""
    if case["kind"] == "moe":
        cfg, t = MoeConfig.mixtral_8x7b(), case["tokens"]
        expert = 3 * cfg.hidden * cfg.ffn
        used = cfg.experts * (1.0 - (1.0 - cfg.topk / cfg.experts) ** t)  # experts that some token picks
        return {"bytes": 2 * (used * expert + cfg.experts * cfg.hidden + 2 * t * cfg.hidden),
                "flops": 2 * t * (cfg.topk * expert + cfg.experts * cfg.hidden)}
    cfg = LlamaConfig.llama3_8b()
    width, kv_width = cfg.heads * cfg.head_dim, cfg.kv_heads * cfg.head_dim
    layer = cfg.hidden * (2 * width + 2 * kv_width + 3 * cfg.ffn)
    if case["kind"] == "prefill":
        t = case["tokens"]
        return {"bytes": 2 * (PREFILL_LAYERS * layer + 2 * t * cfg.hidden),
                "flops": PREFILL_LAYERS * (2 * t * layer + 4 * width * t * (t + 1) // 2)}
    b = case["batch"]
    rows = b * ((case["kv"] + 1) / 2 if case["mixed"] else case["kv"])  # cached rows that are attended
    head = cfg.vocab * cfg.hidden
    return {"bytes": 2 * (DECODE_LAYERS * (layer + 2 * kv_width * (rows + b)) + head + b * (2 * cfg.hidden + cfg.vocab)),
            "flops": 2 * b * (DECODE_LAYERS * layer + head) + 4 * DECODE_LAYERS * width * (rows + b)}


def tolerance(case):
    # bf16 activations and a bf16 residual: every layer rounds a handful of times, and random layers carry a
    # difference of one rounding on at its own size.  Two orders of the same fp32 sums in the linears (this
    # library's GEMM and the vendor's) measured 1.2e-2 apart after 4 such layers and 1.8e-2 after 8.
    if case["kind"] == "decode":
        return {"rel": 2.5e-2, "max": 0.2}
    if case["kind"] == "prefill":
        return {"rel": 2e-2, "max": 0.2}
    return {"rel": 1e-2, "max": 0.2}
