"""Mixtral-8x7B-shaped MoE layer with expert parallelism.

Every rank holds `experts / world` experts (SwiGLU FFNs) and its own tokens.
One forward pass:

    router (top-k of softmax-normalised logits)
    -> routing tables (which row goes where; a tiny all-gather of per-expert counts)
    -> dispatch: rows pushed over NVLink straight into the owners' dense
       expert-input buffers                                   (one kernel)
    -> expert FFN on the received rows (tcgen05 GEMMs of this library)
    -> combine: outputs pushed back to their sources and summed with the gate
       weights in the same kernel                             (one kernel)

`backend="nccl"` does the two exchanges with all_to_all_single (padded to equal
splits is not needed: it uses the split-size form) and the weighted sum as a
separate op – the baseline.  Works with a real communicator (one process per
GPU) or an emulated one (all ranks on one GPU: every tensor argument is then a
list).  The reference has no MoE path; its exchange is a pairwise swap
(csrc/exchange.cu).
"""
from __future__ import annotations

from dataclasses import dataclass
from typing import List

import torch

from .._ext import ops


@dataclass
class MoeConfig:
    hidden: int = 4096
    ffn: int = 14336
    experts: int = 8
    topk: int = 2
    init_std: float = 0.02

    @classmethod
    def mixtral_8x7b(cls):
        return cls()

    @classmethod
    def tiny(cls):
        return cls(hidden=256, ffn=512, experts=8, topk=2)


def route(logits: torch.Tensor, topk: int):
    """Top-k routing: expert ids [T, k] (int32) and gate weights [T, k] (fp32,
    softmax over the selected logits, as Mixtral does).  One kernel for bf16 CUDA logits
    (csrc/moe_routing.cu), torch ops otherwise."""
    if logits.is_cuda and logits.dtype == torch.bfloat16 and logits.is_contiguous() and topk <= 8:
        return ops.moe_route(logits, topk)
    return route_torch(logits, topk)


def route_torch(logits: torch.Tensor, topk: int):
    vals, ids = logits.float().topk(topk, dim=-1)
    return ids.to(torch.int32).contiguous(), torch.softmax(vals, dim=-1).contiguous()


def build_routing(topk_ids: torch.Tensor, experts: int):
    """Sender-side tables for one rank: pairs sorted by expert (stable), per-expert counts.
    One kernel (a counting sort in one thread block) instead of sort + bincount + cumsum."""
    if topk_ids.is_cuda and topk_ids.dtype == torch.int32 and experts <= 256:
        return ops.moe_tables(topk_ids.reshape(-1).contiguous(), experts)
    return build_routing_torch(topk_ids, experts)


def build_routing_torch(topk_ids: torch.Tensor, experts: int):
    flat = topk_ids.reshape(-1).to(torch.int64)
    expert_sorted, order = torch.sort(flat, stable=True)
    counts = torch.bincount(flat, minlength=experts)
    send_off = torch.zeros(experts + 1, dtype=torch.int64, device=flat.device)
    send_off[1:] = counts.cumsum(0)
    return (order.to(torch.int32).contiguous(), expert_sorted.to(torch.int32).contiguous(),
            send_off.to(torch.int32).contiguous(), counts)


def _placement(counts_all: torch.Tensor):
    """placement_device with the ranges of all experts as a device tensor [E, 2] as well."""
    W, E = counts_all.shape
    dst_base, rows, ranges = ops.moe_placement(counts_all.contiguous())
    host = torch.cat([rows, ranges.reshape(-1)]).cpu().tolist()
    rows_per_rank, flat = host[:W], host[W:]
    epr = E // W
    expert_ranges = [[(flat[2 * (d * epr + le)], flat[2 * (d * epr + le) + 1]) for le in range(epr)] for d in range(W)]
    return dst_base, rows_per_rank, expert_ranges, ranges


def placement_device(counts_all: torch.Tensor):
    """`placement` on the device: counts_all [W, E] int32 (CUDA) -> dst_base [W, E] int32 (stays on
    the device for the dispatch kernel), and - the one host round trip of the layer, for the capacity
    check - rows_per_rank and per-rank expert ranges."""
    return _placement(counts_all)[:3]


def placement(counts_all: torch.Tensor, world: int):
    """counts_all[s, e] = rows rank s sends to expert e.  Returns
    dst_base[s, e] (row at e's owner where s's rows of e start), rows_per_rank[d]
    and expert_rows[d] = per-local-expert row ranges (start, end) at rank d.
    Rows at an owner are ordered by local expert, then by source rank."""
    W, E = counts_all.shape
    epr = E // world
    dst_base = torch.zeros_like(counts_all)
    rows_per_rank, expert_ranges = [], []
    for d in range(world):
        base = 0
        ranges = []
        for le in range(epr):
            e = d * epr + le
            start = base
            for s in range(W):
                dst_base[s, e] = base
                base += int(counts_all[s, e])
            ranges.append((start, base))
        rows_per_rank.append(base)
        expert_ranges.append(ranges)
    return dst_base, rows_per_rank, expert_ranges


def expert_tiles(rows: int, experts: int, hidden: int, ffn: int, sms: int):
    """Tile of the grouped GEMMs and cluster of the down projection for `rows` rows on a rank's `experts` experts.

    128-row tiles of single CTAs, 256 columns wide: most experts' rows fill one or two.  256-row tiles of CTA
    pairs once the average expert fills three (8 experts, gate/up + down: 1000 tokens 804 us against 857,
    2000 tokens 1278 / 1379, 3000 tokens 1723 / 1678; at 5 to 500 tokens pairs cost 70 to 90 us of 334 to 510).
    PENNY_GEMM_PAIR=0 leaves them out.

    Where at most half of the SMs have a tile of the down projection, two CTAs share a tile's K steps (hidden 4096, ffn
    14336, down alone: 4 experts 156 us -> 97; with 6 of them 125 -> 146, there are enough tiles then; whole layer
    of 4 experts and 100 rows 292 -> 275).  Handing the sums over costs about 13 of the steps of 64 that half of K
    must save (whole layer, 2 tokens, ffn 1024 / 1664 / 2048 / 4096: 68.3 / 76.0 / 79.3 / 120.1 us without, 69.4 /
    75.8 / 77.7 / 108.4 with), and a cluster works on one row tile."""
    shared = rows <= 128 and 2 * min(rows, experts) * -(-hidden // 256) <= sms and ffn > 2 * 13 * 64
    return (512 if rows > 640 * experts and ops.gemm_pair_enabled() else 256), (2 if shared else 0)


def expert_rows(rows: int, experts: int, hidden: int = 4096, most: int | None = None):
    """Rows per tile of gate/up and of down where one rank's grouped GEMMs have the weight on the M side, 0 where
    `expert_tiles` holds.  `most`: the rows that an expert can have at most (a token picks an expert once), None: as many as
    a tile has.

    There a group's rows are paid to the next 16 instead of 128 or 256, and few rows leave the shared memory to the
    weights; but an expert with more rows than a tile has its weights staged again for each further one, so tiles are as
    long as the longest expert can be, or 128 rows, as `expert_tiles` has them.  Whole layers against `expert_tiles`: 8 experts,
    hidden 4096, ffn 14336 / 16, 6144, 10752 / 64, 2048, 1024 / 64, 2048, 1408 / 128, 2048, 768 / 8, 1024, 3584; in brackets the
    range over them with nearly all rows at as many experts as a token picks.
      up to 64 tokens, tiles that hold them      0.88 to 1.01 (0.77 to 0.99; 16 rows for 24 to 64 of them up to 1.17)
      up to 6 rows per expert, 128 rows          0.97 to 1.00 (0.90 to 0.98; 16 rows 0.97 to 1.01 and up to 1.30)
      15 / 30 rows per expert, 128 in gate/up    0.98 to 1.00 / 0.99 to 1.01 (0.95 to 1.04 / 0.97 to 1.04)
      40 / 48 / 51 / 56                          0.96 to 1.00 / 0.99 to 1.00 / 0.98 to 1.01 / 0.98 to 1.02 (0.96 to 1.09)
      64 / 75, 128 in gate/up; 256 in both       0.99 to 1.02 (0.99 to 1.11); 0.95 to 1.06 (0.89 to 1.05)
      88 / 96 / 105 / 128, 256 in both           8 of 4096: 1.04 / 0.90 / 0.91 / 0.89 (0.86 to 0.97), 16 of 6144: 1.03 / 1.00 / 0.97 / 0.95
                                                 (0.87 to 1.04), hidden 2048: 1.01 to 1.04 / 1.01 to 1.02 / 1.01 to 1.05 / 0.98 to 1.01
      190 / 256 / 512 / 1024, 256 in both        0.84 to 0.99 (0.85 to 1.05), hidden 1024: 0.97 / 1.06 / 1.20 / 1.11 (1.10 to 1.20)
    Layers under hidden 1024 were not timed."""
    per = rows / experts
    if not ops.gemm_pair_enabled() or hidden < 1024:
        return 0, 0
    if most is not None and most <= 64:
        return ((most + 15) // 16 * 16,) * 2
    if per <= 6:
        return (16, 16) if most is None else (128, 128)
    if per <= 52:
        return 128, 0
    return (256, 256) if hidden >= 2048 and per >= (88 if hidden >= 4096 else 128) else (0, 0)


class MoeEPLayer:
    def __init__(self, cfg: MoeConfig, comm, tokens: int, cap_factor: float = 2.0, backend: str = "penny",
                 seed: int = 0, use_own_gemm: bool = True):
        self.cfg, self.comm, self.backend = cfg, comm, backend
        self.world = comm.world_size
        self.views = comm.views
        self.tokens = tokens
        self.epr = cfg.experts // self.world
        assert cfg.experts % self.world == 0
        self.use_own_gemm = use_own_gemm
        dev = torch.device("cuda", torch.cuda.current_device())
        self.dev = dev
        self.sms = torch.cuda.get_device_properties(dev).multi_processor_count
        pairs = tokens * cfg.topk
        self.cap_rows = int(cap_factor * pairs) // 8 * 8
        dt = torch.bfloat16
        # symmetric buffers the peers write into
        self.recv = self._as_views(comm.empty(self.cap_rows, cfg.hidden, dtype=dt))
        self.meta = self._as_views(comm.empty(self.cap_rows, dtype=torch.float32))  # int32 payload
        self.meta = [m.view(torch.int32) for m in self.meta]
        self.comb = self._as_views(comm.empty(pairs, cfg.hidden, dtype=dt))
        self.counts_buf = self._as_views(comm.empty(cfg.experts, dtype=torch.float32))
        self.dst_row_of_pair = [torch.zeros(pairs, dtype=torch.int32, device=dev) for _ in range(self.views)]
        # weights: router replicated; experts sharded
        self.ranks = list(range(self.world)) if comm.emulated else [comm.rank]
        g = torch.Generator(device=dev)
        self.router, self.w13, self.w2 = [], [], []
        for r in self.ranks:
            g.manual_seed(seed * 7919 + 1)
            self.router.append((torch.randn(cfg.experts, cfg.hidden, device=dev, generator=g) * cfg.init_std).to(dt))
            # one tensor per kind and rank, the experts' matrices are views of it: the grouped GEMMs address
            # all of them through one descriptor.  (Weights copied into the views keep that; a list whose entries
            # are replaced by other tensors is taken one expert after another.)
            w13 = torch.empty(self.epr, 2 * cfg.ffn, cfg.hidden, dtype=dt, device=dev)
            w2 = torch.empty(self.epr, cfg.hidden, cfg.ffn, dtype=dt, device=dev)
            for le in range(self.epr):
                g.manual_seed(seed * 7919 + 100 + r * self.epr + le)
                w13[le] = torch.randn(2 * cfg.ffn, cfg.hidden, device=dev, generator=g) * cfg.init_std
                w2[le] = torch.randn(cfg.hidden, cfg.ffn, device=dev, generator=g) * cfg.init_std
            self.w13.append(list(w13))
            self.w2.append(list(w2))

    def _as_views(self, t) -> List[torch.Tensor]:
        return list(t) if isinstance(t, (list, tuple)) else [t]

    def _gemm(self, a, w):
        out = torch.empty(a.shape[0], w.shape[0], dtype=a.dtype, device=a.device)
        if a.shape[0] == 0:
            return out
        if self.use_own_gemm:
            ops.gemm_bf16(a, w, out, 0)
        else:
            torch.matmul(a, w.t(), out=out)
        return out

    def _stacked(self, v: int):
        """Gate/up and down weights of this rank's experts as [experts * rows, K], or None where an entry of the
        lists does not lie behind the one before it (any more)."""
        w13, w2 = ops.stacked_rows(self.w13[v][:self.epr]), ops.stacked_rows(self.w2[v][:self.epr])
        return None if w13 is None or w2 is None else (w13, w2)

    def _experts_grouped(self, w13: torch.Tensor, w2: torch.Tensor, rows: torch.Tensor, ranges: torch.Tensor):
        """SwiGLU FFN of this rank's local experts (stacked) over its received rows in two launches; `ranges`
        [local experts, 2] stays on the device."""
        cfg = self.cfg
        act = torch.empty(rows.shape[0], cfg.ffn, dtype=rows.dtype, device=rows.device)
        y = torch.empty_like(rows)
        block_n, down_cluster = expert_tiles(rows.shape[0], self.epr, cfg.hidden, cfg.ffn, self.sms)
        ops.gemm_tile(rows, w13, act, 1, ranges, block_n=block_n, pdl=True)
        ops.gemm_tile(act, w2, y, 0, ranges, block_n=block_n, pdl=True, cluster=down_cluster)
        return y

    def _experts(self, v: int, rows: torch.Tensor, ranges):
        """SwiGLU FFN of this rank's local experts over its received rows."""
        y = torch.empty_like(rows)
        for le, (s, e) in enumerate(ranges):
            if e <= s:
                continue
            h = self._gemm(rows[s:e], self.w13[v][le])
            act = torch.empty(e - s, self.cfg.ffn, dtype=rows.dtype, device=rows.device)
            ops.silu_mul(h, act)
            y[s:e] = self._gemm(act, self.w2[v][le])
        return y

    def forward(self, x):
        """x: [tokens, hidden], tokens at most those the layer was built for (a list with one tensor per virtual rank
        when emulated)."""
        cfg, comm = self.cfg, self.comm
        xs = self._as_views(x)
        for xv in xs:
            if xv.shape[0] > self.tokens:  # the exchange's buffers and tables are that long
                raise RuntimeError(f"MoE layer built for {self.tokens} tokens, called with {xv.shape[0]}")
        x0, pairs = xs[0], xs[0].shape[0] * cfg.topk
        if (self.world == 1 and self.backend == "penny" and self.use_own_gemm and 0 < pairs <= self.cap_rows
                and x0.dtype == torch.bfloat16 and x0.is_contiguous() and x0.data_ptr() % 16 == 0
                and cfg.topk <= 8 and cfg.experts <= 256):
            out = ops.moe_layer(x0, self.router[0], self.w13[0][:self.epr], self.w2[0][:self.epr], cfg.topk,
                                *expert_tiles(pairs, self.epr, cfg.hidden, cfg.ffn, self.sms),
                                *expert_rows(pairs, self.epr, cfg.hidden, x0.shape[0]))
            if out is not None:
                return [out] if comm.emulated else out
        ids, gates, tables = [], [], []
        for v, xv in enumerate(xs):
            i, g = route(torch.matmul(xv, self.router[v].t()), cfg.topk)
            ids.append(i)
            gates.append(g)
            tables.append(build_routing(i, cfg.experts))
        # every rank learns how many rows each rank sends to each expert
        if self.world > 1:
            for v in range(len(xs)):
                self.counts_buf[v].view(torch.int32).copy_(tables[v][3].to(torch.int32))
            gathered = comm.all_gather(self.counts_buf if comm.emulated else self.counts_buf[0])
            gathered = self._as_views(gathered)
            counts_dev = gathered[0].view(torch.int32).view(self.world, cfg.experts)
        else:
            counts_dev = tables[0][3].to(torch.int32).view(1, cfg.experts)
        dst_base, rows_per_rank, expert_ranges, ranges_dev = _placement(counts_dev)
        if max(rows_per_rank) > self.cap_rows:
            raise RuntimeError(f"MoE capacity exceeded: {max(rows_per_rank)} rows > {self.cap_rows}")
        dst_base_dev = [dst_base[r].contiguous() for r in self.ranks]
        counts_all = counts_dev.cpu() if self.backend != "penny" else None  # the NCCL baseline wants split sizes
        L = (lambda t: t) if comm.emulated else (lambda t: t[0])
        if self.backend == "penny":
            comm.moe_dispatch(L(xs), L([t[0] for t in tables]), L([t[1] for t in tables]), L([t[2] for t in tables]),
                              L(dst_base_dev), L(self.dst_row_of_pair), L(self.recv), L(self.meta), cfg.topk,
                              cfg.experts)
            ys = []
            for v, r in enumerate(self.ranks):
                rows = self.recv[v][:rows_per_rank[r]]
                # (one grouped launch holds up to 256 groups)
                stacked = self._stacked(v) if self.use_own_gemm and rows.shape[0] > 0 and self.epr <= 256 else None
                if stacked is not None:
                    ys.append(self._experts_grouped(*stacked, rows, ranges_dev[r * self.epr:(r + 1) * self.epr]))
                else:
                    ys.append(self._experts(v, rows, expert_ranges[r]))
            outs = [torch.empty_like(xv) for xv in xs]
            comm.moe_combine(L(ys), L(outs), L([i.reshape(-1).contiguous() for i in ids]),
                             L([g.reshape(-1).contiguous() for g in gates]), L(self.meta), L(self.dst_row_of_pair),
                             L(self.comb), [rows_per_rank[r] for r in self.ranks] if comm.emulated
                             else rows_per_rank[self.ranks[0]], cfg.experts)
            return outs if comm.emulated else outs[0]
        return self._forward_nccl(xs[0], ids[0], gates[0], tables[0], counts_all, rows_per_rank, expert_ranges)

    def _forward_nccl(self, x, ids, gates, table, counts_all, rows_per_rank, expert_ranges):
        """Baseline: the same layer with NCCL all_to_all_single for both exchanges."""
        import torch.distributed as dist
        cfg, r = self.cfg, self.comm.rank
        order, expert_sorted, send_off, _ = table
        send_rows = x[(order.long() // cfg.topk)]
        # per-destination split sizes; received rows arrive ordered by source, then expert
        in_splits = [int(counts_all[r, d * self.epr:(d + 1) * self.epr].sum()) for d in range(self.world)]
        out_splits = [int(counts_all[s, r * self.epr:(r + 1) * self.epr].sum()) for s in range(self.world)]
        recv = torch.empty(sum(out_splits), cfg.hidden, dtype=x.dtype, device=x.device)
        dist.all_to_all_single(recv, send_rows, out_splits, in_splits)
        if self.epr == 1:
            ranges = [(0, recv.shape[0])]
            y = self._experts(0, recv, ranges)
        else:  # regroup by expert
            src_expert = torch.cat([torch.repeat_interleave(torch.arange(self.epr, device=x.device),
                                                            counts_all[s, r * self.epr:(r + 1) * self.epr].to(x.device))
                                    for s in range(self.world)])
            perm = torch.argsort(src_expert, stable=True)
            cnt = torch.bincount(src_expert, minlength=self.epr).tolist()
            ranges, b = [], 0
            for c in cnt:
                ranges.append((b, b + c))
                b += c
            y = torch.empty_like(recv)
            y[perm] = self._experts(0, recv[perm], ranges)
        back = torch.empty_like(send_rows)
        dist.all_to_all_single(back, y, in_splits, out_splits)
        per_pair = torch.empty_like(back)
        per_pair[order.long()] = back
        return (per_pair.view(self.tokens, cfg.topk, cfg.hidden).float() * gates[..., None]).sum(1).to(x.dtype)

    def reference(self, xs: List[torch.Tensor], all_w13, all_w2, router):
        """fp32 PyTorch oracle from FULL expert weights (all_w13[e], all_w2[e])."""
        outs = []
        for x in xs:
            ids, gates = route(torch.matmul(x, router.t()), self.cfg.topk)
            out = torch.zeros(x.shape, dtype=torch.float32, device=x.device)
            for k in range(self.cfg.topk):
                for e in range(self.cfg.experts):
                    sel = (ids[:, k] == e).nonzero().squeeze(1)
                    if sel.numel() == 0:
                        continue
                    h = (x[sel].float() @ all_w13[e].float().t()).to(torch.bfloat16).float()
                    act = (torch.nn.functional.silu(h[:, :self.cfg.ffn]) * h[:, self.cfg.ffn:]).to(torch.bfloat16).float()
                    y = (act @ all_w2[e].float().t()).to(torch.bfloat16).float()
                    out[sel] += gates[sel, k, None] * y
            outs.append(out)
        return outs
