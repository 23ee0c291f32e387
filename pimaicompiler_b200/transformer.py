"""Transformer-base greedy translation (configuration C5) for many sequences per GPU, every op through libpimb200.so.

The reference runs its Transformer graph for one sequence (input [1, 11] token ids,
examples/runtime/source/pipeline_manager.cpp:216-217): per generated token the interpreter dispatches each linear as a
batch-1 addmm, each attention as matmul -> softmax -> matmul with per-head reshapes, and grows the key / value cache with
an at::cat (runtime/source/executor/op_executor/aten_ops_executor.cpp:181-216, 2488-2505, 3402-3436, 772-819).  Sequences
are independent, so a GPU runs `group` of them in lock step:

  * encoder: the tokens of the group's sequences, one sequence behind the other without padding, are the rows of every
    product; each layer is one fused q/k/v projection GEMM, one attention launch (a CTA per head and sequence, own rows),
    the output projection, the feed-forward pair (ReLU fused into the first GEMM) and two fused residual-add + layer-norm
    launches;
  * the cross-attention keys and values of all decoder layers come from one GEMM over the encoder output;
  * decoder: all `steps` steps of the group are captured into ONE CUDA graph.  Step t's projection GEMM writes q, k, v
    straight into row t of every sequence's part of a [group, steps, 3d] cache (no append, no device-side position),
    single-query attention reads rows 0..t of it, and the vocabulary projection, the arg max (which writes row t of the
    token table) and the next step's embedding are two launches that leave no logits in memory.

`TransformerTranslator.translate` is the user call; `bench.py --workload c5` times it.
"""
from __future__ import annotations

from typing import List, Optional, Sequence

import numpy as np
import torch

from . import ops
from .gnmt import flat_tokens


def stage_groups(sequences: Sequence[torch.Tensor], G: int, max_len: int, pin: bool = False):
    """Lock-step groups, longest sequences first: dicts of `idx` (sequence indices), `S` (longest length) and the tensors
    `ids` and `pos` (token and position of every row, one sequence behind the other), `lengths` [G] and `row0` [G] (first row
    of every sequence), with `pin` in pinned host memory.  A ragged last group is filled with one-token dummies."""
    n = len(sequences)
    lens = np.fromiter((s.shape[0] for s in sequences), np.int64, n)
    if n and (lens.max() > max_len or lens.min() < 1):
        raise ValueError("sequence length outside 1..max_len")
    order = np.argsort(-lens, kind="stable").tolist()
    keep = (lambda t: t.pin_memory()) if pin else (lambda t: t)
    dummy = torch.full((1,), 4, dtype=torch.int64)
    groups = []
    for g0 in range(0, n, G):
        idx = order[g0:g0 + G]
        lens_g = np.ones(G, np.int64)
        lens_g[:len(idx)] = lens[idx]
        row0 = np.cumsum(lens_g) - lens_g
        ids = torch.cat([flat_tokens([sequences[i] for i in idx])] + [dummy] * (G - len(idx)))
        pos = np.arange(ids.numel()) - np.repeat(row0, lens_g)
        groups.append({"idx": idx, "S": int(lens_g[0]), "ids": keep(ids), "pos": keep(torch.from_numpy(pos)),
                       "lengths": keep(torch.from_numpy(lens_g)), "row0": keep(torch.from_numpy(row0))})
    return groups


class TransformerTranslator:
    def __init__(self, cfg, weights: dict, group: int = 128, device: Optional[torch.device] = None):
        ops.init()
        self.cfg = cfg
        self.G = int(group)
        self.dev = device or torch.device("cuda", torch.cuda.current_device())
        d, G, S, T = cfg.d_model, self.G, cfg.max_len, cfg.max_steps
        self.d = d

        def put(t):
            return t.to(torch.float16).to(self.dev).contiguous()

        w = weights
        self.emb_src, self.emb_tgt, self.pe, self.Wo = put(w["emb_src"]), put(w["emb_tgt"]), put(w["pe"]), put(w["Wo"])

        def fuse(L, names):
            return put(torch.cat([L[n] for n in names])), put(torch.cat([L[n + "_b"] for n in names]))

        self.enc = []
        for L in w["enc"]:
            qkv, qkv_b = fuse(L, ("sq", "sk", "sv"))
            self.enc.append({"qkv": qkv, "qkv_b": qkv_b, **{k: put(L[k]) for k in ("so", "so_b", "f1", "f1_b", "f2", "f2_b")}})
        self.dec = []
        for L in w["dec"]:
            qkv, qkv_b = fuse(L, ("sq", "sk", "sv"))
            self.dec.append({"qkv": qkv, "qkv_b": qkv_b,
                             **{k: put(L[k]) for k in ("so", "so_b", "cq", "cq_b", "co", "co_b", "f1", "f1_b", "f2", "f2_b")}})
        # cross-attention key / value projections of all decoder layers side by side: [layers * 2d, d]
        self.ckv = put(torch.cat([torch.cat([L["ck"], L["cv"]]) for L in w["dec"]]))
        self.ckv_b = put(torch.cat([torch.cat([L["ck_b"], L["cv_b"]]) for L in w["dec"]]))
        f16 = dict(dtype=torch.float16, device=self.dev)
        i64 = dict(dtype=torch.int64, device=self.dev)
        nl = cfg.layers
        self.lengths = torch.ones(G, **i64)
        self.row0 = torch.zeros(G, **i64)                            # first encoder row of every sequence
        self.cross = torch.zeros(G * S, nl * 2 * d, **f16)           # encoder side, packed rows, at its maximum size
        self.cache = [torch.zeros(G, T, 3 * d, **f16) for _ in range(nl)]
        self.toks = torch.zeros(T + 1, G, **i64)                     # row 0: start tokens, row t+1: choice of step t
        self.forced = torch.zeros(T + 1, G, **i64)
        self.x0 = torch.zeros(G, d, **f16)                           # the step's input: embedding of the last token + position
        self.token_ws = ops.greedy_token_workspace(cfg.vocab, G, self.dev)
        self.logits = None                                           # [G, vocab], where the arg max needs them in memory
        self.logits_all = None
        self._graphs = {}
        self.launches_per_step = 0
        torch.cuda.current_stream(self.dev).synchronize()            # weights are in place before a launch reads them ahead of its turn

    # ------------------------------------------------------------------------------------------------ encoder
    def encode(self, group: dict) -> None:
        """One staged group (see stage(); tensors on the device).  Fills the cross-attention keys / values of every decoder
        layer."""
        cfg, d = self.cfg, self.d
        n = group["ids"].numel()
        self.lengths.copy_(group["lengths"])
        self.row0.copy_(group["row0"])
        x = ops.add_f16(ops.gather_rows(self.emb_src, group["ids"]), ops.gather_rows(self.pe, group["pos"]))    # [n, d]
        for L in self.enc:
            qkv = ops.gemm_wx_fixed(L["qkv"], x, L["qkv_b"])
            a = ops.attention_block_packed(qkv[:, :d], qkv[:, d:2 * d], qkv[:, 2 * d:], cfg.heads, self.row0, self.lengths, group["S"])
            x = ops.add_layer_norm(x, ops.gemm_wx_fixed(L["so"], a, L["so_b"]))
            f = ops.gemm_wx_fixed(L["f2"], ops.gemm_wx_fixed(L["f1"], x, L["f1_b"], ops.ACT_RELU), L["f2_b"])
            x = ops.add_layer_norm(x, f)
        ops.gemm_wx_fixed(self.ckv, x, self.ckv_b, out=self.cross[:n])

    # ------------------------------------------------------------------------------------------------ decoder
    def _step(self, t: int, forced: bool, want_logits: bool) -> int:
        cfg, d, G = self.cfg, self.d, self.G
        n = 0
        if t == 0 or forced or want_logits or self.logits is not None:
            x = ops.gather_rows(self.emb_tgt, (self.forced if forced else self.toks)[t]); n += 1
            x = ops.add_f16(x, self.pe[t]); n += 1
        else:
            x = self.x0                                                          # left there by the previous step
        for i, L in enumerate(self.dec):
            row = self.cache[i][:, t]                                            # [G, 3d]: q, k, v of step t
            ops.gemm_wx_fixed(L["qkv"], x, L["qkv_b"], out=row); n += 1
            a = ops.attention_rows(row[:, :d], self.cache[i][:, :, d:2 * d], self.cache[i][:, :, 2 * d:], cfg.heads,
                                   len_add=t + 1); n += 1
            x = ops.add_layer_norm(x, ops.gemm_wx_fixed(L["so"], a, L["so_b"])); n += 2
            cq = ops.gemm_wx_fixed(L["cq"], x, L["cq_b"]); n += 1
            ck = self.cross[:, (2 * i) * d:(2 * i + 1) * d]
            cv = self.cross[:, (2 * i + 1) * d:(2 * i + 2) * d]
            ca = ops.attention_rows_packed(cq, ck, cv, cfg.heads, self.row0, self.lengths, cfg.max_len); n += 1
            x = ops.add_layer_norm(x, ops.gemm_wx_fixed(L["co"], ca, L["co_b"])); n += 2
            f = ops.gemm_wx_fixed(L["f2"], ops.gemm_wx_fixed(L["f1"], x, L["f1_b"], ops.ACT_RELU), L["f2_b"]); n += 2
            x = ops.add_layer_norm(x, f); n += 1
        if not want_logits and self.logits is None:
            nxt = None if forced or t + 1 >= cfg.max_steps else self.pe[t + 1]
            if ops.greedy_token(self.Wo, x, None, self.token_ws, self.toks[t + 1], None if nxt is None else self.emb_tgt, nxt,
                                None if nxt is None else self.x0):
                return n + 2
            self.logits = torch.zeros(G, cfg.vocab, dtype=torch.float16, device=self.dev)
        lg = self.logits_all[t] if want_logits else self.logits
        ops.gemm_wx_fixed(self.Wo, x, out=lg); n += 1
        ops.argmax(lg, out=self.toks[t + 1]); n += 1
        return n

    def _graph(self, steps: int, forced: bool, want_logits: bool):
        key = (steps, forced, want_logits)
        if key in self._graphs:
            return self._graphs[key]
        side = torch.cuda.Stream(device=self.dev)
        side.wait_stream(torch.cuda.current_stream(self.dev))
        with torch.cuda.stream(side):          # eager once: workspaces exist before the capture
            self._step(0, forced, want_logits)
        torch.cuda.current_stream(self.dev).wait_stream(side)
        torch.cuda.synchronize(self.dev)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            for t in range(steps):
                self.launches_per_step = self._step(t, forced, want_logits)
        self._graphs[key] = g
        return g

    def decode(self, steps: int, forced: Optional[torch.Tensor] = None, want_logits: bool = False):
        """All `steps` greedy steps of the encoded group (one graph launch).  Returns the token table [steps, G] (device)
        and, when asked, the logits [steps, G, V]."""
        cfg, G = self.cfg, self.G
        if steps > cfg.max_steps:
            raise ValueError("more steps than the configuration's maximum")
        if want_logits and (self.logits_all is None or self.logits_all.shape[0] < steps):
            self.logits_all = torch.zeros(steps, G, cfg.vocab, dtype=torch.float16, device=self.dev)
            self._graphs = {k: v for k, v in self._graphs.items() if not k[2]}
        self.toks[0].fill_(cfg.bos)
        if forced is not None:
            self.forced[0].fill_(cfg.bos)
            self.forced[1:steps].copy_(forced[:steps - 1].to(self.dev))          # step t is fed the token forced at t - 1
        self._graph(steps, forced is not None, want_logits).replay()
        toks = self.toks[1:steps + 1]
        return (toks, self.logits_all[:steps]) if want_logits else (toks, None)

    # ------------------------------------------------------------------------------------------------ user call
    def stage(self, sequences: Sequence[torch.Tensor]):
        """Packs the sequences into lock-step groups (see stage_groups)."""
        return stage_groups(sequences, self.G, self.cfg.max_len, pin=True)

    def to_device(self, group: dict) -> dict:
        return {k: v.to(self.dev, non_blocking=True) if isinstance(v, torch.Tensor) else v for k, v in group.items()}

    def h2d_bytes(self, group: dict) -> int:
        return 8 * sum(v.numel() for v in group.values() if isinstance(v, torch.Tensor))

    def check_status(self) -> None:
        """Raises if a bounded wait of the tensor-core GEMM gave up since the last check."""
        from . import _lib
        rc = _lib.lib().pimb200_gemm_last_status()
        if rc != 0:
            raise RuntimeError(f"device-side wait timed out (gemm status {rc})")

    def translate(self, sequences: Sequence[torch.Tensor], steps: Optional[int] = None,
                  forced: Optional[Sequence[Sequence[int]]] = None, want_logits: bool = False):
        """sequences: 1-D tensors of source token ids.  Returns one token list per sequence (cut behind the first
        end-of-sequence token unless `steps` is given) and, when asked, each one's logits [steps, V]."""
        cfg, G = self.cfg, self.G
        n = len(sequences)
        run_steps = cfg.max_steps if steps is None else steps
        out_toks: List[Optional[List[int]]] = [None] * n
        out_logits: List[Optional[torch.Tensor]] = [None] * n
        pending = []
        for group in self.stage(sequences):
            idx = group["idx"]
            self.encode(self.to_device(group))
            f = None
            if forced is not None:
                f = torch.zeros(run_steps, G, dtype=torch.int64)
                for j, i in enumerate(idx):
                    f[:, j] = torch.tensor(list(forced[i])[:run_steps], dtype=torch.int64)
            toks, logits = self.decode(run_steps, f, want_logits)
            host = torch.empty(toks.shape, dtype=torch.int64, pin_memory=True)
            host.copy_(toks, non_blocking=True)
            pending.append((idx, host, logits.float().cpu() if want_logits else None))
            torch.cuda.current_stream(self.dev).synchronize()   # the next group reuses the token table
            self.check_status()
        for idx, host, logits in pending:
            rows = host.t().tolist()                        # [G][steps] in one call
            for j, i in enumerate(idx):
                seq = rows[j]
                if steps is None and cfg.eos in seq:
                    seq = seq[:seq.index(cfg.eos) + 1]
                out_toks[i] = seq
                if logits is not None:
                    out_logits[i] = logits[:, j]
        return (out_toks, out_logits) if want_logits else out_toks
