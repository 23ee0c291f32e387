"""GNMT greedy translation (configuration C4) for many sentences per GPU, every op through libpimb200.so.

The reference serves one sentence at a time: its interpreter walks the GNMT graph once per token, each decoder layer one
aten::lstm call with seq_len 1, the attention a chain of add / tanh / matmul / softmax / bmm nodes and the vocabulary
projection a batch-1 addmm (runtime/source/executor/op_executor/aten_ops_executor.cpp:2135-2307, 181-216, 110-166; GNMT
inputs examples/runtime/source/pipeline_manager.cpp:143-151).  Sentences are independent, so a GPU that has to serve
hundreds of them runs `group` sentences in lock step instead:

  * encoder: the group's sentences, sorted by length, go through each layer as packed batches of up to 512 sentences
    (aten::lstm's packed overload, which the library runs as a padded lock-step batch on the persistent weight-stationary
    recurrence, the backward direction of the first layer on the sentences reversed one by one);
  * decoder: one step for the whole group is four cells (each one launch: both products and the gate math; the output, for
    the last two with the residual added, goes straight into the next cell's concatenated input), the query projection, one
    attention launch (which writes the context into the other halves of those inputs), and the vocabulary projection with
    its arg max and the next token's embedding (two launches, no logits in memory).  Sixteen, four, two and one steps are captured
    into CUDA graphs when they are first needed, and any number of steps is made of their replays: the step's number lives
    on the device.  The chosen tokens stay there until the group is done.

`GnmtTranslator.translate` is the user call; `bench.py --workload c4` times it.
"""
from __future__ import annotations

import gc
from typing import List, Optional, Sequence

import numpy as np
import torch

from . import ops


def flat_tokens(sentences: Sequence[torch.Tensor]) -> torch.Tensor:
    """The sentences' tokens one behind the other, as int64 on the host, whatever type and device each sentence has."""
    try:
        flat = torch.cat(list(sentences)) if len(sentences) else torch.zeros(0, dtype=torch.int64)
    except RuntimeError:             # not on one device
        flat = None
    if flat is None or flat.dtype != torch.int64:     # (of several types it would hold them all in a common one)
        flat = torch.cat([s.to("cpu", torch.int64) for s in sentences])
    return flat.cpu()


def stage_groups(sentences: Sequence[torch.Tensor], G: int, enc_batch: int, max_len: int, pin: bool = False):
    """Host-side packing of sentences into lock-step groups of G.  A group is a dict: `idx` (sentence indices, longest
    first), `S` (longest sentence), `lengths` [G] int64, and `slices`: per `enc_batch` sentences the packed token ids
    [sum of lengths] (timestep-major, the order of torch's pack_padded_sequence), `batch_sizes` (CPU int64, one per
    timestep) and `dst`, the row t * G + j of the padded [S, G] buffer each packed row belongs to.  A ragged last group
    is filled with one-token dummies.  With `pin` the tensors that travel to the device are in pinned host memory."""
    keep = (lambda t: t.pin_memory()) if pin else (lambda t: t)
    n = len(sentences)
    lens = np.fromiter((s.shape[0] for s in sentences), np.int64, n)
    if n and (lens.max() > max_len or lens.min() < 1):
        raise ValueError("sentence length outside 1..max_len")
    flat = flat_tokens(sentences).numpy()
    start = np.cumsum(lens) - lens
    order = np.argsort(-lens, kind="stable")
    groups = []
    for g0 in range(0, n, G):
        idx = order[g0:g0 + G]
        lens_all = np.ones(G, np.int64)
        lens_all[:len(idx)] = lens[idx]
        first = np.zeros(G, np.int64)                        # where a sentence's tokens begin in `flat`
        first[:len(idx)] = start[idx]
        slices = []
        for j0 in range(0, G, enc_batch):
            sl_lens, nb = lens_all[j0:j0 + enc_batch], min(enc_batch, G - j0)
            steps_col = np.arange(sl_lens[0])[:, None]
            mask = steps_col < sl_lens                       # [t, b]: sentence b has a step t
            at = (first[j0:j0 + enc_batch] + steps_col)[mask]
            ids = flat[at]
            if j0 + nb > len(idx):                           # one-token dummies
                ids[(steps_col * 0 + np.arange(j0, j0 + nb))[mask] >= len(idx)] = 4
            dst = (steps_col * G + np.arange(j0, j0 + nb))[mask]
            slices.append({"ids": keep(torch.from_numpy(ids)), "dst": keep(torch.from_numpy(dst)),
                           "batch_sizes": torch.from_numpy(mask.sum(1))})
        groups.append({"idx": idx.tolist(), "S": int(lens_all[0]), "lengths": keep(torch.from_numpy(lens_all)), "slices": slices})
    return groups


class GnmtTranslator:
    def __init__(self, cfg, weights: dict, group: int = 128, device: Optional[torch.device] = None):
        ops.init()
        self.cfg = cfg
        self.G = int(group)
        self.dev = device or torch.device("cuda", torch.cuda.current_device())
        H, V, G, S = cfg.hidden, cfg.vocab, self.G, cfg.max_len
        self.H, self.V, self.S = H, V, S

        def put(t):
            return t.to(torch.float16).to(self.dev).contiguous()

        self.w = {k: ([put(t) for t in v] if isinstance(v, list) else put(v)) for k, v in weights.items()}
        self.v_norm = put(weights["att_v"] / weights["att_v"].norm() * float(weights["att_g"]))
        self.lstm = {"enc0": ops.Lstm(self.w["enc0_f"] + self.w["enc0_r"], 1, True, H, H, True)}   # bidirectional first layer
        for name in ("enc1", "enc2", "enc3", "dec0", "dec1", "dec2", "dec3"):
            p = self.w[name]
            self.lstm[name] = ops.Lstm(p, 1, False, p[0].shape[1], H, True)
        self.enc_batch = min(self.ENC_BATCH, max(128, min(self.lstm[f"enc{i}"].packed_capacity() for i in range(4))))
        f16 = dict(dtype=torch.float16, device=self.dev)
        i64 = dict(dtype=torch.int64, device=self.dev)
        # encoder outputs / attention keys of the current group, time-major, at their maximum size
        self.enc_out = torch.zeros(S, G, H, **f16)
        self.keys_proj = torch.zeros(S, G, H, **f16)
        self.lengths = torch.ones(G, **i64)
        # decoder step buffers (addresses fixed: the steps are replayed from a CUDA graph)
        self.x = torch.zeros(G, H, **f16)
        self.q = torch.zeros(G, H, **f16)
        self.scores = torch.zeros(G, S, dtype=torch.float32, device=self.dev)
        self.y = [torch.zeros(1, G, H, **f16) for _ in range(4)]
        self.r2 = torch.zeros(G, H, **f16)
        self.r3 = torch.zeros(G, H, **f16)
        self.cats = torch.zeros(G, 3, 2 * H, **f16)                     # inputs [previous output | context] of the last three cells
        self.cat = [self.cats[:, i] for i in range(3)]
        self.state = [[torch.zeros(1, G, H, **f16) for _ in range(8)] for _ in range(2)]   # h0..3, c0..3, two sets
        self.step_no = torch.zeros(2, **i64)                            # the step's number: word t & 1 for step t, which sets the other
        self.token_ws = ops.greedy_token_workspace(V, G, self.dev)
        self.start = torch.zeros(G, **i64)
        self.toks = torch.zeros(max(cfg.max_steps, 1), G, **i64)        # row t: choice of step t
        self.forced = torch.zeros(cfg.max_steps + 1, G, **i64)          # row t: token fed to step t
        self.tok = torch.zeros(1, G, **i64)                             # a step's tokens, where the arg max is a launch of its own
        self.logits = None                                              # [G, V], there
        self.logits_out = None
        self._graphs = {}
        self.launches_per_step = 0

    # ------------------------------------------------------------------------------------------------ encoder
    ENC_BATCH = 512          # sequences per packed aten::lstm call, where the lock-step recurrences take as many

    def encode(self, group: dict) -> int:
        """One staged group (see stage(); tensors on the device).  Every slice of up to 512 sentences goes through the
        encoder as a PACKED batch (the aten::lstm overload the reference's GNMT graph uses for its encoder): rows of
        padding never reach a GEMM or an add, and the library runs the packed batch on the lock-step recurrences.  The
        encoder states are scattered into the padded time-major buffer the attention kernel reads.  Returns S_g."""
        H, G = self.H, self.G
        Sg = group["S"]
        self.lengths.copy_(group["lengths"])
        flat = self.enc_out.view(-1, H)
        for sl in group["slices"]:
            x = ops.gather_rows(self.w["emb_src"], sl["ids"])                       # packed rows [sum of lengths, H]
            y0, _, _ = self.lstm["enc0"].forward_packed(x, sl["batch_sizes"])       # [rows, 2H]
            y1, _, _ = self.lstm["enc1"].forward_packed(y0, sl["batch_sizes"])
            y2, _, _ = self.lstm["enc2"].forward_packed(y1, sl["batch_sizes"])
            y2 = ops.add_f16(y2, y1)
            y3, _, _ = self.lstm["enc3"].forward_packed(y2, sl["batch_sizes"])
            ops.scatter_rows(flat, sl["dst"], ops.add_f16(y3, y2))                  # row (t, j) of the padded buffer
        n = Sg * G
        ops.gemm_wx(self.w["Wk"], self.enc_out[:Sg].view(n, H), out=self.keys_proj[:Sg].view(n, H))
        return Sg

    # ------------------------------------------------------------------------------------------------ decoder
    def _step(self, t: int, forced: bool, want_logits: bool) -> int:
        """A decode step of the whole group; of its number t only the last bit matters, so that replays of a graph can stand
        for any step.  Returns its launch count."""
        H, G, w = self.H, self.G, self.w
        src, dst = self.state[t & 1], self.state[1 - (t & 1)]
        step, next_step = self.step_no[t & 1:(t & 1) + 1], self.step_no[1 - (t & 1):2 - (t & 1)]
        row, half = 3 * 2 * H * 2, H * 2        # bytes from row to row of a concatenated input, of half of it
        n = 0
        cat = self.cat
        if forced:                              # teacher forcing: the token comes from a table
            ops.gather_rows(self.forced, step, out=self.tok)
            ops.gather_rows(w["emb_tgt"], self.tok[0], out=self.x); n += 2
        # groups of 8 or more sentences: every cell writes its output (the last two with their residual added) straight
        # into the first half of the next cell's concatenated input, as the reference's labelled GNMT graph does
        fused = self.lstm["dec0"].forward_step(self.x, src[0][0], src[4][0], cat[0][:, :H], dst[0][0], dst[4][0])
        n += 1
        y0 = cat[0][:, :H]
        if not fused:
            self.lstm["dec0"].forward(self.x.view(1, G, H), src[0], src[4], out=(self.y[0], dst[0], dst[4]))
            ops.copy_2d(self.cats, 0, row, self.y[0], 0, half, half, G); n += 1
        ops.gemm_wx_fixed(w["Wq"], y0, out=self.q); n += 1
        ops.additive_attention(self.q, self.keys_proj, self.enc_out, self.lengths, self.v_norm, w["att_b"],
                               out=cat[0][:, H:], scores=self.scores, copies=3, copy_stride=2 * H); n += 1
        if fused:
            self.lstm["dec1"].forward_step(cat[0], src[1][0], src[5][0], cat[1][:, :H], dst[1][0], dst[5][0])
            self.lstm["dec2"].forward_step(cat[1], src[2][0], src[6][0], cat[2][:, :H], dst[2][0], dst[6][0],
                                           residual=cat[1][:, :H])
            self.lstm["dec3"].forward_step(cat[2], src[3][0], src[7][0], self.r3, dst[3][0], dst[7][0],
                                           residual=cat[2][:, :H]); n += 3
        else:
            def cell(i):                         # of whole rows: the concatenated input is a slice
                x = cat[i - 1].contiguous().view(1, G, 2 * H)
                self.lstm[f"dec{i}"].forward(x, src[i], src[4 + i], out=(self.y[i], dst[i], dst[4 + i]))
                return self.y[i].view(G, H)
            y1 = cell(1)
            ops.copy_2d(self.cats, 2 * half, row, y1, 0, half, half, G)
            ops.add_f16(cell(2), y1, out=self.r2)
            ops.copy_2d(self.cats, 4 * half, row, self.r2, 0, half, half, G)
            ops.add_f16(cell(3), self.r2, out=self.r3); n += 10
        nxt = (None, None) if forced else (w["emb_tgt"], self.x)
        if not want_logits and self.logits is None:
            if ops.greedy_token(w["Wc"], self.r3, w["bc"], self.token_ws, self.toks, nxt[0], None, nxt[1], step, next_step):
                return n + 2
        if self.logits is None:
            self.logits = torch.zeros(G, self.V, dtype=torch.float16, device=self.dev)
        ops.gemm_wx(w["Wc"], self.r3, w["bc"], out=self.logits)
        ops.argmax(self.logits, out=self.tok[0])
        ops.scatter_rows(self.toks, step, self.tok); n += 3
        if want_logits:
            ops.scatter_rows(self.logits_out.view(self.logits_out.shape[0], -1), step, self.logits.view(1, -1)); n += 1
        if not forced:
            ops.gather_rows(w["emb_tgt"], self.tok[0], out=self.x); n += 1
        torch.add(step, 1, out=next_step)
        return n + 1

    CHUNKS = (16, 4, 2, 1)   # steps per graph: of the last one, if any, the state ends up in the other set

    def _graph(self, steps: int, forced: bool, want_logits: bool):
        """`steps` steps, captured once per (steps, forced, logits) mode."""
        key = (steps, forced, want_logits)
        if key in self._graphs:
            return self._graphs[key]
        side = torch.cuda.Stream(device=self.dev)
        side.wait_stream(torch.cuda.current_stream(self.dev))
        with torch.cuda.stream(side):
            if not any(k[1:] == key[1:] for k in self._graphs):
                self.step_no.zero_()
                self._step(0, forced, want_logits)   # outside the capture: buffers of the LSTM handles grow here
            side.synchronize()
            g = torch.cuda.CUDAGraph()
            collecting = gc.isenabled()
            gc.disable()                             # (a handle of some garbage would free device memory inside the capture)
            try:
                g.capture_begin()
                try:
                    for t in range(steps):
                        self.launches_per_step = self._step(t, forced, want_logits)
                finally:
                    g.capture_end()
            finally:
                if collecting:
                    gc.enable()
        torch.cuda.current_stream(self.dev).wait_stream(side)
        self._graphs[key] = g
        return g

    def decode(self, steps: int, forced: Optional[torch.Tensor] = None, want_logits: bool = False):
        """Greedy decode of the encoded group for `steps` steps.  Returns the token table [steps, G] (device, int64) and,
        when asked, the logits [steps, G, V]."""
        cfg, G = self.cfg, self.G
        if steps > cfg.max_steps:
            raise ValueError("more steps than the configuration's maximum")
        if not want_logits:
            if self.logits_out is not None:          # 2.6 GB for 512 sentences
                self.logits_out = None
                self._graphs = {k: v for k, v in self._graphs.items() if not k[2]}
        elif self.logits_out is None or self.logits_out.shape[0] < steps:
            self.logits_out = torch.zeros(steps, G, self.V, dtype=torch.float16, device=self.dev)
            self._graphs = {k: v for k, v in self._graphs.items() if not k[2]}
        if forced is not None:
            self.forced[0].fill_(cfg.bos)
            self.forced[1:max(steps, 1)].copy_(forced[:max(steps - 1, 0)].to(self.dev))   # step t is fed the token forced at t - 1
        graphs, left = [], max(steps, 0)
        for c in self.CHUNKS:
            graphs += [self._graph(c, forced is not None, want_logits)] * (left // c) if left >= c else []
            left %= c
        for s in self.state[0]:
            s.zero_()
        self.step_no.zero_()
        self.start.fill_(cfg.bos)
        ops.gather_rows(self.w["emb_tgt"], self.start, out=self.x)
        for g in graphs:
            g.replay()
        toks = self.toks[:steps]
        return (toks, self.logits_out[:steps]) if want_logits else (toks, None)

    # ------------------------------------------------------------------------------------------------ user call
    def stage(self, sentences: Sequence[torch.Tensor]):
        """Sorts the sentences by length and packs them into lock-step groups (see stage_groups)."""
        return stage_groups(sentences, self.G, self.enc_batch, self.S, pin=True)

    def to_device(self, group: dict) -> dict:
        """The group's tensors copied to the device (batch_sizes stays on the host, as aten::lstm takes it)."""
        mv = lambda t: t.to(self.dev, non_blocking=True)
        return {"idx": group["idx"], "S": group["S"], "lengths": mv(group["lengths"]),
                "slices": [{"ids": mv(sl["ids"]), "dst": mv(sl["dst"]), "batch_sizes": sl["batch_sizes"]} for sl in group["slices"]]}

    def h2d_bytes(self, group: dict) -> int:
        return 8 * (group["lengths"].numel() + sum(sl["ids"].numel() + sl["dst"].numel() for sl in group["slices"]))

    def run_group(self, group_dev: dict, steps: int, forced: Optional[torch.Tensor] = None, want_logits: bool = False):
        """Encoder + greedy decode of one staged group whose tensors are already on the device."""
        self.encode(group_dev)
        return self.decode(steps, forced, want_logits)

    def check_status(self) -> None:
        """Raises if a bounded device-side wait of a recurrence or of the tensor-core GEMM gave up since the last check
        (the launches that followed have run, but the results of the one that gave up are not valid)."""
        from . import _lib
        bad = [name for name, h in self.lstm.items() if h.last_status() != 0]
        rc = _lib.lib().pimb200_gemm_last_status()
        if bad or rc != 0:
            raise RuntimeError(f"device-side wait timed out (recurrences: {bad}, gemm status {rc})")

    def translate(self, sentences: Sequence[torch.Tensor], steps: Optional[int] = None,
                  forced: Optional[Sequence[Sequence[int]]] = None, want_logits: bool = False):
        """sentences: 1-D tensors of source token ids.  Returns one token list per sentence (cut behind the
        first end-of-sentence token unless `steps` is given, which decodes exactly that many steps) and, when asked,
        the logits [steps, V] of each."""
        cfg, G = self.cfg, self.G
        n = len(sentences)
        run_steps = cfg.max_steps if steps is None else steps
        out_toks: List[Optional[List[int]]] = [None] * n
        out_logits: List[Optional[torch.Tensor]] = [None] * n
        pending = []
        for group in self.stage(sentences):
            idx = group["idx"]
            f = None
            if forced is not None:
                f = torch.zeros(run_steps, G, dtype=torch.int64)
                for j, i in enumerate(idx):
                    f[:, j] = torch.tensor(list(forced[i])[:run_steps], dtype=torch.int64)
            toks, logits = self.run_group(self.to_device(group), run_steps, f, want_logits)
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
