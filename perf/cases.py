"""The work that users of this framework have it do, as cases to be timed: single ``aten::linear`` and ``aten::lstm``
calls, RNN-T greedy decoding, and greedy translation with the GNMT and the Transformer model.

Sizes come from the repository's benchmark configurations (``pimaicompiler_b200/synthetic.py``, ``bench.py``).  Weights
are random, but decisions have the margins of a trained model instead of the near-ties of random logits, so that two
correct implementations choose the same tokens: some units of the RNN-T encoder relay what the features say about speech and
label, and the translators' output layers favour successors of the last target token, among which (in the Transformer) a
topic that runs through the source sentence chooses.  The rest of the network overrules that now and then.
"""
import itertools
import math

import numpy as np
import torch

from pimaicompiler_b200 import ops, synthetic
from pimaicompiler_b200.gnmt import GnmtTranslator
from pimaicompiler_b200.rnnt import RnntDecoder
from pimaicompiler_b200.transformer import TransformerTranslator

DEV = "cuda"
RNNT, GNMT, TRANSFORMER = synthetic.RnntConfig(), synthetic.GnmtConfig(), synthetic.TransformerConfig()
LISTED_UTTERANCES, LISTED_FRAMES = 1024, 1000        # the benchmark's RNN-T job; drawn ones are no larger
GNMT_MARGIN, TRANSFORMER_MARGIN = 1.2, 1.2           # how strongly the output layers favour the successor token
TOPICS, TOPIC_DIMS = 8, 3                            # the Transformer's last dimensions hold the topic's three bits
LABEL_BITS = 5


def listed():
    return [
        # one decoder layer's matrix times one vector, bias and ReLU fused: the shortest call that is used in earnest
        {"name": "linear 4096x1024, 1 row", "kind": "linear", "form": "mv", "n": 4096, "k": 1024, "rows": 1, "relu": True},
        # the vocabulary projection of a decode step of 32 streams
        {"name": "linear 32320x1024, 32 rows", "kind": "linear", "form": "wx", "n": 32320, "k": 1024, "rows": 32, "relu": False},
        # one token of one stream through a decoder layer with attention context
        {"name": "lstm step, 1 stream", "kind": "lstm", "layers": 1, "bidirectional": False, "input": 2048, "hidden": 1024,
         "steps": 1, "batch": 1, "packed": False},
        # the RNN-T pre-net on two seconds of speech, one stream
        {"name": "lstm 2 layers, 200 steps", "kind": "lstm", "layers": 2, "bidirectional": False, "input": 240, "hidden": 1024,
         "steps": 200, "batch": 1, "packed": False},
        # the first encoder layer of the GNMT model over a batch of sentences of 20 to 50 tokens
        {"name": "lstm bidirectional, packed", "kind": "lstm", "layers": 1, "bidirectional": True, "input": 1024, "hidden": 1024,
         "steps": 50, "batch": 96, "packed": True},
        # dictation: one utterance of 10 s, latency is all that counts
        {"name": "rnnt 1 utterance", "kind": "rnnt", "utterances": 1, "frames": 1000, "voiced": 0.35},
        # a server's batch of shorter utterances
        {"name": "rnnt 37 utterances", "kind": "rnnt", "utterances": 37, "frames": 727, "voiced": 0.35},
        # the benchmark's job on one GPU, where every frame emits a label
        {"name": "rnnt 1024 utterances", "kind": "rnnt", "utterances": LISTED_UTTERANCES, "frames": LISTED_FRAMES, "voiced": 1.0},
        # an interactive translation service: a handle for 16 sentences, nine requests waiting
        {"name": "gnmt 9 sentences", "kind": "gnmt", "sentences": 9, "group": 16, "steps": 80},
        # the benchmark's job on one GPU
        {"name": "gnmt 512 sentences", "kind": "gnmt", "sentences": 512, "group": 512, "steps": 80},
        {"name": "transformer 20 sentences", "kind": "transformer", "sentences": 20, "group": 20, "steps": 64},
        {"name": "transformer 2048 sentences", "kind": "transformer", "sentences": 2048, "group": 2048, "steps": 64},
    ]


def _between(rng, lo, hi):
    """A whole number of lo..hi, spread evenly over the logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("linear", "linear", "lstm", "lstm", "rnnt", "gnmt", "transformer"))
    if kind == "linear":
        form = rng.choice(("mv", "vm", "wx", "wx"))
        k = _between(rng, 64, 4096)
        return {"kind": kind, "form": form, "n": _between(rng, 29, 32768), "k": k if rng.random() < 0.25 else k // 8 * 8,
                "rows": 1 if form != "wx" else _between(rng, 2, 2048), "relu": rng.random() < 0.5}
    if kind == "lstm":
        packed = rng.random() < 0.3
        return {"kind": kind, "layers": rng.choice((1, 1, 2, 3)), "bidirectional": rng.random() < 0.25,
                "input": rng.choice((240, 320, 512, 1024, 2048)), "hidden": rng.choice((320, 512, 1024, 1024)),
                "steps": _between(rng, 20, 64) if packed else rng.choice((1, _between(rng, 2, 600))), "batch": _between(rng, 1, 128), "packed": packed}
    if kind == "rnnt":
        frames = _between(rng, 100, 1600)
        return {"kind": kind, "utterances": _between(rng, 1, LISTED_UTTERANCES * LISTED_FRAMES // max(frames, LISTED_FRAMES)), "frames": frames,
                "voiced": round(rng.uniform(0.2, 1.0), 2)}
    n = _between(rng, 1, 512 if kind == "gnmt" else 2048)
    group = rng.choice((n, n, -(-n // 16) * 16, max(1, -(-n // 2))))
    return {"kind": kind, "sentences": n, "group": group, "steps": rng.randint(20, 80 if kind == "gnmt" else 64)}


# ------------------------------------------------------------------------------------------------------------- weights
def _uniform(gen, shape, fan_in, gain=1.0):
    return (torch.rand(*shape, generator=gen, device=DEV) * 2 - 1).mul_(gain / math.sqrt(fan_in)).half()


def _normal(gen, shape, scale=1.0):
    return (torch.randn(*shape, generator=gen, device=DEV) * scale).half()


def _lstm_weights(gen, layers, directions, inputs, hidden, gain=1.0):
    ps = []
    for layer in range(layers):
        for _ in range(directions):
            n = inputs if layer == 0 else directions * hidden
            ps += [_uniform(gen, (4 * hidden, n), hidden, gain), _uniform(gen, (4 * hidden, hidden), hidden, gain),
                   _uniform(gen, (4 * hidden,), hidden, gain), _uniform(gen, (4 * hidden,), hidden, gain)]
    return ps


def _relay_units(ps, hidden, n):
    """Unit j < n of every layer passes on the sign of its input's element j, without memory: input and output gates
    open, forget gate shut."""
    for layer in range(len(ps) // 4):
        w_ih, w_hh, b_ih, b_hh = ps[4 * layer:4 * layer + 4]
        for gate, bias in enumerate((6.0, -6.0, 0.0, 6.0)):
            unit = slice(gate * hidden, gate * hidden + n)
            w_ih[unit], w_hh[unit], b_ih[unit], b_hh[unit] = 0.0, 0.0, bias, 0.0
        w_ih[2 * hidden:2 * hidden + n, :n].fill_diagonal_(8.0)


def _rnnt_decoder(gen):
    c, gain, sharp = RNNT, 2.0, 8.0
    pre = _lstm_weights(gen, c.pre_layers, 1, c.feat_dim, c.enc_hidden, gain)
    post = _lstm_weights(gen, c.post_layers, 1, c.stack_factor * c.enc_hidden, c.enc_hidden, gain)
    _relay_units(pre, c.enc_hidden, 1 + LABEL_BITS)
    _relay_units(post, c.enc_hidden, 1 + LABEL_BITS)
    fan = c.enc_hidden + c.pred_hidden
    w1, b1 = _uniform(gen, (c.joint_hidden, fan), fan, gain), _uniform(gen, (c.joint_hidden,), fan, gain)
    w2, b2 = (_uniform(gen, s, c.joint_hidden, gain * sharp) for s in ((c.vocab, c.joint_hidden), (c.vocab,)))
    n = 2 * (1 + LABEL_BITS)                  # a relayed sign takes two hidden units of the joint network, one for +, one for -
    w1[:n], b1[:n], w2[:, :n] = 0.0, 0.0, 0.0
    w1[0:n:2, :n // 2].fill_diagonal_(8.0)
    w1[1:n:2, :n // 2].fill_diagonal_(-8.0)
    w2[c.blank, 0], b2[c.blank] = -8.0, 24.0  # speech takes the blank from +24 to -24
    bits = _label_bits(torch.arange(c.vocab, device=DEV))
    w2[:c.blank, 2:n:2], w2[:c.blank, 3:n:2] = 0.4 * bits[:c.blank], -0.4 * bits[:c.blank]
    return RnntDecoder(c, pre, post, _normal(gen, (c.vocab, c.pred_hidden)),
                       _lstm_weights(gen, c.pred_layers, 1, c.pred_hidden, c.pred_hidden), w1, b1, w2, b2)


def _label_bits(label):
    """The bits of a label as signs, in a last dimension of their own."""
    return ((label[..., None] >> torch.arange(LABEL_BITS, device=label.device)) & 1).half() * 2 - 1


def _gnmt_weights(gen):
    H, V = GNMT.hidden, GNMT.vocab
    lstm = lambda inputs: _lstm_weights(gen, 1, 1, inputs, H, 1.5)  # noqa: E731
    w = {"emb_src": _normal(gen, (V, H), 0.5), "emb_tgt": _normal(gen, (V, H), 0.5), "enc0_f": lstm(H), "enc0_r": lstm(H),
         "enc1": lstm(2 * H), "enc2": lstm(H), "enc3": lstm(H), "dec0": lstm(H), "dec1": lstm(2 * H), "dec2": lstm(2 * H),
         "dec3": lstm(2 * H), "Wq": _uniform(gen, (H, H), H), "Wk": _uniform(gen, (H, H), H), "att_b": _uniform(gen, (H,), H),
         "att_v": _uniform(gen, (H,), H), "att_g": torch.tensor(1.0), "bc": _uniform(gen, (V,), H)}

    def cell(name, x):      # the layer's output from a zero state and a zero attention context
        w_ih, _, b_ih, b_hh = w[name]
        i, _, g, o = (x @ w_ih[:, :H].T + (b_ih + b_hh)).float().chunk(4, 1)
        return (o.sigmoid() * (i.sigmoid() * g.tanh()).tanh()).half()

    # the row of a token's successor points to where that token alone takes the decoder's output
    x = cell("dec1", cell("dec0", w["emb_tgt"]))
    for name in ("dec2", "dec3"):
        x = x + cell(name, x)
    x = x.float() - x.float().mean(0)
    out = torch.empty(V, H, device=DEV)
    out[torch.randperm(V, generator=gen, device=DEV)] = GNMT_MARGIN * x / x.norm(dim=1, keepdim=True)
    w["Wc"] = (out + _uniform(gen, (V, H), H, 2.0)).half()
    return w


def _transformer_weights(gen):
    d, f, V, n = TRANSFORMER.d_model, TRANSFORMER.ffn, TRANSFORMER.vocab, TRANSFORMER.layers

    def layer(names):
        shapes = dict({name: (d, d) for name in names}, f1=(f, d), f2=(d, f))
        w = {name: _uniform(gen, s, s[1]) for name, s in shapes.items()}
        return dict(w, **{name + "_b": _uniform(gen, s[:1], s[1]) for name, s in shapes.items()})

    self_names, V8 = ("sq", "sk", "sv", "so"), V // TOPICS
    emb_src, emb_tgt, bucket = _normal(gen, (V, d), 0.3), _normal(gen, (V, d), 0.4), _normal(gen, (V8, d), 0.6)
    emb_tgt += bucket[torch.randperm(V, generator=gen, device=DEV) % V8]      # what may follow this token: eight tokens, one per topic
    out = (TRANSFORMER_MARGIN * bucket.float() / bucket.float().norm(dim=1, keepdim=True)).repeat_interleave(TOPICS, 0)
    out += _uniform(gen, (V, d), d)
    pe = synthetic.positional_table(max(TRANSFORMER.max_len, TRANSFORMER.max_steps), d)
    enc, dec = [layer(self_names) for _ in range(n)], [layer(self_names + ("cq", "ck", "cv", "co")) for _ in range(n)]
    # the topic's dimensions: set by the source embedding, left alone by every layer, passed on by the cross-attention
    topic = slice(d - TOPIC_DIMS, d)
    signs = ((torch.arange(V, device=DEV)[:, None] >> torch.arange(TOPIC_DIMS, device=DEV)) & 1) * 2.0 - 1
    emb_src[:, topic], emb_tgt[:, topic], pe[:, topic], out[:, topic] = (2 * signs).half(), 0.0, 0.0, 0.25 * signs
    for w in enc + dec:
        for name in ("so", "f2", "cv", "co"):
            if name in w:
                w[name][topic], w[name + "_b"][topic] = 0.0, 0.0
                if name in ("cv", "co"):
                    w[name][topic, topic].fill_diagonal_(1.0)
    return {"emb_src": emb_src, "emb_tgt": emb_tgt, "pe": pe, "Wo": out.half(), "enc": enc, "dec": dec}


# ------------------------------------------------------------------------------------------------------------- prepare
def prepare(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    rnd = np.random.RandomState(seed % (1 << 32))
    ops.init()
    state = {"case": case}
    if case["kind"] == "linear":
        n, k, rows = case["n"], case["k"], case["rows"]
        state["w"] = _uniform(gen, (k, n) if case["form"] == "vm" else (n, k), k)
        state["x"] = _normal(gen, (rows, k) if case["form"] == "wx" else (k,))
        state["b"] = _uniform(gen, (n,), k)
    elif case["kind"] == "lstm":
        L, D, H, B, T = case["layers"], 2 if case["bidirectional"] else 1, case["hidden"], case["batch"], case["steps"]
        state["lstm"] = ops.Lstm(_lstm_weights(gen, L, D, case["input"], H), L, D == 2, case["input"], H)
        rows = (T, B)
        if case["packed"]:
            sizes = _batch_sizes(case)
            state["batch_sizes"] = torch.from_numpy(sizes)
            rows = (int(sizes.sum()),)
        state["x"] = _normal(gen, rows + (case["input"],))
        state["h"], state["c"] = _normal(gen, (L * D, B, H), 0.1), _normal(gen, (L * D, B, H), 0.1)
    elif case["kind"] == "rnnt":
        n, T = case["utterances"], case["frames"]
        state["decoder"] = _rnnt_decoder(gen)
        state["x"] = torch.randn(n, T, RNNT.feat_dim, generator=gen, device=DEV, dtype=torch.float16)
        pairs = (n, T // 2 + 1)
        speech = (torch.rand(*pairs, generator=gen, device=DEV) < case["voiced"]).half() * 2 - 1
        label = torch.randint(0, RNNT.blank, pairs, generator=gen, device=DEV)
        said = torch.cat([speech[..., None], _label_bits(label)], 2)
        state["x"][:, :, :1 + LABEL_BITS] = said.repeat_interleave(2, 1)[:, :T]
        state["tokens"] = torch.zeros(n, T // RNNT.stack_factor, dtype=torch.int32, device=DEV)
        state["counts"] = torch.zeros(n, dtype=torch.int32, device=DEV)
    else:
        cfg, make, translator = ((GNMT, _gnmt_weights, GnmtTranslator) if case["kind"] == "gnmt"
                                 else (TRANSFORMER, _transformer_weights, TransformerTranslator))
        state["translator"] = translator(cfg, make(gen), group=case["group"])
        lengths = rnd.randint(cfg.min_len, cfg.max_len + 1, case["sentences"])
        topics = rnd.randint(0, TOPICS, case["sentences"]).repeat(lengths)
        ids = torch.from_numpy(rnd.randint(1, cfg.vocab // TOPICS, int(lengths.sum())) * TOPICS + topics)
        state["sentences"] = list(ids.split(lengths.tolist()))
    return state


def _batch_sizes(case):
    """Lengths spread evenly from all steps down to two fifths of them, as sequences per step."""
    lengths = case["steps"] - np.arange(case["batch"]) * (case["steps"] * 3 // 5) // case["batch"]
    return (lengths[:, None] > np.arange(case["steps"])).sum(0)


def run(state):
    case = state["case"]
    if case["kind"] == "linear":
        act = ops.ACT_RELU if case["relu"] else ops.ACT_NONE
        if case["form"] == "mv":
            return ops.gemv_mv(state["w"], state["x"], state["b"], act)
        if case["form"] == "vm":
            return ops.gemv_vm(state["x"], state["w"], state["b"], act)
        return ops.gemm_wx(state["w"], state["x"], state["b"], act)
    if case["kind"] == "lstm":
        if case["packed"]:
            return state["lstm"].forward_packed(state["x"], state["batch_sizes"], state["h"], state["c"])
        return state["lstm"].forward(state["x"], state["h"], state["c"])
    if case["kind"] == "rnnt":
        state["decoder"].decode_into(state["x"], state["tokens"], state["counts"])
        return {"tokens": state["tokens"], "counts": state["counts"]}
    lists = state["translator"].translate(state["sentences"], steps=case["steps"])
    flat = np.fromiter(itertools.chain.from_iterable(lists), np.int64, case["sentences"] * case["steps"])
    return flat.reshape(case["sentences"], case["steps"])


# ---------------------------------------------------------------------------------------------------------------- work
def _lstm_size(layers, directions, inputs, hidden):
    return sum(directions * 4 * hidden * ((inputs if layer == 0 else directions * hidden) + hidden + 2) for layer in range(layers))


def work(case):
    """Every input, weight and output once (a translator's and the RNN-T's weights once per pass, although every step
    needs them: they could stay on the chip), and two operations per weight and row that it is applied to."""
    if case["kind"] == "linear":
        n, k, rows = case["n"], case["k"], case["rows"]
        return {"bytes": 2 * (n * k + n + rows * (n + k)), "flops": 2 * n * k * rows}
    if case["kind"] == "lstm":
        L, D, I, H = case["layers"], 2 if case["bidirectional"] else 1, case["input"], case["hidden"]
        rows = int(_batch_sizes(case).sum()) if case["packed"] else case["batch"] * case["steps"]
        size = _lstm_size(L, D, I, H)
        return {"bytes": 2 * (size + rows * (I + D * H) + 4 * L * D * case["batch"] * H), "flops": 2 * size * rows}
    if case["kind"] == "rnnt":
        c, n, T = RNNT, case["utterances"], case["frames"]
        pre, post = _lstm_size(c.pre_layers, 1, c.feat_dim, c.enc_hidden), _lstm_size(c.post_layers, 1, c.stack_factor * c.enc_hidden, c.enc_hidden)
        enc, out = c.joint_hidden * c.enc_hidden, c.joint_hidden * c.vocab
        pred = _lstm_size(c.pred_layers, 1, c.pred_hidden, c.pred_hidden) + c.joint_hidden * c.pred_hidden
        frames = T // c.stack_factor
        return {"bytes": 2 * (pre + post + enc + out + pred + n * T * c.feat_dim) + 4 * n * frames,
                "flops": 2 * n * (pre * T + frames * (post + enc + out + case["voiced"] * pred))}
    n, steps = case["sentences"], case["steps"]
    if case["kind"] == "gnmt":
        H, V, S = GNMT.hidden, GNMT.vocab, (GNMT.min_len + GNMT.max_len) / 2
        enc = _lstm_size(1, 2, H, H) + _lstm_size(1, 1, 2 * H, H) + 2 * _lstm_size(1, 1, H, H) + H * H
        dec = _lstm_size(1, 1, H, H) + 3 * _lstm_size(1, 1, 2 * H, H) + H * H + V * H
        # the attention keys and values of every sentence are read anew by every step
        return {"bytes": 2 * (enc + dec + n * (S + steps) * H + 2 * n * steps * S * H), "flops": 2 * n * (enc * S + steps * (dec + 2 * S * H))}
    d, f, V, S, L = TRANSFORMER.d_model, TRANSFORMER.ffn, TRANSFORMER.vocab, (TRANSFORMER.min_len + TRANSFORMER.max_len) / 2, TRANSFORMER.layers
    enc, dec = L * (4 * d * d + 2 * d * f), L * (6 * d * d + 2 * d * f) + V * d
    # so are the keys and values of the source and of the tokens so far
    rows = steps * (S + steps / 2)
    return {"bytes": 2 * (enc + L * 2 * d * d + dec + n * (S + steps) * d + 2 * n * L * rows * d),
            "flops": 2 * n * (S * (enc + L * 2 * d * d) + steps * dec + 2 * L * rows * d)}


def tolerance(case):
    """fp16 in and out, 32-bit sums: half a unit in the last place is 2.4e-4 to 4.9e-4; a recurrence feeds its rounded
    state back, step after step.  Tokens are whole numbers; a near-tie may fall the other way and take the tokens behind
    it along."""
    if case["kind"] == "linear":
        return {"rel": 1e-3, "max": 1e-2}
    if case["kind"] == "lstm":
        return {"rel": 2e-3, "max": 4e-2}
    return {"rel": 0.0, "differ": 0.01}
