"""
The work that this framework is measured by: its layers and losses, each through the entry point that a model calls, one beam-search
ranking, the feature extraction, and one whole training pass of the Conformer-CTC model.

Sizes are those of the training configurations of this repository (Conformer-CTC 12x512 and BLSTM-CTC 6x1024 on 40k / 20k frames per
batch, 10k BPE labels; Transformer MT 512 with 32k labels on 25k tokens per batch) and, for the drawn cases, the range around them from
one short utterance to a full batch. Sequence lengths are ragged as in those configurations. Dropout is off throughout: with it the
outputs are random numbers that two programs cannot be compared by.
"""

from __future__ import annotations
from typing import Any, Dict, List
import math
import numpy
import torch
import torch.nn.functional as F

from returnn_b200.models.packing import PackInfo

DEV = "cuda"


# ---------------------------------------------------------------------------------------------------------------- the cases


def listed() -> List[Dict[str, Any]]:
    return [
        # the up-projection of a feed-forward block with its activation, one training pass over a full Conformer batch (40k feature
        # frames after 6x subsampling)
        dict(name="linear_ff_train", kind="linear", rows=6656, n_in=512, n_out=2048, act="silu", train=True),
        # self-attention of one Transformer MT encoder layer, one training pass over 25k tokens: many short sentences
        dict(name="attention_mt_train", kind="attention", batch=250, t_q=100, t_k=100, heads=8, causal=False, lens=True, train=True),
        # causal self-attention of one decoder / language model layer over long sequences
        dict(name="attention_lm_train", kind="attention", batch=8, t_q=1000, t_k=1000, heads=8, causal=True, lens=False, train=True),
        # relative-position self-attention of one Conformer layer over a full batch
        dict(name="rel_pos_train", kind="rel_pos", batch=36, t=333, heads=8, train=True),
        # the middle of one Conformer convolution module (GLU, depthwise convolution, BatchNorm, SiLU) over a full batch
        dict(name="conv_module_train", kind="conv_module", batch=36, t=333, channels=512, taps=32, train=True),
        # one layer norm, a training pass over a full batch
        dict(name="layer_norm_train", kind="layer_norm", rows=6656, n=512, dtype="bf16", train=True),
        # CTC loss and its gradient over a full batch, 10k labels + blank
        dict(name="ctc_train", kind="ctc", batch=36, t=333, vocab=10001, labels_per_frame=0.2),
        # smoothed cross entropy of the MT model's output layer with its gradient
        dict(name="cross_entropy_train", kind="cross_entropy", rows=6001, vocab=32000, smoothing=0.1),
        # one bidirectional LSTM layer of the BLSTM-CTC model after its time reductions, training pass
        dict(name="blstm_train", kind="blstm", batch=16, t=400, n_in=2048, hidden=1024, train=True),
        # log-mel features of a batch of 10 s utterances at 16 kHz
        dict(name="log_mel", kind="log_mel", batch=64, samples=160000),
        # the ranking of one label step of a beam search: the smallest call, where launches and latency count
        dict(name="beam_rank", kind="beam_rank", batch=1, beam=12, vocab=10001),
        # forward and backward pass of the whole Conformer-CTC model: features to logits, loss and all gradients
        dict(name="conformer_ctc_train", kind="conformer", batch=36, t=2000, layers=12),
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> Dict[str, Any]:
    kind = rng.choice(["linear", "linear", "attention", "attention", "attention", "rel_pos", "rel_pos", "conv_module", "conv_module", "layer_norm", "ctc",
                       "cross_entropy", "blstm", "log_mel", "beam_rank", "conformer"])
    train = rng.random() < 0.7
    if kind == "linear":
        n_in, n_out = rng.choice([(512, 512), (512, 1024), (512, 1536), (512, 2048), (2048, 512), (512, 10000), (1024, 4096)])
        return dict(kind=kind, rows=_log_int(rng, 1, 25000), n_in=n_in, n_out=n_out, act=rng.choice([None, "silu", "relu"]), train=train)
    if kind == "attention":
        t_q = _log_int(rng, 5, 1000)
        causal = rng.random() < 0.4
        t_k = t_q if (causal or rng.random() < 0.5) else _log_int(rng, 10, 1000)
        most = min(250, max(1, 25000 // max(t_q, t_k)), max(1, 8_000_000 // (t_q * t_k)))
        return dict(kind=kind, batch=_log_int(rng, 1, most), t_q=t_q, t_k=t_k, heads=rng.choice([4, 8, 12]), causal=causal, lens=not causal or rng.random() < 0.3,
                    train=train)
    if kind == "rel_pos":
        t = _log_int(rng, 20, 500)
        return dict(kind=kind, batch=_log_int(rng, 1, max(1, 12000 // t)), t=t, heads=rng.choice([4, 6, 8]), train=train)
    if kind == "conv_module":
        t = _log_int(rng, 20, 1000)
        return dict(kind=kind, batch=_log_int(rng, 1, max(1, 12000 // t)), t=t, channels=rng.choice([256, 512]), taps=rng.choice([7, 9, 15, 31, 32]), train=train)
    if kind == "layer_norm":
        return dict(kind=kind, rows=_log_int(rng, 1, 25000), n=rng.choice([256, 384, 512, 768, 1024]), dtype=rng.choice(["bf16", "bf16", "f32"]), train=train)
    if kind == "ctc":
        t = _log_int(rng, 20, 400)
        return dict(kind=kind, batch=_log_int(rng, 1, max(1, 12000 // t)), t=t, vocab=rng.choice([80, 1001, 5001, 10001]),
                    labels_per_frame=rng.choice([0.1, 0.2, 0.3]))
    if kind == "cross_entropy":
        return dict(kind=kind, rows=_log_int(rng, 10, 6000), vocab=rng.choice([1000, 10000, 10025, 32000]), smoothing=rng.choice([0.0, 0.1]))
    if kind == "blstm":
        return dict(kind=kind, batch=_log_int(rng, 1, 40), t=_log_int(rng, 20, 400), n_in=rng.choice([80, 512, 1024, 2048]), hidden=rng.choice([512, 1024]),
                    train=train)
    if kind == "log_mel":
        return dict(kind=kind, batch=_log_int(rng, 1, 64), samples=_log_int(rng, 8000, 160000))
    if kind == "beam_rank":
        return dict(kind=kind, batch=_log_int(rng, 1, 64), beam=rng.choice([1, 4, 8, 12]), vocab=rng.choice([1001, 5000, 10001, 32000]))
    return dict(kind="conformer", batch=_log_int(rng, 1, 16), t=_log_int(rng, 300, 1500), layers=rng.choice([1, 2, 4]))


# ---------------------------------------------------------------------------------------------------------------- inputs


def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device=DEV).manual_seed(seed)


def _randn(g, *shape, scale: float = 1.0, dtype=torch.float32) -> torch.Tensor:
    return (torch.randn(*shape, generator=g, device=DEV) * scale).to(dtype)


def _lengths(seed: int, batch: int, t: int, lo: float = 0.15) -> torch.Tensor:
    """
    uniform lengths up to t, the longest of them t itself (a padded batch is as long as its longest sequence); the seed orders them, so
    that the number of valid frames is that of the case
    """
    lens = numpy.random.RandomState(1000 * batch + t).randint(max(1, int(t * lo)), t + 1, size=(batch,))
    lens[0] = t
    return torch.tensor(numpy.random.RandomState(seed % (2 ** 31)).permutation(lens), dtype=torch.int32)


def _leaf(t: torch.Tensor, train: bool) -> torch.Tensor:
    return t.requires_grad_(True) if train else t


class _Norm:
    """the fields of a BatchNorm module that the convolution module reads"""

    class _P:
        def __init__(self, raw):
            self.raw_tensor = raw

    def __init__(self, gamma, beta, mean, var):
        self.affine, self.eps = True, 1e-3
        self.momentum = 1.0  # the running statistics of a pass are then those of its batch, whatever was there before: comparable
        self.gamma, self.beta, self.running_mean, self.running_variance = (self._P(x) for x in (gamma, beta, mean, var))


def prepare(case: Dict[str, Any], seed: int) -> Dict[str, Any]:
    g = _gen(seed)
    bf = torch.bfloat16
    kind, train = case["kind"], bool(case.get("train", True))
    st: Dict[str, Any] = {"case": case}
    if kind == "linear":
        m, n_in, n_out = case["rows"], case["n_in"], case["n_out"]
        st["x"] = _leaf(_randn(g, m, n_in, dtype=bf), train)
        st["w"] = _leaf(_randn(g, n_in, n_out, scale=n_in ** -0.5), train)  # fp32 master weights, as under mixed precision
        st["b"] = _leaf(_randn(g, n_out, scale=0.1), train)
        st["dy"] = _randn(g, m, n_out, dtype=bf)
    elif kind == "attention":
        b, tq, tk, h = case["batch"], case["t_q"], case["t_k"], case["heads"]
        # the slices of a fused projection, as the attention modules pass them
        if tq == tk:
            qkv = _leaf(_randn(g, b, tq, h, 3 * 64, dtype=bf), train)
            st["leaves"] = [qkv]
        else:
            st["leaves"] = [_leaf(_randn(g, b, tq, h, 64, dtype=bf), train), _leaf(_randn(g, b, tk, h, 2 * 64, dtype=bf), train)]
        st["k_lens"] = _lengths(seed, b, tk, 0.1).to(DEV) if case["lens"] else None
        st["dy"] = _randn(g, b, tq, h, 64, dtype=bf)
    elif kind == "rel_pos":
        h = case["heads"]
        pack = PackInfo(_lengths(seed, case["batch"], case["t"]), DEV)
        st["pack"] = pack
        st["qkv"] = _leaf(_randn(g, pack.n, h * 3 * 64, dtype=bf), train)
        st["pos"] = _leaf(_randn(g, 2 * pack.max_len - 1, h * 64, dtype=bf), train)
        st["u"] = _leaf(_randn(g, h, 64, scale=0.2), train)
        st["v"] = _leaf(_randn(g, h, 64, scale=0.2), train)
        st["dy"] = _randn(g, pack.n, h * 64, dtype=bf)
    elif kind == "conv_module":
        c, k = case["channels"], case["taps"]
        pack = PackInfo(_lengths(seed, case["batch"], case["t"]), DEV)
        st["pack"] = pack
        st["x"] = _leaf(_randn(g, pack.n, 2 * c, dtype=bf), train)
        st["filt"] = _leaf(_randn(g, c, 1, k, scale=k ** -0.5), train)
        # BatchNorm takes the bias out again: its gradient in training is rounding noise around 0, which is not compared
        st["bias"] = _randn(g, c, scale=0.1)
        st["gamma"] = _leaf(_randn(g, c, scale=0.2) + 1.0, train)
        st["beta"] = _leaf(_randn(g, c, scale=0.2), train)
        st["bn"] = _Norm(st["gamma"], st["beta"], _randn(g, c, scale=0.1), torch.rand(c, generator=g, device=DEV) * 0.4 + 0.1)
        st["dy"] = _randn(g, pack.n, c, dtype=bf)
    elif kind == "layer_norm":
        dt = bf if case["dtype"] == "bf16" else torch.float32
        st["x"] = _leaf(_randn(g, case["rows"], case["n"], dtype=dt), train)
        st["gamma"] = _leaf((_randn(g, case["n"], scale=0.2) + 1.0).to(dt), train)
        st["beta"] = _leaf(_randn(g, case["n"], scale=0.2, dtype=dt), train)
        st["dy"] = _randn(g, case["rows"], case["n"], dtype=dt)
    elif kind == "ctc":
        lens = _lengths(seed, case["batch"], case["t"])
        pack = PackInfo(lens, DEV)
        tl = torch.clamp((lens.float() * case["labels_per_frame"]).to(torch.int32), min=1)
        st.update(pack=pack, target_lens=tl, logits=_leaf(_randn(g, pack.n, case["vocab"], dtype=bf), True))
        st["targets"] = torch.randint(0, case["vocab"] - 1, (case["batch"], int(tl.max())), generator=g, device=DEV, dtype=torch.int32)
    elif kind == "cross_entropy":
        st["logits"] = _leaf(_randn(g, case["rows"], case["vocab"], dtype=bf), True)
        st["targets"] = torch.randint(0, case["vocab"], (case["rows"],), generator=g, device=DEV)
        st["dy"] = torch.full((case["rows"],), 1.0 / case["rows"], device=DEV)
    elif kind == "blstm":
        b, t, n_in, h = case["batch"], case["t"], case["n_in"], case["hidden"]
        st["x"] = _leaf(_randn(g, t, b, n_in, dtype=bf), train)
        st["lens"] = _lengths(seed, b, t, 0.3)
        st["params"] = [_leaf(_randn(g, 4 * h, k, scale=k ** -0.5) if k else _randn(g, 4 * h, scale=0.1), train) for k in (n_in, h, 0, n_in, h, 0)]
        st["zero"] = torch.zeros(b, h, device=DEV)
        st["dy"] = [_randn(g, t, b, h, dtype=bf), _randn(g, t, b, h, dtype=bf)]
    elif kind == "log_mel":
        st["audio"] = _randn(g, case["batch"], case["samples"], scale=0.1)
    elif kind == "beam_rank":
        st["logits"] = _randn(g, case["batch"], case["beam"], case["vocab"], scale=2.0)
        st["prev"] = -torch.rand(case["batch"], case["beam"], generator=g, device=DEV) * 10.0
        st["finished"] = torch.rand(case["batch"], case["beam"], generator=g, device=DEV) < 0.1
    elif kind == "conformer":
        _prepare_conformer(st, case, seed, g)
    else:
        raise ValueError(kind)
    return st


def _prepare_conformer(st, case, seed: int, g):
    from returnn_b200.models.conformer_ctc import ConformerCtcModel
    from returnn_b200.parallel.arena import ParamArena
    from returnn_b200.tensor import Dim
    from returnn_b200.torch.frontend.bridge import rf_module_to_pt_module
    from returnn_b200.utils.basic import BehaviorVersion

    if not BehaviorVersion.is_set():
        BehaviorVersion.set(24)  # what a configuration file would ask for: convolutions do not see padded frames
    model = ConformerCtcModel(in_dim=Dim(80, name="feature"), vocab_dim=Dim(10000, name="vocab"), num_layers=case["layers"], dropout=0.0, att_dropout=0.0)
    model.encoder.input_dropout = 0.0
    st["model"] = model
    st["module"] = rf_module_to_pt_module(model).to(DEV)
    with torch.no_grad():  # random weights of this seed: variance 1 / fan-in, as the initialisation gives them, and small biases
        for name, p in st["module"].named_parameters():
            if name.endswith(("scale", "gamma")):
                p.fill_(1.0)
            elif p.dim() == 1 or "pos_bias" in name:
                p.copy_(_randn(g, *p.shape, scale=0.05))
            else:
                fan = p[0].numel() if name.endswith("filter") else p.shape[0]
                p.copy_(_randn(g, *p.shape, scale=fan ** -0.5))
    st["arena"] = ParamArena(list(st["module"].named_parameters()))
    st["lens"] = _lengths(seed, case["batch"], case["t"])
    st["feats"] = _randn(g, case["batch"], case["t"], 80)
    frames = (st["lens"] + 5) // 6
    tl = torch.clamp((frames.float() * 0.2).to(torch.int32), min=1)
    st["target_lens"] = tl
    st["targets"] = torch.randint(0, 9999, (case["batch"], int(tl.max())), generator=g, device=DEV, dtype=torch.int32)


# ---------------------------------------------------------------------------------------------------------------- one pass


def _attention_slices(leaves):
    if len(leaves) == 1:
        return leaves[0][..., :64], leaves[0][..., 64:128], leaves[0][..., 128:]
    return leaves[0], leaves[1][..., :64], leaves[1][..., 64:]


def run(st: Dict[str, Any]):
    case = st["case"]
    kind, train = case["kind"], bool(case.get("train", True))
    if kind == "linear":
        from returnn_b200.ops.linear import linear

        y = linear(st["x"], st["w"], st["b"], case["act"])
        return [y.detach(), *torch.autograd.grad(y, [st["x"], st["w"], st["b"]], st["dy"])] if train else [y]
    if kind == "attention":
        from returnn_b200.ops.sdpa import sdpa_heads

        q, k, v = _attention_slices(st["leaves"])
        y = sdpa_heads(q, k, v, k_lens=st["k_lens"], causal=case["causal"])
        return [y.detach(), *torch.autograd.grad(y, st["leaves"], st["dy"])] if train else [y]
    if kind == "rel_pos":
        from returnn_b200.ops.attention_packed import rel_pos_attention_packed

        y = rel_pos_attention_packed(st["qkv"], st["pos"], st["u"], st["v"], st["pack"], num_heads=case["heads"], head_dim=64, scale=0.125)
        return [y.detach(), *torch.autograd.grad(y, [st["qkv"], st["pos"], st["u"], st["v"]], st["dy"])] if train else [y]
    if kind == "conv_module":
        from returnn_b200.ops.conv_module import glu_dwconv_bn_silu

        bn = st["bn"]
        y = glu_dwconv_bn_silu(st["x"], st["filt"], st["bias"], bn, st["pack"], training=train)
        if not train:
            return [y]
        return [y.detach(), bn.running_mean.raw_tensor, bn.running_variance.raw_tensor,
                *torch.autograd.grad(y, [st["x"], st["filt"], st["gamma"], st["beta"]], st["dy"])]
    if kind == "layer_norm":
        from returnn_b200.ops.layer_norm import layer_norm

        y = layer_norm(st["x"], st["gamma"], st["beta"], 1e-6)
        return [y.detach(), *torch.autograd.grad(y, [st["x"], st["gamma"], st["beta"]], st["dy"])] if train else [y]
    if kind == "ctc":
        from returnn_b200.ops.ctc import ctc_loss_packed

        loss = ctc_loss_packed(st["logits"], st["pack"], st["targets"], st["target_lens"], blank_index=case["vocab"] - 1)
        return [loss.detach(), *torch.autograd.grad(loss.sum(), [st["logits"]])]
    if kind == "cross_entropy":
        from returnn_b200.ops.softmax_ce import softmax_cross_entropy

        loss = softmax_cross_entropy(st["logits"], st["targets"], case["smoothing"])
        return [loss.detach(), *torch.autograd.grad(loss, [st["logits"]], st["dy"])]
    if kind == "blstm":
        from returnn_b200.ops.lstm import blstm

        p, zero = st["params"], st["zero"]
        (yf, _hf, cf), (yb, _hb, cb) = blstm(st["x"], st["lens"], tuple(p[:3]), tuple(p[3:]), zero, zero, zero, zero)
        if not train:
            return [yf, cf, yb, cb]
        return [yf.detach(), cf.detach(), yb.detach(), cb.detach(), *torch.autograd.grad([yf, yb], [st["x"], *p], st["dy"])]
    if kind == "log_mel":
        from returnn_b200.ops.logmel import log_mel

        return [log_mel(st["audio"], sampling_rate=16000, window=400, step=160, n_fft=512, n_mel=80, f_min=0.0, f_max=8000.0)]
    if kind == "beam_rank":
        from returnn_b200.ops.seq_ops import beam_topk

        return list(beam_topk(st["logits"], st["prev"], finished=st["finished"], eos=0, k=case["beam"]))
    from returnn_b200.ops.ctc import ctc_loss_packed

    arena, model = st["arena"], st["model"]
    arena.zero_grad()
    logits, pack = model.fused_logits(st["feats"], st["lens"], training=True)
    loss = ctc_loss_packed(logits, pack, st["targets"], st["target_lens"], blank_index=model.blank_idx)
    loss.sum().backward()
    arena.relink_grads()
    return [logits.detach()[:, : model.blank_idx + 1], loss.detach(), arena.flat_grad]  # (the computed logits may carry a few padding classes)


# ---------------------------------------------------------------------------------------------------------------- what it needs


def work(case: Dict[str, Any]) -> Dict[str, float]:
    """input read once, output written once (no intermediate result), and the arithmetic of the definition over an average ragged batch"""
    kind, train = case["kind"], bool(case.get("train", True))
    if kind == "linear":
        m, i, o = case["rows"], case["n_in"], case["n_out"]
        byt = 2.0 * (m * i + m * o) + 4.0 * (i * o + o)
        fl = 2.0 * m * i * o
        return {"bytes": byt + (2.0 * (m * o + m * i) + 4.0 * (i * o + o) if train else 0.0), "flops": fl * (3 if train else 1)}
    if kind == "attention":
        b, tq, tk, h = case["batch"], case["t_q"], case["t_k"], case["heads"]
        share = (0.55 if case["lens"] else 1.0) * (0.5 if case["causal"] else 1.0)
        byt = 2.0 * 64 * h * b * (2 * tq + 2 * tk)
        fl = 4.0 * 64 * h * b * tq * tk * share
        return {"bytes": byt * (2 if train else 1), "flops": fl * (3.5 if train else 1)}
    if kind == "rel_pos":
        h, t, b = case["heads"], case["t"], case["batch"]
        n = 0.575 * b * t
        sq = b * t * t * 0.39  # mean of the squared lengths
        byt = 2.0 * 64 * h * (4 * n + 2 * t)
        fl = 6.0 * 64 * h * sq
        return {"bytes": byt * (2 if train else 1), "flops": fl * (10.0 / 3 if train else 1)}
    if kind == "conv_module":
        n, c = 0.575 * case["batch"] * case["t"], case["channels"]
        byt = 2.0 * n * 3 * c
        fl = 2.0 * n * c * case["taps"]
        return {"bytes": byt * (2 if train else 1), "flops": fl * (3 if train else 1)}
    if kind == "layer_norm":
        s = 2 if case["dtype"] == "bf16" else 4
        return {"bytes": float(s) * case["rows"] * case["n"] * (4 if train else 2), "flops": case["rows"] * case["n"] * (20.0 if train else 8.0)}
    if kind == "ctc":
        n = 0.575 * case["batch"] * case["t"]
        return {"bytes": 2.0 * n * case["vocab"] * 2, "flops": 6.0 * n * case["vocab"]}
    if kind == "cross_entropy":
        return {"bytes": 2.0 * case["rows"] * case["vocab"] * 2, "flops": 6.0 * case["rows"] * case["vocab"]}
    if kind == "blstm":
        b, t, i, h = case["batch"], case["t"], case["n_in"], case["hidden"]
        byt = 2.0 * t * b * (i + 2 * h) + 2 * 4.0 * 4 * h * (i + h + 1)
        fl = 2 * 2.0 * t * b * 4 * h * (i + h)
        return {"bytes": byt * (2 if train else 1), "flops": fl * (3 if train else 1)}
    if kind == "log_mel":
        frames = case["batch"] * max(0, (case["samples"] - 400) // 160 + 1)
        return {"bytes": 4.0 * case["batch"] * case["samples"] + 4.0 * frames * 80, "flops": frames * (2.5 * 512 * 9 + 2.0 * 257 * 2)}
    if kind == "beam_rank":
        n = case["batch"] * case["beam"]
        return {"bytes": 4.0 * n * case["vocab"] + 12.0 * n, "flops": 4.0 * n * case["vocab"]}
    rows, frames, d = 0.575 * case["batch"] * case["t"] / 6, 0.575 * case["batch"] * case["t"], 512
    per_row = 4 * 2 * d * 2048 + 2 * d * (3 * d + d + 2 * d + d)  # feed-forward blocks, attention and convolution projections
    att = 6.0 * d * 0.39 * case["batch"] * (case["t"] / 6.0) ** 2 / 0.575 * 0.575
    front = 2.0 * 40 * (frames * 2 * 9 * 32 + frames / 3 * 9 * 32 * 64 + rows * 9 * 64 * 64)
    params = case["layers"] * 6.35e6 + 512 * 10001 + 40 * 64 * 512
    fl = 3.0 * (case["layers"] * (rows * per_row + att) + front + 2.0 * rows * (d * 10001 + 2560 * d))
    return {"bytes": 4.0 * frames * 80 + 8.0 * params + 4.0 * rows * 10001, "flops": fl}


def tolerance(case: Dict[str, Any]):
    """about four times the distance to the 64-bit result (bf16 operands and results, 32-bit sums)"""
    kind = case["kind"]
    if kind == "beam_rank":
        return {"rel": 1e-5, "differ": 0.02}  # ranks of nearly equal scores may swap
    if kind == "layer_norm":
        return {"rel": 1.2e-2 if case["dtype"] == "bf16" else 1e-5}
    if kind == "log_mel":
        return {"rel": 2e-5}
    if kind == "conformer":
        return {"rel": 1.5e-1}
    if kind == "cross_entropy":
        return {"rel": 1e-2}
    return {"rel": 2e-2}


# ---------------------------------------------------------------------------------------------------------------- in 64 bits


def exact(case: Dict[str, Any], seed: int):
    kind, train = case["kind"], bool(case.get("train", True))
    st = prepare(case, seed)

    def up(t):  # a 64-bit copy that takes part in differentiation
        return t.detach().double().requires_grad_(train)

    def grads(ys, xs, dys):
        if not train:
            return []
        return list(torch.autograd.grad(ys, xs, [d.double() for d in dys]))

    if kind == "linear":
        x, w, b = up(st["x"]), up(st["w"]), up(st["b"])
        # the operands are the 16-bit values that mixed precision multiplies
        w16 = w + (w.detach().bfloat16().double() - w.detach())
        y = x @ w16 + b
        if case["act"]:
            y = {"silu": F.silu, "relu": torch.relu}[case["act"]](y)
        return [y.detach(), *grads([y], [x, w, b], [st["dy"]])]
    if kind == "attention":
        b, tq, tk = case["batch"], case["t_q"], case["t_k"]
        leaves = [up(t) for t in st["leaves"]]
        kl = st["k_lens"]
        out, gr = [], [torch.zeros_like(t) for t in leaves]
        pos_q, pos_k = torch.arange(tq, device=DEV)[:, None], torch.arange(tk, device=DEV)[None, :]
        for i in range(b):  # one sequence after another: bounded memory
            li = [t.detach()[i].requires_grad_(train) for t in leaves]
            q, k, v = (t.transpose(0, 1) for t in _attention_slices(li))
            s = q @ k.transpose(1, 2) * 0.125
            ok = torch.ones(tq, tk, dtype=torch.bool, device=DEV)
            if kl is not None:
                ok = ok & (pos_k < kl[i])
            if case["causal"]:
                ok = ok & (pos_k <= pos_q + (tk - tq))
            y = (torch.softmax(s.masked_fill(~ok, float("-inf")), -1) @ v).transpose(0, 1)
            out.append(y.detach())
            for o, gi in zip(gr, grads([y], li, [st["dy"][i]])):
                o[i] = gi
        return [torch.stack(out), *(gr if train else [])]
    if kind == "rel_pos":
        h, pack = case["heads"], st["pack"]
        qkv, pos, u, v = (up(st[k]) for k in ("qkv", "pos", "u", "v"))
        ys, lo = [], 0
        for n in pack.lens_host.tolist():
            ys.append(_rel_pos(qkv[lo: lo + n].view(n, h, 3, 64), pos.view(-1, h, 64), u, v, 0.125))
            lo += n
        y = torch.cat(ys)
        return [y.detach(), *grads([y], [qkv, pos, u, v], [st["dy"]])]
    if kind == "conv_module":
        x, filt, gamma, beta = (up(st[k]) for k in ("x", "filt", "gamma", "beta"))
        bn = st["bn"]
        stats = None if train else (bn.running_mean.raw_tensor.double(), bn.running_variance.raw_tensor.double())
        y, mean, var = _conv_middle(x, filt, st["bias"].double(), gamma, beta, st["pack"], stats, bn.eps)
        return [y.detach(), *([mean.detach(), var.detach()] if train else []), *grads([y], [x, filt, gamma, beta], [st["dy"]])]
    if kind == "layer_norm":
        x, gamma, beta = (up(st[k]) for k in ("x", "gamma", "beta"))
        y = F.layer_norm(x, (case["n"],), gamma, beta, 1e-6)
        return [y.detach(), *grads([y], [x, gamma, beta], [st["dy"]])]
    if kind == "ctc":
        x = up(st["logits"])
        loss = _ctc(x, st["pack"].lens_host, st["targets"], st["target_lens"], case["vocab"] - 1)
        return [loss.detach(), *torch.autograd.grad(loss.sum(), [x])]
    if kind == "cross_entropy":
        x, tg, s, v = up(st["logits"]), st["targets"], case["smoothing"], case["vocab"]
        lp = torch.log_softmax(x, -1)
        lt = lp.gather(1, tg[:, None])[:, 0]
        loss = -(1 - s) * lt - s / (v - 1) * (lp.sum(-1) - lt)
        return [loss.detach(), *grads([loss], [x], [st["dy"]])]
    if kind == "blstm":
        if case["t"] * (3 if train else 1) > 1300:
            return None
        x, p = up(st["x"]), [up(t) for t in st["params"]]
        yf, cf = _lstm(x, st["lens"].to(DEV), *p[:3], False)
        yb, cb = _lstm(x, st["lens"].to(DEV), *p[3:], True)
        return [yf.detach(), cf.detach(), yb.detach(), cb.detach(), *grads([yf, yb], [x, *p], st["dy"])]
    if kind == "log_mel":
        return [_log_mel(st["audio"].double())]
    if kind == "beam_rank":
        b, k, v = case["batch"], case["beam"], case["vocab"]
        lp = torch.log_softmax(st["logits"].double(), -1) + st["prev"].double()[..., None]
        ended = torch.full_like(lp, float("-inf"))
        ended[:, :, 0] = st["prev"].double()
        top, idx = torch.topk(torch.where(st["finished"][..., None], ended, lp).reshape(b, -1), k, -1)
        return [top, (idx // v).to(torch.int32), (idx % v).to(torch.int32)]
    return _conformer(case, st)


def _rel_pos(qkv, pos, u, v, scale):
    """one sequence: qkv [n, H, 3, 64], pos [2L-1, H, 64] (row r: distance r - (L-1))"""
    n, h = qkv.shape[:2]
    q, k, val = (qkv[:, :, i].transpose(0, 1) for i in range(3))
    mid = (pos.shape[0] - 1) // 2
    ac = (q + u[:, None]) @ k.transpose(1, 2)
    bd = (q + v[:, None]) @ pos[mid - n + 1: mid + n].permute(1, 2, 0)  # [H, n, 2n-1]
    at = torch.arange(n, device=DEV)
    bd = torch.gather(bd, 2, (at[None, :] - at[:, None] + n - 1).expand(h, n, n))
    return (torch.softmax((ac + bd) * scale, -1) @ val).transpose(0, 1).reshape(n, -1)


def _conv_middle(x, filt, bias, gamma, beta, pack, stats, eps):
    c, k = filt.shape[0], filt.shape[-1]
    a = pack.unpack(x[:, :c] * torch.sigmoid(x[:, c:])).transpose(1, 2)
    left = (k - 1) // 2
    y = torch.einsum("bctk,ck->bct", F.pad(a, (left, k - 1 - left)).unfold(2, k, 1), filt[:, 0]) + bias[None, :, None]
    y = pack.pack(y.transpose(1, 2))
    mean, var = (y.mean(0), y.var(0, unbiased=False)) if stats is None else stats
    return F.silu((y - mean) * torch.rsqrt(var + eps) * gamma + beta), mean, var


def _ctc(rows, lens, targets, target_lens, blank):
    """one loss per sequence; rows [N, V] of all sequences back to back"""
    lp = torch.log_softmax(rows, -1)
    res, lo = [], 0
    for i, (n, s) in enumerate(zip(lens.tolist(), target_lens.tolist())):
        res.append(F.ctc_loss(lp[lo: lo + n, None], targets[i: i + 1, :s].long(), torch.tensor([n]), torch.tensor([s]), blank=blank, reduction="none",
                              zero_infinity=True))
        lo += n
    return torch.cat(res)


def _lstm(x, lens, w_ff, w_rec, bias, reverse):
    t, b, _ = x.shape
    z_in = x @ w_ff.t() + bias
    h = c = x.new_zeros(b, w_rec.shape[1])
    ys = [None] * t
    for i in reversed(range(t)) if reverse else range(t):
        gi, gf, gg, go = (z_in[i] + h @ w_rec.t()).chunk(4, -1)
        c2 = torch.sigmoid(gf) * c + torch.sigmoid(gi) * torch.tanh(gg)
        h2 = torch.sigmoid(go) * torch.tanh(c2)
        m = (lens > i)[:, None]
        c, h = torch.where(m, c2, c), torch.where(m, h2, h)
        ys[i] = torch.where(m, h2, torch.zeros_like(h2))
    return torch.stack(ys), c


def _log_mel(audio):
    frames = audio.unfold(-1, 400, 160) * torch.hann_window(400, periodic=True, dtype=torch.float64, device=DEV)
    power = torch.fft.rfft(frames, n=512).abs().square()
    mel = lambda f: 1127.0 * numpy.log1p(f / 700.0)  # noqa: E731
    pts = numpy.linspace(mel(0.0), mel(8000.0), 82)
    at = mel(numpy.linspace(0.0, 8000.0, 257))[:, None]
    fb = numpy.maximum(0.0, numpy.minimum((at - pts[None, :-2]) / (pts[1:-1] - pts[:-2]), (pts[None, 2:] - at) / (pts[2:] - pts[1:-1])))
    return torch.log10(torch.clamp(power @ torch.tensor(fb, device=DEV), min=1e-10))


def _conformer(case, st):
    """the whole model in plain 64-bit operations over the same parameters"""
    arena = st["arena"]
    par = {s.name: arena.flat_param[s.offset: s.offset + s.numel].view(s.shape).detach().double().requires_grad_(True) for s in arena.slots}
    lens, d = st["lens"].long(), 512
    x = st["feats"].bfloat16().double()[:, None]
    n = lens.to(DEV)

    def masked(y, m):
        return y * (torch.arange(y.shape[2], device=DEV)[None, :] < m[:, None]).double()[:, None, :, None]

    x = masked(x, n)
    for i, (stride, pool) in enumerate(((1, 2), (3, 1), (2, 1))):
        f, b = par["encoder.input_layer.conv_layers.%i.filter" % i], par["encoder.input_layer.conv_layers.%i.bias" % i]
        x = torch.relu(F.conv2d(x, f, b, stride=(stride, 1), padding=1))
        if pool > 1:
            x = F.max_pool2d(x, (1, pool))
        n = -(-n // stride)
        x = masked(x, n)
    pack = PackInfo(n.cpu().to(torch.int32), DEV, padded_len=x.shape[2])
    x = pack.pack(x.permute(0, 2, 3, 1).reshape(x.shape[0], x.shape[2], -1)) @ par["encoder.input_projection.weight"]
    dist = torch.arange(-(pack.max_len - 1), pack.max_len, device=DEV, dtype=torch.float64)
    arg = dist[:, None] * torch.exp(torch.arange(d // 2, device=DEV, dtype=torch.float64) * -(2.0 * math.log(1e4) / d))[None]
    sinus = torch.cat([torch.sin(arg), torch.cos(arg)], -1)

    def norm(y, name):
        return F.layer_norm(y, (d,), par[name + ".scale"], par[name + ".bias"], 1e-6)

    def lin(y, name):
        w = par[name + ".weight"]
        return y @ w + par[name + ".bias"] if name + ".bias" in par else y @ w

    for i in range(case["layers"]):
        p = "encoder.layers.%i." % i
        x = x + 0.5 * lin(F.silu(lin(norm(x, p + "ffn1_layer_norm"), p + "ffn1.linear_ff")), p + "ffn1.linear_out")
        qkv = lin(norm(x, p + "self_att_layer_norm"), p + "self_att.qkv")
        pos = lin(sinus, p + "self_att.linear_pos").view(-1, 8, 64)
        ys, lo = [], 0
        for m in pack.lens_host.tolist():
            ys.append(_rel_pos(qkv[lo: lo + m].view(m, 8, 3, 64), pos, par[p + "self_att.pos_bias_u"], par[p + "self_att.pos_bias_v"], 0.125))
            lo += m
        x = x + lin(torch.cat(ys), p + "self_att.proj")
        c = p + "conv_block."
        y, _, _ = _conv_middle(lin(norm(x, p + "conv_layer_norm"), c + "positionwise_conv1"), par[c + "depthwise_conv.filter"], par[c + "depthwise_conv.bias"],
                               par[c + "norm.gamma"], par[c + "norm.beta"], pack, None, 1e-3)
        x = x + lin(y, c + "positionwise_conv2")
        x = x + 0.5 * lin(F.silu(lin(norm(x, p + "ffn2_layer_norm"), p + "ffn2.linear_ff")), p + "ffn2.linear_out")
        x = norm(x, p + "final_layer_norm")
    logits = lin(x, "logits")
    loss = _ctc(logits, pack.lens_host, st["targets"], st["target_lens"], 10000)
    flat = torch.zeros(arena.total, dtype=torch.float64, device=DEV)
    for s, gr in zip(arena.slots, torch.autograd.grad(loss.sum(), [par[s.name] for s in arena.slots])):
        flat[s.offset: s.offset + s.numel] = gr.reshape(-1)
    return [logits.detach(), loss.detach(), flat]
