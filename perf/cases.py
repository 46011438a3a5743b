"""The workloads whose speed this repository cares about, as plain data and four functions over it.

A case names an entry point (`kind`), its sizes and the options used in earnest.  `listed()` is the fixed set,
`draw(rng)` picks one more from the same ranges, `prepare(case, seed)` makes what a program holds before it calls the
library (inputs, weights, plans), `run(state)` is one call through the public entry points, `work(case)` the bytes and
operations the path cannot do without and `tolerance(case)` how far another correct implementation may be off.
"""
from __future__ import annotations

import math

import torch

from souffle_models_b200 import bert, efficientnet, lstm, swin

SEQS = (16, 32, 48, 64, 80, 96, 112, 128, 256, 384)          # the sequence lengths a BERT plan takes
HIDDEN_HEADS = (2, 4, 8, 12, 16)                             # times 64 = the hidden sizes a BERT plan takes
SE_SHAPES = ((112, 32, 8), (56, 96, 4), (56, 144, 6), (28, 144, 6), (28, 240, 10), (14, 240, 10), (14, 480, 20),
             (14, 672, 28), (7, 672, 28), (7, 1152, 48))     # (side, channels, reduced channels) of an EfficientNet-B0


def listed():
    return [
        # one encoder layer, one sequence: the latency the library is quoted on
        dict(name="bert_layer_b1_s128", kind="bert", batch=1, seq=128, heads=12, ffn=3072, layers=1, ragged=False),
        # the whole encoder over a small batch with an unusual length (rows are no multiple of a tile), as a server
        # with little traffic runs it
        dict(name="bert_base_b7_s112", kind="bert", batch=7, seq=112, heads=12, ffn=3072, layers=12, ragged=True),
        # the benchmark's step: the whole encoder over 64 sequences of ragged lengths, the throughput case
        dict(name="bert_base_b64_s128", kind="bert", batch=64, seq=128, heads=12, ffn=3072, layers=12, ragged=True),
        # the drop-in call of the reference's binding: one layer at its fixed length, all six stage outputs returned
        dict(name="bert_dropin_s384", kind="bert_dropin", batch=1, seq=384, heads=12, ffn=3072),
        # the reference's stacked LSTM through its drop-in call (fp32 tensors, inputs one step late)
        dict(name="lstm_10x256x100", kind="lstm_dropin", layers=10, hidden=256, steps=100),
        # a shallow stack of another width with bias, an odd number of steps, through the plan
        dict(name="lstm_3x128x37", kind="lstm", layers=3, hidden=128, steps=37),
        # a pair of Swin blocks (plain and shifted windows) on one image
        dict(name="swin_pair_b1", kind="swin", batch=1, res=14, dim=512, window=7, blocks=2, merge=False),
        # stage 3 of a Swin-B with the patch merging that ends it, on four images
        dict(name="swin_stage3_b4", kind="swin", batch=4, res=14, dim=512, window=7, blocks=18, merge=True),
        # the reference's fused MLP call, at its own shape
        dict(name="swin_mlp_m256", kind="mlp", rows=256, dim=512, ffn=2048),
        # one large product with an odd number of rows through the GEMM call
        dict(name="gemm_m8191_n3072_k768", kind="gemm", rows=8191, cols=3072, inner=768),
        # squeeze-and-excite at the network's first and largest image, batch 1 as the reference calls it: the smallest call
        dict(name="se_b1_112x112x32", kind="se", batch=1, side=112, channels=32, reduce=8),
        # the same module over a batch, bound by memory
        dict(name="se_b32_56x56x144", kind="se", batch=32, side=56, channels=144, reduce=6),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    most = max(work(c)["flops"] for c in listed())
    kind = rng.choice(("bert", "bert", "bert", "bert_dropin", "lstm", "lstm_dropin", "swin", "swin", "mlp", "gemm", "se"))
    while True:
        if kind == "bert":
            heads = rng.choice(HIDDEN_HEADS)
            c = dict(kind=kind, batch=_log_int(rng, 1, 64), seq=rng.choice(SEQS), heads=heads,
                     ffn=64 * _log_int(rng, heads, 4 * heads), layers=rng.choice((1, 2, 3, 6, 12)), ragged=rng.random() < 0.5)
        elif kind == "bert_dropin":
            c = dict(kind=kind, batch=1, seq=rng.choice(SEQS), heads=12, ffn=3072)
        elif kind in ("lstm", "lstm_dropin"):
            c = dict(kind=kind, layers=rng.randint(1, 12), hidden=rng.choice((64, 128, 256)), steps=_log_int(rng, 4, 200))
        elif kind == "swin":
            window = rng.choice((7, 7, 8))
            stage = rng.randrange(4)                       # a grid of 8, 4, 2 or 1 windows per side
            c = dict(kind=kind, batch=_log_int(rng, 1, 16), res=window << (3 - stage), dim=128 << stage, window=window,
                     blocks=rng.choice((1, 2, 2, 6, 18)), merge=stage < 3 and rng.random() < 0.5)
        elif kind == "mlp":
            c = dict(kind=kind, rows=_log_int(rng, 1, 8192), dim=64 * rng.randint(2, 16), ffn=64 * _log_int(rng, 4, 64))
        elif kind == "gemm":
            c = dict(kind=kind, rows=_log_int(rng, 1, 8192), cols=64 * _log_int(rng, 1, 64), inner=64 * _log_int(rng, 1, 64))
        else:
            side, channels, reduce = rng.choice(SE_SHAPES)
            c = dict(kind=kind, batch=_log_int(rng, 1, 32), side=side, channels=channels, reduce=reduce)
        if work(c)["flops"] <= most:
            return c


class _Make:
    """Seeded tensors on the GPU."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(self, *shape, scale=1.0, base=0.0, dtype=torch.float16):
        return (torch.randn(*shape, generator=self.gen, device="cuda") * scale + base).to(dtype)

    def uniform(self, *shape, scale):
        return (torch.rand(*shape, generator=self.gen, device="cuda") - 0.5) * (2.0 * scale)

    def bert_layer(self, H, F):
        w = lambda *s: self.normal(*s, scale=0.02)
        v = lambda *s, base=0.0: self.normal(*s, scale=0.05, base=base)
        return dict(qkv_w=w(3, H, H), qkv_b=v(3, H), proj_w=w(H, H), proj_b=v(H), ln1_g=v(H, base=1.0), ln1_b=v(H), fc1_w=w(H, F),
                    fc1_b=v(F), fc2_w=w(F, H), fc2_b=v(H), ln2_g=v(H, base=1.0), ln2_b=v(H))

    def swin_block(self, C, heads, window):
        w = lambda *s: self.normal(*s, scale=0.02)
        v = lambda *s, base=0.0: self.normal(*s, scale=0.05, base=base)
        return dict(ln1_g=v(C, base=1.0), ln1_b=v(C), qkv_w=w(C, 3 * C), qkv_b=v(3 * C), rel_bias=w((2 * window - 1) ** 2, heads),
                    proj_w=w(C, C), proj_b=v(C), ln2_g=v(C, base=1.0), ln2_b=v(C), fc1_w=w(C, 4 * C), fc1_b=v(4 * C),
                    fc2_w=w(4 * C, C), fc2_b=v(C))


def prepare(case, seed):
    make = _Make(seed)
    kind = case["kind"]
    s = dict(kind=kind)
    if kind in ("bert", "bert_dropin"):
        H, F = 64 * case["heads"], case["ffn"]
        s["x"] = make.normal(case["batch"], case["seq"], H)
        if kind == "bert":
            layers = [make.bert_layer(H, F) for _ in range(case["layers"])]
            s["layers"] = layers
            s["plan"] = bert.BertEncoder(case["batch"], case["seq"], case["heads"], 64, F, layers)
            s["lens"] = None
            if case["ragged"]:                             # valid lengths in [S/4, S]
                S = case["seq"]
                s["lens"] = torch.randint(S // 4, S + 1, (case["batch"],), generator=make.gen, device="cuda", dtype=torch.int32)
        else:
            w = make.bert_layer(H, F)
            s["w"] = [w[k] for k in ("qkv_w", "proj_w", "fc1_w", "fc2_w")]
    elif kind in ("lstm", "lstm_dropin"):
        L, H, T = case["layers"], case["hidden"], case["steps"]
        # weights on the scale 1 / sqrt(hidden), as a trained or freshly initialised stack has them; values of fp16 in fp32
        # tensors, which is what the drop-in call keeps exactly
        w = [make.uniform(4 * L, H, H, scale=1.0 / math.sqrt(H)).half().float() for _ in range(2)]
        s["x"] = make.normal(1, T, H, dtype=torch.float32)
        if kind == "lstm":
            s["bias"] = make.normal(L, H, scale=0.1, dtype=torch.float32)
            s["plan"] = lstm.LstmStack(w[0], w[1], T, bias=s["bias"])
        s["w"] = w
    elif kind == "swin":
        C, heads, window = case["dim"], case["dim"] // 32, case["window"]
        blocks = [make.swin_block(C, heads, window) for _ in range(case["blocks"])]
        merge = None
        if case["merge"]:
            merge = dict(norm_g=make.normal(4 * C, scale=0.05, base=1.0), norm_b=make.normal(4 * C, scale=0.05),
                         reduction_w=make.normal(4 * C, 2 * C, scale=0.02))
        shift = window // 2 if case["res"] > window else 0         # a grid of one window is not shifted
        s["plan"] = swin.SwinBlock(case["batch"], case["res"], C, heads, window, 0, blocks, shift_alt=shift, merge=merge)
        s["x"] = make.normal(case["batch"] * case["res"] ** 2, C)
        s["blocks"], s["merge"] = blocks, merge
    elif kind == "mlp":
        s["x"] = make.normal(case["rows"], case["dim"])
        s["w"] = [make.normal(case["dim"], case["ffn"], scale=0.02), make.normal(case["ffn"], case["dim"], scale=0.02)]
    elif kind == "gemm":
        s["x"] = make.normal(case["rows"], case["inner"])
        s["w"] = make.normal(case["inner"], case["cols"], scale=0.02)
    else:
        C, R = case["channels"], case["reduce"]
        s["x"] = make.normal(case["batch"], C, case["side"], case["side"], dtype=torch.float32)
        s["w"] = [make.normal(R, C, scale=0.2, dtype=torch.float32), make.normal(C, R, scale=0.5, dtype=torch.float32)]
    return s


def run(state):
    kind = state["kind"]
    if kind == "bert":
        return state["plan"].forward(state["x"], state["lens"])
    if kind == "bert_dropin":
        return bert.souffle_bert_layer(state["x"], *state["w"], 4)
    if kind == "lstm":
        return state["plan"].forward(state["x"])
    if kind == "lstm_dropin":
        return lstm.fused_lstm(state["x"], *state["w"])
    if kind == "swin":
        return state["plan"].forward(state["x"])
    if kind == "mlp":
        return swin.swin_fused_feed_mlp(state["x"], *state["w"])
    if kind == "gemm":
        return swin.gemm(state["x"], state["w"])
    return efficientnet.se_module(state["x"], *state["w"])


def work(case):
    kind = case["kind"]
    if kind in ("bert", "bert_dropin"):
        B, S, H, F, L = case["batch"], case["seq"], 64 * case["heads"], case["ffn"], case.get("layers", 1)
        M = B * S
        flops = L * (2 * M * H * 3 * H + 4 * B * S * S * H + 2 * M * H * H + 4 * M * H * F)
        nbytes = L * 2 * (4 * H * H + 2 * H * F + 9 * H + F) + 2 * 2 * M * H
        if kind == "bert_dropin":                          # q, k, v, probabilities, attention output, first half, hidden layer
            nbytes += 2 * (3 * M * H + B * case["heads"] * S * S + 2 * M * H + M * F)
        return dict(bytes=nbytes, flops=flops)
    if kind in ("lstm", "lstm_dropin"):
        L, H, T = case["layers"], case["hidden"], case["steps"]
        return dict(bytes=2 * 8 * L * H * H + 2 * 4 * T * H, flops=2 * 8 * L * H * H * T)
    if kind == "swin":
        C, w, n = case["dim"], case["window"], case["blocks"]
        T = case["batch"] * case["res"] ** 2
        flops = n * (2 * T * C * 12 * C + 4 * T * w * w * C)
        nbytes = n * 2 * (12 * C * C + 13 * C + (2 * w - 1) ** 2 * (C // 32)) + 2 * 2 * T * C
        if case["merge"]:
            flops += 2 * (T // 4) * 4 * C * 2 * C
            nbytes += 2 * (8 * C * C + 8 * C) - 2 * T * C // 2
        return dict(bytes=nbytes, flops=flops)
    if kind == "mlp":
        M, C, F = case["rows"], case["dim"], case["ffn"]
        return dict(bytes=2 * (2 * M * C + M * F + 2 * C * F), flops=4 * M * C * F)
    if kind == "gemm":
        M, N, K = case["rows"], case["cols"], case["inner"]
        return dict(bytes=2 * (M * K + K * N + M * N), flops=2 * M * N * K)
    B, C, R, hw = case["batch"], case["channels"], case["reduce"], case["side"] ** 2
    return dict(bytes=4 * (2 * B * C * hw + B * C + 2 * R * C), flops=2 * B * C * hw + 4 * B * R * C)


def tolerance(case):
    """Measured against the same path in double precision (inputs as given, nothing rounded in between), times four."""
    kind = case["kind"]
    if kind == "bert":                                     # every activation handed on is fp16: 4.4e-4 for a layer, 1.4e-3 for twelve
        n = math.sqrt(case["layers"])
        return dict(rel=1.8e-3 * n, max=1.0e-2 * n)
    if kind == "bert_dropin":                              # worst of the six stage outputs
        return dict(rel=1.5e-3, max=7e-3)
    if kind == "lstm":                                     # hidden states of order 0.1: fp32 throughout
        return dict(rel=1e-5, max=5e-5)
    if kind == "lstm_dropin":                              # no bias: hidden states shrink with every layer to 1e-3 and below, where
        return dict(rel=5e-4, max=2e-3)                    # the 1e-7 of a fast tanh or sigmoid counts (measured 6e-5 to 1.2e-4)
    if kind == "swin":                                     # 4.4e-4 for two blocks, 1.3e-3 for eighteen
        n = math.sqrt(case["blocks"] + 1)
        return dict(rel=1.2e-3 * n, max=6e-3 * n)
    if kind == "mlp":                                      # the hidden layer and the output are fp16
        return dict(rel=1.2e-3, max=6e-3)
    if kind == "gemm":
        return dict(rel=8e-4, max=2e-3)
    return dict(rel=1e-6, max=4e-6)                        # fp32 sums
