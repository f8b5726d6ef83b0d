"""The work a user has this package do, as cases that can be timed and compared.

Every case goes through the public entry points only: the operators of `algebraic_transformer_b200`,
their differentiable forms in `algebraic_transformer_b200.autograd`, and `prefill.Prefill`.  Sizes come from the
model presets of `prefill.py`, the benchmark configurations of `bench.py` and the tests; `draw` spreads
more of them over the same ranges, off the tile grids as often as on them.

A case is a dict of plain values; `kind` says which path it takes:

    decode       one new token against a KV cache that is partly filled
    attention    guarded attention forward over q, k, v that are normalised already (inference, bf16)
    layer        QK-norm + rotation + guarded attention in one call (inference, float32 or bf16)
    train_layer  QK-norm and attention, forward and backward through torch.autograd
    train_ops    the same with the operator pairs called directly (any sequence length)
    score_head   likelihood head forward (evaluation)
    train_head   likelihood head, forward and backward through torch.autograd
    prompt       a model's hidden states for a prompt
    score        a model's loss and per-token negative log-likelihoods over a batch
"""

import math

import torch

import algebraic_transformer_b200 as A
from algebraic_transformer_b200 import autograd as G
from algebraic_transformer_b200.prefill import SIZES, Prefill, PrefillConfig

DEVICE = "cuda"
ATTN = dict(n=16, c=8.0)      # the `algebraic` preset's attention link
HEAD = dict(n=8, c=2.0)       # and its head link


def listed():
    return [
        # the first tokens of a generation by the 125M model: the smallest call there is, all latency
        dict(name="decode_start", kind="decode", B=1, H=12, Tk=333, D=64),
        # a serving batch of the 350M model, a couple of thousand tokens into its sequences
        dict(name="decode_batch", kind="decode", B=16, H=16, Tk=1900, D=64),
        # configuration 5's decode: one sequence against a 32768-token cache
        dict(name="decode_long", kind="decode", B=1, H=16, Tk=32768, D=128),
        # configuration 5: long-context attention forward
        dict(name="attention_long", kind="attention", B=1, H=16, T=8192, D=128),
        # configuration 1: one layer's attention in float32, as in evaluation against the float32 reference
        dict(name="layer_float32", kind="layer", dtype="float32", B=4, H=12, T=1024, D=64),
        # a training step of the 125M model's attention (one layer, its batch of 16 x 1024)
        dict(name="train_layer_125m", kind="train_layer", B=16, H=12, T=1024, D=64),
        # fine-tuning on documents of whatever length they have, head_dim 128
        dict(name="train_ragged", kind="train_ops", B=2, H=16, T=1837, D=128),
        # configuration 2's head in training: forward, both gradients, a float32 embedding that the optimizer owns
        dict(name="train_head", kind="train_head", head="alg_ce", N=8192, d=768, V=50304),
        # evaluation of a handful of documents with the softmax control head, off every tile grid
        dict(name="score_head_ragged", kind="score_head", head="ce", N=2741, d=1024, V=32000),
        # a user's prompt through the 125M model
        dict(name="prompt_125m", kind="prompt", size="125m", V=50304, B=1, T=613),
        # configuration 3: the 125M model's prefill
        dict(name="score_125m", kind="score", size="125m", V=50304, B=16, T=1024),
        # configuration 4's larger model
        dict(name="score_1b", kind="score", size="1b", V=32000, B=8, T=2048),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case; sizes are redrawn until the work fits the listed range."""
    kind = rng.choice(["decode", "attention", "layer", "train_layer", "train_ops", "score_head", "train_head", "prompt",
                       "score"])
    while True:
        B, H, D = _log_int(rng, 1, 32), rng.choice([6, 12, 16, 24]), rng.choice([64, 128])
        if kind == "decode":
            case = dict(kind=kind, B=B, H=H, Tk=_log_int(rng, 32, 65536), D=D)
            fits = work(case)["bytes"] <= 6e8
        elif kind == "attention":
            case = dict(kind=kind, B=B, H=H, T=_log_int(rng, 64, 16384), D=D)
            fits = work(case)["flops"] <= 6e11
        elif kind == "layer":
            case = dict(kind=kind, dtype=rng.choice(["float32", "bfloat16"]), B=B, H=H, T=_log_int(rng, 64, 4096), D=D)
            fits = work(case)["flops"] <= 1e11
        elif kind == "train_layer":      # the differentiable form takes lengths up to 512 and multiples of 512
            T = _log_int(rng, 64, 8192)
            case = dict(kind=kind, B=B, H=H, T=T if T <= 512 else 512 * round(T / 512), D=D)
            fits = work(case)["flops"] <= 1e12
        elif kind == "train_ops":
            case = dict(kind=kind, B=B, H=H, T=_log_int(rng, 64, 6000), D=D)
            fits = work(case)["flops"] <= 1e12
        elif kind in ("score_head", "train_head"):
            size = rng.choice(list(SIZES))
            case = dict(kind=kind, head=rng.choice(["alg_ce", "alg_ce", "ce"]), N=_log_int(rng, 64, 16384),
                        d=SIZES[size]["d_model"], V=rng.choice([32000, 32768, 50304]))
            fits = work(case)["flops"] <= 3e12
        else:
            lo, hi = (1, 4) if kind == "prompt" else (1, 16)
            sizes = ["proxy", "125m", "350m"] if kind == "prompt" else list(SIZES)
            case = dict(kind=kind, size=rng.choice(sizes), V=rng.choice([32000, 50304]), B=_log_int(rng, lo, hi),
                        T=_log_int(rng, 64, 2048))
            fits = work(case)["flops"] <= 2.5e13
        if fits:
            return case


# ------------------------------------------------------------------------------------------- inputs

class _Inputs:
    """Seeded tensors on the GPU."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEVICE).manual_seed(int(seed))

    def normal(self, *shape, dtype=torch.float32, scale=1.0, shift=0.0):
        x = torch.randn(shape, generator=self.g, device=DEVICE)
        return x.mul_(scale).add_(shift).to(dtype)

    def ints(self, hi, *shape):
        return torch.randint(0, hi, shape, generator=self.g, device=DEVICE)

    def heads(self, B, H, T, D, dtype=torch.bfloat16):
        """(B,H,T,D), as the (B,T,H,D) output of a projection is viewed."""
        return self.normal(B, T, H, D, dtype=dtype).transpose(1, 2)


def _model(r, case):
    """A model with weights of the init scale and gains and sinks as training leaves them."""
    cfg = PrefillConfig.preset(case["size"], vocab_size=case["V"])
    L, d, f, V, H, D = cfg.n_layers, cfg.d_model, cfg.d_ff, cfg.vocab_size, cfg.n_heads, cfg.head_dim
    s = cfg.init_std
    params = {
        "embed": r.normal(V, d, scale=s),
        "embed_gain": r.normal(d, scale=0.1, shift=1.0), "final_gain": r.normal(d, scale=0.1, shift=1.0),
        "w_q": r.normal(L, d, d, scale=s), "w_k": r.normal(L, d, d, scale=s), "w_v": r.normal(L, d, d, scale=s),
        "w_o": r.normal(L, d, d, scale=s), "w_g": r.normal(L, d, f, scale=s), "w_u": r.normal(L, d, f, scale=s),
        "w_d": r.normal(L, f, d, scale=s),
        "ln1": r.normal(L, d, scale=0.1, shift=1.0), "ln2": r.normal(L, d, scale=0.1, shift=1.0),
        "q_gain": r.normal(L, D, scale=0.1, shift=1.0), "k_gain": r.normal(L, D, scale=0.1, shift=1.0),
        "sink": r.normal(L, H, scale=0.02),
    }
    return Prefill(cfg, params, DEVICE, seq_len=case["T"])


def prepare(case, seed):
    r, kind = _Inputs(seed), case["kind"]
    s = {"case": case}
    if kind in ("prompt", "score"):
        s["model"] = _model(r, case)
        s["tokens"] = r.ints(case["V"], case["B"], case["T"])
        if kind == "score":
            s["targets"] = r.ints(case["V"], case["B"], case["T"])
        return s
    if kind in ("score_head", "train_head"):
        N, d, V = case["N"], case["d"], case["V"]
        s["h"], s["embed"] = r.normal(N, d, dtype=torch.bfloat16), r.normal(V, d, scale=0.02)
        s["targets"] = r.ints(V, N).to(torch.int32)
        if kind == "train_head":
            s["h"].requires_grad_(True), s["embed"].requires_grad_(True)
        else:
            s["embed"] = s["embed"].bfloat16()            # an evaluator keeps the cast copy
        return s
    B, H, D = case["B"], case["H"], case["D"]
    s["sink"] = r.normal(H, scale=0.02)
    if kind == "decode":
        room = 1 << (case["Tk"] - 1).bit_length()         # the cache is allocated ahead of what is filled
        s["q"] = r.normal(B, H, 1, D, dtype=torch.bfloat16)
        s["k"], s["v"] = (r.normal(B, H, room, D, dtype=torch.bfloat16)[:, :, :case["Tk"]] for _ in range(2))
        return s
    T = case["T"]
    dtype = torch.float32 if case.get("dtype") == "float32" else torch.bfloat16
    if kind == "attention":                               # what a QK-norm leaves: dense, rows of unit mean square
        s["q"], s["k"], s["v"] = (r.normal(B, H, T, D, dtype=dtype) for _ in range(3))
        return s
    s["q"], s["k"], s["v"] = (r.heads(B, H, T, D, dtype) for _ in range(3))
    s["q_gain"], s["k_gain"] = (r.normal(D, scale=0.1, shift=1.0) for _ in range(2))
    if kind == "layer":
        s["cos"], s["sin"] = A.cayley_table_geometric(D, T, device=DEVICE)
        return s
    s["d_o"] = r.heads(B, H, T, D)                        # the out-projection hands its gradient back in this layout
    if kind == "train_layer":
        for name in ("q", "k", "v", "q_gain", "k_gain", "sink"):
            s[name].requires_grad_(True)
    return s


# --------------------------------------------------------------------------------------------- run

def run(s):
    kind = s["case"]["kind"]
    if kind == "decode":
        return A.decode_attention(s["q"], s["k"], s["v"], s["sink"], **ATTN)
    if kind == "attention":
        return A.flash_attention(s["q"], s["k"], s["v"], s["sink"], kind="asinh", block=s["case"]["T"], range_guard=True,
                                 **ATTN)
    if kind == "layer":
        return A.flash_attention(s["q"], s["k"], s["v"], s["sink"], kind="asinh", block=s["case"]["T"], range_guard=True,
                                 q_gain=s["q_gain"], k_gain=s["k_gain"], cos=s["cos"], sin=s["sin"], **ATTN)
    if kind == "train_layer":
        o = G.attention(G.qk_norm(s["q"], s["q_gain"]), G.qk_norm(s["k"], s["k_gain"]), s["v"], s["sink"], **ATTN)
        grads = torch.autograd.grad(o, [s[x] for x in ("q", "k", "v", "q_gain", "k_gain", "sink")], s["d_o"])
        return [o.detach(), *grads]
    if kind == "train_ops":
        q, k = A.qk_rms_norm(s["q"], s["q_gain"]), A.qk_rms_norm(s["k"], s["k_gain"])
        o, stat, which = A.flash_attention(q, k, s["v"], s["sink"], kind="asinh", block=s["case"]["T"], range_guard=True,
                                           return_stat=True, **ATTN)
        dqn, dkn, dv, dsink = A.flash_attention_backward(q, k, s["v"], o, s["d_o"], stat, which, s["sink"], **ATTN)
        dq, dqg = A.qk_rms_norm_backward(s["q"], s["q_gain"], dqn)
        dk, dkg = A.qk_rms_norm_backward(s["k"], s["k_gain"], dkn)
        return [o, dq, dk, dv, dqg, dkg, dsink]
    if kind == "score_head":
        obj, tel, nll = A.fused_head(s["h"], s["embed"], s["targets"], kind=s["case"]["head"], block_n=s["case"]["N"],
                                     want_nll=True, **HEAD)
        return [obj, tel, nll]
    if kind == "train_head":
        obj, tel = G.head_loss(s["h"], s["embed"], s["targets"], kind=s["case"]["head"], **HEAD)
        return [obj.detach(), tel, *torch.autograd.grad(obj, [s["h"], s["embed"]])]
    if kind == "prompt":
        return s["model"].hidden(s["tokens"])
    obj, _, nll = s["model"].loss(s["tokens"], s["targets"], want_nll=True)
    return [obj, nll]


# ------------------------------------------------------------------------------- work and tolerance

def work(case):
    """What one pass cannot do without: every input and output once, the causal half of the score matrix."""
    kind = case["kind"]
    if kind in ("prompt", "score"):
        cfg = PrefillConfig.preset(case["size"], vocab_size=case["V"])
        L, d, f, V, n_tok = cfg.n_layers, cfg.d_model, cfg.d_ff, case["V"], case["B"] * case["T"]
        matrices = L * (4 * d * d + 3 * d * f)
        flops = 2.0 * n_tok * matrices + L * 2.0 * n_tok * (case["T"] + 1) * d
        if kind == "prompt":
            return {"bytes": 2.0 * matrices + n_tok * (8.0 + 2 * 2 * d), "flops": flops}
        return {"bytes": 2.0 * (matrices + V * d) + n_tok * 24.0, "flops": flops + 2.0 * n_tok * V * d}
    if kind in ("score_head", "train_head"):
        N, d, V = case["N"], case["d"], case["V"]
        if kind == "score_head":
            return {"bytes": 2.0 * N * d + 2.0 * V * d + 12.0 * N, "flops": 2.0 * N * d * V}
        # forward and both gradients; h, dh in bf16, the embedding and its gradient in float32
        return {"bytes": 4.0 * N * d + 8.0 * V * d + 8.0 * N, "flops": 6.0 * N * d * V}
    B, H, D = case["B"], case["H"], case["D"]
    if kind == "decode":
        return {"bytes": 4.0 * B * H * (case["Tk"] + 1) * D, "flops": 4.0 * B * H * case["Tk"] * D}
    T = case["T"]
    size = 4.0 if case.get("dtype") == "float32" else 2.0
    rows, forward = float(B) * H * T * D, 2.0 * B * H * T * (T + 1) * D
    if kind in ("attention", "layer"):
        return {"bytes": 4.0 * rows * size, "flops": forward}
    # q, k, v, d_o in; o and three gradients out; the backward's products are 2.5 times the forward's
    return {"bytes": 8.0 * rows * size, "flops": 3.5 * forward}


def tolerance(case):
    """About four times what each path differs by from itself in float64 (the models: from the same weights with
    the norms and projections as separate steps, which moves where bf16 rounds; deep ones at random weights
    amplify that)."""
    kind = case["kind"]
    if kind == "decode":
        return {"rel": 0.007}                             # seen 1.7e-3: the rounding of the output
    if kind == "attention":
        return {"rel": 0.01}                              # 2.3e-3: weights and output in bf16
    if kind == "layer":                                   # 8.6e-6; 6.6e-3: q and k rounded after norm and rotation
        return {"rel": 4e-5} if case["dtype"] == "float32" else {"rel": 0.025}
    if kind in ("train_layer", "train_ops"):
        return {"rel": 0.025}                             # 6.8e-3 (the sink's gradient), 5.2e-3 elsewhere
    if kind == "score_head":
        return {"rel": 1e-5}                              # 2.0e-6: float32 sums over the vocabulary
    if kind == "train_head":
        return {"rel": 0.01}                              # 2.4e-3: bf16 logit gradients
    if kind == "score":
        return {"rel": 0.025}                             # 1.2e-3 (125m), 6.4e-3 (1b)
    return {"rel": 0.03}                                  # 1.2e-2 (125m), 2.4e-2 (350m)
