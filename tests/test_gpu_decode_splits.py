"""Decode at the sizes where its grid rule turns or a ring slot, a tile or a split is not full: one key, one tile and one
key more, one CTA per head and several, one and two CTAs per SM, more heads than CTAs fit."""

import math
import os
import subprocess
import sys

import pytest
import torch

import algebraic_transformer_b200 as A
from oracle import algebraic_ref as R

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rel_l2(a, b):
    a, b = a.detach().double().cpu(), b.detach().double().cpu()
    return float((a - b).norm() / b.norm().clamp_min(1e-30))


def randn(shape, seed, dtype=torch.float32, scale=1.0):
    return (torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * scale).to(dtype)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,H,Tk", [(1, 1, 1), (1, 1, 33), (13, 23, 65), (32, 12, 200), (2, 74, 129), (10, 15, 385), (1, 2, 20000)])
def test_decode_splits(B, H, Tk, D):
    q, k, v = (randn((B, H, n, D), 31 + i, torch.bfloat16) for i, n in enumerate((1, Tk + 3, Tk)))
    k = k.to(DEV)[:, :, :Tk]                                       # a cache with room to grow
    for sink in (randn((H,), 34, scale=0.5), None):
        want = R.asinh_attention(q, k.cpu(), v, n=16, c=8.0, sink_logit=sink, causal=False)
        got = A.decode_attention(q.to(DEV), k, v.to(DEV), None if sink is None else sink.to(DEV), n=16, c=8.0)
        assert rel_l2(got, want) < 5e-3                            # the output's bf16 rounding: 2^-9 an element at most
        again = A.decode_attention(q.to(DEV), k, v.to(DEV), None if sink is None else sink.to(DEV), n=16, c=8.0)
        assert torch.equal(got, again)


@pytest.mark.parametrize("D", [64, 128])
def test_decode_extremes(D):
    """Scores far apart (the running maximum moves, weights underflow) and an infinite value."""
    q, k, v = (randn((1, 2, n, D), 41 + i, torch.bfloat16) for i, n in enumerate((1, 700, 700)))
    k = (k.float() * torch.logspace(-3, 3, 700)[None, None, :, None]).bfloat16()
    want = R.asinh_attention(q, k, v, n=16, c=8.0, causal=False)
    args = [t.to(DEV) for t in (q, k, v)]
    assert rel_l2(A.decode_attention(*args, n=16, c=8.0), want) < 5e-3
    args[2][0, 0, 5, 3] = float("inf")
    args[1][0, 0, 5] = args[0][0, 0, 0]                            # a key with weight
    got = A.decode_attention(*args, n=16, c=8.0).float()
    assert got[0, 0, 0, 3] == float("inf") and torch.isfinite(got[0, 1]).all() and torch.isfinite(got[0, 0, 0, :3]).all()


@pytest.mark.parametrize("D", [64, 128])
def test_decode_weights_keep_their_bits(D):
    """Two keys whose contributions cancel to about 2^-14: the output's rounding is far below the error of the weights.

    n = 2, so that nothing multiplies the error of a weight up: one score (2^-22 of it), one rho on either side of the shift
    (2^-22 each, approximate square root), a power of two and fp32 sums: below 2^-20 of the terms' size.  Weights cut to 16
    bits are off by up to 2^-18."""
    B, H, c = 4, 64, 8.0
    q, k = (randn((B, H, n, D), 61 + i, torch.bfloat16) for i, n in enumerate((1, 2)))
    x = (k.double() @ q.double().transpose(-1, -2))[..., 0] / (math.sqrt(D) * c)
    w = (x + torch.sqrt(1 + x * x)) ** 2
    ratio = w[..., :1] / w[..., 1:]
    v0 = torch.arange(128, 256).double() / 128                     # every mantissa of a bf16
    e = 2.0 ** torch.floor(torch.log2(ratio * v0))
    v1 = (ratio * v0 / e * 128).round() / 128 * e                  # the bf16 nearest to what would cancel it
    best = ((ratio * v0 - v1).abs() / v1).argsort(-1)[..., :D]
    v = torch.stack([v0[best], -torch.gather(v1, -1, best)], 2).bfloat16()
    got = A.decode_attention(q.to(DEV), k.to(DEV), v.to(DEV), n=2, c=c).cpu().double()[:, :, 0]
    terms = w[..., None] * v.double() / w.sum(-1)[..., None, None]
    want, size = terms.sum(2), terms.abs().sum(2)
    rounding = want.abs() * 2.0 ** -8                              # a bf16 next to the nearest one
    seen = rounding < 2.0 ** -22 * size                            # where the output shows the weights' error
    assert int(seen.sum()) > 1000
    assert float(((got - want).abs() / size)[seen].max()) < 2.0 ** -20 + 2.0 ** -22


STALE_WORDS = """
import torch
from algebraic_transformer_b200 import _lib as L
B, H, Tk, D = 1, 64, 1000, 64
q, k, v = (torch.randn(B, H, n, D, device="cuda").bfloat16() for n in (1, Tk, Tk))
o, want = torch.empty_like(q), None
lib = L.load()
a = L.DecodeArgs(q=q.data_ptr(), k=k.data_ptr(), v=v.data_ptr(), o=o.data_ptr(), B=B, H=H, Tk=Tk, D=D, n=16, c=8.0,
                 k_stride=L.I64x3(*k.stride()[:3]), v_stride=L.I64x3(*v.stride()[:3]))
size = lib.alg_decode_workspace_bytes(a)
splits = (size - B * H * 8) // (B * H * (D + 2) * 4)
assert splits > 1
for _ in range(H):
    ws = torch.full((size // 8,), -1, dtype=torch.int64, device="cuda")          # states: NaN
    ws[-H:] = (torch.arange(H, device="cuda") + 1) * 65536 + splits - 1          # "all but one split of call 1, 2, ..."
    a.workspace, a.workspace_bytes = ws.data_ptr(), size
    assert lib.alg_attn_decode(a, torch.cuda.current_stream().cuda_stream) == 0
    want = o.clone() if want is None else want
    assert torch.isfinite(o).all() and torch.equal(o, want)
"""


def test_stale_arrival_words():
    """A workspace that holds what the first calls of a process would leave, were their numbers counted from one."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", STALE_WORDS], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
