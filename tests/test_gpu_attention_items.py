"""Short problems, where an item is one query tile: lengths around the tile, one head and enough of them to turn the rule,
both head_dims, with the saved statistic, against the oracle."""

import pytest
import torch

import algebraic_transformer_b200 as A
from oracle import algebraic_ref as R

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rel_l2(a, b):
    a, b = a.detach().double().cpu(), b.detach().double().cpu()
    return float((a - b).norm() / b.norm().clamp_min(1e-30))


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,H,T", [(1, 1, 1), (1, 3, 128), (1, 2, 129), (2, 3, 300), (4, 12, 385), (1, 2, 1025), (12, 16, 257)])
def test_short_attention(B, H, T, D):
    g = torch.Generator().manual_seed(T + D)
    q, k, v = (torch.randn((B, H, T, D), generator=g).bfloat16() for _ in range(3))
    sink = torch.randn(H, generator=g) * 0.5
    want = R.asinh_attention(q, k, v, n=16, c=8.0, sink_logit=sink)
    out = torch.full((B, H, T + 2, D), 7.0, dtype=torch.bfloat16, device=DEV)
    got, stat, which = A.flash_attention(q.to(DEV), k.to(DEV), v.to(DEV), sink.to(DEV), kind="asinh", n=16, c=8.0, block=T,
                                         range_guard=True, return_stat=True, out=out[:, :, :T])
    assert rel_l2(got, want) < 1e-2 and (out[:, :, T:] == 7.0).all()
    mma = A.flash_attention(q.to(DEV), k.to(DEV), v.to(DEV), sink.to(DEV), kind="asinh", n=16, c=8.0, block=T, range_guard=True,
                            return_stat=True, impl="mma")
    assert rel_l2(stat, mma[1]) < 1e-2 and int(which) == int(mma[2])
