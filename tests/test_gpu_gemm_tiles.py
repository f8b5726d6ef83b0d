"""The projection and head GEMMs at the sizes where their tiles, CTA pairs and rounds turn: one row block and its
neighbours, an odd number of row blocks, ragged columns, more tiles than CTAs."""

import pytest
import torch

import algebraic_transformer_b200 as A
from algebraic_transformer_b200 import ops
from oracle import algebraic_ref as R

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rel_l2(a, b):
    a, b = a.detach().double().cpu(), b.detach().double().cpu()
    return float((a - b).norm() / b.norm().clamp_min(1e-30))


def randn(shape, seed, dtype=torch.float32, scale=1.0):
    return (torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * scale).to(dtype)


@pytest.mark.parametrize("M,K,N", [(1, 64, 128), (129, 128, 192), (257, 1024, 256), (613, 768, 768), (640, 2048, 768),
                                   (3000, 64, 320), (20000, 128, 768)])
def test_projections(M, K, N):
    x, w = randn((M, K), 41, torch.bfloat16).to(DEV), randn((N, K), 42, torch.bfloat16, 0.05).to(DEV)
    resid = randn((M, N), 43, torch.bfloat16).to(DEV)
    y, ss = ops.resid_projection(x, w, resid)
    want = (x.float() @ w.float().t() + resid.float()).bfloat16()
    assert rel_l2(y, want) < 1e-3                                  # sums in another order: an ulp of bf16 here and there
    assert rel_l2(ss.sum(0), y.double().square().sum(1)) < 1e-5
    f = 1024 if M > 4000 else 256
    wg, wu = (randn((f, K), 44 + i, torch.bfloat16, 0.05).to(DEV) for i in range(2))
    got = ops.glu_projection(x, ops.interleave_gate_up(wg, wu))
    want = ops.alu_glu((x.float() @ wg.float().t()).bfloat16(), (x.float() @ wu.float().t()).bfloat16())
    assert rel_l2(got, want) < 6e-3
    for D, H in ((64, 3), (128, 2)):
        cos, sin = (t.to(DEV) for t in R.cayley_table_geometric(D, M))
        w3 = randn((3 * H * D, K), 46, torch.bfloat16, 0.05).to(DEV)
        got = ops.qkv_projection(x, w3, H, M, cos.bfloat16(), sin.bfloat16()).view(M, 3, H, D)
        qkv = (x.float() @ w3.float().t()).bfloat16().view(1, M, 3, H, D)
        for i in range(3):
            want = qkv[:, :, i].transpose(1, 2)
            if i < 2:
                want = A.qk_rms_norm(want, None, cos=cos, sin=sin)
            assert rel_l2(got[:, i], want[0].transpose(0, 1)) < 6e-3


@pytest.mark.parametrize("kind", ["alg_ce", "ce"])
@pytest.mark.parametrize("N,d,V", [(1, 64, 8), (129, 128, 1000), (300, 192, 4104), (5000, 64, 6280)])
def test_head(N, d, V, kind):
    h, e = randn((N, d), 51, torch.bfloat16).to(DEV), randn((V, d), 52, torch.bfloat16, 0.1).to(DEV)
    t = torch.randint(0, V, (N,), generator=torch.Generator().manual_seed(53)).to(torch.int32).to(DEV)
    stats = ops.head_statistic(h, e, t, n=8, c=2.0, kind=kind)
    z = h.double() @ e.double().t()
    x = z / 2.0
    want = torch.logsumexp(z, 1) if kind == "ce" else ((x + torch.sqrt(1 + x * x)) ** 8).sum(1)
    assert rel_l2(stats[0], want) < 2e-5                           # fp32 products and sums over d and V
    assert rel_l2(stats[1], z.gather(1, t.long()[:, None])[:, 0]) < 2e-5
    dh, de = ops.fused_head_backward(h, e, t, stats, n=8, c=2.0, kind=kind)
    y = torch.zeros_like(z).scatter_(1, t.long()[:, None], 1.0)
    if kind == "ce":
        dz = (torch.softmax(z, 1) - y) / N
    else:
        r = 1 / torch.sqrt(1 + x * x)
        dz = (4.0 / N) * r * ((x + 1 / r) ** 8 / want[:, None] - y)
    assert rel_l2(dh, dz @ e.double()) < 1e-2 and rel_l2(de, dz.t() @ h.double()) < 1e-2
