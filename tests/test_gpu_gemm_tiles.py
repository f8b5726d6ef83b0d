"""The projection and head GEMMs at the sizes where their tiles and rounds turn: one row block and its neighbours, an odd
number of row blocks, ragged columns, more tiles than CTAs.  Short K or few rows leave a tile to one CTA; the sizes
of the tests named `pairs` are those at which two share one, which they ask the library."""

import ctypes as C
import math

import pytest
import torch

import algebraic_transformer_b200 as A
from algebraic_transformer_b200 import _lib as L
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


QKV, GLU, DZ, RESID, HEAD = range(5)


def plan(op, M, K, N, D=64):
    """(tile width, CTAs that share a tile, parts of K)"""
    out = [C.c_int() for _ in range(3)]
    assert L.load().alg_gemm_plan(op, M, K, N, D, *out) == L.ALG_OK
    return tuple(x.value for x in out)


def worst_row(a, b):
    """Largest relative error of a row: one wrong row among thousands would pass as a norm over all of them."""
    a, b = a.double(), b.double()
    return float(((a - b).norm(dim=-1) / b.norm(dim=-1).clamp_min(1e-30)).max())


# Rows: an odd number of 128-row blocks (the last pair's second CTA has none), the last one 37 rows; an even one, the last
# one 57 rows.  Columns: the last tile's second half of weight rows outside the matrix, or partly.
@pytest.mark.parametrize("M,K,H,D", [(100 * 128 + 37, 1536, 3, 64), (101 * 128 + 57, 1536, 3, 64), (148 * 128 + 37, 1536, 1, 128),
                                     (149 * 128 + 57, 1536, 1, 128)])
def test_qkv_pairs(M, K, H, D):
    assert plan(QKV, M, K, 3 * H * D, D)[:2] == (256, 2)
    x, w = randn((M, K), 71, torch.bfloat16).to(DEV), randn((3 * H * D, K), 72, torch.bfloat16, 0.05).to(DEV)
    T = 1000
    cos, sin = (t.to(DEV) for t in R.cayley_table_geometric(D, T))
    gq, gk = (randn((D,), 73 + i, scale=0.1).add_(1.0).to(DEV) for i in range(2))
    pad = -M % T                                                   # the stand-alone kernel wants whole sequences
    z = x.float() @ w.float().t()
    for row_ss in (None, ops.row_sumsq(x)):
        words = torch.zeros(4, dtype=torch.int32, device=DEV)
        got = ops.qkv_projection(x, w, H, T, cos.bfloat16(), sin.bfloat16(), gq, gk, guard_words=words, row_ss=row_ss).view(M, 3, H, D)
        zr = z if row_ss is None else z * torch.rsqrt(x.float().square().mean(1, keepdim=True) + 1e-5)
        ref = torch.nn.functional.pad(zr.bfloat16(), (0, 0, 0, pad)).view(-1, T, 3, H, D)
        for i in range(3):
            want = ref[:, :, i].transpose(1, 2)
            if i < 2:
                want = A.qk_rms_norm(want, (gq, gk)[i], cos=cos, sin=sin)
            want = want.transpose(1, 2).reshape(-1, H, D)[:M]
            # three roundings to bf16 (projection, norm, rotation), the rotation mixing two of them: 3 * 2^-9 * sqrt(2)
            assert worst_row(got[:, i], want) < 1e-2
        q2, k2, vmax = words[:3].view(torch.float32).tolist()
        scale = 1 / (math.sqrt(D) * 8.0)
        assert abs(q2 / float((got[:, 0].float() * scale).square().sum(-1).max()) - 1) < 1e-2
        assert abs(k2 / float(got[:, 1].float().square().sum(-1).max()) - 1) < 1e-2
        assert vmax == float(got[:, 2].float().abs().max())


@pytest.mark.parametrize("M", [100 * 128 + 37, 101 * 128 + 57])
def test_glu_pairs(M):
    K, f = 1536, 384
    assert plan(GLU, M, K, 2 * f)[:2] == (256, 2)
    x = randn((M, K), 81, torch.bfloat16).to(DEV)
    wg, wu = (randn((f, K), 82 + i, torch.bfloat16, 0.05).to(DEV) for i in range(2))
    w = ops.interleave_gate_up(wg, wu)
    for row_ss in (None, ops.row_sumsq(x)):
        tau = 1.0 if row_ss is None else torch.rsqrt(x.float().square().mean(1, keepdim=True) + 1e-5)
        want = ops.alu_glu((x.float() @ wg.float().t() * tau).bfloat16(), (x.float() @ wu.float().t() * tau).bfloat16())
        assert worst_row(ops.glu_projection(x, w, row_ss=row_ss), want) < 1e-2     # gate, up, activation, product: bf16 each


@pytest.mark.parametrize("M,N", [(88 * 128 + 37, 1152), (87 * 128 + 57, 1152), (100 * 128 + 37, 704)])
@pytest.mark.parametrize("in_place", [False, True])
def test_resid_pairs(M, N, in_place):
    K = 1536
    assert plan(RESID, M, K, N)[:2] == (256, 2)
    x, w = randn((M, K), 91, torch.bfloat16).to(DEV), randn((N, K), 92, torch.bfloat16, 0.05).to(DEV)
    resid = randn((M, N), 93, torch.bfloat16).to(DEV)
    want = (x.float() @ w.float().t() + resid.float()).bfloat16()
    y, ss = ops.resid_projection(x, w, resid, out=resid if in_place else None)
    assert worst_row(y, want) < 1e-3                               # sums in another order: an ulp of bf16 here and there
    assert rel_l2(ss.sum(0), y.double().square().sum(1)) < 1e-5


@pytest.mark.parametrize("kind", ["alg_ce", "ce"])
@pytest.mark.parametrize("N,d,V", [(16 * 128 + 37, 1536, 4984), (17 * 128 + 57, 1536, 5000), (34 * 128 + 37, 256, 19976)])
def test_head_pairs(N, d, V, kind):
    assert plan(HEAD, N, d, V)[1] == 2
    if d == 1536:
        assert plan(DZ, N, d, V)[:2] == (256, 2)
    h, e = randn((N, d), 94, torch.bfloat16).to(DEV), randn((V, d), 95, torch.bfloat16, 1.6 / math.sqrt(d)).to(DEV)
    t = torch.randint(0, V, (N,), generator=torch.Generator().manual_seed(96)).to(torch.int32).to(DEV)
    stats = ops.head_statistic(h, e, t, n=8, c=2.0, kind=kind)
    z = h.double() @ e.double().t()
    x = z / 2.0
    want = torch.logsumexp(z, 1) if kind == "ce" else ((x + torch.sqrt(1 + x * x)) ** 8).sum(1)
    assert worst_row(stats[0, :, None], want[:, None]) < 2e-5      # fp32 products and sums over d and V
    assert rel_l2(stats[1], z.gather(1, t.long()[:, None])[:, 0]) < 2e-5
    dh, de = ops.fused_head_backward(h, e, t, stats, n=8, c=2.0, kind=kind)
    y = torch.zeros_like(z).scatter_(1, t.long()[:, None], 1.0)
    if kind == "ce":
        dz = (torch.softmax(z, 1) - y) / N
    else:
        r = 1 / torch.sqrt(1 + x * x)
        dz = (4.0 / N) * r * ((x + 1 / r) ** 8 / want[:, None] - y)
    # bf16 dz (2^-9 an element, of either sign) and bf16 results; rows that no target falls into are small, not wrong
    assert worst_row(dh, dz @ e.double()) < 1e-2 and worst_row(de, dz.t() @ h.double()) < 1e-2
