"""The tcgen05 attention backward over sequence lengths around its tiles: 128 resident rows, 64 or 128
streamed ones (TMA zero fill past the end, masked statistics, masked stores)."""

import pytest
import torch

import algebraic_transformer_b200 as A
from oracle import algebraic_ref as R

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rel_l2(a, b):
    a, b = a.detach().double().cpu(), b.detach().double().cpu()
    return float((a - b).norm() / b.norm().clamp_min(1e-30))


def randn(shape, seed, dtype=torch.float32):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed)).to(dtype)


@pytest.mark.parametrize("T", [1, 63, 65, 128, 193, 300, 900])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("form,n", [("guard", 16), ("shift", 16), ("guard", 8)])
def test_backward_lengths(T, D, form, n):
    """Gradients against autograd through the oracle; every gradient tensor sits in front of a sentinel row that
    must survive, and a second run must repeat the first bit for bit.  Tolerance: the weights, dS and the
    outputs are rounded to bf16 (three roundings of at most 2^-9 relative each), as in the existing tests."""
    B, H = 2, 3
    q, k, v, d_o = (randn((B, H, T, D), 40 + i, torch.bfloat16) for i in range(4))
    sink = randn((H,), 44) * 0.5
    qf, kf, vf = (t.float().requires_grad_(True) for t in (q, k, v))
    sf = sink.clone().requires_grad_(True)
    R.asinh_attention(qf, kf, vf, n=n, c=8.0, sink_logit=sf).backward(d_o.float())
    # one row more than T per (batch, head), so that gradients (allocated with these strides) have a row behind them
    pad = [torch.zeros((B, H, T + 1, D), dtype=torch.bfloat16, device=DEV) for _ in range(3)]
    for buf, t in zip(pad, (q, k, v)):
        buf[:, :, :T] = t.to(DEV)
    qd, kd, vd = (buf[:, :, :T] for buf in pad)
    o, stat, kind = A.flash_attention(qd, kd, vd, sink.to(DEV), kind="asinh", n=n, c=8.0, block=T,
                                      range_guard=form == "guard", shift=True if form == "shift" else None,
                                      return_stat=True)
    runs = [A.flash_attention_backward(qd, kd, vd, o, d_o.to(DEV), stat, kind, sink.to(DEV), n=n, c=8.0) for _ in range(2)]
    for got, want in zip(runs[0], (qf.grad, kf.grad, vf.grad)):
        assert torch.isfinite(got).all() and rel_l2(got, want) < 2e-2
    # dsink = -sum_i delta_i p_sink,i n / (c sqrt(1 + (b/c)^2)) is a sum that cancels: the rounding of o to bf16 moves
    # delta_i = dO_i . o_i by at most 2^-9 sum_d |dO_id o_id|, and that bounds the sum
    x = (q.double() @ k.double().transpose(-1, -2)) / (D ** 0.5 * 8.0)
    bs = (sink.double() / 8.0).view(1, H, 1)
    p_sink = R.rho(bs) ** n / ((R.rho(x) ** n).tril().sum(-1) + R.rho(bs) ** n)
    slope = n / 8.0 / (1 + bs * bs).sqrt()
    bound = (p_sink * slope * (d_o.double().abs() * o.cpu().double().abs()).sum(-1)).sum((0, 2)) * 2.0 ** -9
    assert ((runs[0][3].cpu().double() - sf.grad.double()).abs() <= bound + 1e-4).all()
    for a, b in zip(runs[0][:3], runs[1][:3]):
        assert torch.equal(a, b)
    mma = A.flash_attention_backward(qd, kd, vd, o, d_o.to(DEV), stat, kind, sink.to(DEV), n=n, c=8.0, impl="mma")
    for got, want in zip(runs[0], mma):
        assert rel_l2(got, want) < (2e-2 if got.ndim == 4 else 1e-3)


@pytest.mark.parametrize("D", [64, 128])
def test_backward_stores_nothing_past_the_end(D):
    B, H, T = 1, 2, 70
    q, k, v, d_o = (randn((B, H, T, D), 50 + i, torch.bfloat16).to(DEV) for i in range(4))
    o, stat, kind = A.flash_attention(q, k, v, None, kind="asinh", n=16, c=8.0, block=T, range_guard=True, return_stat=True)
    want = A.flash_attention_backward(q, k, v, o, d_o, stat, kind, None, n=16, c=8.0)
    from algebraic_transformer_b200 import _lib as L
    outs = [torch.full((B * H * T * D + 128 * D,), 7.0, dtype=torch.bfloat16, device=DEV) for _ in range(3)]
    a = L.AttnBwdArgs(q=q.data_ptr(), k=k.data_ptr(), v=v.data_ptr(), o=o.data_ptr(), d_o=d_o.data_ptr(), stat=stat.data_ptr(),
                      stat_kind=kind.data_ptr(), dq=outs[0].data_ptr(), dk=outs[1].data_ptr(), dv=outs[2].data_ptr(), B=B, H=H,
                      Tq=T, Tk=T, D=D, n=16, c=8.0, causal=1)
    lib = L.load()
    ws = torch.empty(lib.alg_attn_bwd_workspace_bytes(a), dtype=torch.uint8, device=DEV)
    a.workspace, a.workspace_bytes = ws.data_ptr(), ws.numel()
    L.check(lib.alg_attn_bwd(a, torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    for got, w in zip(outs, want):
        assert torch.equal(got[:B * H * T * D].view(B, H, T, D), w)
        assert (got[B * H * T * D:] == 7.0).all()


@pytest.mark.parametrize("D", [64, 128])
def test_statistic_is_not_amplified(D):
    """The sink's gradient, the one fp32 output, for single rows: with a zero sink and one element of `d_o` it is a product of
    exact numbers, n, 1 / c and the saved 1 / l: five roundings.  l^(-1/n) raised to n again would be off by up to 16."""
    H, n, c = 512, 16, 8.0
    q, k, v = (randn((1, H, 1, D), 71 + i, torch.bfloat16).to(DEV) for i in range(3))
    sink = torch.zeros(H, device=DEV)
    o, stat, which = A.flash_attention(q, k, v, sink, kind="asinh", n=n, c=c, block=1, range_guard=True, return_stat=True)
    d_o = torch.zeros_like(o)
    d_o[..., 3] = 1.0
    assert int(which) == 1                                         # the unshifted form
    dsink = A.flash_attention_backward(q, k, v, o, d_o, stat, which, sink, n=n, c=c)[3]
    want = -(o[0, :, 0, 3].double() * stat[0, :, 0].double() * n / c)
    assert float(((dsink.double() - want) / want).abs().max()) < 5 * 2.0 ** -24
