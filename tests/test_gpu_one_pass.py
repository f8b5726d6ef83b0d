"""Passes that were joined or taken out: the head gradient's scale, the fp32 layer's preparation, the copy of an output
gradient in another layout."""

import pytest
import torch

import algebraic_transformer_b200 as A
from algebraic_transformer_b200 import autograd as G
from algebraic_transformer_b200 import ops
from oracle import algebraic_ref as R

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rel_l2(a, b):
    a, b = a.detach().double().cpu(), b.detach().double().cpu()
    return float((a - b).norm() / b.norm().clamp_min(1e-30))


def randn(shape, seed, dtype=torch.float32, scale=1.0):
    return (torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * scale).to(dtype)


@pytest.mark.parametrize("n,offset", [(0, 0), (1, 0), (7, 0), (4099, 0), (4099, 1)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_scale_by(n, offset, dtype):
    x, s = randn((n + offset,), 61, torch.bfloat16).to(DEV)[offset:], torch.tensor(1.7, device=DEV)
    assert torch.equal(ops.scale_by(x, s, dtype), (x.float() * s).to(dtype))


@pytest.mark.parametrize("embed_dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_head_loss_scales_its_gradients(embed_dtype):
    h, e = randn((65, 64), 62, torch.bfloat16).to(DEV).requires_grad_(True), randn((72, 64), 63, embed_dtype).to(DEV).requires_grad_(True)
    t = torch.arange(65, device=DEV)
    obj, _ = G.head_loss(h, e, t)
    one = torch.autograd.grad(obj, (h, e), retain_graph=True)
    two = torch.autograd.grad(obj * 3, (h, e), retain_graph=True)
    many = torch.autograd.grad(obj, (h, e), torch.tensor([1.0, 3.0], device=DEV), retain_graph=True, is_grads_batched=True)
    slope = torch.autograd.grad(obj * 3, (h, e), create_graph=True)
    for a, b, c, s in zip(one, two, many, slope):
        assert a.dtype == b.dtype and rel_l2(b, 3 * a.float()) < 5e-3      # a bf16 rounding
        assert torch.equal(c[0], a) and torch.equal(c[1], b) and torch.equal(s, b)


# in range (tcgen05 on the hi | lo copies) and out of range (the max-shifted form reads the fp32 rows)
@pytest.mark.parametrize("vscale", [1.0, 1e9])
@pytest.mark.parametrize("B,H,T", [(1, 1, 1), (2, 9, 130), (1, 3, 515)])
def test_fp32_layer_preparation(B, H, T, vscale):
    q, k, v = (randn((B, T, H, 64), 71 + i).transpose(1, 2) for i in range(3))
    v = v * vscale
    gain, sink = 0.5 + torch.rand(64, generator=torch.Generator().manual_seed(74)), randn((H,), 75, scale=0.5)
    cos, sin = R.cayley_table_geometric(64, T)
    want = R.asinh_attention(R.apply_rotary(R.rms_norm(q, gain), cos, sin), R.apply_rotary(R.rms_norm(k, gain), cos, sin), v,
                             n=16, c=8.0, sink_logit=sink)
    q, k, v, gain, sink, cos, sin = (t.to(DEV) for t in (q, k, v, gain, sink, cos, sin))
    got = A.flash_attention(q, k, v, sink, kind="asinh", n=16, c=8.0, block=T, range_guard=True, q_gain=gain, k_gain=gain,
                            cos=cos, sin=sin)
    assert rel_l2(got, want) < 1e-4                                # 16 mantissa bits of weights and values
    q, k = (A.qk_rms_norm(x, gain, cos=cos, sin=sin) for x in (q, k))
    assert torch.equal(got, A.flash_attention(q, k, v, sink, kind="asinh", n=16, c=8.0, block=T, range_guard=True))


# dense, (B, T, H, D) rows, rows apart by more than D, misaligned rows, an expanded gradient; both kernel families
@pytest.mark.parametrize("layout", ["dense", "bthd", "wide", "odd", "expanded"])
@pytest.mark.parametrize("impl", ["auto", "mma"])
def test_output_gradient_layouts(layout, impl):
    B, H, T, D = 2, 3, 130, 64
    q, k, v = (randn((B, H, T, D), 81 + i, torch.bfloat16).to(DEV) for i in range(3))
    sink, g = randn((H,), 84, scale=0.3).to(DEV), randn((B, T, H, D), 85, torch.bfloat16).to(DEV)
    o, stat, which = A.flash_attention(q, k, v, sink, kind="asinh", n=16, c=8.0, block=T, range_guard=True, return_stat=True)
    if layout == "bthd":
        g = g.transpose(1, 2)
    elif layout in ("wide", "odd"):
        g = torch.zeros((B, H, T, D + (8 if layout == "wide" else 2)), dtype=torch.bfloat16, device=DEV)[..., :D].copy_(g.transpose(1, 2))
    elif layout == "expanded":
        g = g[:, :1, :1, :1].expand(B, H, T, D)
    else:
        g = g.transpose(1, 2).contiguous()
    got = ops.flash_attention_backward(q, k, v, o, g, stat, which, sink, impl=impl)
    want = ops.flash_attention_backward(q, k, v, o, g.contiguous(), stat, which, sink, impl=impl)
    for a, b in zip(got[:3], want[:3]):
        assert torch.equal(a, b)
    assert rel_l2(got[3], want[3]) < 1e-5                          # the sink's gradient adds its blocks in any order


def test_backward_in_a_thread_without_a_context():
    """The first CUDA work of a thread may be the backward call: nothing before it has bound a context there."""
    import threading
    B, H, T, D = 1, 2, 64, 64
    q, k, v = (randn((B, H, T, D), 91 + i, torch.bfloat16).to(DEV) for i in range(3))
    o, stat, which = A.flash_attention(q, k, v, None, kind="asinh", n=16, c=8.0, block=T, range_guard=True, return_stat=True)
    want, got = ops.flash_attention_backward(q, k, v, o, o, stat, which), []
    t = threading.Thread(target=lambda: got.extend(ops.flash_attention_backward(q, k, v, o, o, stat, which)[:3]))
    t.start(), t.join()
    assert len(got) == 3 and all(torch.equal(a, b) for a, b in zip(got, want))
