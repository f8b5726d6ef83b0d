"""The prefill's native loop over the blocks is its operators called in turn, bit for bit."""

import pytest
import torch

import algebraic_transformer_b200 as A
from algebraic_transformer_b200 import ops
from algebraic_transformer_b200 import prefill as P

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("B,T,D", [(1, 1, 64), (3, 77, 64), (2, 129, 128), (5, 1100, 64)])
def test_prefill_blocks_are_the_operators_in_turn(B, T, D):
    cfg = P.PrefillConfig(vocab_size=320, d_model=2 * D, n_layers=2, n_heads=2, d_ff=256)
    m = P.Prefill(cfg, P.init_params(cfg, seed=3), DEV, seq_len=T)
    tokens = torch.randint(0, 320, (B, T), generator=torch.Generator().manual_seed(81)).to(DEV)
    d, H, p = cfg.d_model, cfg.n_heads, m.p
    x = ops.rms_norm(p["embed"][tokens], p["embed_gain"]).view(B * T, d)
    ss = ops.row_sumsq(x)
    for i in range(cfg.n_layers):
        words = torch.zeros(4, dtype=torch.int32, device=DEV)
        qkv = ops.qkv_projection(x, p["w_qkv_t"][i], H, T, m.cos_lp, m.sin_lp, p["q_gain"][i], p["k_gain"][i],
                                 guard_words=words, row_ss=ss).view(B, T, 3, H, D)
        q, k, v = (qkv[:, :, j].transpose(1, 2) for j in range(3))
        o = torch.empty((B, T, H, D), dtype=torch.bfloat16, device=DEV)
        A.flash_attention(q, k, v, p["sink"][i], kind="asinh", n=cfg.attn_n, c=cfg.attn_c, block=T, range_guard=True,
                          guard_words=words, out=o.transpose(1, 2))
        x, ss = ops.resid_projection(o.view(B * T, d), p["w_o_t"][i], x)
        x, ss = ops.resid_projection(ops.glu_projection(x, p["w_gu_t"][i], cfg.alu_beta, row_ss=ss), p["w_d_t"][i], x)
    assert torch.equal(m.hidden(tokens), ops.rms_norm(x, p["final_gain"]).view(B, T, d))
    with pytest.raises(ValueError):
        m.hidden(torch.zeros((1, T + 1), dtype=torch.int64, device=DEV))   # longer than the rotation tables
