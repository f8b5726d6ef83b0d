"""Failure detection without a GPU fault: a device-side wait that can never be satisfied
runs out after its budget, the kernel reports ALG_DEV_TIMEOUT through the status word and
returns, and the context stays usable for the next launch.  A result that such a wait concerns is not a plausible one."""

import pytest
import torch

import algebraic_transformer_b200 as A
from algebraic_transformer_b200 import _lib as L

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def test_bounded_wait_times_out_and_reports_status():
    lib = L.load()
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    waited = torch.zeros(1, dtype=torch.int64, device=DEV)
    budget_ns = 5_000_000                                  # 5 ms
    stream = torch.cuda.current_stream().cuda_stream
    assert lib.alg_selftest_bounded_wait(status.data_ptr(), budget_ns, waited.data_ptr(), stream) == L.ALG_OK
    torch.cuda.synchronize()                               # returns: the kernel did not hang
    assert int(status) == 1                                # ALG_DEV_TIMEOUT
    assert budget_ns <= int(waited) < 100 * budget_ns
    # the context is intact: a real kernel runs right after and gives the right answer
    x = torch.randn(4, 2, 16, 64, device=DEV)
    y = A.qk_rms_norm(x, torch.ones(64, device=DEV))
    want = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-5)
    assert torch.allclose(y, want, rtol=1e-5, atol=1e-6)
    # bad arguments are refused on the host
    assert lib.alg_selftest_bounded_wait(None, budget_ns, None, stream) == L.ALG_ERR_INVALID
    assert lib.alg_selftest_bounded_wait(status.data_ptr(), 5_000_000_000, None, stream) == L.ALG_ERR_INVALID


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("H,Tk,sink", [(296, 400, False), (296, 400, True), (4, 6000, True)])   # whole heads, and splits
def test_decode_timeout_leaves_no_plausible_row(H, Tk, D, sink):
    lib = L.load()
    q, k, v = (torch.randn(1, H, n, D, device=DEV).bfloat16() for n in (1, Tk, Tk))
    s = torch.randn(H, device=DEV) if sink else None
    want = A.decode_attention(q, k, v, s)
    o, status = torch.zeros_like(q), torch.zeros(1, dtype=torch.int32, device=DEV)
    a = L.DecodeArgs(q=q.data_ptr(), k=k.data_ptr(), v=v.data_ptr(), o=o.data_ptr(), sink=s.data_ptr() if sink else None, B=1,
                     H=H, Tk=Tk, D=D, n=16, c=8.0, k_stride=L.I64x3(*k.stride()[:3]), v_stride=L.I64x3(*v.stride()[:3]))
    ws = torch.zeros(lib.alg_decode_workspace_bytes(a), dtype=torch.uint8, device=DEV)
    a.workspace, a.workspace_bytes = ws.data_ptr(), ws.numel()
    stream = torch.cuda.current_stream().cuda_stream
    assert lib.alg_attn_decode_status(a, status.data_ptr(), stream) == L.ALG_OK
    torch.cuda.synchronize()
    assert int(status) == 0 and torch.equal(o, want)
    assert lib.alg_selftest_decode_timeout(a, 1, 2_000_000, status.data_ptr(), stream) == L.ALG_OK   # one tile of each split
    torch.cuda.synchronize()
    assert int(status) == 1 and torch.isnan(o).all()               # ALG_DEV_TIMEOUT
    assert torch.equal(A.decode_attention(q, k, v, s), want)
    assert lib.alg_selftest_decode_timeout(a, 1, 2_000_000, None, stream) == L.ALG_ERR_INVALID
    assert lib.alg_selftest_decode_timeout(a, 1, 5_000_000_000, status.data_ptr(), stream) == L.ALG_ERR_INVALID
