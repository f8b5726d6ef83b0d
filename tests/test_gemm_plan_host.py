"""What the GEMM kernels choose, asked of the library (148 SMs where there is no GPU)."""

import ctypes as C

import pytest

from algebraic_transformer_b200 import _lib as L

QKV, GLU, DZ, RESID, HEAD = range(5)


def plan(op, M, K, N, D=64):
    """(tile width, CTAs that share a tile, parts of K)"""
    out = [C.c_int() for _ in range(3)]
    assert L.load().alg_gemm_plan(op, M, K, N, D, *out) == L.ALG_OK
    return tuple(x.value for x in out)


def rounds(M, N, width):
    return -(-(-(-M // 128) * -(-N // width)) // 148)


@pytest.mark.parametrize("N", [768, 1024, 1536, 2048])
def test_residual_tile_follows_the_rounds_alone(N):
    """Equal rounds, equal tile: a row more or less changes nothing unless it changes the rounds."""
    seen = {}
    for M in range(128, 24577, 128):
        key = (rounds(M, N, 256), rounds(M, N, 128))
        width = plan(RESID, M, 768, N)[0]
        assert seen.setdefault(key, width) == width, (M, key)
        assert L.load().alg_resid_proj_ss_slots(M, N) == 2 * -(-N // width)
    assert seen[1, 1] == 128 and seen[2, 3] == 256 and seen[3, 5] == 256


def test_pairs_and_parts():
    assert plan(QKV, 16384, 1536, 4608) == (256, 2, 1) and plan(QKV, 613, 768, 2304) == (128, 1, 1)
    assert plan(GLU, 16384, 768, 4096) == (256, 2, 1) and plan(GLU, 613, 768, 4096)[1] == 1
    assert plan(RESID, 613, 2048, 768) == (128, 1, 4) and plan(RESID, 16384, 2048, 768) == (256, 2, 1)
    assert plan(HEAD, 8192, 768, 50304)[1] == 2 and plan(DZ, 8192, 768, 50304) == (256, 2, 1)
    assert L.load().alg_gemm_plan(5, 128, 64, 128, 64, None, None, None) == L.ALG_ERR_INVALID
    assert L.load().alg_gemm_plan(RESID, 2**31 - 1, 64, 2**31 - 1, 64, None, None, None) == L.ALG_ERR_INVALID
    assert L.load().alg_gemm_plan(RESID, 128, 65, 128, 64, None, None, None) == L.ALG_ERR_INVALID
