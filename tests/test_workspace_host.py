"""Which calls may share a scratch buffer: only calls that run one after the other."""

import threading

import pytest
import torch

from algebraic_transformer_b200 import ops

CPU = torch.device("cpu")


@pytest.fixture
def place(monkeypatch):
    """The stream that is current and whether it is being captured."""
    at = {"stream": 1, "capturing": False}
    monkeypatch.setattr(ops, "_raw_stream", lambda index: at["stream"], raising=False)
    monkeypatch.setattr(ops, "_capturing", lambda: at["capturing"], raising=False)
    monkeypatch.setattr(ops, "_kept", threading.local(), raising=False)
    return at


def take(nbytes=1000, tag="decode"):
    return ops._workspace(CPU, nbytes, tag)


def test_one_stream_keeps_its_buffer(place):
    first = take()
    assert take() is first and take(500) is first
    assert take(2000).numel() >= 2000 and take(tag="attn") is not take()


def test_streams_do_not_share(place):
    first = take()
    place["stream"] = 2
    assert take() is not first
    place["stream"] = 1
    assert take() is first


def test_threads_do_not_share(place):
    first, seen = take(), []
    t = threading.Thread(target=lambda: seen.append(take()))
    t.start()
    t.join()
    assert seen[0] is not first


def test_capture_has_a_buffer_of_its_own(place):
    first = take()
    place["capturing"] = True
    captured = take()
    assert captured is not first and take() is not captured
    place["capturing"] = False
    assert take() is first


def test_what_is_kept_is_bounded(place):
    big = take(ops._KEEP_BYTES + 1)
    assert big.numel() > ops._KEEP_BYTES and take(ops._KEEP_BYTES + 1) is not big
    for stream in range(3 * ops._KEEP_BUFFERS):
        place["stream"] = stream
        take()
        assert len(ops._kept.__dict__) <= ops._KEEP_BUFFERS
    for stream in range(20):
        place["stream"] = stream
        take(ops._KEEP_BYTES)
        assert sum(b.numel() for b in ops._kept.__dict__.values()) <= ops._KEEP_TOTAL
