"""A decode step that fails while it is being captured: the capture ends, the error comes through, the engine stays usable."""
import contextlib

import pytest
import torch

from qllm2_b200 import model as M
from qllm2_b200 import serving


class _Fake:
    """Stands in for torch.cuda: one stream that is in capture between capture_begin and capture_end."""

    def __init__(self, end_fails=False):
        self.log, self.capturing, self.end_fails = [], False, end_fails

    def Stream(self):
        return self

    def wait_stream(self, other):
        self.log.append("wait")

    def current_stream(self):
        return self

    def stream(self, side):
        return contextlib.nullcontext()

    def is_current_stream_capturing(self):
        return self.capturing

    def CUDAGraph(self):
        return self

    def capture_begin(self):
        self.log.append("begin")
        self.capturing = True

    def capture_end(self):
        self.log.append("end")
        self.capturing = False
        if self.end_fails:
            raise RuntimeError("the capture was invalidated")


@pytest.mark.parametrize("begin,end_fails", [(True, False), (True, True), (False, False)])
def test_capture_ends_when_its_body_fails(monkeypatch, begin, end_fails):
    fake = _Fake(end_fails)
    monkeypatch.setattr(serving.torch, "cuda", fake)
    with pytest.raises(ValueError, match="the body's error"):
        with serving._captured() as graph:
            if begin:
                graph.capture_begin()
            raise ValueError("the body's error")
    assert not fake.capturing
    assert fake.log == (["wait", "begin", "end", "wait"] if begin else ["wait", "wait"])


def test_capture_ends_once_when_its_body_succeeds(monkeypatch):
    fake = _Fake()
    monkeypatch.setattr(serving.torch, "cuda", fake)
    with serving._captured() as graph:
        graph.capture_begin()
    assert fake.log == ["wait", "begin", "end", "wait"]


@pytest.mark.gpu
def test_engine_survives_an_error_under_capture(monkeypatch):
    torch.manual_seed(0)
    cfg = M.V11Config(vocab_size=101, dim=64, n_heads=1, head_dim=64, n_layers=1, dropout=0.0, gradient_checkpointing=False, max_seq_len=64)
    net = M.V11LM(cfg).to("cuda").bfloat16().eval()

    def tokens(eng):
        rid = eng.submit([5, 9, 2, 77], 6)
        return eng.run()[rid]

    want = tokens(serving.ContinuousBatcher(net, n_slots=2, max_position=64))
    eng = serving.ContinuousBatcher(net, n_slots=2, cuda_graph=True, max_position=64)
    step = eng._decode_tensors

    def failing(*args):
        if torch.cuda.is_current_stream_capturing():
            raise ValueError("host error under capture")
        return step(*args)

    monkeypatch.setattr(eng, "_decode_tensors", failing)
    with pytest.raises(ValueError, match="under capture"):
        eng.warmup()
    assert eng._graph is None and not torch.cuda.is_current_stream_capturing()
    torch.cuda.synchronize()
    monkeypatch.undo()
    assert tokens(eng) == want
