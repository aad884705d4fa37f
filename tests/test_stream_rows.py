"""Which steps add to the residual stream and prepare the norms inside their products: rows, width and kind of step decide."""
from types import SimpleNamespace

import pytest
import torch

from llmserver_b200.parts.block import PreNormBlock


class RecordingNorm:
    def __init__(self):
        self.asked, self.unscaled = 0, []

    def sink(self, residual, consumer):
        self.asked += 1
        return SimpleNamespace(added=True)

    def add_norm(self, residual, delta, unscaled=False):
        self.unscaled.append(unscaled)
        return residual


class Consumer:
    takes_unscaled = feeds_stream = True

    def forward(self, x, *args, sink=None):
        return None if sink is not None else x


def inside(rows, width, max_q_len):
    norms = [RecordingNorm() for _ in range(3)]
    block = PreNormBlock({}, {"mixer": Consumer(), "feed_forward": Consumer(), "mixer_norm": norms[0], "feed_forward_norm": norms[1]})
    block.forward(torch.empty((rows, width)), None, SimpleNamespace(n_tokens=rows, max_q_len=max_q_len), None, after=(norms[2], None))
    taken = {norm.asked > 0 for norm in norms} | set(norms[0].unscaled + norms[1].unscaled)
    assert len(taken) == 1, "one way for the whole block"
    return taken.pop()


@pytest.mark.parametrize("rows,width,max_q_len,want", [
    (1, 4096, 1, True), (17, 4096, 1, True), (64, 4096, 1, True), (64, 5120, 1, True),
    (65, 4096, 1, False), (128, 2048, 1, False), (128, 5120, 1, False),            # replayed: the device decides
    (65, 4096, 65, True), (128, 4096, 128, True), (128, 2048, 100, True),          # prompts bound by their launches
    (64, 5120, 64, True), (65, 5120, 65, False), (128, 8192, 128, False),          # wide models are bound by the device
    (129, 4096, 129, False), (129, 4096, 1, False)])
def test_steps_inside_the_products(rows, width, max_q_len, want):
    assert inside(rows, width, max_q_len) is want


def test_the_environment_sets_the_bound_for_all(monkeypatch):
    from llmserver_b200.ops import stream
    for bound in (0, 16, 40, 128):
        monkeypatch.setattr(stream, "STREAM_ROWS", bound)
        monkeypatch.setattr(stream, "STREAM_MANY_ROWS", bound)
        assert {stream.stream_rows(width, decode) for width in (2048, 8192) for decode in (False, True)} == {bound}
