"""Who says that recurrent states may be read before the kernel in front has ended: the engine's steps, which run every layer once
behind the copy of their batch, and nobody who does not ask for it."""
import torch

from llmserver_b200 import ops
from llmserver_b200.cache import CacheManager
from llmserver_b200.engine.batch import SequenceSlice, build_batch
from llmserver_b200.engine.step import StepFunction
from llmserver_b200.ops import attention_bf16
from llmserver_b200.sampling import SamplingRow
from stubs import ArgmaxSampler, StubModel
from test_decode_rows import DeviceStyleSampler


def test_a_state_is_read_early_only_when_the_caller_says_so(monkeypatch):
    launches = []
    monkeypatch.setattr(ops, "check", lambda tensor, *_, **__: tensor)
    monkeypatch.setattr(ops, "stream_handle", lambda: 0)
    monkeypatch.setattr(ops, "call", lambda name, *args: launches.append((name, args)))
    batch = build_batch([SequenceSlice("r", [1], 4, [0], [[0, 1]], 0)], 1, "cpu")
    assert batch.keys_settled and not batch.states_settled

    def early(**given):
        ops.gla_recurrent(torch.zeros((1, 384), dtype=torch.bfloat16), 0, 64, 128, 256, torch.zeros((1, 64)), None, torch.ones(128),
                          torch.zeros((1, 1, 64, 128)), batch, 1, 64, 128, 16.0, 0.125, 1e-5, **given)
        name, args = launches.pop()
        assert name == "llm_gla_recurrent" and args[-3] == 1      # single tokens
        return args[-2]

    assert early() == 0 and early(settled=False) == 0 and early(settled=True) == 1
    monkeypatch.setattr(attention_bf16, "EARLY_KEYS", False)
    assert early(settled=True) == 0


def test_steps_of_the_engine_say_so():
    model = StubModel()
    cache = CacheManager(model.cache_needs(), 4, 8, num_slots=2, prefix_sharing=False)
    model.bind_cache(cache)
    seen, step_of = [], model.step
    model.step = lambda batch: (seen.append(batch.states_settled), step_of(batch))[1]
    step = StepFunction(model, cache)
    step.admit("r")
    step.run([("r", [1, 2, 3], [2])])
    step.run_and_sample([("r", [4], [0])], [SamplingRow()], sampler=DeviceStyleSampler())
    step.run_and_sample([("r", [5], [0])], [SamplingRow()], sampler=ArgmaxSampler())
    assert seen == [True] * 3
