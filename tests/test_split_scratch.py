"""The scratch of decode attention, without a GPU: what each layer of a step is handed must hold a place for everything that the
layer's launch writes, in whatever order the layers come."""
import itertools
import types

import pytest
import torch

from llmserver_b200.ops import attention_bf16

# (heads, key/value heads, size of keys, of values, window, bias by distance)
LAYERS = {"windowed": (32, 8, 128, 128, 256, False), "narrow": (32, 8, 64, 64, 0, False), "wide values": (32, 8, 64, 128, 0, False),
          "narrow values": (32, 4, 128, 64, 0, False), "bias": (32, 8, 128, 128, 0, True)}


@pytest.fixture
def launches(monkeypatch):
    """The wrapper on a GPU of 148 SMs whose launches are written down instead."""
    made = []
    monkeypatch.setattr(attention_bf16, "_sm_count", lambda device: 148)
    monkeypatch.setattr(attention_bf16, "check", lambda tensor, *_: tensor)
    monkeypatch.setattr(attention_bf16, "stream_handle", lambda: 0)
    monkeypatch.setattr(attention_bf16, "wait_error_flag", lambda device: torch.zeros(1, dtype=torch.int32))
    monkeypatch.setattr(attention_bf16, "call", lambda name, *args: made.append((name, args)))
    return made


def run(layer, batch):
    heads, kv_heads, dim, value_dim, window, bias = layer
    k_pages, v_pages = (torch.zeros((4, kv_heads, 16, size), dtype=torch.bfloat16) for size in (dim, value_dim))
    q_stride = heads * dim + kv_heads * (dim + value_dim)
    attention_bf16.try_attention_precise(torch.zeros((batch.n_tokens, q_stride), dtype=torch.bfloat16), q_stride, batch,
                                         torch.zeros((batch.n_seqs, 200), dtype=torch.int32), k_pages, v_pages, heads, kv_heads, dim, value_dim,
                                         dim ** -0.5, window, None, bias_log2=torch.zeros((heads, 64)) if bias else None)


@pytest.mark.parametrize("q_lens,contexts", [([100, 1, 1], [100, 1400, 1400]), ([512] + [1] * 13, [512] + [1500] * 13), ([1, 1, 100], [1400, 1400, 100]),
                                             ([1] * 5, [3000] * 5)])
@pytest.mark.parametrize("order", list(itertools.permutations(LAYERS, 2)), ids=" then ".join)
def test_every_layer_gets_scratch_of_its_own_size(launches, order, q_lens, contexts):
    starts = [0] + list(itertools.accumulate(q_lens))
    batch = types.SimpleNamespace(q_lens=q_lens, context_lens=contexts, n_seqs=len(q_lens), n_tokens=sum(q_lens), scratch={},
                                  q_start=torch.tensor(starts, dtype=torch.int32), context_len=torch.tensor(contexts, dtype=torch.int32))
    for name in order:
        launches.clear()
        run(LAYERS[name], batch)
        (_, args), = [launch for launch in launches if launch[0] == "llm_attention_mma_sinks"]
        split_len, max_splits, out, statistics, counters = args[28:33]
        if max_splits <= 1:
            continue
        by_length = 0 < -split_len < max_splits
        assert bool(counters) == by_length
        heads, value_dim = LAYERS[name][0], LAYERS[name][3]
        last = batch.n_seqs - 1 if by_length else max(start for start, count in zip(starts, q_lens) if count == 1)
        held = {tensor.data_ptr(): tensor for entry in batch.scratch.values() if isinstance(entry, tuple) for tensor in entry if torch.is_tensor(tensor)}
        assert held[out].numel() >= (last + 1) * heads * max_splits * value_dim, name
        assert held[statistics].numel() >= (last + 1) * heads * max_splits * 2, name
