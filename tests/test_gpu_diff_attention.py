"""Differential attention with maps of 64 and values of 128: the tcgen05 prompt kernel and the TMA decode kernel with the kernel
that subtracts the maps, against the kernel for every size."""
import pytest
import torch

from test_gpu_serving_sizes import DEVICE, HostBatch

pytestmark = pytest.mark.gpu


def case(seed, q_lens, contexts, heads, kv_heads, page_size, window):
    """Rows [heads x 2 x 64 | gate | padding] and shuffled pages; rows behind a context, and pages that the window has given back (their
    table entries are 0, page 0 belongs to nobody), hold NaN."""
    generator = torch.Generator(device=DEVICE).manual_seed(seed)
    counts = [-(-context // page_size) for context in contexts]
    pages = torch.randperm(sum(counts), generator=torch.Generator().manual_seed(seed)) + 1
    k_pages = torch.randn((sum(counts) + 1, kv_heads, page_size, 128), generator=generator, device=DEVICE).to(torch.bfloat16)
    v_pages = torch.randn((sum(counts) + 1, kv_heads, page_size, 128), generator=generator, device=DEVICE).to(torch.bfloat16)
    tables = torch.zeros((len(contexts), max(counts) + 1), dtype=torch.int32)
    k_pages[0] = v_pages[0] = float("nan")
    for row, (count, context, q_len) in enumerate(zip(counts, contexts, q_lens)):
        tables[row, :count], pages = pages[:count].to(torch.int32), pages[count:]
        last = int(tables[row, count - 1])
        k_pages[last, :, (context - 1) % page_size + 1:] = v_pages[last, :, (context - 1) % page_size + 1:] = float("nan")
        if window:
            tables[row, :max(0, context - q_len - window + 1) // page_size] = 0
    width = heads * 128 + -(-heads // 8) * 8 + 8
    qkv = torch.randn((sum(q_lens), width), generator=generator, device=DEVICE)
    qkv[:, :heads * 128] *= 2.0
    batch = HostBatch(q_lens, contexts)
    batch.max_q_len, batch.keys_settled = max(q_lens), True
    batch.positions = torch.cat([torch.arange(c - n, c) for c, n in zip(contexts, q_lens)]).to(torch.int32).to(DEVICE)
    batch.seq_of_token = torch.cat([torch.full((n,), row) for row, n in enumerate(q_lens)]).to(torch.int32).to(DEVICE)
    return qkv.to(torch.bfloat16), k_pages, v_pages, tables.to(DEVICE), batch


def both(heads, kv_heads, page_size, window, cap, q_lens, contexts, gate):
    from llmserver_b200 import ops
    from llmserver_b200.ops import attention_bf16
    from llmserver_b200.ops.library import check_wait_errors
    qkv, k_pages, v_pages, tables, batch = case(len(contexts) + window, q_lens, contexts, heads, kv_heads, page_size, window)
    out = {}
    for kernel in ("tcgen05", "generic"):
        before, attention_bf16.DIFF_KERNEL = attention_bf16.DIFF_KERNEL, kernel
        try:
            out[kernel] = ops.attention_diff(qkv, heads * 128 if gate else None, batch, tables, k_pages, v_pages, heads, kv_heads, 64, 128, 0.125,
                                             cap, window, 0.41, 1e-6, 0.8).double()
        finally:
            attention_bf16.DIFF_KERNEL = before
    torch.cuda.synchronize()
    check_wait_errors()
    got, want = out["tcgen05"], out["generic"]
    assert torch.isfinite(got).all() and torch.isfinite(want).all()
    # one rounding to bfloat16 each, and weights of 16 bits: the head norm divides by the size of a difference of two maps, here not
    # below a tenth of a map's, so 2^-16 of a map is at most 2^-12 of the row
    error = (got - want).abs() / torch.maximum(want.abs(), 0.05 * want.abs().amax(dim=-1, keepdim=True))
    assert error.max() <= 2.0 ** -7 + 0.05 * 2.0 ** -4, f"{float(error.max()):.2e}"


@pytest.mark.parametrize("pairing", [True, False])
@pytest.mark.parametrize("heads,kv_heads,page_size,window,cap", [(4, 4, 8, 0, 0.0), (8, 2, 16, 70, 30.0), (16, 2, 16, 1024, 50.0), (6, 2, 64, 129, 30.0),
                                                                 (3, 1, 32, 1, 0.0)])
def test_prompt_portions(heads, kv_heads, page_size, window, cap, pairing):
    """Whole prompts on both sides of a row tile and of a key tile, portions behind cached tokens, single tokens beside them."""
    from llmserver_b200.ops import attention_bf16
    attention_bf16.FORCE_PAIRING = pairing
    try:
        both(heads, kv_heads, page_size, window, cap, [1, 33, 64, 65, 2, 127, 200, 1], [1, 33, 64, 65, 300, 1400, 200, 2500], True)
        both(heads, kv_heads, page_size, window, cap, [17], [17], False)
    finally:
        attention_bf16.FORCE_PAIRING = None


MANY = [1, 63, 64, 65, 127, 128, 129, 700, 3000, 2, 1025, 1087, 1088, 1089]


@pytest.mark.parametrize("heads,kv_heads,page_size,contexts", [(4, 4, 8, [1]), (8, 1, 16, [2500]), (32, 8, 16, [900, 64, 2100]), (16, 2, 64, MANY),
                                                               (32, 8, 32, MANY * 5)])
@pytest.mark.parametrize("window,cap", [(0, 0.0), (1024, 30.0), (100, 50.0)])
def test_single_tokens(heads, kv_heads, page_size, contexts, window, cap):
    """From one block to more than a wave of them; contexts of one split, of several, and beyond the window."""
    both(heads, kv_heads, page_size, window, cap, [1] * len(contexts), contexts, True)


def test_single_tokens_beside_portions_run_the_decode_kernel(monkeypatch):
    """In one block of the prompt kernel a token would walk all of its context; results as in the tests above."""
    from llmserver_b200.ops import attention_bf16
    launch, launched = attention_bf16.call, []
    monkeypatch.setattr(attention_bf16, "call", lambda name, *args: (launched.append(name), launch(name, *args))[1])
    for q_lens, contexts in (([1, 40, 1], [3000, 700, 64]), ([200, 1], [200, 2500]), ([64], [64]), ([1, 1], [9, 900])):
        del launched[:]
        both(8, 2, 16, 0, 30.0, q_lens, contexts, True)
        kernels = [name for name in launched if "diff" in name]
        assert ("llm_attention_diff_decode" in kernels) == (1 in q_lens) and ("llm_attention_diff_prefill" in kernels) == (max(q_lens) > 1)
