"""The TMA decode kernel's form with 16-bit-grade weights (sinks, chunks, kept first keys, gates) against the kernel for every
size, and the order in which its blocks take sequences."""
import pytest
import torch

from test_gpu_serving_sizes import DEVICE, HostBatch, paged_case, plain_rows, relative_error

pytestmark = pytest.mark.gpu

MANY = [1, 63, 64, 65, 127, 128, 129, 700, 4096, 2, 1025, 2047, 2048, 2049, 191, 192, 193]


def decode_batch(contexts):
    batch = HostBatch([1] * len(contexts), contexts)
    batch.max_q_len, batch.keys_settled = 1, True
    batch.positions, batch.seq_of_token = batch.context_len - 1, torch.arange(len(contexts), dtype=torch.int32, device=DEVICE)
    return batch


# no limit, windows on and off a tile's edge, with kept first keys, chunks, a gate, sinks
FORMS = [dict(), dict(sinks=True), dict(window=1024, gate=True), dict(window=100, keep=5, sinks=True), dict(window=129, keep=70, gate=True),
         dict(chunk=128), dict(chunk=1000, sinks=True, gate=True)]


@pytest.mark.parametrize("form", FORMS, ids=lambda form: "-".join(form) or "plain")
@pytest.mark.parametrize("heads,kv_heads,dim,page_size,contexts", [
    (4, 4, 128, 16, [1]), (16, 1, 128, 16, [3000]), (32, 8, 128, 16, [900, 64, 2500]), (10, 2, 64, 8, MANY), (8, 8, 128, 64, MANY),
    (32, 8, 128, 32, MANY * 4), (16, 1, 64, 16, MANY * 7)])
@pytest.mark.parametrize("shared", [False, True])
def test_precise_decode_attention(form, heads, kv_heads, dim, page_size, contexts, shared):
    """From one block to more than a wave of them (sequences then start longest first; 119 sequences are just what that rule
    takes), values of their own and values that are the keys.  Rows of the pages behind a context hold NaN: nothing of
    them may reach a result.  The bound: weights of 16 bits against 32, and one rounding of the output to bfloat16."""
    from llmserver_b200 import ops
    from llmserver_b200.ops import attention_bf16
    from llmserver_b200.ops.library import check_wait_errors
    batch = decode_batch(contexts)
    qkv, q_stride, k_pages, v_pages, tables = paged_case(len(contexts) + dim, [1] * len(contexts), contexts, heads, kv_heads, dim, page_size, 2.0)
    for row, context in enumerate(contexts):
        last = int(tables[row, (context - 1) // page_size])
        for pages in (k_pages, v_pages):
            pages[last, :, (context - 1) % page_size + 1:] = float("nan")
    if shared:
        v_pages = k_pages
    assert attention_bf16.decode_by_tma(k_pages, v_pages)
    given = dict(window=form.get("window", 0), chunk=form.get("chunk", 0), keep=form.get("keep", 0),
                 sinks=torch.linspace(-2.0, 3.0, heads, device=DEVICE) if form.get("sinks") else None,
                 gate=torch.randn((len(contexts), heads * dim), device=DEVICE).to(torch.bfloat16) if form.get("gate") else None)
    got = ops.attention(qkv, batch, tables, k_pages, v_pages, heads, kv_heads, dim, dim ** -0.5, precise=True, q_stride=q_stride, **given)
    want = ops.attention_generic(qkv, q_stride, k_pages, v_pages, tables, batch.seq_of_token, batch.positions, heads, kv_heads, dim,
                                 dim ** -0.5, **given)
    torch.cuda.synchronize()
    check_wait_errors()
    got, want = got.double(), want.double()
    assert torch.isfinite(got).all()
    # both are rounded to bfloat16 once: they differ by at most one step of 2^-8 where the 32-bit results straddle a boundary,
    # beside 2^-16 of weight error on sums whose size is the row's largest value
    error = (got - want).abs() / torch.maximum(want.abs(), 0.05 * want.abs().amax(dim=-1, keepdim=True))
    assert error.max() <= 2.0 ** -7, f"{float(error.max()):.2e}"


@pytest.mark.parametrize("n_seqs", [127, 128, 129])
def test_longest_first_takes_every_sequence_once(n_seqs):
    """Up to 128 sequences are taken longest first; among them equal lengths, in an order that is neither rising nor falling."""
    from llmserver_b200.ops import attention_bf16
    heads, kv_heads, dim, page_size = 8, 4, 128, 16
    contexts = [1 + (37 * row) % 50 * 20 for row in range(n_seqs)]
    batch = decode_batch(contexts)
    qkv, q_stride, k_pages, v_pages, tables = paged_case(n_seqs, [1] * n_seqs, contexts, heads, kv_heads, dim, page_size)
    out = attention_bf16.try_attention(qkv, q_stride, batch, tables, k_pages, v_pages, heads, kv_heads, dim, dim ** -0.5, 0)
    worst = 0.0
    for row, context in enumerate(contexts):
        want = plain_rows(qkv, k_pages, v_pages, tables[row], context, context - 1, [0], heads, kv_heads, dim, page_size, dim ** -0.5, row)
        worst = max(worst, relative_error(out[row:row + 1], want))
    assert worst <= 2e-2, f"relative error {worst:.3e}"


# (contexts, tokens of prompt portions in front of them): lengths around a tile and around the shortest part, one much longer than
# all others, equal ones, a sequence without tokens, rows of a padded step, as many sequences as are divided by length
UNEVEN = [([4000] + [1] * 20, 0), ([64 * k + k % 3 - 1 for k in range(1, 34)], 0), ([3000] * 17, 0), ([2500, 0, 70, 900, 0] * 4, 0),
          ([1 + 31 * k for k in range(128)], 0), ([700, 4096, 33, 1900, 128, 129, 191, 192, 193, 2000] * 2, 150)]


@pytest.mark.parametrize("form", [None, dict(), dict(sinks=True, gate=True), dict(window=300, keep=70)], ids=["narrow", "precise", "sinks-gate", "window"])
@pytest.mark.parametrize("case", range(len(UNEVEN)))
@pytest.mark.parametrize("heads,dim", [(32, 128), (10, 64)])
@pytest.mark.parametrize("settled", [False, True])
def test_parts_by_length(form, case, heads, dim, settled):
    """Sequences of unequal length on up to a wave of blocks: the longer ones are divided into more parts, and the part that comes
    last adds them.  Launches on the same counters give the same bits, and what the kernel for every size gives but for
    the rounding of weights.  Settled: as an engine's step says, the older keys are read before the kernel in front, which writes
    the newest, has ended; the bits are those of the plain order."""
    from llmserver_b200 import ops
    from llmserver_b200.ops import attention_bf16
    from llmserver_b200.ops.library import check_wait_errors
    contexts, portion = UNEVEN[case]
    kv_heads, page_size = (2 if len(contexts) > 37 else 8) if dim == 128 else 2, 16
    q_lens = ([portion] if portion else []) + [1] * len(contexts)
    contexts = ([portion + 77] if portion else []) + contexts
    batch = HostBatch(q_lens, contexts)
    batch.max_q_len, batch.keys_settled = max(q_lens), False
    batch.seq_of_token = torch.repeat_interleave(torch.arange(len(q_lens), dtype=torch.int32), torch.tensor(q_lens)).to(DEVICE)
    batch.positions = torch.cat([torch.arange(context - count, context) for context, count in zip(contexts, q_lens)]).clamp_min(0).to(torch.int32).to(DEVICE)
    qkv, q_stride, k_pages, v_pages, tables = paged_case(case, q_lens, [max(c, 1) for c in contexts], heads, kv_heads, dim, page_size, 2.0)
    given = dict(window=0) if form is None else dict(
        window=form.get("window", 0), keep=form.get("keep", 0), sinks=torch.linspace(-2.0, 3.0, heads, device=DEVICE) if form.get("sinks") else None,
        gate=torch.randn((batch.n_tokens, heads * dim), device=DEVICE).to(torch.bfloat16) if form.get("gate") else None)
    planned = attention_bf16.plan(batch, heads // kv_heads, kv_heads, torch.device(DEVICE), by_length=True,
                                  span=attention_bf16.key_span(given["window"], 0, given.get("keep", 0)))
    singles = sum(count == 1 for count in q_lens)
    assert (0 < -planned[3] < planned[4]) == (296 // (singles * kv_heads) <= attention_bf16.UNEVEN_SPLITS), planned
    results, page_error = [], torch.zeros(1, dtype=torch.int32, device=DEVICE)
    newest = batch.positions.long()
    places = tables[batch.seq_of_token.long(), newest // page_size].long(), newest % page_size
    torch.cuda.synchronize()
    for launch in range(5 if settled else 3):
        if settled:
            batch.keys_settled = launch > 0
            for pages in (k_pages, v_pages):
                pages[places[0], :, places[1]] = 99.0
            ops.qk_norm_rope_kv_write(qkv, None, None, None, batch.positions, batch.seq_of_token, tables, k_pages, v_pages, heads, kv_heads, dim, 1e-6,
                                      True, page_error)
        if form is None:
            results.append(attention_bf16.try_attention(qkv, q_stride, batch, tables, k_pages, v_pages, heads, kv_heads, dim, dim ** -0.5, 0))
        else:
            results.append(ops.attention(qkv, batch, tables, k_pages, v_pages, heads, kv_heads, dim, dim ** -0.5, precise=True, q_stride=q_stride, **given))
    want = ops.attention_generic(qkv, q_stride, k_pages, v_pages, tables, batch.seq_of_token, batch.positions, heads, kv_heads, dim, dim ** -0.5, **given)
    torch.cuda.synchronize()
    check_wait_errors()
    assert int(page_error) == 0 and all(torch.equal(result, results[0]) for result in results)
    got, want = results[0].double(), want.double()
    for context, row in zip(contexts, batch.q_start.tolist()):
        if context == 0:
            assert not got[row].any()
            want[row] = 0
    assert torch.isfinite(got).all()
    # as above; weights of 8 bits (narrow) are off by 2^-9 each, at most that much of the row's largest value
    error = (got - want).abs() / torch.maximum(want.abs(), 0.05 * want.abs().amax(dim=-1, keepdim=True).clamp_min(1e-30))
    assert error.max() <= (2.0 ** -7 if form is not None else 2.0 ** -7 + 20 * 2.0 ** -9), f"{float(error.max()):.2e}"


@pytest.mark.parametrize("q_lens,contexts,layers", [
    ([100, 1, 1], [100, 1400, 1400], [(32, 8, 128, 128, 256), (32, 8, 64, 128, 0)]), ([512] + [1] * 13, [512] + [1500] * 13, [(32, 8, 64, 64, 0), (32, 4, 128, 64, 0)])])
@pytest.mark.parametrize("turned", [False, True])
def test_layers_of_other_kinds_in_one_step(q_lens, contexts, layers, turned):
    """Two layers whose single tokens, behind a prompt portion, are divided by length in one and into equal parts of the cp.async kernel in
    the other, with the same heads, value size and number of parts: each against the kernel for every size."""
    from llmserver_b200 import ops
    from llmserver_b200.ops.library import check_wait_errors
    batch = HostBatch(q_lens, contexts)
    batch.max_q_len = max(q_lens)
    batch.seq_of_token = torch.repeat_interleave(torch.arange(len(q_lens), dtype=torch.int32), torch.tensor(q_lens)).to(DEVICE)
    batch.positions = torch.cat([torch.arange(context - count, context) for context, count in zip(contexts, q_lens)]).to(torch.int32).to(DEVICE)
    for seed, (heads, kv_heads, dim, value_dim, window) in enumerate(layers[::-1] if turned else layers):
        qkv, q_stride, k_pages, _, tables = paged_case(seed, q_lens, contexts, heads, kv_heads, dim, 16, 2.0)
        v_pages = torch.randn((*k_pages.shape[:3], value_dim), device=DEVICE).to(torch.bfloat16)
        got = ops.attention(qkv, batch, tables, k_pages, v_pages, heads, kv_heads, dim, dim ** -0.5, window, value_dim, precise=True, q_stride=q_stride)
        want = ops.attention_generic(qkv, q_stride, k_pages, v_pages, tables, batch.seq_of_token, batch.positions, heads, kv_heads, dim, dim ** -0.5,
                                     window, value_dim=value_dim)
        torch.cuda.synchronize()
        check_wait_errors()
        got, want = got.double(), want.double()
        error = (got - want).abs() / torch.maximum(want.abs(), 0.05 * want.abs().amax(dim=-1, keepdim=True))
        assert error.max() <= 2.0 ** -7, f"{float(error.max()):.2e}"      # as in the first test


@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("precise", [False, True])
@pytest.mark.parametrize("contexts", [[900], [3000, 700]])
def test_pages_that_tma_cannot_describe(monkeypatch, dim, precise, contexts):
    """A pool said to have 2^31 - 1 pages (every table entry names one of those that exist) has more rows than a tensor map can: the
    step runs the other kernel, whose splits do not merge in a cluster, and its results are written all the same."""
    from llmserver_b200 import ops
    from llmserver_b200.ops import attention_bf16
    from llmserver_b200.ops.library import check_wait_errors
    heads, kv_heads, page_size = 16, 4, 16
    batch = decode_batch(contexts)
    qkv, q_stride, k_pages, v_pages, tables = paged_case(3, [1] * len(contexts), contexts, heads, kv_heads, dim, page_size)
    torch.full((len(contexts), heads * dim), float("nan"), dtype=torch.bfloat16, device=DEVICE)      # what the allocator hands out next
    launch, launched = attention_bf16.call, []

    def call(name, *args):
        launched.append(name)
        place = {"llm_attention_mma": 14, "llm_attention_mma_sinks": 15}[name]
        assert args[place] == k_pages.shape[0]
        launch(name, *args[:place], 2 ** 31 - 1, *args[place + 1:])

    monkeypatch.setattr(attention_bf16, "call", call)
    got = ops.attention(qkv, batch, tables, k_pages, v_pages, heads, kv_heads, dim, dim ** -0.5, precise=precise, q_stride=q_stride)
    torch.cuda.synchronize()
    check_wait_errors()
    assert launched == ["llm_attention_mma_sinks" if precise else "llm_attention_mma"]
    for row, context in enumerate(contexts):
        want = plain_rows(qkv, k_pages, v_pages, tables[row], context, context - 1, [0], heads, kv_heads, dim, page_size, dim ** -0.5, row)
        assert relative_error(got[row:row + 1], want) <= 2e-2      # of bfloat16 weights and results, as in the test above
