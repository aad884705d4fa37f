"""The product kernel for few rows at 65 to 128 rows (one K atom per stage, twice the tensor memory) and its fused epilogues from 17
rows on, where a warp finishes several tokens and a lane adds a token's sums of squares."""
import pytest
import torch

from test_gpu_kernels import DEVICE, close, rand

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [17, 63, 64, 65, 96, 97, 127, 128])
@pytest.mark.parametrize("cols,inner,split", [(130, 72, 1), (256, 64, 1), (1000, 520, 2), (4096, 1024, 8)])
def test_product(rows, cols, inner, split):
    from llmserver_b200.ops import gemm_bf16
    from llmserver_b200.ops.library import call, check_wait_errors, stream_handle
    x, w = rand((rows, inner), torch.bfloat16, 12), rand((cols, inner), torch.bfloat16, 13, 0.05)
    for out_dtype in (torch.float32, torch.bfloat16):
        out = torch.full((rows, cols), float("nan"), dtype=out_dtype, device=DEVICE)
        call("llm_gemm_small_m", x.data_ptr(), w.data_ptr(), out.data_ptr(), rows, cols, inner, cols, int(out_dtype == torch.float32), split,
             *gemm_bf16.NO_SCALE, gemm_bf16.error_flag(DEVICE).data_ptr(), stream_handle())
        torch.cuda.synchronize()
        check_wait_errors()
        close(out, x.double() @ w.double().T, out_dtype, f"{rows, cols, inner, split}", factor=4.0 if out_dtype == torch.float32 else 1.0)


@pytest.mark.parametrize("rows", [16, 17, 18, 47, 64, 65])
@pytest.mark.parametrize("tiles,inner,split", [(296, 136, 1), (297, 136, 1), (149, 520, 2), (99, 264, 3), (38, 1032, 8)])
def test_three_blocks_an_sm(rows, tiles, inner, split):
    """Launches around two blocks per SM of 148, beyond which 17 to 64 rows run three of them with stages of one atom, K split or not:
    plain sums, the gated form and the sums added to a stream, each with a last tile that is not full (the gated form's are)."""
    from llmserver_b200.ops import gemm_bf16
    from llmserver_b200.ops.library import call, check_wait_errors, stream_handle
    cols = tiles * 128 - 126
    x, w = rand((rows, inner), torch.bfloat16, 1), rand((tiles * 128, inner), torch.bfloat16, 2, inner ** -0.5)
    flag, exact = gemm_bf16.error_flag(DEVICE).data_ptr(), x.double() @ w.double().T
    out = torch.full((rows, cols), float("nan"), dtype=torch.float32, device=DEVICE)
    call("llm_gemm_small_m", x.data_ptr(), w.data_ptr(), out.data_ptr(), rows, cols, inner, cols, 1, split, *gemm_bf16.NO_SCALE, flag, stream_handle())
    close(out, exact[:, :cols], torch.float32, "sums", factor=4.0)
    gated = torch.full((rows, tiles * 64), float("nan"), dtype=torch.bfloat16, device=DEVICE)
    call("llm_gemm_gate_up_silu", x.data_ptr(), w.data_ptr(), gated.data_ptr(), rows, tiles * 128, inner, tiles * 64, split, *gemm_bf16.NO_SCALE, flag,
         stream_handle())
    pairs = exact.view(rows, tiles, 2, 64)
    close(gated, (pairs[:, :, 0] * torch.sigmoid(pairs[:, :, 0]) * pairs[:, :, 1]).flatten(1), torch.bfloat16, "gates")
    stream, norm = rand((rows, cols), torch.float32, 3), rand((cols,), torch.bfloat16, 4)
    want = stream.double() + exact[:, :cols]
    scaled, parts = torch.zeros((rows, cols), dtype=torch.bfloat16, device=DEVICE), torch.zeros((tiles, 128), dtype=torch.float32, device=DEVICE)
    call("llm_gemm_into_stream", x.data_ptr(), w.data_ptr(), stream.data_ptr(), rows, cols, inner, split, norm.data_ptr(), 0, scaled.data_ptr(),
         parts.data_ptr(), 128, flag, stream_handle())
    torch.cuda.synchronize()
    check_wait_errors()
    close(stream, want, torch.float32, "stream", factor=4.0)
    close(scaled, want * norm.double(), torch.bfloat16, "the next norm's input")
    close(parts[:, :rows].sum(0), (want * want).sum(-1), torch.float32, "sums of squares", factor=4.0)


@pytest.mark.parametrize("rows", [1, 8, 16])
@pytest.mark.parametrize("split", [1, 3, 8])
def test_few_rows_add_in_the_order_of_k(rows, split):
    """Up to 16 rows a feature's sum does not depend on the tile that it lies in: tiles of equal weights give equal bits."""
    from llmserver_b200.ops import gemm_bf16
    from llmserver_b200.ops.library import call, check_wait_errors, stream_handle
    tiles, inner = 9, 4096
    x, w = rand((rows, inner), torch.bfloat16, 1), rand((128, inner), torch.bfloat16, 2, inner ** -0.5).repeat(tiles, 1)
    out = torch.full((rows, tiles * 128), float("nan"), dtype=torch.float32, device=DEVICE)
    call("llm_gemm_small_m", x.data_ptr(), w.data_ptr(), out.data_ptr(), rows, tiles * 128, inner, tiles * 128, 1, split, *gemm_bf16.NO_SCALE,
         gemm_bf16.error_flag(DEVICE).data_ptr(), stream_handle())
    torch.cuda.synchronize()
    check_wait_errors()
    for tile in range(1, tiles):
        assert torch.equal(out[:, tile * 128:(tile + 1) * 128], out[:, :128])


@pytest.mark.parametrize("rows", [16, 17, 64, 65, 128])
@pytest.mark.parametrize("tiles,inner,split", [(148, 136, 1), (149, 136, 1), (33, 1032, 4), (34, 1032, 4), (3, 200, 2), (22, 520, 6)])
def test_one_block_an_sm(rows, tiles, inner, split):
    """Launches around one block per SM, which run a long ring of two-atom stages beyond 16 rows, where the
    tiles begin at different places of their shares of K."""
    from llmserver_b200.ops import gemm_bf16
    from llmserver_b200.ops.library import call, check_wait_errors, stream_handle
    cols = tiles * 128 - 126
    x, w = rand((rows, inner), torch.bfloat16, 1), rand((cols, inner), torch.bfloat16, 2, inner ** -0.5)
    flag, exact = gemm_bf16.error_flag(DEVICE).data_ptr(), x.double() @ w.double().T
    out = torch.full((rows, cols), float("nan"), dtype=torch.float32, device=DEVICE)
    call("llm_gemm_small_m", x.data_ptr(), w.data_ptr(), out.data_ptr(), rows, cols, inner, cols, 1, split, *gemm_bf16.NO_SCALE, flag, stream_handle())
    stream = rand((rows, cols), torch.float32, 3)
    want = stream.double() + exact
    call("llm_gemm_into_stream", x.data_ptr(), w.data_ptr(), stream.data_ptr(), rows, cols, inner, split, 0, 0, 0, 0, 0, flag, stream_handle())
    torch.cuda.synchronize()
    check_wait_errors()
    close(out, exact, torch.float32, "sums", factor=4.0)
    close(stream, want, torch.float32, "stream", factor=4.0)


@pytest.mark.parametrize("rows", [16, 17, 33, 64, 65, 119, 128])
def test_stream_and_scaled_rows(rows):
    """x W^T added to the stream, the sums of squares it leaves, and the gated product that divides by them: against the same in 64
    bits.  A stream of 640 columns leaves five sums per token."""
    from llmserver_b200 import ops
    from llmserver_b200.ops import gemm_bf16
    from llmserver_b200.ops.library import check_wait_errors
    width, inner, features, eps = 640, 512, 320, 1e-6
    x, w = rand((rows, inner), torch.bfloat16, 1), rand((width, inner), torch.bfloat16, 2, inner ** -0.5)
    stream, norm = rand((rows, width), torch.float32, 3, 2.0), rand((width,), torch.bfloat16, 4, 0.1) + 1
    gate, up = rand((features, width), torch.bfloat16, 5, width ** -0.5), rand((features, width), torch.bfloat16, 6, width ** -0.5)
    want = stream.double() + x.double() @ w.double().T
    sink = ops.StreamSink(stream, norm, eps)
    assert gemm_bf16.linear_into_stream(x, w, sink) and sink.added
    close(stream, want, torch.float32, "the stream", factor=4.0)
    normed = want / torch.sqrt((want * want).mean(-1, keepdim=True) + eps) * norm.double()
    g, u = normed @ gate.double().T, normed @ up.double().T
    out = ops.gate_up_silu(sink.scaled, ops.interleave_gate_up(gate, up), ops.GATE_UP_GROUP)
    torch.cuda.synchronize()
    check_wait_errors()
    close(out, g * torch.sigmoid(g) * u, torch.bfloat16, "the gated product of scaled rows")


@pytest.mark.parametrize("rows", [17, 40, 64, 65, 128])
def test_fused_heads(rows):
    """The q/k/v epilogue for the tokens of several sequences, each warp finishing several: queries and cache rows as the two
    kernels that it stands for leave them (which round the product to bfloat16 first)."""
    from llmserver_b200 import ops
    from llmserver_b200.ops import gemm_bf16
    heads, kv_heads, dim, inner, page_size = 4, 2, 128, 256, 16
    width = (heads + 2 * kv_heads) * dim
    x, w = rand((rows, inner), torch.bfloat16, 1), rand((width, inner), torch.bfloat16, 2, inner ** -0.5)
    q_norm, k_norm = rand((dim,), torch.bfloat16, 3, 0.1) + 1, rand((dim,), torch.bfloat16, 4, 0.1) + 1
    inv_freq = (1e6 ** (-torch.arange(0, dim, 2) / dim)).float().to(DEVICE)
    seq = (torch.arange(rows) % 3).to(torch.int32).to(DEVICE)
    positions = (torch.arange(rows) // 3 * 7 % 300 + torch.arange(rows) // 3).to(torch.int32).to(DEVICE)
    tables = (torch.randperm(90, generator=torch.Generator().manual_seed(1)).view(3, 30)).to(torch.int32).to(DEVICE)
    parts = torch.empty((1, 128), dtype=torch.float32, device=DEVICE)
    parts[0, :rows] = (x.float() ** 2).sum(-1)
    normed = (x.float() / torch.sqrt((x.float() ** 2).mean(-1, keepdim=True) + 1e-6)).to(torch.bfloat16)
    results = []
    for fused in (True, False):
        k_pages = torch.zeros((90, kv_heads, page_size, dim), dtype=torch.bfloat16, device=DEVICE)
        v_pages, error = torch.zeros_like(k_pages), torch.zeros(1, dtype=torch.int32, device=DEVICE)
        if fused:
            out = gemm_bf16.qkv_rope_fused(ops.RowScaled(x, parts, 1e-6), w, q_norm, k_norm, inv_freq, positions, seq, tables, k_pages,
                                           v_pages, heads, kv_heads, dim, 1e-6, True, error)
        else:
            out = torch.matmul(normed, w.t())
            ops.qk_norm_rope_kv_write(out, q_norm, k_norm, inv_freq, positions, seq, tables, k_pages, v_pages, heads, kv_heads, dim, 1e-6, True, error)
        assert int(error) == 0
        results.append((out[:, :heads * dim], k_pages, v_pages))
    for name, got, want in zip(("queries", "keys", "values"), *results):
        close(got, want, torch.bfloat16, name, factor=2.0)      # either side is rounded where the other is not


@pytest.mark.parametrize("n_parts", [1, 5, 32, 40, 64, 200])
def test_a_row_is_divided_alike_in_every_step(n_parts):
    """The sums of squares that a row's scale is made of are added in the order that their number gives, whether the step has up to
    16 rows, up to 64 or more: the same row and parts give the same bits."""
    from llmserver_b200 import ops
    from llmserver_b200.ops import gemm_bf16
    from llmserver_b200.ops.library import call, check_wait_errors, stream_handle
    cols, inner = 256, 512
    w = rand((cols, inner), torch.bfloat16, 2, inner ** -0.5)
    x = rand((16, inner), torch.bfloat16, 1)
    parts = rand((n_parts, 16), torch.float32, 3).abs() * torch.logspace(-3, 1, n_parts, device=DEVICE)[:, None]
    results = []
    for rows in (16, 17, 64, 65, 128):
        many = x.repeat(8, 1)[:rows].contiguous()
        scaled = ops.RowScaled(many, parts.repeat(1, 8).contiguous(), 1e-6)
        out = torch.empty((rows, cols), dtype=torch.float32, device=DEVICE)
        call("llm_gemm_small_m", many.data_ptr(), w.data_ptr(), out.data_ptr(), rows, cols, inner, cols, 1, 1, *scaled.scale_args(),
             gemm_bf16.error_flag(DEVICE).data_ptr(), stream_handle())
        torch.cuda.synchronize()
        check_wait_errors()
        results.append(out[:16])
    assert all(torch.equal(result, results[0]) for result in results)


def test_steps_of_more_than_64_rows(tiny_folders, monkeypatch):
    """A prompt of 100 tokens runs without stand-alone norms (but for the first layer's input and the final norm); a step that decodes
    96 requests runs with them, eagerly and replayed; all against the plain implementation."""
    from helpers import assert_close, plain_logits, tokens_for
    from llmserver_b200 import ops
    from llmserver_b200.cache import CacheManager
    from llmserver_b200.engine.step import StepFunction
    from llmserver_b200.models import load_model
    from llmserver_b200.sampling import SamplingRow
    folder, rows = tiny_folders["e"], 96
    model = load_model(folder, "bfloat16", "cuda:0")
    cache = CacheManager(model.cache_needs(), 16, 3 * rows + 16, num_slots=rows, prefix_sharing=False)
    cache.materialize(model.runtime.device, model.runtime.dtype)
    step = StepFunction(model, cache)
    step.enable_graphs(64, rows)
    norm, calls = ops.add_rmsnorm, []
    monkeypatch.setattr(ops, "add_rmsnorm", lambda *args, **kwargs: (calls.append(1), norm(*args, **kwargs))[1])
    vocab, layers = model.spec.vocab_size, len(model.spec.schedule)
    tokens = tokens_for(vocab, 100, 3)
    step.admit("prompt")
    got = step.run([("prompt", tokens, list(range(100)))])
    assert len(calls) == 2
    assert_close(got.float().cpu().numpy(), plain_logits(folder, tokens), "bfloat16", "a prompt of 100 tokens")
    step.release("prompt")
    prompts = [tokens_for(vocab, 3 + row % 30, 100 + row) for row in range(rows)]
    for row, prompt in enumerate(prompts):
        step.admit(row)
        step.run([(row, prompt, [])])
    want = {row: plain_logits(folder, prompts[row] + [row])[-1:] for row in (0, 1, 50, 95)}
    for turn in range(4):      # the third replays
        del calls[:]
        entries = [(row, [row], [0]) for row in range(rows)]
        if turn == 0:
            logits = step.run(entries)
        else:
            step.run_and_sample(entries, [SamplingRow()] * rows)
            graph = step.graphs.graphs.get(rows)
            logits = graph.logits if graph is not None else None
        if turn != 3:
            assert len(calls) == 2 * layers + 1
        for row in range(rows):
            step.computed[row] -= 1      # the same step again
        if logits is not None:
            for row, expected in want.items():
                assert_close(logits[row:row + 1].float().cpu().numpy(), expected, "bfloat16", f"turn {turn}, row {row}")
    assert step.graph_steps > 0
    step.check_errors()


def test_prompts_of_more_than_64_tokens_time_nothing():
    """The splits of products that only prompts run at these rows follow from the shape: the first such prompt does not stop for them."""
    from llmserver_b200 import ops
    from llmserver_b200.ops import gemm_bf16
    x, w = rand((100, 1032), torch.bfloat16, 1), rand((392, 1032), torch.bfloat16, 2, 1032 ** -0.5)
    stream = rand((100, 392), torch.float32, 3)
    want = stream.double() + x.double() @ w.double().T
    before = gemm_bf16.tunings()
    assert gemm_bf16.linear_into_stream(x, w, ops.StreamSink(stream))
    assert gemm_bf16.tunings() == before
    close(stream, want, torch.float32, "the stream", factor=4.0)
