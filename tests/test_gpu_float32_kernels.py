"""The 32-bit path's product for few rows and the attention kernel's forms by value size, at the edges of their ranges."""
import pytest
import torch

from test_gpu_kernels import DEVICE, DTYPES, close, paged, rand

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 4, 5, 8, 9, 16, 17, 32])
@pytest.mark.parametrize("cols,inner", [(1, 4), (31, 124), (33, 128), (64, 132), (509, 384), (40, 388), (100, 1540)])
def test_few_rows_give_the_sums_of_many_rows(rows, cols, inner):
    """Every output is one running sum over ascending k in both kernels: equal bit for bit, whatever the number of rows
    (33 rows run in tiles), and so is a product whose operands are not 16-byte aligned (which also runs in tiles)."""
    from llmserver_b200 import ops
    x, w = rand((33, inner), torch.float32, 8), rand((cols, inner), torch.float32, 9)
    many = ops.gemm_f32(x, w)
    few = ops.gemm_f32(x[:rows].contiguous(), w)
    assert torch.equal(few, many[:rows])
    close(few, x[:rows].double() @ w.double().T, torch.float32, f"product {rows, cols, inner}", factor=max(1.0, inner / 200))
    shifted = torch.empty(cols * inner + 1, dtype=torch.float32, device=DEVICE)[1:].view(cols, inner).copy_(w)
    assert torch.equal(ops.gemm_f32(x[:rows].contiguous(), shifted), few)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("dim,value_dim", [(32, 32), (36, 33), (64, 64), (72, 65), (30, 128), (128, 129), (96, 256), (66, 257), (512, 512)])
def test_attention_by_value_size(dtype, dim, value_dim):
    """Value sizes on both sides of each form's limit, key rows with and without whole 16-byte pieces, contexts of one, of
    exactly two and of several rounds of 32 keys."""
    from llmserver_b200 import ops
    heads, kv_heads, page_size, scale = 3, 1, 8, dim ** -0.5
    contexts, q_lens = [1, 64, 65, 150], [1, 2, 1, 3]
    dense_k = [rand((c, kv_heads, dim), dtype, 20 + i).cpu() for i, c in enumerate(contexts)]
    dense_v = [rand((c, kv_heads, value_dim), dtype, 30 + i).cpu() for i, c in enumerate(contexts)]
    k_pages, _, tables = paged(dense_k, dense_k, page_size, 1, dtype)
    v_pages, _, _ = paged(dense_v, dense_v, page_size, 1, dtype)
    queries = [rand((n, heads, dim), dtype, 40 + i).cpu() for i, n in enumerate(q_lens)]
    q_stride = heads * dim + 5
    packed = torch.zeros((sum(q_lens), q_stride), dtype=dtype)
    packed[:, :heads * dim] = torch.cat(queries).reshape(-1, heads * dim)
    positions = torch.cat([torch.arange(c - n, c) for c, n in zip(contexts, q_lens)]).to(torch.int32).to(DEVICE)
    seq_of_token = torch.cat([torch.full((n,), i) for i, n in enumerate(q_lens)]).to(torch.int32).to(DEVICE)
    out = ops.attention_generic(packed.to(DEVICE), q_stride, k_pages, v_pages, tables, seq_of_token, positions, heads, kv_heads, dim,
                                scale, 0, value_dim=value_dim)

    def plain(q, k, v, first):
        scores = torch.einsum("qhd,kd->hqk", q.double(), k[:, 0].double()) * scale
        hidden = torch.arange(len(k))[None, :] > torch.arange(first, first + len(q))[:, None]
        weights = torch.softmax(scores.masked_fill(hidden, float("-inf")), dim=-1)
        return torch.einsum("hqk,kd->qhd", weights, v[:, 0].double()).flatten(1)

    want = torch.cat([plain(q, k, v, c - n) for q, k, v, c, n in zip(queries, dense_k, dense_v, contexts, q_lens)])
    close(out, want, dtype, f"attention {dim, value_dim}")


OPTIONS = [dict(), dict(window=70, keep=9), dict(chunk=50), dict(sinks=True, gate=True), dict(bias=True)]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("dim,value_dim", [(32, 32), (36, 33), (96, 128), (66, 257), (512, 512)])
@pytest.mark.parametrize("options", OPTIONS, ids=lambda options: "-".join(options) or "plain")
def test_many_tokens_give_the_bits_of_few(dtype, dim, value_dim, options):
    """A launch of many (token, head) pairs, where a warp makes all parts of a pair, against launches of few, where four do: positions
    with one round of 32 keys and with up to nine, scores of -inf (from a bias) in whole rounds."""
    from llmserver_b200 import ops
    heads, kv_heads, page_size, count, step = 36, 3, 8, 260, 14
    assert count * heads >= 8192 > step * heads * 16      # as many columns as the widest values have
    pages = -(-count // page_size)
    k_pages, v_pages = rand((pages, kv_heads, page_size, dim), dtype, 1), rand((pages, kv_heads, page_size, value_dim), dtype, 2)
    table = torch.randperm(pages, generator=torch.Generator().manual_seed(3)).to(torch.int32).view(1, -1).to(DEVICE)
    q = rand((count, heads * dim), dtype, 4)
    given = {key: value for key, value in options.items() if key in ("window", "keep", "chunk")}
    if "sinks" in options:
        given["sinks"] = torch.linspace(-2.0, 3.0, heads, device=DEVICE)
    if "bias" in options:
        given["bias"] = rand((heads, 200), torch.float32, 5)
        given["bias"][:, 30:130] = -float("inf")
    gate = rand((count, heads * value_dim), dtype, 6) if "gate" in options else None
    positions, sequence = torch.arange(count, dtype=torch.int32, device=DEVICE), torch.zeros(count, dtype=torch.int32, device=DEVICE)

    def run(first, last):
        return ops.attention_generic(q[first:last].contiguous(), heads * dim, k_pages, v_pages, table, sequence[first:last].contiguous(),
                                     positions[first:last].contiguous(), heads, kv_heads, dim, dim ** -0.5, value_dim=value_dim,
                                     gate=None if gate is None else gate[first:last].contiguous(), **given)

    many = run(0, count)
    assert torch.isfinite(many).all()
    for first in range(0, count, step):
        assert torch.equal(run(first, min(count, first + step)), many[first:first + step])
