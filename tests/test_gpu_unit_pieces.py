"""Bias, norm, rotation and cache write of whole units in 16-byte pieces, against the kernel for every size: the same numbers in rows
that are one element wider, which that kernel takes."""
import pytest
import torch

from test_gpu_kernels import DEVICE, rand

pytestmark = pytest.mark.gpu


def places(tokens, page_size):
    positions = (torch.arange(tokens) * 7 % 500).to(torch.int32).to(DEVICE)
    seq = (torch.arange(tokens) % 2).to(torch.int32).to(DEVICE)
    pages = -(-500 // page_size)
    tables = torch.randperm(2 * pages, generator=torch.Generator().manual_seed(3)).view(2, pages).to(torch.int32).to(DEVICE)
    return positions, seq, tables, 2 * pages


# one piece a thread and several, fewer pieces than threads, regions that end inside a warp, more blocks than one per token
@pytest.mark.parametrize("tokens", [1, 5, 255, 256, 300])
@pytest.mark.parametrize("heads,kv_heads,maps,dim,value_dim", [(1, 1, 1, 64, 8), (3, 1, 1, 128, 72), (32, 8, 2, 64, 128), (6, 3, 2, 128, 64), (96, 4, 1, 128, 128)])
@pytest.mark.parametrize("parts", ["all", "turn", "norm", "bias"])
def test_units(tokens, heads, kv_heads, maps, dim, value_dim, parts):
    from llmserver_b200 import ops
    page_size = 16
    positions, seq, tables, pages = places(tokens, page_size)
    used = (heads + kv_heads) * maps * dim + kv_heads * value_dim
    rows = rand((tokens, used), torch.bfloat16, 1)
    weight_type = torch.float32 if heads == 3 else torch.bfloat16
    given = dict(eps=1e-6)
    if parts in ("all", "norm"):
        given.update(q_weight=rand((dim,), weight_type, 2, 0.1) + 1, k_weight=rand((dim,), weight_type, 3, 0.1) + 1)
    if parts in ("all", "bias"):
        given.update(bias=rand((used,), torch.float32, 4))
    if parts in ("all", "turn"):
        given.update(inv_freq=(5e5 ** (-torch.arange(0, dim, 2) / dim)).float().to(DEVICE), rotary_dim=dim)
    results = []
    for extra in (8, 9):
        qkv = torch.zeros((tokens, used + extra), dtype=torch.bfloat16, device=DEVICE)
        qkv[:, :used] = rows
        k_pages = torch.zeros((pages, kv_heads, page_size, maps * dim), dtype=torch.bfloat16, device=DEVICE)
        v_pages = torch.zeros((pages, kv_heads, page_size, value_dim), dtype=torch.bfloat16, device=DEVICE)
        error = torch.zeros(1, dtype=torch.int32, device=DEVICE)
        ops.norm_rope_units(qkv, positions, seq, tables, k_pages, v_pages, heads, kv_heads, maps, dim, dim, value_dim, error, **given)
        assert int(error) == 0 and not qkv[:, used:].any()
        results.append((qkv[:, :heads * maps * dim].float(), k_pages.float(), v_pages.float()))
    for name, got, want in zip(("queries", "keys", "values"), *results):
        # the sums of squares are added in another order: the 32-bit results differ by 2^-20 of a unit's largest value (a turned element is
        # a difference of two), and where a rounding to bfloat16 flips by one step of it, 2^-7 of the value at most
        assert ((got - want).abs() <= 2.0 ** -7 * want.abs() + 2.0 ** -20 * want.abs().max()).all(), name
        assert (got != want).float().mean() < 0.01, name


@pytest.mark.parametrize("tokens", [1, 300])
@pytest.mark.parametrize("heads,kv_heads,dim,value_dim", [(4, 2, 64, 64), (32, 8, 128, 128), (5, 5, 128, 64)])
def test_turned_heads(tokens, heads, kv_heads, dim, value_dim):
    """The rotation with a magnitude, and a page outside the pool, which is reported and written to nobody's page."""
    from llmserver_b200 import ops
    page_size, magnitude = 16, 1.25
    positions, seq, tables, pages = places(tokens, page_size)
    inv_freq = (1.5e5 ** (-torch.arange(0, dim, 2) / dim)).float().to(DEVICE)
    rows = rand((tokens, (heads + kv_heads) * dim + kv_heads * value_dim), torch.bfloat16, 1)
    qkv = rows.clone()
    k_pages = torch.zeros((pages, kv_heads, page_size, dim), dtype=torch.bfloat16, device=DEVICE)
    v_pages = torch.zeros((pages, kv_heads, page_size, value_dim), dtype=torch.bfloat16, device=DEVICE)
    error = torch.zeros(1, dtype=torch.int32, device=DEVICE)
    ops.rope_kv_write_split(qkv, inv_freq, magnitude, positions, seq, tables, k_pages, v_pages, heads, kv_heads, dim, value_dim, True, error)
    angle = (positions.float()[:, None] * inv_freq).double()[:, None]
    units = rows[:, :(heads + kv_heads) * dim].double().view(tokens, heads + kv_heads, dim)
    low, high = units[..., :dim // 2], units[..., dim // 2:]
    cos, sin = torch.cos(angle) * magnitude, torch.sin(angle) * magnitude
    want = torch.cat([low * cos - high * sin, high * cos + low * sin], dim=-1)
    page, slot = tables[seq.long(), (positions // page_size).long()].long(), (positions % page_size).long()
    got = torch.cat([qkv[:, :heads * dim].view(tokens, heads, dim), k_pages[page, :, slot]], dim=1).double()
    assert ((got - want).abs() <= 2.0 ** -8 * want.abs() + 2e-6 * want.abs().max()).all()
    assert torch.equal(v_pages[page, :, slot].flatten(1), rows[:, (heads + kv_heads) * dim:])
    before = k_pages.clone(), v_pages.clone()
    ops.rope_kv_write_split(rows.clone(), inv_freq, magnitude, positions, seq, tables * 0 + pages, k_pages, v_pages, heads, kv_heads, dim, value_dim, True, error)
    assert int(error) > 0 and torch.equal(before[0], k_pages) and torch.equal(before[1], v_pages)
