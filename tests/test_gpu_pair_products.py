"""The products that pairs of SMs make: the gated product of many rows and the expert products on tiles of 256 rows."""
import math

import pytest
import torch

from test_gpu_kernels import DEVICE, rand

pytestmark = pytest.mark.gpu


def gated(x, gate, up, limit, alpha, shift):
    g, u = x.double() @ gate.double().T, x.double() @ up.double().T
    g, u = g.clamp(max=limit), u.clamp(-limit, limit)
    return g * torch.sigmoid(alpha * g) * (u + shift)


# rows on both sides of a block's 128 and a pair's 256, features that fill no tile, an inner size that ends inside a stage, more
# row tiles than one group, fewer tiles than pairs
@pytest.mark.parametrize("rows,features,inner", [(1, 8, 64), (127, 64, 64), (128, 192, 72), (129, 320, 200), (255, 128, 128), (256, 136, 512),
                                                 (257, 1000, 1000), (1537, 640, 4096), (4400, 704, 2048)])
@pytest.mark.parametrize("interleave", [0, 64])
def test_gated_product(rows, features, inner, interleave):
    from llmserver_b200 import ops
    from llmserver_b200.ops.library import call, check_wait_errors, library, stream_handle, wait_error_flag
    if not library().llm_gemm_pair_supports(features, inner, interleave):
        assert interleave and features % 64
        return
    x, gate, up = rand((rows, inner), torch.bfloat16, 1), rand((features, inner), torch.bfloat16, 2, inner ** -0.5), rand((features, inner), torch.bfloat16, 3, inner ** -0.5)
    weight = ops.interleave_gate_up(gate, up) if interleave else torch.cat([gate, up]).contiguous()
    for limit, alpha, shift in ((math.inf, 1.0, 0.0), (0.7, 1.702, 1.0)):
        out = torch.full((rows, features), float("nan"), dtype=torch.bfloat16, device=DEVICE)
        call("llm_gemm_pair_gated", x.data_ptr(), weight.data_ptr(), out.data_ptr(), rows, features, inner, interleave, limit, alpha, shift,
             wait_error_flag(torch.device(DEVICE)).data_ptr(), stream_handle())
        torch.cuda.synchronize()
        check_wait_errors()
        want = gated(x, gate, up, limit, alpha, shift)
        # 32-bit sums and one rounding to 8 bits
        error = (out.double() - want).abs() / (want.abs() + 0.01 * want.abs().max())
        assert error.max() <= 2.0 ** -8, f"{float(error.max()):.2e}"


@pytest.mark.parametrize("by_pairs", [False, True])
def test_gate_over_its_range(by_pairs):
    """Products of one term each, so that gates and values are the weights themselves: gates from -88.5, whose exponential is still a
    number, to 88.  The bound: the hardware's exponential is off by up to 2 + 1.17 |x| units in the last place at x, beside one rounding to 8 bits."""
    from llmserver_b200 import ops
    from llmserver_b200.ops.library import check_wait_errors
    features, inner, tokens = 256, 64, 256
    gate = torch.cat([torch.arange(-88.5, -80.0, 0.5), torch.linspace(-80.0, 88.0, features - 17)]).to(torch.bfloat16).to(DEVICE)
    up = torch.linspace(-8.0, 8.0, features).to(torch.bfloat16).to(DEVICE)
    weight = torch.zeros((1, 2 * features, inner), dtype=torch.bfloat16, device=DEVICE)
    weight[0, :features, 0], weight[0, features:, 0] = gate, up
    x = torch.zeros((tokens, inner), dtype=torch.bfloat16, device=DEVICE)
    x[:, 0] = 1.0
    plan = ops.moe_plan(torch.zeros((tokens, 1), dtype=torch.int32, device=DEVICE), 1, ops.MOE_PAIR_TILE_ROWS if by_pairs else ops.MOE_TILE_ROWS)
    got = ops.moe_grouped(x, weight, plan, gather_div=1, gated=(100.0, 1.0)).double()
    torch.cuda.synchronize()
    check_wait_errors()
    g, u = gate.double(), up.double()
    want = g * torch.sigmoid(g) * (u + 1.0)
    assert ((got - want).abs() <= (2.0 ** -8 + 106 * 2.0 ** -23) * want.abs()).all(), f"{got[0, :20]} {want[:20]}"


@pytest.mark.parametrize("by_pairs", [False, True])
def test_gates_that_are_not_finite(by_pairs):
    """A gate beyond the type's range has its limit: itself upwards, 0 downwards as far as the exponential is infinite and the gate a number."""
    from llmserver_b200 import ops
    gate = torch.tensor([-3e38, -1000.0, -89.0, 0.0, 1000.0, 3e38, float("inf"), float("nan")]).to(torch.bfloat16).to(DEVICE)
    weight = torch.zeros((1, 16, 64), dtype=torch.bfloat16, device=DEVICE)
    weight[0, :8, 0] = gate
    x = torch.zeros((256, 64), dtype=torch.bfloat16, device=DEVICE)
    x[:, 0] = 1.0
    plan = ops.moe_plan(torch.zeros((256, 1), dtype=torch.int32, device=DEVICE), 1, ops.MOE_PAIR_TILE_ROWS if by_pairs else ops.MOE_TILE_ROWS)
    got = ops.moe_grouped(x, weight, plan, gather_div=1, gated=(math.inf, 1.0)).float()
    assert (got[:, :4] == 0.0).all() and torch.equal(got[:, 4:7], gate[4:7].float().expand(256, 3))
    assert not by_pairs or torch.isnan(got[:, 7]).all()      # the tiles of 128 rows take the limit of a gate that is no number


def test_gated_product_keeps_nan():
    """Without a limit a NaN in the gate stays one (a minimum with infinity would drop it)."""
    from llmserver_b200.ops import gemm_bf16
    from llmserver_b200 import ops
    x, gate, up = rand((2000, 256), torch.bfloat16, 1), rand((1152, 256), torch.bfloat16, 2), rand((1152, 256), torch.bfloat16, 3)
    x[1700, 3] = float("nan")
    out = gemm_bf16.gated_by_pairs(x, ops.interleave_gate_up(gate, up), 64, math.inf, 1.0, 0.0)
    assert torch.isnan(out[1700]).all() and torch.isfinite(out[:1700]).all() and torch.isfinite(out[1701:]).all()


def test_which_products_are_fused():
    """Few rows, few features, a large inner size, operands that are no bfloat16 rows in one piece: the caller's two kernels."""
    from llmserver_b200.ops import gemm_bf16
    weight = rand((2 * 1536, 512), torch.bfloat16, 2)      # 72 tiles at the fewest rows: a wave of 74 pairs
    take = lambda x, w=weight: gemm_bf16.gated_by_pairs(x, w, 0, math.inf, 1.0, 0.0)  # noqa: E731
    assert take(rand((gemm_bf16.PAIR_MIN_ROWS, 512), torch.bfloat16, 1)) is not None
    assert take(rand((gemm_bf16.PAIR_MIN_ROWS - 1, 512), torch.bfloat16, 1)) is None
    assert take(rand((gemm_bf16.PAIR_MIN_ROWS, 512), torch.bfloat16, 1), weight[:256]) is None
    assert take(rand((2000, 1024), torch.bfloat16, 1)[:, :512]) is None
    wide = gemm_bf16.PAIR_MAX_INNER + 64
    assert take(rand((2000, wide), torch.bfloat16, 1), rand((3072, wide), torch.bfloat16, 2)) is None


@pytest.mark.parametrize("tokens,experts,top,features,inner", [(5, 4, 2, 64, 64), (300, 3, 2, 136, 128), (700, 5, 3, 320, 192), (2048, 16, 4, 256, 256)])
def test_expert_products_on_tiles_of_256_rows(tokens, experts, top, features, inner):
    """Every pair gets the sums that the kernel for tiles of 128 rows gives it, bit for bit (both add along K in the order of the
    tensor core's steps); one expert is chosen by nearly all tokens, one by none."""
    from llmserver_b200 import ops
    from llmserver_b200.ops.library import check_wait_errors
    generator = torch.Generator().manual_seed(tokens)
    chosen = torch.stack([torch.randperm(experts - 1, generator=generator)[:top] for _ in range(tokens)])
    chosen[: tokens * 9 // 10, 0] = 0
    chosen = torch.where((chosen[:, 1:] == chosen[:, :1]).any(1, keepdim=True) & (torch.arange(top) > 0), chosen * 0 + experts - 2, chosen) if top == 2 else chosen
    chosen = chosen.to(torch.int32).to(DEVICE)
    x = rand((tokens, inner), torch.bfloat16, 4)
    gate_up, down = rand((experts, 2 * features, inner), torch.bfloat16, 5, inner ** -0.5), rand((experts, inner, features), torch.bfloat16, 6, features ** -0.5)
    up_only = rand((experts, features, inner), torch.bfloat16, 7, inner ** -0.5)
    got = {}
    for rows in (ops.MOE_TILE_ROWS, ops.MOE_PAIR_TILE_ROWS):
        plan = ops.moe_plan(chosen, experts, rows)
        hidden = ops.moe_grouped(x, gate_up, plan, gather_div=top, gated=(7.0, 1.702))
        squared = ops.moe_grouped(x, up_only, plan, gather_div=top, squared_relu=True)
        place = plan.row_of_pair.long()
        got[rows] = hidden[place], squared[place], ops.moe_grouped(hidden, down, plan)[place]
    torch.cuda.synchronize()
    check_wait_errors()
    few, many = got[ops.MOE_TILE_ROWS], got[ops.MOE_PAIR_TILE_ROWS]
    assert torch.equal(many[1], few[1])
    assert torch.equal(many[0], few[0])
    assert torch.equal(many[2], few[2])
