"""Residual add + norm at widths on both sides of each arrangement: one, two and four pieces per thread, ragged last pieces, the widest
row that the vector form takes, and a width that it does not take."""
import pytest
import torch

from test_gpu_kernels import DEVICE, DTYPES, close, rand

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("width", [8, 248, 2552, 2560, 2568, 5112, 5120, 5128, 7680, 10248, 16384, 16392, 5121])
def test_widths(dtype, width):
    from llmserver_b200 import ops
    rows, eps = 5, 1e-6
    residual, delta = rand((rows, width), torch.float32, 1, 2.0), rand((rows, width), dtype, 2)
    weight, post, bias = rand((width,), dtype, 3, 0.1) + 1, rand((width,), dtype, 4, 0.1) + 1, rand((width,), torch.float32, 5, 0.1)

    def norm(x, w):
        return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w.double()

    work = residual.clone()
    out = ops.add_rmsnorm(work, delta, weight, eps)
    want = residual.double() + delta.double()
    close(work, want, torch.float32, "stream")
    close(out, norm(want, weight), dtype, "norm")
    alone = ops.add_rmsnorm(residual[2:3].clone(), delta[2:3].contiguous(), weight, eps)
    assert torch.equal(alone[0], out[2])
    for extra in (None, rand((rows, width), torch.float32, 6)):
        work = residual.clone()
        out = ops.normed_add_rmsnorm(work, delta, post, eps, weight, eps, extra=extra, act_dtype=dtype, delta_bias=bias)
        want = residual.double() + norm(delta.double() + bias.double(), post) + (0.0 if extra is None else extra.double())
        close(work, want, torch.float32, "stream with a normed delta", factor=2.0)
        close(out, norm(want, weight), dtype, "norm of it", factor=2.0)
