"""Rows of a norm at the widths and counts where the kernel that takes them changes."""
import pytest
import torch

from test_kernels_gpu import _ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 15, 16, 17, 128, 129, 300])
@pytest.mark.parametrize("width", [1024, 1028, 1600, 2044, 2048, 2052])
@pytest.mark.parametrize("beta", [True, False])
def test_layernorm_of_wide_rows(rows, width, beta):
    ops = _ops()
    g = torch.Generator(device="cuda").manual_seed(rows + width)
    x = torch.randn(rows, width, device="cuda", generator=g) * 3 + 1
    gamma = torch.randn(width, device="cuda", generator=g)
    bias = torch.randn(width, device="cuda", generator=g) if beta else None
    ref = torch.nn.functional.layer_norm(x.double(), (width,), gamma.double(),
                                         None if bias is None else bias.double(), 1e-5)
    for dtype, tol in ((torch.float32, 2e-5), (torch.bfloat16, 2.0 ** -8)):
        out = torch.full((rows, width), float("nan"), device="cuda", dtype=dtype)
        ops.layernorm(out, x, gamma, bias, 1e-5)
        # (bfloat16 rounds once: half of 2^-8 of the value; float32: the statistics' rounding)
        assert bool(((out.double() - ref).abs() <= tol * ref.abs().clamp(min=1.0)).all())
