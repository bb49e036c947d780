"""Kernels that may start while the kernel ahead of them still runs read what that kernel wrote:
each is launched directly behind a kernel that signals at once and then writes its operand."""
import pytest
import torch

from test_kernels_gpu import _ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(8, 768, 768), (3, 2304, 100), (1, 700, 33), (65, 768, 3072), (40, 130, 33)])
def test_gemm_f32_reads_weights_written_by_the_kernel_before_it(m, n, k):
    ops = _ops()
    g = torch.Generator(device="cuda").manual_seed(n + k)
    a = torch.randn(m, k, device="cuda", generator=g)
    sources = [torch.randn(n, k, device="cuda", generator=g) for _ in range(8)]
    wants = []
    for src in sources:
        want = torch.empty(m, n, device="cuda")
        torch.cuda.synchronize()
        ops.gemm_f32(want, a, src, settled=True)
        torch.cuda.synchronize()
        wants.append(want)
    w = torch.zeros(n, k, device="cuda")
    outs = [torch.empty(m, n, device="cuda") for _ in sources]
    torch.cuda.synchronize()
    for src, out in zip(sources, outs):
        ops.bias_act(w, src, None, None, None)
        ops.gemm_f32(out, a, w)
    for out, want in zip(outs, wants):
        assert torch.equal(out, want)
