"""Products whose reduction is shared by a thread-block cluster: what their owners store."""
import pytest
import torch

from test_kernels_gpu import _ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,heads,kv_heads,dh,ps,k", [(17, 12, 12, 64, 64, 768), (64, 6, 3, 32, 16, 128),
                                                      (40, 5, 1, 24, 32, 320), (1, 2, 2, 8, 1, 64),
                                                      (23, 16, 16, 64, 64, 1024)])
def test_gemm_midm_scatters_keys_and_values_to_the_cache(m, heads, kv_heads, dh, ps, k):
    """The key and value columns of a fused QKV product reach the cache slots bit for bit as the
    output holds them; a token without a slot reaches nothing; with the cache alone the query
    columns are as before."""
    ops = _ops()
    g = torch.Generator(device="cuda").manual_seed(m)
    pages = (m + ps - 1) // ps + 3
    q_width, kv_width = heads * dh, kv_heads * dh
    n = q_width + 2 * kv_width
    a = torch.randn(m, k, device="cuda", generator=g).to(torch.bfloat16)
    w = (torch.randn(n, k, device="cuda", generator=g) * 0.2).to(torch.bfloat16)
    bias = torch.randn(n, device="cuda", generator=g)
    slots = torch.randperm(pages * ps, device="cuda", generator=g)[:m].to(torch.int32)
    if m > 3:
        slots[3] = -1
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    plain = torch.zeros(m, n, device="cuda", dtype=torch.bfloat16)
    ops.gemm_midm(plain, a, w, bias=bias, status=status)
    k1, v1, k2, v2 = (torch.zeros(pages, kv_heads, ps, dh, device="cuda", dtype=torch.bfloat16) for _ in range(4))
    ops.kv_append(k1, v1, plain[:, q_width:q_width + kv_width], plain[:, q_width + kv_width:], slots, m, status)
    out = torch.zeros_like(plain)
    ops.gemm_midm(out, a, w, bias=bias, kv_scatter=(k2, v2, slots, q_width), status=status)
    assert torch.equal(out, plain) and torch.equal(k1, k2) and torch.equal(v1, v2)
    k3, v3 = torch.zeros_like(k1), torch.zeros_like(k1)
    out = torch.full_like(plain, 7.0)
    ops.gemm_midm(out, a, w, bias=bias, kv_scatter=(k3, v3, slots, q_width, True), status=status)
    assert torch.equal(k1, k3) and torch.equal(v1, v3) and torch.equal(out[:, :q_width], plain[:, :q_width])
    assert status.tolist() == [0, 0, 0, 0]
    with pytest.raises(ops.KernelArgumentError):
        ops.gemm_midm(torch.zeros(m, n, device="cuda"), a, w, kv_scatter=(k3, v3, slots, q_width))
