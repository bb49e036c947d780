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


@pytest.mark.parametrize("tile_n,pair", [(224, False), (192, True)])
@pytest.mark.parametrize("m,n,k", [(129, 230, 64), (300, 1000, 1280), (257, 449, 1288), (650, 4800, 1600)])
@pytest.mark.parametrize("act", [None, "gelu"])
def test_gemm_bf16_with_eight_or_sixteen_epilogue_warps(tile_n, pair, m, n, k, act):
    """The tiles whose epilogue has eight warps or sixteen, by activation and reduction."""
    ops = _ops()
    g = torch.Generator(device="cuda").manual_seed(n + k)
    a = torch.randn(m, k, device="cuda", generator=g).to(torch.bfloat16)
    w = (torch.randn(n, k, device="cuda", generator=g) / k ** 0.5).to(torch.bfloat16)
    bias = torch.randn(n, device="cuda", generator=g)
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    out = torch.full((m, n + 8 - n % 8), float("nan"), device="cuda", dtype=torch.bfloat16)
    ops.gemm_bf16(out[:, :n], a, w, bias=bias, act=act, tile_n=tile_n, pair=pair, status=status)
    ref = a.double() @ w.double().t() + bias.double()
    if act:
        ref = torch.nn.functional.gelu(ref)
    # bfloat16 rounds once (2^-9 of the value); the 32-bit sum of k products of size 1 / sqrt(k)
    assert bool(((out[:, :n].double() - ref).abs() <= 2.0 ** -8 * ref.abs().clamp(min=0.25)).all())
    assert bool(torch.isnan(out[:, n:]).all()) and status.tolist() == [0, 0, 0, 0]
