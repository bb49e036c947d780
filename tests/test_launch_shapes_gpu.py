"""Kernels whose work is dealt out by the sizes of a launch, at the sizes where that turns: strips and
pieces of the weight-streaming product, runs of K of the 32-bit tiles, rows of the norm."""
import pytest
import torch

from test_kernels_gpu import _ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 8, 9, 16])
@pytest.mark.parametrize("n,k", [(16, 64), (4736, 64), (4737, 128), (9473, 768), (50257, 768), (2368, 2048),
                                 (300, 6400), (4800, 1600)])
@pytest.mark.parametrize("norm", [False, True])
def test_weight_streaming_product_of_many_strips(m, n, k, norm):
    """One strip a CTA, a second one for some, many; a ring that is used again; pieces of a strip."""
    ops = _ops()
    if norm and k > ops.smallm_limits()[1]:
        pytest.skip("too wide for the fused norm")
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    w = (torch.randn(n, k, device="cuda", generator=g) * 0.1).to(torch.bfloat16)
    bias = torch.randn(n, device="cuda", generator=g)
    out = torch.full((m, n), float("nan"), device="cuda")
    if norm:
        x = torch.randn(m, k, device="cuda", generator=g) * 2.0 + 0.5
        gamma, beta = torch.rand(k, device="cuda", generator=g) + 0.5, torch.randn(k, device="cuda", generator=g)
        ops.gemm_smallm(out, w, norm_input=x, gamma=gamma, beta=beta, eps=1e-6, bias=bias)
        a = torch.nn.functional.layer_norm(x, (k,), gamma, beta, 1e-6).to(torch.bfloat16)
    else:
        a = (torch.randn(m, k, device="cuda", generator=g) * 0.5).to(torch.bfloat16)
        resid = torch.randn(m, n, device="cuda", generator=g)
        out.copy_(resid)
        ops.gemm_smallm(out, w, a=a, bias=bias, resid=out)
        bias = bias + resid
    ref = a.float() @ w.float().t() + bias
    # without the norm only the order of 32-bit sums differs; a normed number may round to the other
    # of two neighbouring bfloat16 numbers (2^-8 of it) in either
    tol = 3e-2 if norm else 2e-4
    assert float((out - ref).abs().max()) <= tol * max(1.0, float(ref.abs().max()))


@pytest.mark.parametrize("n,k", [(4800, 768), (50257, 768), (1600, 1600), (3072, 1600), (4096, 1600), (50257, 1600)])
def test_a_second_place_for_sums_costs_no_cta_and_no_piece(n, k):
    """16 rows without the norm: a strip in one piece, two CTAs an SM where K allows it, whatever place is left."""
    ops = _ops()
    ctas, pieces, sets = ops.smallm_plan(16, False, n, k)
    strips, sms = -(-n // 16), ops.sm_count()
    assert pieces == 1 and sets == 1
    most = 2 * sms if k == 768 or strips <= 2 * sms else sms     # (two strips of 1,600 take one CTA an SM)
    assert ctas == -(-strips // -(-strips // most))
    assert ops.smallm_plan(8, False, n, k)[2] == 2 and ops.smallm_plan(16, True, n, k)[2] == 2


@pytest.mark.parametrize("m,n,k", [(17, 1, 1), (64, 128, 32), (65, 129, 128), (129, 257, 132), (100, 300, 260),
                                   (130, 512, 768)])
def test_float32_tiles_of_one_and_of_two_runs_a_cta_give_the_same_bits(m, n, k):
    """Also with runs of K that are empty, and with rows that no copy engine's map describes."""
    ops = _ops()
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = torch.randn(m, k, device="cuda", generator=g)
    wide = torch.randn(n, k + 1, device="cuda", generator=g)
    resid = torch.randn(m, n, device="cuda", generator=g)
    out = []
    for kernel in (0, 2, 3, 4, 5):
        for w in (wide[:, :k].contiguous(), wide[:, :k]):
            out.append(torch.full((m, n), float("nan"), device="cuda"))
            ops.gemm_f32(out[-1], a, w, resid=resid, kernel=kernel)
    few = torch.full((m, n), float("nan"), device="cuda")
    for i in range(0, m, 16):
        ops.gemm_f32(few[i:i + 16], a[i:i + 16], wide[:, :k].contiguous(), resid=resid[i:i + 16].contiguous())
    for other in out[1:] + [few]:
        assert torch.equal(out[0], other)


@pytest.mark.parametrize("k", [768, 1600, 3072])
def test_float32_tiles_turn_where_a_round_of_clusters_is_full(k):
    """Columns of 64 x 128, by the clusters that the device says run side by side: 64 x 64 while its clusters take one
    round, then one run a CTA while those do; two runs where that saves a round."""
    ops = _ops()
    _kind, (small, one, two) = ops.gemm_f32_tiles(64, 128, k)
    assert 2 * one > small and two > one
    for tiles, kind in ((1, 3), (small // 2, 3), (small // 2 + 1, 4), (one, 4), (one + 1, 3), (two, 5), (9 * two, 5)):
        assert ops.gemm_f32_tiles(64 * tiles, 128, k)[0] == kind, tiles


@pytest.mark.parametrize("rows", [128, 129, 149, 2368, 2369, 5000])
@pytest.mark.parametrize("width", [4, 768, 1024, 1028, 1600, 2048])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_norm_of_many_rows(rows, width, dtype):
    """More than 128 rows by the kernel of a CTA an SM: the same bits as a few at a time, and right."""
    ops = _ops()
    g = torch.Generator(device="cuda").manual_seed(rows + width)
    x = torch.randn(rows, width, device="cuda", generator=g) * 3.0 + 1.0
    gamma, beta = torch.randn(width, device="cuda", generator=g), torch.randn(width, device="cuda", generator=g)
    out = torch.full((rows, width), float("nan"), device="cuda", dtype=dtype)
    few = torch.full_like(out, float("nan"))
    ops.layernorm(out, x, gamma, beta, 1e-5)
    for i in range(0, rows, 100):
        ops.layernorm(few[i:i + 100], x[i:i + 100], gamma, beta, 1e-5)
    assert torch.equal(out, few)
    ref = torch.nn.functional.layer_norm(x.double(), (width,), gamma.double(), beta.double(), 1e-5)
    # 32-bit statistics of rows around 1: a few roundings of 2^-24 of numbers up to 3, or bfloat16's own
    tol = 1e-5 if dtype == torch.float32 else 2.0 ** -8
    assert bool(((out.double() - ref).abs() <= tol * (1.0 + ref.abs())).all())


@pytest.mark.parametrize("m", [1, 4, 8, 13, 16])
@pytest.mark.parametrize("heads,kv_heads,dh,ps", [(6, 3, 64, 16), (2, 1, 20, 24), (3, 3, 7, 1), (12, 12, 64, 64)])
def test_float32_product_scatters_keys_and_values(m, heads, kv_heads, dh, ps):
    """The key and value columns of a fused QKV product reach the cache as the append kernel brings them."""
    ops = _ops()
    g = torch.Generator(device="cuda").manual_seed(m + dh)
    q_width, kv_width, k = heads * dh, kv_heads * dh, 96
    n, pages = q_width + 2 * kv_width, 2 + 140 // ps
    a, w = torch.randn(m, k, device="cuda", generator=g), torch.randn(n, k, device="cuda", generator=g)
    bias = torch.randn(n, device="cuda", generator=g)
    slots = torch.randperm(pages * ps, generator=torch.Generator().manual_seed(m))[:m].to(torch.int32)
    slots[m // 2] = -1
    slots = slots.cuda()
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    cache = [torch.zeros(pages, kv_heads, ps, dh, device="cuda") for _ in range(4)]
    out = [torch.full((m, n), float("nan"), device="cuda") for _ in range(2)]
    ops.gemm_f32(out[0], a, w, bias=bias, status=status, kv_scatter=(cache[0], cache[1], slots, q_width))
    ops.gemm_f32(out[1], a, w, bias=bias)
    ops.kv_append(cache[2], cache[3], out[1][:, q_width:q_width + kv_width], out[1][:, q_width + kv_width:], slots,
                  m, status)
    assert torch.equal(out[0], out[1]) and torch.equal(cache[0], cache[2]) and torch.equal(cache[1], cache[3])
    assert status.tolist() == [0, 0, 0, 0]
    slots[0] = pages * ps                                  # a slot outside the pool is recorded, not written
    ops.gemm_f32(out[0], a, w, bias=bias, status=status, kv_scatter=(cache[0], cache[1], slots, q_width))
    assert status.tolist()[0] == 3
    many = torch.zeros(17, k, device="cuda")               # more rows than the kernel that does it takes
    with pytest.raises(ops.KernelArgumentError, match="size"):
        ops.gemm_f32(torch.zeros(17, n, device="cuda"), many, w,
                     kv_scatter=(cache[0], cache[1], torch.zeros(17, dtype=torch.int32, device="cuda"), q_width))


@pytest.mark.parametrize("m", [1, 5, 16])
@pytest.mark.parametrize("k", [8192, 8224, 8225, 16384, 16640, 40000])
def test_float32_product_says_where_it_scatters(m, k):
    """The widest rows: where the answer is yes the product brings keys and values to the cache, however its rows
    are aligned, and where it is no it refuses."""
    ops = _ops()
    g = torch.Generator(device="cuda").manual_seed(m + k)
    dh, ps = 8, 16
    a, w = torch.randn(m, k + 1, device="cuda", generator=g), torch.randn(3 * dh, k, device="cuda", generator=g)
    slots = torch.arange(m, dtype=torch.int32, device="cuda")
    want = ops.gemm_f32_scatters(m, 3 * dh, k)
    assert want or k > 8225
    for rows in (a[:, :k], a[:, :k].contiguous()):
        keys, values = torch.zeros(2, 1, ps, dh, device="cuda"), torch.zeros(2, 1, ps, dh, device="cuda")
        out = torch.zeros(m, 3 * dh, device="cuda")
        if want:
            ops.gemm_f32(out, rows, w, kv_scatter=(keys, values, slots, dh))
            assert torch.equal(keys.view(-1, dh)[:m], out[:, dh:2 * dh])
            assert torch.equal(values.view(-1, dh)[:m], out[:, 2 * dh:])
            # (a sum of k products of numbers around 1, chunk by chunk)
            assert float((out.double() - rows.double() @ w.double().t()).abs().max()) <= 1e-6 * k
        else:
            with pytest.raises(ops.KernelArgumentError, match="size"):
                ops.gemm_f32(out, rows, w, kv_scatter=(keys, values, slots, dh))
    assert not ops.gemm_f32_scatters(17, 3 * dh, 64)


@pytest.mark.parametrize("heads", [20, 25, 32])
def test_a_few_requests_keep_32_bit_weights(heads):
    """Fewer than 16 tokens of up to two (token, head) pairs an SM stay with the kernel that multiplies the values
    by 32-bit weights; the other one rounds them to bfloat16."""
    ops = _ops()
    for tokens in range(1, 16):
        for context in (256, 512, 768, 1024):
            if tokens * heads < 2 * ops.sm_count():
                assert not ops.decode_ring_prefers(tokens, heads, context)
    assert ops.decode_ring_prefers(16, 12, 1024) and not ops.decode_ring_prefers(16, 12, 512)
