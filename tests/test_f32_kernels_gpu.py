"""The kernels of the float32 path: one order of sums whichever kernel runs, at the sizes where
tiles, chunks and stages end."""
import pytest
import torch

from test_kernels_gpu import _ops, _paged_case, _ref_attention

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 2, 3, 4, 5, 8, 9, 16, 17, 64, 65, 129])
@pytest.mark.parametrize("n,k", [(1, 1), (70, 20), (130, 33), (768, 768), (257, 3072), (300, 6400),
                                 (2304, 100), (5000, 96)])
def test_gemm_f32_kernels_give_the_same_bits(m, n, k):
    ops = _ops()
    g = torch.Generator(device="cuda").manual_seed(m * 7 + n + k)
    wide = torch.randn(m, k + 3, device="cuda", generator=g)          # rows that start off 16 bytes
    a = wide[:, :k].contiguous()
    w = torch.randn(n, k, device="cuda", generator=g)
    bias = torch.randn(n, device="cuda", generator=g)
    resid = torch.randn(m, n, device="cuda", generator=g)
    torch.cuda.synchronize()
    out = [torch.full((m, n), float("nan"), device="cuda") for _ in range(4)]
    for which in range(4):
        ops.gemm_f32(out[which], a, w, bias=bias, resid=resid, kernel=which)
    strided = torch.full((m, n), float("nan"), device="cuda")
    ops.gemm_f32(strided, wide[:, :k], w, bias=bias, resid=resid)
    exact = a.double() @ w.double().t() + bias.double() + resid.double()
    # a sum of k products in chains of at most 32 and runs of k / 128 + 2: each addition rounds
    # by 2^-24 of the partial sum, which is at most the sum of the magnitudes
    size = a.abs().double() @ w.abs().double().t() + bias.abs().double() + resid.abs().double()
    assert bool(((out[0].double() - exact).abs() <= size * 2.0 ** -24 * (40 + k // 128)).all())
    for other in out[1:] + [strided]:
        assert torch.equal(out[0], other)


@pytest.mark.parametrize("m", [1, 7, 16, 40])
@pytest.mark.parametrize("pitch", [0, 4, 64, 100, 132])
def test_gemm_f32_of_weight_rows_that_overlap_or_lie_apart(m, pitch):
    ops = _ops()
    g = torch.Generator(device="cuda").manual_seed(pitch)
    n, k = 300, 96
    a = torch.randn(m, k, device="cuda", generator=g)
    w = torch.randn(n * 132 + k, device="cuda", generator=g).as_strided((n, k), (pitch, 1))
    out, want = (torch.full((m, n), float("nan"), device="cuda") for _ in range(2))
    ops.gemm_f32(out, a, w)
    ops.gemm_f32(want, a, w.clone(memory_format=torch.contiguous_format))
    assert torch.equal(out, want)


CASES = [
    # heads, kv heads, head size, page size, window
    (12, 12, 64, 64, None), (4, 4, 16, 16, None), (6, 2, 64, 64, 70), (5, 1, 48, 32, 300),
    (2, 2, 128, 128, None), (8, 4, 80, 64, 100), (3, 1, 4, 1, None), (2, 1, 100, 24, 256),
]


@pytest.mark.parametrize("nh,nkv,dh,ps,window", CASES)
def test_attention_f32(nh, nkv, dh, ps, window):
    """Tiles and single tokens against the plain reference, the same bits from both for the same
    query; what lies behind a request's last token is poisoned."""
    ops = _ops()
    lengths, portions = [1, 63, 64, 65, 257, 300, 1000, 129], [1, 5, 64, 1, 17, 1, 33, 129]
    q, k, v, table, seq, pos = _paged_case(3, nh, nkv, dh, ps, lengths, portions, torch.float32)
    for b, n in enumerate(lengths):
        if n % ps:
            page = int(table[b, n // ps])
            k[page, :, n % ps:] = float("nan")
            v[page, :, n % ps:] = float("nan")
    t = q.shape[0]
    tiles, at = [], 0
    for p in portions:
        tiles += [(at + r, min(128, p - r)) for r in range(0, p, 128)]
        at += p
    ints = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")  # noqa: E731
    row0, rows = ints([a for a, _ in tiles] + [0]), ints([b for _, b in tiles] + [0])
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    by_tile, single = torch.full_like(q, float("nan")), torch.full_like(q, float("nan"))
    for out, n, count, lists in ((by_tile, len(tiles) + 1, ints([len(tiles)]), dict(tiles=(row0, rows))),
                                 (single, t, ints([t]), dict(token_list=torch.arange(t, dtype=torch.int32,
                                                                                     device="cuda")))):
        # (bounds on the context of one and of two to eight groups of keys: another split, same bits)
        ops.attention_f32(out, q, k, v, table, seq, pos, count, n, nh, 0.3, window, 1024, status, **lists)
        for bound in [4000] + ([window, window + 1] if window else []):   # (windowed: positions lie behind it)
            again = torch.full_like(q, float("nan"))
            ops.attention_f32(again, q, k, v, table, seq, pos, count, n, nh, 0.3, window, bound, status, **lists)
            assert torch.equal(out, again)
    assert status.tolist() == [0, 0, 0, 0]
    assert torch.equal(by_tile, single)
    ref = _ref_attention(q, k, v, table, seq, pos, nh, 0.3, window)
    assert float((by_tile - ref).abs().max()) <= 2e-5


def test_attention_f32_records_what_is_out_of_range():
    ops = _ops()
    q, k, v, table, seq, pos = _paged_case(4, 2, 2, 64, 64, [100, 200], [1, 20], torch.float32)
    table[0, 1] = -1                                       # request 0's second page is missing
    pos[5] = 5000                                          # beyond the block table
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    one = torch.tensor([1], dtype=torch.int32, device="cuda")
    out = torch.full_like(q, float("nan"))
    ops.attention_f32(out, q, k, v, table, seq, pos, one, 1, 2, 0.1, None, 256, status,
                      token_list=torch.zeros(1, dtype=torch.int32, device="cuda"))
    assert status.tolist()[0] == 4 and bool(torch.isfinite(out[0]).all())
    status.zero_()
    ops.attention_f32(out, q, k, v, table, seq, pos, one, 1, 2, 0.1, None, 256, status,
                      tiles=(one, one * 20))
    assert status.tolist()[:3] == [2, 5, 5000] and float(out[5].abs().max()) == 0.0
    assert bool(torch.isfinite(out[1:21]).all())
    assert not ops.attention_f32_supports(130, 1024, None) and not ops.attention_f32_supports(62, 1024, None)
    assert ops.attention_f32_supports(64, 1024, None)


@pytest.mark.parametrize("window,far,context", [(70, 900, 1024), (300, 4000, 4096), (20, 260, 512), (600, 30000, 32768)])
def test_attention_f32_refuses_a_tile_whose_tokens_are_not_consecutive(window, far, context):
    """A windowed tile is planned for the keys that consecutive tokens see; positions further apart are
    recorded and leave zeros, and the tile beside it is as it is alone."""
    ops = _ops()
    q, k, v, table, seq, pos = _paged_case(6, 2, 2, 16, 64, [context, 300], [20, 20], torch.float32)
    pos[:20] = torch.arange(10, 30, device="cuda")
    pos[19] = far
    ints = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")  # noqa: E731
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    out, alone = torch.full_like(q, float("nan")), torch.full_like(q, float("nan"))
    ops.attention_f32(alone, q, k, v, table, seq, pos, ints([1]), 1, 2, 0.3, window, context, status,
                      tiles=(ints([20]), ints([20])))
    assert status.tolist() == [0, 0, 0, 0]
    ops.attention_f32(out, q, k, v, table, seq, pos, ints([2]), 2, 2, 0.3, window, context, status,
                      tiles=(ints([0, 20]), ints([20, 20])))
    room = (window + 31 + 254) // 256 + 1                # groups of 256 keys that 32 tokens' windows touch
    ctas = min(room, 8, context // 256)
    if far // 256 + 1 > -(-room // ctas) * ctas:
        assert status.tolist() == [2, 0, far, context] and float(out[:20].abs().max()) == 0.0
    else:
        assert status.tolist() == [0, 0, 0, 0] and bool(torch.isfinite(out[:20]).all())
    assert torch.equal(out[20:], alone[20:])


@pytest.mark.parametrize("n", [1, 64, 65, 257, 300])
@pytest.mark.parametrize("what", ["last key", "a chunk of keys", "query", "infinite value of no weight",
                                  "infinite value far below", "infinite score", "lowest scores"])
def test_attention_f32_of_values_that_are_no_numbers(n, what):
    """What is not finite reaches a result as it does in the kernel that walks all keys at once."""
    ops = _ops()
    q, k, v, table, seq, pos = _paged_case(7, 2, 2, 16, 64, [n], [min(n, 40)], torch.float32)
    at = lambda j: (int(table[0, j // 64]), slice(None), j % 64)  # noqa: E731
    if what == "last key":
        k[at(n - 1)] = float("nan")
    elif what == "a chunk of keys":
        k[int(table[0, 0])] = float("nan")
    elif what == "query":
        q[0, 3] = float("nan")
    elif what == "infinite value of no weight":
        q[:] = 1.0
        k[at(0)] = -1e20
        v[at(0)] = float("inf")
    elif what == "infinite value far below":
        q[:] = 1.0
        k[:] = 0.0
        k[int(table[0, 0])] = -40.0                     # (a whole chunk e^-192 below the next)
        v[at(0)] = float("inf")
    elif what == "infinite score":
        q[:] = 1.0
        k[at(n // 2)] = float("inf")
    else:
        q[:] = 1.0
        k[:] = -torch.finfo(torch.float32).max
    t = q.shape[0]
    ints = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")  # noqa: E731
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    want = torch.empty_like(q)
    ops.attention_generic(want, q, k, v, table, seq, pos, t, 2, 0.3, None, 512, status)
    for lists, count in ((dict(tiles=(ints([0]), ints([t]))), 1),
                         (dict(token_list=torch.arange(t, dtype=torch.int32, device="cuda")), t)):
        out = torch.empty_like(q)
        ops.attention_f32(out, q, k, v, table, seq, pos, ints([count]), count, 2, 0.3, None, 512, status, **lists)
        assert torch.allclose(out, want, rtol=1e-5, atol=1e-6, equal_nan=True)
    assert status.tolist() == [0, 0, 0, 0]
