"""Kernels that may start while the kernel ahead of them still runs read what that kernel wrote:
each is launched directly behind a kernel that signals at once and then writes its operand."""
import pytest
import torch

from test_kernels_gpu import _ops, _paged_case

pytestmark = pytest.mark.gpu


def _sources(g, n, k, count=8):
    """Operands of products whose results are the [n, k] tensors to be written."""
    return [(torch.randn(n, 640, device="cuda", generator=g), torch.randn(k, 640, device="cuda", generator=g))
            for _ in range(count)]


def _write(ops, out, source):
    """out <- a product, by a kernel that lets its successor start before it has written anything."""
    ops.gemm_f32(out, source[0], source[1], settled=True)


def _compare(write, read, shape, sources):
    """``read`` directly behind ``write``, for one source after the other, against the two with a
    synchronisation between them."""
    wants, outs = ([torch.zeros(shape, device="cuda") for _ in sources] for _ in range(2))
    for src, want in zip(sources, wants):
        torch.cuda.synchronize()
        write(src)
        torch.cuda.synchronize()
        read(want)
    torch.cuda.synchronize()
    for src, out in zip(sources, outs):
        write(src)
        read(out)
    for out, want in zip(outs, wants):
        assert torch.equal(out, want)


@pytest.mark.parametrize("m,n,k", [(8, 768, 768), (3, 2304, 100), (1, 700, 33), (65, 768, 3072), (40, 130, 33)])
def test_gemm_f32_reads_weights_written_by_the_kernel_before_it(m, n, k):
    ops = _ops()
    g = torch.Generator(device="cuda").manual_seed(n + k)
    a = torch.randn(m, k, device="cuda", generator=g)
    w = torch.zeros(n, k, device="cuda")
    _compare(lambda src: _write(ops, w, src), lambda out: ops.gemm_f32(out, a, w), (m, n), _sources(g, n, k))


@pytest.mark.parametrize("rows,width", [(1, 768), (100, 1024), (20, 1600), (3, 2052), (129, 768), (2369, 1600)])
def test_layernorm_reads_parameters_written_by_the_kernel_before_it(rows, width):
    ops = _ops()
    g = torch.Generator(device="cuda").manual_seed(rows + width)
    x = torch.randn(rows, width, device="cuda", generator=g)
    w = torch.zeros(2, width, device="cuda")
    _compare(lambda src: _write(ops, w, src), lambda out: ops.layernorm(out, x, w[0], w[1], 1e-5), (rows, width),
             _sources(g, 2, width))


@pytest.mark.parametrize("rows,width", [(1, 768), (128, 1024), (129, 768), (149, 1600), (2369, 1024)])
def test_layernorm_of_settled_parameters_reads_rows_written_by_the_kernel_before_it(rows, width):
    ops = _ops()
    g = torch.Generator(device="cuda").manual_seed(rows + width)
    x = torch.zeros(rows, width, device="cuda")
    gamma, beta = torch.randn(width, device="cuda", generator=g), torch.randn(width, device="cuda", generator=g)
    _compare(lambda src: _write(ops, x, src), lambda out: ops.layernorm(out, x, gamma, beta, 1e-5, settled=True),
             (rows, width), _sources(g, rows, width))


@pytest.mark.parametrize("m,n,k,kernel", [(16, 768, 768, 0), (65, 768, 768, 3), (65, 768, 3072, 4), (690, 2304, 768, 4),
                                          (690, 2304, 768, 5), (129, 1027, 260, 5), (130, 700, 33, 0)])
def test_gemm_f32_of_settled_weights_reads_rows_written_by_the_kernel_before_it(m, n, k, kernel):
    """Its weights may be read while the kernel ahead still runs, its rows of A may not."""
    ops = _ops()
    g = torch.Generator(device="cuda").manual_seed(n + k + kernel)
    w = torch.randn(n, k, device="cuda", generator=g)
    a = torch.zeros(m, k, device="cuda")
    _compare(lambda src: _write(ops, a, src), lambda out: ops.gemm_f32(out, a, w, kernel=kernel, settled=True), (m, n),
             _sources(g, m, k))


@pytest.mark.parametrize("rows,width", [(1, 768), (100, 1600), (5, 4100)])
def test_norm_pair_reads_parameters_written_by_the_kernel_before_it(rows, width):
    ops = _ops()
    g = torch.Generator(device="cuda").manual_seed(rows + width)
    y = torch.randn(rows, width, device="cuda", generator=g)
    w = torch.zeros(4, width, device="cuda")

    def read(out):                                       # (x is zero at first)
        ops.norm_pair(out[:rows], y, 0.5, w[0], w[1], 1e-5, True, out=out[rows:],
                      next_norm=(w[2], w[3], 1e-5, True))

    _compare(lambda src: _write(ops, w, src), read, (2 * rows, width), _sources(g, 4, width))


@pytest.mark.parametrize("heads,kv_heads,dh", [(12, 12, 64), (4, 1, 128), (3, 3, 20)])
def test_attention_f32_reads_rows_written_by_the_kernel_before_it(heads, kv_heads, dh):
    ops = _ops()
    lengths = [250, 129, 64, 33, 7, 1]
    q, k, v, table, seq, pos = _paged_case(5, heads, kv_heads, dh, 64, lengths, [1] * len(lengths), torch.float32)
    t = len(lengths)
    g = torch.Generator(device="cuda").manual_seed(dh)
    held = torch.cat([table[b, torch.arange(n, device="cuda") // 64] * 64 + torch.arange(n, device="cuda") % 64
                      for b, n in enumerate(lengths)]).to(torch.int32)          # every slot the requests hold
    sources = [torch.randn(len(held), 2 * kv_heads * dh, device="cuda", generator=g) for _ in range(8)]
    tokens, count = torch.arange(t, dtype=torch.int32, device="cuda"), torch.tensor([t], dtype=torch.int32, device="cuda")
    status = torch.zeros(4, dtype=torch.int32, device="cuda")

    def write(src):
        ops.kv_append(k, v, src[:, :kv_heads * dh], src[:, kv_heads * dh:], held, len(held), status)

    def read(out):
        ops.attention_f32(out, q, k, v, table, seq, pos, count, t, heads, 0.2, None, 256, status, token_list=tokens)

    _compare(write, read, tuple(q.shape), sources)
    assert status.tolist() == [0, 0, 0, 0]


@pytest.mark.parametrize("rows,n", [(1, 2048), (24, 3072)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_gated_pair_reads_what_the_kernel_before_it_wrote(rows, n, dtype):
    ops = _ops()
    g = torch.Generator(device="cuda").manual_seed(n)
    pair = torch.zeros(rows, 2 * n + 64, device="cuda")                 # gate, up, a scale for 64 columns each
    half = torch.empty(rows, n, device="cuda", dtype=dtype)

    def read(out):
        ops.gated_pair(half, pair, 0, n, n, scale=pair[:, 2 * n:], group=64)
        out.copy_(half)

    _compare(lambda src: _write(ops, pair, src), read, (rows, n), _sources(g, rows, 2 * n + 64))


@pytest.mark.parametrize("rows,n", [(1, 2048), (24, 3072), (5, 1030)])
def test_act_columns_reads_what_the_kernel_before_it_wrote(rows, n):
    ops = _ops()
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.zeros(rows, n, device="cuda")
    _compare(lambda src: _write(ops, x, src), lambda out: ops.act_columns(out, x), (rows, n),
             _sources(g, rows, n))


@pytest.mark.parametrize("m,n,k", [(300, 768, 768), (1200, 1600, 512), (130, 1027, 768), (280, 768, 3072)])
def test_gemm_bf16_reads_the_residual_the_kernel_before_it_wrote(m, n, k):
    ops = _ops()
    g = torch.Generator(device="cuda").manual_seed(n)
    a = torch.randn(m, k, device="cuda", generator=g).to(torch.bfloat16)
    w = torch.randn(n, k, device="cuda", generator=g).to(torch.bfloat16)
    x = torch.zeros(m, n, device="cuda")

    def read(out):
        ops.gemm_bf16(x, a, w, resid=x)
        out.copy_(x)

    _compare(lambda src: _write(ops, x, src), read, (m, n), _sources(g, m, n))
