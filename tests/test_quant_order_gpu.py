"""The quantizer's launch starts early but keeps stream order with what writes its weights and reads or overwrites its
results."""
import pytest
import torch

from gemmlib_b200 import capi, ms_blkq4linear_ext
from gemmlib_b200.ms_blkq4linear import BlkQ4Linear

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("colwise", [True, False])
def test_quantizer_keeps_stream_order(colwise):
    K, N, block = 4096, 2048, 64
    g = torch.Generator(device="cuda").manual_seed(0)
    src = [(torch.randn(N, K, generator=g, device="cuda") * 0.02).half() for _ in range(6)]
    meta = K * N // block

    def outputs():
        return (torch.empty(K * N // 2, dtype=torch.uint8, device="cuda"), torch.empty(meta, dtype=torch.float16, device="cuda"),
                torch.empty(meta, dtype=torch.uint8, device="cuda"))

    want = []
    for w in src:
        q = outputs()
        capi.quant(block, colwise, K, N, K, w, *q)
        torch.cuda.synchronize()
        want.append(q)
    # one weight buffer rewritten, and one set of outputs copied away, between launches that are all queued at once
    w, q, got = torch.empty_like(src[0]), outputs(), []
    for x in src:
        w.copy_(x)
        capi.quant(block, colwise, K, N, K, w, *q)
        got.append([t.clone() for t in q])
    # back to back into one set of outputs: the last one stays
    for x in src:
        capi.quant(block, colwise, K, N, K, x, *q)
    torch.cuda.synchronize()
    for a, b in zip(want + [want[-1]], got + [list(q)]):
        for s, t in zip(a, b):
            assert torch.equal(s.view(torch.uint8), t.view(torch.uint8))


@pytest.mark.parametrize("block,N", [(32, 64 * 32768 + 32), (128, 128 * 32768 + 128), (16, 64 * 32768 - 32)])
def test_row_wise_tiles_beyond_one_grid_layer(block, N):
    """The column tiles fold into the grid's third dimension: what lies behind the fold against the same columns alone."""
    K, tail = 64, 4096
    g = torch.Generator(device="cuda").manual_seed(1)
    w = (torch.randn(N, K, generator=g, device="cuda") * 0.02).half()

    def quant(x):
        n = x.size(0)
        q = (torch.empty(K * n // 2, dtype=torch.uint8, device="cuda"), torch.empty(K * n // block, dtype=torch.float16, device="cuda"),
             torch.empty(K * n // block, dtype=torch.uint8, device="cuda"))
        capi.quant(block, False, K, n, K, x, *q)
        torch.cuda.synchronize()
        return q

    start = (N - tail) // 128 * 128  # a shard of the columns is a contiguous range of bytes
    for whole, part in zip(quant(w), quant(w[start:].contiguous())):
        assert torch.equal(whole[-part.numel():].view(torch.uint8), part.view(torch.uint8))


def weight(N, K, seed):
    return (torch.randn(N, K, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda") * 0.02).half()


def packed(K, N, block):
    meta = K * N // block
    return (torch.empty(K * N // 2, dtype=torch.uint8, device="cuda"), torch.empty(meta, dtype=torch.float16, device="cuda"),
            torch.empty(meta, dtype=torch.uint8, device="cuda"))


def same(a, b):
    return torch.equal(a.view(torch.uint8), b.view(torch.uint8))


def long_gemm(M, N, K):
    """Activations, and a function that multiplies them into a tensor: a kernel of about 100 us that lets its successor start at once."""
    layer = BlkQ4Linear(64, True, False, weight(N, K, 11))
    a = torch.randn(M, K, generator=torch.Generator(device="cuda").manual_seed(12), device="cuda").half()
    stream = torch.cuda.current_stream().cuda_stream
    return a, lambda out: capi.gemm(64, True, M, N, K, a, layer.q_weights, layer.q_scales, layer.q_zp, out, stream=stream)


@pytest.mark.parametrize("col_wise", [True, False])
def test_quantizer_waits_for_the_kernel_that_writes_its_weights(col_wise):
    """The weights are the result of a GEMM, which lets the quantizer start before it has written anything."""
    M, N, K = 2048, 4096, 8192
    _, gemm = long_gemm(M, N, K)
    out, want = torch.empty(M, N, dtype=torch.float16, device="cuda"), packed(N, M, 64)
    gemm(out)
    torch.cuda.synchronize()
    capi.quant(64, col_wise, N, M, N, out, *want)
    for _ in range(5):
        got = packed(N, M, 64)
        out.fill_(float("nan"))
        torch.cuda.synchronize()
        torch.cuda._sleep(400_000)  # both launches are queued before the first starts
        gemm(out)
        capi.quant(64, col_wise, N, M, N, out, *got)
        torch.cuda.synchronize()
        assert all(same(a, b) for a, b in zip(want, got))


@pytest.mark.parametrize("col_wise", [True, False])
def test_quantizer_waits_for_the_kernel_that_reads_what_it_overwrites(col_wise):
    """The scales of the quantizer take the place of the activations of the GEMM before it."""
    M, N, K = 256, 28672, 8192
    n, k, block = 8192, 4096, 16  # as many scales as activations
    a, gemm = long_gemm(M, N, K)
    w, keep = weight(n, k, 13), a.clone()
    out, want = torch.empty(M, N, dtype=torch.float16, device="cuda"), torch.empty(M, N, dtype=torch.float16, device="cuda")
    gemm(want)
    q = packed(k, n, block)
    assert q[1].numel() == a.numel()
    for _ in range(5):
        a.copy_(keep)
        out.fill_(float("nan"))
        torch.cuda.synchronize()
        torch.cuda._sleep(400_000)
        gemm(out)
        capi.quant(block, col_wise, k, n, k, w, q[0], a.view(-1), q[2])
        torch.cuda.synchronize()
        assert same(out, want) and not same(a, keep)


def test_captured_copy_quantizer_and_gemm():
    """Replays of one graph that copies new weights in, quantizes them and multiplies with the early weight fetch."""
    N, K, M = 2048, 2048, 4
    x = torch.randn(M, K, generator=torch.Generator(device="cuda").manual_seed(7), device="cuda").half()
    src, w = weight(N, K, 0), torch.empty(N, K, dtype=torch.float16, device="cuda")
    layer = BlkQ4Linear(64, True, False, src)
    layer(x)
    graph, stream, out = torch.cuda.CUDAGraph(), torch.cuda.Stream(), torch.empty(M, N, dtype=torch.float16, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        w.copy_(src)
        capi.quant(64, True, K, N, K, w, layer.q_weights, layer.q_scales, layer.q_zp, stream=stream.cuda_stream)
        layer(x, out=out)
    for seed in range(1, 5):
        new = weight(N, K, seed)
        src.copy_(new)
        graph.replay()
        torch.cuda.synchronize()
        assert same(out, BlkQ4Linear(64, True, False, new)(x))


@pytest.mark.parametrize("col_wise,N,K", [(True, 2048, 2048), (False, 1024, 2048), (True, 512, 4096)])
@pytest.mark.parametrize("M", [1, 12, 40])
def test_early_weight_fetch_behind_the_quantizer(M, col_wise, N, K):
    """A layer whose first (plain) call ran on a side stream, and a layer whose packed tensors were replaced, are called with
    the early weight fetch right behind the quantizer of those tensors, all queued behind a long kernel."""
    x = torch.randn(M, K, generator=torch.Generator(device="cuda").manual_seed(7), device="cuda").half()
    ws = [weight(N, K, s) for s in range(4)]
    want = []
    for w in ws:
        layer = BlkQ4Linear(64, col_wise, False, w)
        torch.cuda.synchronize()
        want.append(layer(x))
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    got = []
    for w in ws:
        torch.cuda._sleep(2_000_000)  # about a millisecond: the calls below are queued before the quantizer starts
        layer = BlkQ4Linear(64, col_wise, False, w)
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            layer(x)
        assert layer._settled and layer.early_weight_fetch
        got.append(layer(x))
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    replaced = []
    for w in ws:
        torch.cuda._sleep(2_000_000)
        layer.q_weights, layer.q_scales, layer.q_zp = ms_blkq4linear_ext.quant(64, col_wise, True, w)
        replaced.append(layer(x))
    torch.cuda.synchronize()
    for a, b, c in zip(want, got, replaced):
        assert torch.equal(a.view(torch.int16), b.view(torch.int16)) and torch.equal(a.view(torch.int16), c.view(torch.int16))
