"""The quantizer's launch starts early but keeps stream order with what writes its weights and reads its results."""
import pytest
import torch

from gemmlib_b200 import capi

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
