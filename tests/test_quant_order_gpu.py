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
