"""Several weight matrices in one launch: every part bit for bit what its own call gives."""
import pytest
import torch

from gemmlib_b200 import capi
from gemmlib_b200.ms_blkq4linear import BlkQ4Linear
from gemmlib_b200.stack import LinearStack, llama_like_stack

pytestmark = pytest.mark.gpu


def make(N, K, block, zp, seed, bias, colwise=True):
    g = torch.Generator(device="cuda").manual_seed(seed)
    w = (torch.randn(N, K, generator=g, device="cuda") * 0.02).half()
    meta = N * K // block
    q = (torch.empty(N * K // 2, dtype=torch.uint8, device="cuda"), torch.empty(meta, dtype=torch.float16, device="cuda"),
         torch.empty(meta, dtype=torch.uint8, device="cuda") if zp else None)
    capi.quant(block, colwise, K, N, K, w, *q)
    return N, q, (torch.randn(N, generator=g, device="cuda") * 0.02).half() if bias else None


# tiles of 16 columns: fewer than the CTAs, as many, many rounds; parts of one tile; the shortest K and long ones
DECODE = [(1, 2048, 64, True, (32, 32)), (1, 4096, 64, False, (4096, 4096, 4096)), (2, 4096, 128, True, (2368, 32, 96, 1024)),
          (3, 4096, 64, True, (11008, 11008)), (4, 8192, 128, False, (4736, 2368)), (8, 2304, 64, True, (1056, 544, 2016)),
          (5, 11008, 64, False, (2048, 256))]


@pytest.mark.parametrize("flags", [0, capi.EARLY_WEIGHT_FETCH], ids=["plain", "early_fetch"])
@pytest.mark.parametrize("M,K,block,zp,widths", DECODE)
def test_group_equals_its_parts(M, K, block, zp, widths, flags):
    assert capi.gemm_group_supported(block, True, M, K, widths)
    a = torch.randn(M, K, generator=torch.Generator(device="cuda").manual_seed(1), device="cuda").half()
    parts = [make(n, K, block, zp, i, i % 2 == 1) for i, n in enumerate(widths)]
    want = [torch.empty(M, n, dtype=torch.float16, device="cuda") for n in widths]
    got = [torch.full((M, n), float("nan"), dtype=torch.float16, device="cuda") for n in widths]
    for (n, q, b), o in zip(parts, want):
        capi.gemm(block, True, M, n, K, a, *q, o, bias=b)
    torch.cuda.synchronize()
    for _ in range(2):
        capi.gemm_group(block, True, M, K, a, [(n, *q, o, b) for (n, q, b), o in zip(parts, got)], flags=flags)
    torch.cuda.synchronize()
    assert capi.last_kernel_status() == 0
    for n, w, o in zip(widths, want, got):
        assert torch.equal(w.view(torch.int16), o.view(torch.int16)), n


def test_misaligned_scales_of_a_group_are_refused():
    N, q, _ = make(64, 2048, 64, False, 0, False)
    shifted = torch.empty(q[1].numel() + 1, dtype=torch.float16, device="cuda")[1:]
    a, o = torch.zeros(1, 2048, dtype=torch.float16, device="cuda"), torch.empty(2, 1, 64, dtype=torch.float16, device="cuda")
    with pytest.raises(capi.BlkQ4Error, match="Misaligned"):
        capi.gemm_group(64, True, 1, 2048, a, [(64, *q, o[0], None), (64, q[0], shifted, None, o[1], None)])


# column tiles of 128 (pairs of 256) with remainders, in one and in several rounds of both tensor-core kernels
PREFILL = [(17, 512, 32, True, True, (96, 32, 2080)), (64, 1024, 64, True, False, (1024, 1024, 1024)),
           (100, 4096, 128, True, True, (11008, 11008)), (200, 960, 32, False, True, (2080, 4128)),
           (333, 2048, 16, True, False, (7200, 544)), (300, 1024, 64, False, True, (9536, 192, 2048, 64)),
           (512, 1024, 64, True, True, (4096, 4096, 4096)),
           # up to 64 rows and 16 steps a CTA or more (four dequantizer groups): whole rounds, balanced ranges, row-wise blocks
           (64, 4096, 64, True, True, (4096, 4096, 4096)), (33, 4096, 32, True, False, (11008, 11008)),
           (48, 2048, 32, False, True, (2080, 4128))]


@pytest.mark.parametrize("M,K,block,colwise,zp,widths", PREFILL)
def test_prefill_group_equals_its_parts(M, K, block, colwise, zp, widths):
    """Without a workspace bit for bit; with one K is split over all tiles together, another order of the fp32 sums."""
    assert capi.gemm_group_supported(block, colwise, M, K, widths)
    a = torch.randn(M, K, generator=torch.Generator(device="cuda").manual_seed(1), device="cuda").half()
    parts = [make(n, K, block, zp, i, i % 2 == 1, colwise) for i, n in enumerate(widths)]
    want = [torch.empty(M, n, dtype=torch.float16, device="cuda") for n in widths]
    for (n, q, b), o in zip(parts, want):
        capi.gemm(block, colwise, M, n, K, a, *q, o, bias=b)
    need = capi.gemm_group_workspace_size(block, colwise, M, K, widths)
    ws = torch.zeros(need, dtype=torch.uint8, device="cuda") if need else None
    for workspace in (None, ws):
        for flags in (0, capi.EARLY_WEIGHT_FETCH):
            got = [torch.full((M, n), float("nan"), dtype=torch.float16, device="cuda") for n in widths]
            capi.gemm_group(block, colwise, M, K, a, [(n, *q, o, b) for (n, q, b), o in zip(parts, got)], flags=flags,
                            workspace=workspace)
            torch.cuda.synchronize()
            assert capi.last_kernel_status() == 0
            for n, w, o in zip(widths, want, got):
                if workspace is None:
                    assert torch.equal(w.view(torch.int16), o.view(torch.int16)), n
                else:  # one unit of the rounded result, and of the bias added to it
                    d = (w.float() - o.float()).abs()
                    assert bool((d <= 2.0 ** -9 * torch.clamp(w.float().abs(), min=1.0)).all()), (n, float(d.max()))
    if ws is not None:
        assert not ws[:768].any()  # the flag words of balanced ranges are back to zero


@pytest.mark.parametrize("M", [1, 7, 9, 40, 300])
def test_stack_equals_its_layers(M):
    """q, k, v and gate, up are runs of their own, in one launch up to 16 rows and where no layer splits K; the buffers are
    those of one call per layer, bit for bit."""
    stack = llama_like_stack(2048, 2304, 2, 64, True, False, torch.device("cuda"))
    x = torch.randn(M, 2048, device="cuda").half()
    stack.forward(x, "h1")
    got = {k: v.clone() for k, v in stack.buffers(M).items()}
    runs = [len(r) for r in stack._groups(M)]
    assert sum(runs) == 14 and max(runs) == (1 if 8 < M <= 16 else 3)
    for lyr, src, dst in stack.steps[7:]:  # the first block's buffers but "h0" were overwritten by the second's
        want = lyr(got[src])
        assert torch.equal(got[dst].view(torch.int16), want.view(torch.int16)), dst


# (hidden, ffn, rows, launches of a block): layers split K otherwise than a group; balanced ranges; no split, or the same one, so q, k, v
# and gate, up go together, but not gate and up where short tiles would change to the pair kernel without saving a round
@pytest.mark.parametrize("hidden,ffn,M,launches", [(2048, 2304, 40, 7), (2048, 2304, 300, 7), (1024, 19200, 300, 5),
                                                   (512, 768, 17, 4), (512, 768, 333, 4), (2048, 5632, 333, 7),
                                                   (2048, 5632, 512, 6), (2048, 9472, 300, 6), (1024, 5632, 333, 4),
                                                   (1024, 2816, 40, 4), (1024, 2816, 128, 4), (1536, 2816, 100, 4)])
def test_prefill_stack_keeps_every_bit(hidden, ffn, M, launches):
    stack = llama_like_stack(hidden, ffn, 1, 64, True, False, torch.device("cuda"))
    x = torch.randn(M, hidden, device="cuda").half()
    stack.forward(x, "h0")
    got = stack.buffers(M)
    assert len(stack._launches(M)) == launches
    for lyr, src, dst in stack.steps:
        assert torch.equal(got[dst].view(torch.int16), lyr(got[src]).view(torch.int16)), dst


def test_what_keeps_layers_of_a_stack_apart():
    def layer(n, block=64, zp=True):
        return BlkQ4Linear(block, True, not zp, (torch.randn(n, 2048, device="cuda") * 0.02).half())

    def runs(steps, between=None):
        s = LinearStack(steps, between)
        s.buffers(1)
        return [len(r) for r in s._groups(1)]

    a, b, c = layer(64), layer(2048), layer(128)
    assert runs([(a, "x", "p"), (c, "x", "q")]) == [2]
    assert runs([(a, "x", "p"), (c, "x", "q")], {0: lambda bufs: None}) == [1, 1]   # a hook between them
    assert runs([(b, "x", "p"), (c, "p", "q")]) == [1, 1]                           # another input
    assert runs([(b, "x", "p"), (c, "x", "q"), (b, "x", "p")]) == [2, 1]            # one output twice
    assert runs([(c, "x", "p"), (b, "x", "x")]) == [1, 1]                           # the input overwritten
    assert runs([(a, "x", "p"), (layer(64, 128), "x", "q")]) == [1, 1]              # another block size
    assert runs([(a, "x", "p"), (layer(64, 64, False), "x", "q")]) == [1, 1]        # zero points, and none
    assert runs([(layer(64), "x", f"o{i}") for i in range(6)]) == [4, 2]
    hooked = layer(64)
    hooked.register_forward_hook(lambda *_: None)
    assert runs([(a, "x", "p"), (hooked, "x", "q")]) == [1, 1]
