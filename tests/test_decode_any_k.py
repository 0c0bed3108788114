"""The decode kernel where K is not whole groups of four steps for each of its eight warps."""
import re

import numpy as np
import pytest

from oracle import blkq4_oracle as O
from tests._util import bits, gaussian_act, gaussian_weight
from tests.test_gemm_gpu import gpu_gemm, kat_problem, only_kernel_node, to_cuda

pytestmark = pytest.mark.gpu


def check_bias(block, a, N, packed, plain):
    """A bias is added in fp16 to the rounded result, and changes nothing else."""
    torch = pytest.importorskip("torch")
    from gemmlib_b200 import capi

    bias = gaussian_act(1, N, seed=3).numpy().ravel()
    out = torch.full((a.shape[0], N), float("nan"), dtype=torch.float16, device="cuda")
    capi.gemm(block, True, a.shape[0], N, a.shape[1], to_cuda(a), *(to_cuda(x) for x in packed), out, bias=to_cuda(bias))
    torch.cuda.synchronize()
    assert (bits(out.cpu().numpy()) == bits(plain + bias)).all()


# one step; fewer groups than warps, the last one short or not; one group each and a short one; an uneven slice; N of one tile and many
@pytest.mark.parametrize("K", [64, 128, 192, 256, 320, 1024, 1856, 1984, 2112, 2176, 2240, 4160, 10944])
@pytest.mark.parametrize("block,has_zp", [(64, True), (64, False), (128, True), (128, False)])
def test_any_k(K, block, has_zp):
    """Within one fp16 rounding and the fp32 sums of K terms of the exact product, for every row count class; the early weight fetch
    and a bias change nothing else."""
    from gemmlib_b200 import capi

    if K % block:
        pytest.skip("not whole blocks")
    N = 32 if K > 2000 else 2528
    w = gaussian_weight(N, K, seed=1)
    packed = O.quant_prepack(block, True, w.numpy(), has_zp)
    ideal = O.dequant_ideal(block, True, K, N, *packed).T
    for M in (1, 2, 3, 8):
        a = gaussian_act(M, K, seed=M).numpy()
        want = a.astype(np.float64) @ ideal
        # the partial sums carry up to 1024 + 8 in place of a weight q - 8
        tol = 2.0 ** -11 * np.abs(want).max() + K ** 0.5 * 1032 * float(np.abs(a).max()) * 2.0 ** -24 * float(np.abs(packed[1]).max())
        got = gpu_gemm(block, True, a, N, *packed)
        assert np.abs(got - want).max() <= tol, M
        assert (bits(gpu_gemm(block, True, a, N, *packed, flags=capi.EARLY_WEIGHT_FETCH)) == bits(got)).all(), M
        check_bias(block, a, N, packed, got)


@pytest.mark.parametrize("block,N,K", [(64, 352, 576), (64, 96, 1088), (128, 160, 640)])
@pytest.mark.parametrize("has_zp", [True, False])
def test_known_answers(block, N, K, has_zp):
    for M in (1, 2, 5, 8):
        a, *packed = kat_problem(block, True, has_zp, M, N, K)
        assert (bits(gpu_gemm(block, True, a, N, *packed)) == bits(O.dequant_gemm(block, True, a, N, *packed))).all(), M


def launch_parameters(M, N, K):
    """Of a plain call, block 64, symmetric."""
    torch, driver = pytest.importorskip("torch"), pytest.importorskip("cuda.bindings.driver")
    from gemmlib_b200 import capi

    a, out = torch.zeros(M, K, dtype=torch.float16, device="cuda"), torch.empty(M, N, dtype=torch.float16, device="cuda")
    qw, qs = torch.zeros(K * N // 2, dtype=torch.uint8, device="cuda"), torch.zeros(K * N // 64, dtype=torch.float16, device="cuda")
    graph, stream = torch.cuda.CUDAGraph(keep_graph=True), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=stream):
        capi.gemm(64, True, M, N, K, a, qw, qs, None, out, stream=stream.cuda_stream)
    return only_kernel_node(driver, graph)


@pytest.mark.parametrize("K", [4096, 1024])
def test_few_instances_are_loaded_together(K):
    """The first launch of a process loads every kernel of the file that has the launched one: 92 in one file took 12.4 ms, 40 take 2.5."""
    driver = pytest.importorskip("cuda.bindings.driver")
    params = launch_parameters(1, 32, K)
    func = params.func
    if int(params.kern):
        err, func = driver.cuKernelGetFunction(params.kern)
        assert int(err) == 0
    err, module = driver.cuFuncGetModule(func)
    assert int(err) == 0
    err, count = driver.cuModuleGetFunctionCount(module)
    assert int(err) == 0 and count <= 48, count


@pytest.mark.parametrize("M,N,K,ring", [(1, 4096, 8192, 2), (1, 11008, 4096, 2), (2, 1024, 2048, 2), (1, 2048, 8192, 4), (1, 14336, 11008, 4),
                                        (2, 3584, 5120, 4), (1, 1024, 4160, 4), (4, 3584, 8192, 2), (1, 8192, 4160, 2)])
def test_rings(M, N, K, ring):
    """A CTA alone on its SM has four groups of steps in flight where a slice of K is longer than two."""
    slot = 2048 + 4 * 48  # a group's weights, scales and zero points
    smem = launch_parameters(M, N, K).sharedMemBytes
    steps, rows = K // 64, M + M % 2
    rest = steps * 64 + 2 * 8 * 16 * rows * 4 + 256 + M * (K + 8) * 2
    assert smem == 8 * ring * slot + rest, (smem - rest) / 8 / slot


@pytest.mark.parametrize("K,together", [(2048, True), (6144, True), (6400, False), (7168, False), (7232, True), (8256, False)])
def test_staging_of_two_rows(K, together):
    """Two rows are staged together where that is faster: up to three whole groups of steps a warp, and below 8192 k with short groups."""
    driver = pytest.importorskip("cuda.bindings.driver")
    params = launch_parameters(2, 32, K)
    err, name = driver.cuKernelGetName(params.kern) if int(params.kern) else driver.cuFuncGetName(params.func)
    # gemv_stream_kernel<zero points, groups per ring, rows staged at a time, ...>
    assert int(err) == 0 and re.search(rb"Li[24]ELi([28])E", name).group(1) == (b"8" if together else b"2"), name
