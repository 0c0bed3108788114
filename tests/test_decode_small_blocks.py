"""Decode kernel on column-wise blocks of 32 and 16."""
import numpy as np
import pytest

from oracle import blkq4_oracle as O
from tests._util import bits, gaussian_act, gaussian_weight
from tests.test_decode_any_k import check_bias
from tests.test_gemm_gpu import gpu_gemm, kat_problem, only_kernel_node

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def launched_kernel(block, M, N, K, has_zp):
    driver = pytest.importorskip("cuda.bindings.driver")
    from gemmlib_b200 import capi

    a, out = torch.zeros(M, K, dtype=torch.float16, device="cuda"), torch.empty(M, N, dtype=torch.float16, device="cuda")
    qw = torch.zeros(K * N // 2, dtype=torch.uint8, device="cuda")
    qs = torch.zeros(K * N // block, dtype=torch.float16, device="cuda")
    qz = torch.zeros(K * N // block, dtype=torch.uint8, device="cuda") if has_zp else None
    graph, stream = torch.cuda.CUDAGraph(keep_graph=True), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=stream):
        capi.gemm(block, True, M, N, K, a, qw, qs, qz, out, stream=stream.cuda_stream)
    params = only_kernel_node(driver, graph)
    err, name = driver.cuKernelGetName(params.kern) if int(params.kern) else driver.cuFuncGetName(params.func)
    assert int(err) == 0
    return name


# fewer groups than warps, the last one short or not; one group each; an uneven slice
@pytest.mark.parametrize("N,K", [(512, 512), (2528, 576), (544, 1984), (2400, 2048), (1056, 2112), (512, 4160)])
@pytest.mark.parametrize("block,has_zp", [(32, True), (32, False), (16, True), (16, False)])
def test_results(N, K, block, has_zp):
    """Within one fp16 rounding and the fp32 sums of K terms of the exact product (the generic kernel: of that with weights of two fp16 roundings)."""
    from gemmlib_b200 import capi

    w = gaussian_weight(N, K, seed=1)
    packed = O.quant_prepack(block, True, w.numpy(), has_zp)
    ideal = O.dequant_ideal(block, True, K, N, *packed).T
    generic = O.dequant(block, True, K, N, *packed, kernel_formula=True).astype(np.float64).T
    for M in (1, 2, 3, 8):
        a = gaussian_act(M, K, seed=M).numpy()
        want = a.astype(np.float64) @ ideal
        # the partial sums carry up to 1024 + 8 in place of a weight q - 8
        tol = 2.0 ** -11 * np.abs(want).max() + K ** 0.5 * 1032 * float(np.abs(a).max()) * 2.0 ** -24 * float(np.abs(packed[1]).max())
        got = gpu_gemm(block, True, a, N, *packed)
        if b"gemv_kernel" in launched_kernel(block, M, N, K, has_zp):
            want = a.astype(np.float64) @ generic  # the generic kernel's two fp16 roundings of a weight
        assert np.abs(got - want).max() <= tol, M
        assert (bits(gpu_gemm(block, True, a, N, *packed, flags=capi.EARLY_WEIGHT_FETCH)) == bits(got)).all(), M
        check_bias(block, a, N, packed, got)


@pytest.mark.parametrize("block,N,K", [(32, 544, 576), (16, 512, 1088), (32, 544, 2112)])
@pytest.mark.parametrize("has_zp", [True, False])
def test_known_answers(block, N, K, has_zp):
    for M in (1, 2, 4):
        a, *packed = kat_problem(block, True, has_zp, M, N, K)
        assert (bits(gpu_gemm(block, True, a, N, *packed)) == bits(O.dequant_gemm(block, True, a, N, *packed))).all(), M


@pytest.mark.parametrize("block,M,N,K,has_zp,kernel", [(32, 8, 512, 512, True, b"gemv_stream"), (32, 8, 512, 2048, True, b"gemv_kernel"),
                                                       (32, 8, 512, 4096, False, b"gemv_stream"), (32, 4, 4096, 4096, True, b"gemv_stream"),
                                                       (16, 1, 4096, 4096, True, b"gemv_stream"), (16, 2, 4096, 4096, True, b"gemv_kernel"),
                                                       (16, 2, 4096, 4096, False, b"gemv_stream"), (16, 2, 14720, 576, True, b"gemv_kernel"),
                                                       (16, 4, 1024, 1984, False, b"gemv_stream"), (16, 8, 1024, 1984, False, b"gemv_kernel"),
                                                       (32, 1, 480, 512, True, b"gemv_kernel"), (32, 1, 512, 448, True, b"gemv_kernel"),
                                                       (32, 1, 11008, 4096, True, b"gemm_tc_kernel")])
def test_which_kernel(block, M, N, K, has_zp, kernel):
    assert kernel in launched_kernel(block, M, N, K, has_zp)
