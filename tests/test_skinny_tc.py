"""Tensor-core kernel of up to 16 rows, column-wise blocks of 64 and 128: integers times activations, scaled in fp32 per block."""
import numpy as np
import pytest

from oracle import blkq4_oracle as O
from tests._util import bits, gaussian_act, gaussian_weight
from tests.test_decode_any_k import check_bias
from tests.test_gemm_gpu import gpu_gemm, kat_problem, only_kernel_node

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def check(block, has_zp, M, N, K):
    from gemmlib_b200 import capi

    w, a = gaussian_weight(N, K, seed=1), gaussian_act(M, K, seed=M).numpy()
    packed = O.quant_prepack(block, True, w.numpy(), has_zp)
    want = a.astype(np.float64) @ O.dequant_ideal(block, True, K, N, *packed).T
    # one fp16 rounding, and fp32 sums of K terms of up to 15 scales each
    tol = 2.0 ** -11 * np.abs(want).max() + K ** 0.5 * 15 * float(np.abs(a).max()) * 2.0 ** -23 * float(np.abs(packed[1]).max())
    got = gpu_gemm(block, True, a, N, *packed)
    assert np.abs(got - want).max() <= tol, (M, N, K)
    assert (bits(gpu_gemm(block, True, a, N, *packed, flags=capi.EARLY_WEIGHT_FETCH)) == bits(got)).all(), (M, N, K)
    check_bias(block, a, N, packed, got)


# K: half a step; one; an odd number of 64; parts of a cluster, even and not; N: part of a tile; several; more tiles than SMs (two rounds)
@pytest.mark.parametrize("N,K", [(32, 64), (160, 128), (96, 192), (544, 1088), (320, 2112), (2080, 4160), (128, 8256), (19200, 192), (28672, 1024)])
@pytest.mark.parametrize("block,has_zp", [(64, True), (64, False), (128, True), (128, False)])
def test_results(N, K, block, has_zp):
    if K % block:
        pytest.skip("not whole blocks")
    for M in (9, 13, 16):
        check(block, has_zp, M, N, K)


@pytest.mark.parametrize("M,N,K", [(3, 2048, 8256), (6, 4096, 8256), (8, 32, 11072), (8, 1024, 13056)])
def test_long_k_of_few_rows(M, N, K):
    """Few column tiles, and activations that do not fit the decode kernel's shared memory."""
    check(64, True, M, N, K)


@pytest.mark.parametrize("M,N,K", [(5, 96, 64), (3, 4768, 192), (8, 160, 320), (7, 18976, 448), (4, 4800, 512), (8, 4768, 1088),
                                   (6, 14336, 1984), (7, 544, 2112), (8, 14336, 2112), (5, 544, 4160), (3, 96, 6208)])
@pytest.mark.parametrize("has_zp", [True, False])
def test_few_rows(M, N, K, has_zp):
    check(64, has_zp, M, N, K)


@pytest.mark.parametrize("block,N,K", [(64, 352, 2048), (128, 160, 3072), (64, 96, 1088), (64, 2080, 576)])
@pytest.mark.parametrize("has_zp", [True, False])
def test_known_answers(block, N, K, has_zp):
    for M in (9, 12, 16):
        a, *packed = kat_problem(block, True, has_zp, M, N, K)
        assert (bits(gpu_gemm(block, True, a, N, *packed)) == bits(O.dequant_gemm(block, True, a, N, *packed))).all(), M


# few rows: on either side of the rules, K below 512 and not in whole groups
@pytest.mark.parametrize("M,N,K,kernel", [(1, 11008, 64, b"skinny_tc"), (2, 9472, 192, b"gemv_stream"), (1, 18976, 256, b"gemv_stream"), (2, 11008, 320, b"gemv_stream"),
                                          (3, 4768, 64, b"skinny_tc"), (8, 2048, 64, b"skinny_tc"), (4, 2048, 192, b"gemv_stream"),
                                          (5, 2048, 192, b"skinny_tc"), (3, 4768, 448, b"skinny_tc"), (6, 160, 256, b"gemv_stream"),
                                          (7, 160, 448, b"skinny_tc"), (3, 18976, 256, b"skinny_tc"), (5, 18976, 320, b"skinny_tc"),
                                          (4, 18976, 320, b"gemv_stream"), (3, 6144, 640, b"skinny_tc"), (8, 4096, 640, b"gemv_stream"),
                                          (5, 11008, 1024, b"skinny_tc"), (6, 8192, 1024, b"gemv_stream"), (7, 8192, 1024, b"skinny_tc"),
                                          (5, 11008, 1536, b"gemv_stream"), (8, 11008, 1536, b"gemv_stream"), (6, 14336, 1536, b"skinny_tc"), (8, 18976, 768, b"gemv_stream"),
                                          (7, 3072, 2112, b"skinny_tc"), (6, 3072, 2112, b"gemv_stream"), (8, 11008, 2112, b"gemv_stream"),
                                          (5, 2048, 5184, b"skinny_tc"), (5, 4096, 5184, b"gemv_stream"), (6, 4096, 5184, b"skinny_tc"),
                                          (3, 2048, 6208, b"skinny_tc"), (7, 8192, 6208, b"skinny_tc"), (8, 8192, 8192, b"gemv_stream"),
                                          (9, 4096, 4096, b"skinny_tc"), (8, 4096, 4096, b"gemv_stream"), (5, 2048, 11008, b"gemv_stream"),
                                          (5, 2048, 8256, b"skinny_tc"), (2, 2048, 8256, b"gemv_stream"), (6, 8192, 8256, b"gemv_stream")])
def test_which_kernel(M, N, K, kernel):
    driver = pytest.importorskip("cuda.bindings.driver")
    from gemmlib_b200 import capi

    a, out = torch.zeros(M, K, dtype=torch.float16, device="cuda"), torch.empty(M, N, dtype=torch.float16, device="cuda")
    qw = torch.zeros(K * N // 2, dtype=torch.uint8, device="cuda")
    qs = torch.zeros(K * N // 64 + 1, dtype=torch.float16, device="cuda")
    for scales, want in ((qs[:-1], kernel), (qs[1:], b"gemv_kernel")):  # scales that are not 16-byte aligned: the generic kernel
        graph, stream = torch.cuda.CUDAGraph(keep_graph=True), torch.cuda.Stream()
        with torch.cuda.graph(graph, stream=stream):
            capi.gemm(64, True, M, N, K, a, qw, scales, None, out, stream=stream.cuda_stream)
        params = only_kernel_node(driver, graph)
        err, name = driver.cuKernelGetName(params.kern) if int(params.kern) else driver.cuFuncGetName(params.func)
        assert int(err) == 0 and want in name, name


@pytest.mark.parametrize("block,N,K", [(64, 160, 512), (128, 96, 2176)])
def test_any_byte_as_zero_point(block, N, K):
    """The quantizer's zero points have four bits, but callers may bring their own: any byte, as up to eight rows."""
    w = gaussian_weight(N, K, seed=1)
    packed, scales, _ = O.quant_prepack(block, True, w.numpy(), True)
    zp = (np.arange(K // block * N) * 37 % 256).astype(np.uint8)
    ideal = O.dequant_ideal(block, True, K, N, packed, scales, zp).T
    for M in (1, 8, 9, 16):
        a = gaussian_act(M, K, seed=M).numpy()
        want = a.astype(np.float64) @ ideal
        # one fp16 rounding, and fp32 sums of K terms of up to 255 scales each (up to eight rows 1024 + 15)
        tol = 2.0 ** -11 * np.abs(want).max() + K ** 0.5 * 1039 * float(np.abs(a).max()) * 2.0 ** -23 * float(np.abs(scales).max())
        assert np.abs(gpu_gemm(block, True, a, N, packed, scales, zp) - want).max() <= tol, M
