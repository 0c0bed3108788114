"""The decode kernel where K is not whole groups of four steps for each of its eight warps."""
import numpy as np
import pytest

from oracle import blkq4_oracle as O
from tests._util import bits, gaussian_act, gaussian_weight
from tests.test_gemm_gpu import gpu_gemm, kat_problem

pytestmark = pytest.mark.gpu


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


@pytest.mark.parametrize("block,N,K", [(64, 352, 576), (64, 96, 1088), (128, 160, 640)])
@pytest.mark.parametrize("has_zp", [True, False])
def test_known_answers(block, N, K, has_zp):
    for M in (1, 2, 5, 8):
        a, *packed = kat_problem(block, True, has_zp, M, N, K)
        assert (bits(gpu_gemm(block, True, a, N, *packed)) == bits(O.dequant_gemm(block, True, a, N, *packed))).all(), M
