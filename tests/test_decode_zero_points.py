"""Decode kernel with zero points: up to two rows they have sums of their own, from three rows on they are subtracted step by step."""
import numpy as np
import pytest

from oracle import blkq4_oracle as O
from tests._util import gaussian_act, gaussian_weight
from tests.test_gemm_gpu import gpu_gemm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("block", [64, 128])
@pytest.mark.parametrize("M", [1, 2, 3, 4, 5, 7, 8])
def test_zero_points(M, block):
    """One group of steps per warp and uneven numbers of them, a few tiles and many: within one fp16 rounding and the fp32 sums of
    K terms of the exact product (on known answers: test_decode_kernel_exact_on_known_answers)."""
    for N, K in [(32, 2048), (2528, 2304)]:
        a, w = gaussian_act(M, K, seed=M).numpy(), gaussian_weight(N, K, seed=1)
        packed = O.quant_prepack(block, True, w.numpy(), True)
        want = a.astype(np.float64) @ O.dequant_ideal(block, True, K, N, *packed).T
        # the partial sums carry up to 1024 + 8 in place of a weight q - 8
        tol = 2.0 ** -11 * np.abs(want).max() + K ** 0.5 * 1032 * float(np.abs(a).max()) * 2.0 ** -24 * np.abs(packed[1].astype(np.float64)).max()
        assert np.abs(gpu_gemm(block, True, a, N, *packed) - want).max() <= tol, (N, K)
