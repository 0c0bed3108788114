"""Infinite and NaN activations up to sixteen rows: a weight that is not zero times an infinite activation is infinite."""
import numpy as np
import pytest

from oracle import blkq4_oracle as O
from tests._util import bits, gaussian_act, gaussian_weight
from tests.test_gemm_gpu import gpu_gemm, to_cuda

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


# blocks of 32 and 16, whole groups of steps and not; blocks of 64 and 128 with K below 512, and not a multiple of 256; one tile and many
@pytest.mark.parametrize("block,N,K", [(32, 512, 2048), (32, 2528, 576), (16, 544, 512), (16, 512, 1984), (64, 32, 64), (64, 4768, 448),
                                       (128, 160, 384), (64, 96, 2112), (128, 352, 1152)])
@pytest.mark.parametrize("has_zp", [True, False])
def test_non_finite(block, N, K, has_zp):
    """Rows with one infinity (in the first, a middle and the last step), two of either sign, a NaN, infinities all over, and rows of
    finite values beside them, which keep every bit."""
    from gemmlib_b200 import capi

    w = gaussian_weight(N, K, seed=1)
    packed = O.quant_prepack(block, True, w.numpy(), has_zp)
    formula = O.dequant(block, True, K, N, *packed, kernel_formula=True).astype(np.float64)
    ideal = O.dequant_ideal(block, True, K, N, *packed)
    bias = gaussian_act(1, N, seed=9).numpy().ravel()
    for M in (1, 2, 4, 8, 9, 16):
        finite = gaussian_act(M, K, seed=M).numpy()
        a = finite.copy()
        spoilt = [(0, 0, np.inf), (1, K // 2 + 3, -np.inf), (2, K - 1, np.inf), (2, 17, -np.inf), (4, 40, np.nan), (5, K - 9, -np.inf),
                  (15, K - 60, np.inf)]
        for m, k, v in spoilt:
            if m < M:
                a[m, k] = v
        if M > 7:
            a[7] = np.where(np.arange(K) % 2 == 0, np.inf, -np.inf)
        got = gpu_gemm(block, True, a, N, *packed)
        own = gpu_gemm(block, True, finite, N, *packed)
        fused = torch.empty(M, N, dtype=torch.float16, device="cuda")
        capi.gemm(block, True, M, N, K, to_cuda(a), *(to_cuda(x) for x in packed), fused, bias=to_cuda(bias))
        with np.errstate(invalid="ignore"):
            assert (bits(fused.cpu().numpy())[~np.isnan(got)] == bits(got + bias)[~np.isnan(got)]).all(), M
            for m in range(M):
                ks = np.flatnonzero(~np.isfinite(a[m]))
                if len(ks) == 0:
                    assert (bits(got[m]) == bits(own[m])).all(), (M, m)
                    continue
                want = (a[m, ks].astype(np.float64) * formula[:, ks]).sum(1)
                sure = (ideal[:, ks] != 0).all(1)  # a weight q = zp is 0, or what two fp16 roundings leave of it
                assert (np.isnan(got[m]) == np.isnan(want))[sure].all(), (M, m)
                inf = sure & ~np.isnan(want)
                assert (got[m] == want)[inf].all() and inf.any() == (not np.isnan(want[sure]).all()), (M, m)
                assert not np.isfinite(got[m]).any(), (M, m)
