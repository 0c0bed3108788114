"""Problems of fewer than 48 steps of 64 k: lower tiles and fewer parts of K than one tile per 256 rows gives."""
import pytest

from gemmlib_b200 import capi

BIG = 1 << 30
# M, N, K and what is launched with a workspace: rows of a tile, tiles, parts of K
PLANS = [(65, 1024, 1024, 48, 16, 1), (256, 1024, 1024, 64, 32, 1), (257, 512, 512, 64, 20, 1), (1000, 4096, 1024, 256, 128, 1),
         (430, 672, 1088, 48, 54, 2),    # fewer than eight column tiles keep their parts
         (92, 9344, 1408, 48, 146, 1),   # one part instead of two
         (64, 1024, 2048, 64, 8, 4),     # three parts and more stay up to 64 rows
         (100, 1920, 3008, 64, 30, 4),   # above, five or more become four
         (599, 6368, 896, 128, 250, 1),  # balanced ranges of pairs before
         (100, 1920, 3072, 112, 15, 6)]  # as high as possible again


@pytest.mark.parametrize("M,N,K,rows,tiles,parts", PLANS)
def test_plan(M, N, K, rows, tiles, parts):
    p = capi.gemm_plan(M, N, K, BIG)
    assert p["kernel"] == "one-cta" and not p["balanced"]
    assert (p["rows_per_tile"], p["tiles"], p["split"]) == (rows, tiles, parts), p
    assert capi.gemm_plan(M, N, K, 0)["split"] == 1  # the workspace is the opt-in to a split


@pytest.mark.gpu
@pytest.mark.parametrize("block,colwise,has_zp", [(64, True, True), (16, False, False)])
@pytest.mark.parametrize("M,N,K", [p[:3] for p in PLANS] + [(49, 1024, 512), (129, 1184, 1984), (333, 5632, 2048), (700, 672, 704)])
def test_results(M, N, K, block, colwise, has_zp):
    """Against the oracle; where K is not cut, the same bits with and without a workspace (every tile height sums in one order)."""
    import torch

    from oracle import blkq4_oracle as O
    from tests._util import bits, gaussian_act, gaussian_weight
    from tests.test_gemm_gpu import check_gaussian, gpu_gemm

    need = capi.gemm_workspace_size(M, N, K)
    ws = torch.zeros(max(need, 256), dtype=torch.uint8, device="cuda")
    if M * N * K < 1 << 30:
        check_gaussian(block, colwise, has_zp, M, N, K, workspace=ws)
    a, w = gaussian_act(M, K, seed=M).numpy(), gaussian_weight(N, K, seed=1)
    packed = O.quant_prepack(block, colwise, w.numpy(), has_zp)
    plain = gpu_gemm(block, colwise, a, N, *packed)
    rows = slice(0, None, 37)
    want = a[rows].astype("f8") @ O.dequant(block, colwise, K, N, *packed, kernel_formula=True).astype("f8").T
    # one fp16 rounding and fp32 sums of K terms in any order
    tol = (2.0 ** -11 + K * 2.0 ** -24) * abs(want).max() + 2.0 ** -11
    assert abs(plain[rows] - want).max() <= tol
    if capi.gemm_plan(M, N, K, need)["split"] == 1 and not capi.gemm_plan(M, N, K, need)["balanced"]:
        assert (bits(gpu_gemm(block, colwise, a, N, *packed, workspace=ws)) == bits(plain)).all()
    assert not ws[:256].any()
