"""Tiles of one height above 256 rows, and the exchange of a split tile in groups of four rows."""
import pytest

from gemmlib_b200 import capi

BIG = 1 << 30


def test_tiles_of_a_problem_have_one_height():
    for m, n, k, rows, kernel in ((256, 4096, 4096, 256, "one-cta"), (257, 1024, 4096, 144, "one-cta"), (333, 2080, 4032, 176, "one-cta"),
                                  (513, 512, 4096, 176, "one-cta"), (257, 28672, 4096, 160, "pair"), (512, 11008, 4096, 256, "pair"),
                                  (1100, 11008, 4096, 224, "pair"), (2049, 11008, 4096, 256, "pair")):
        p = capi.gemm_plan(m, n, k, BIG)
        assert (p["kernel"], p["rows_per_tile"]) == (kernel, rows), (m, n, k)
        column_tiles = -(-n // 128) if kernel == "one-cta" else -(-n // 256)
        assert p["tiles"] == -(-m // 256) * column_tiles


def test_workspace_sizes_do_not_follow_the_tile_height():
    """256 rows a partial tile, as when the tiles had that height."""
    assert capi.gemm_workspace_size(300, 1024, 4096) == 256 + 16 * 3 * 256 * 128 * 4  # the even four-way split of 16 tiles
    assert capi.gemm_workspace_size(300, 1024, 4096) == capi.gemm_workspace_size(512, 1024, 4096)
    assert capi.gemm_workspace_size(300, 11008, 4096) == 768 + 148 * 256 * 128 * 4    # balanced ranges


@pytest.mark.gpu
@pytest.mark.parametrize("case", [(32, True, True, 257, 160, 1024), (64, True, False, 273, 96, 2048), (16, False, True, 333, 2080, 1024),
                                  (32, False, False, 511, 672, 1024), (64, True, True, 513, 512, 4096),   # one CTA per tile, split
                                  (16, True, True, 257, 18944, 128), (32, False, True, 513, 9504, 192),  # pairs of CTAs
                                  (128, True, False, 289, 18976, 256),
                                  (64, True, True, 17, 96, 4096), (64, True, True, 66, 128, 4096), (32, True, True, 131, 128, 4096),
                                  (32, True, True, 13, 4096, 4096),
                                  (32, False, True, 64, 160, 2048), (16, True, False, 40, 96, 1984)],  # 16 steps a CTA: four groups
                         ids=lambda c: "-".join(map(str, c)))
def test_ragged_rows(case):
    """Against the oracle, with the split (workspace) and without; both runs of a split agree bit for bit."""
    import torch

    from tests.test_gemm_gpu import check_gaussian

    block, colwise, has_zp, M, N, K = case
    check_gaussian(block, colwise, has_zp, M, N, K)
    need = capi.gemm_workspace_size(M, N, K)
    if need:
        check_gaussian(block, colwise, has_zp, M, N, K, workspace=torch.zeros(need, dtype=torch.uint8, device="cuda"))
