"""Decode kernel with zero points.  Where K is whole groups of steps for every warp, their terms have sums of their own for one and two
rows; from three rows on, and for other K, they are subtracted step by step."""
import numpy as np
import pytest

from oracle import blkq4_oracle as O
from tests._util import bits, gaussian_act, gaussian_weight
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


def integer_problem(M, N, K, block, seed=1):
    """Small integers as activations and weights close to their zero points: the sums of q and of the zero points are some hundred
    times their difference, so that an fp16 result shows in which order the fp32 sums were added."""
    rng = np.random.default_rng(seed)
    a = rng.integers(1, 9, (M, K))
    zp = rng.integers(1, 15, (K // block, N))
    q = np.repeat(zp, block, axis=0) + rng.integers(-1, 2, (K, N))
    scales = rng.uniform(0.001, 0.01, (K // block, N)).astype(np.float16)
    packed = np.zeros((N // 2, K), np.uint8)
    for k in range(K):
        r = k % 16
        for hi in (0, 1):  # columns n and n + 8 of a packed column's sixteen bytes
            cols = np.arange(N).reshape(-1, 16)[:, 8 * hi:8 * hi + 8].ravel()
            packed[:, k - r + r % 8 // 2 * 4 + r % 2 * 2 + hi] |= (q[k, cols] << (r // 8 * 4)).astype(np.uint8)
    return a, q, scales, zp, packed


def sums_of_their_own(a, q, scales, zp, block):
    """The kernel's fp32 sums: eight warps' slices of K in groups of four steps of 64; in a slice the scaled sums of q, step by step
    (block by block for blocks of 128), and the terms of the zero points of the first and the second half of each group; then the
    warps' sums and after them their zero-point terms.  Products and step sums are integers here, exact in fp32; fp64 holds an fp32
    product and its addend exactly, so that rounding its sum is an fma."""
    def fma(x, y, z):
        return (x.astype(np.float64) * y + z).astype(np.float32)

    M, K = a.shape
    groups, per = K // 256, block // 64
    sums, terms = [], []
    for w in range(8):
        total = np.zeros((M, q.shape[1]), np.float32)
        half = [np.zeros_like(total), np.zeros_like(total)]
        for j in range(groups * w // 8, groups * (w + 1) // 8):
            for u in range(0, 4, per):
                row = (4 * j + u) * 64 // block
                s, nsz = scales[row].astype(np.float32), -scales[row].astype(np.float32) * zp[row].astype(np.float32)
                k = slice((4 * j + u) * 64, (4 * j + u + per) * 64)
                total = fma(s[None, :], a[:, k] @ q[k], total)
                for v in range(u, u + per):
                    asum = a[:, (4 * j + v) * 64:(4 * j + v + 1) * 64].sum(1)
                    half[u // 2] = fma(nsz[None, :], asum[:, None], half[u // 2])
        sums.append(total)
        terms.append(half[0] + half[1])
    out = np.zeros_like(sums[0])
    for t in sums + terms:
        out = out + t
    return out.astype(np.float16)


@pytest.mark.parametrize("M,block,K", [(1, 64, 2048), (1, 64, 4096), (1, 64, 8448), (1, 128, 4096), (2, 64, 2304), (2, 128, 4096),
                                       (2, 64, 8192), (2, 128, 8448)])
def test_order_of_sums_of_one_and_two_rows(M, block, K):
    """Results of a layer do not change from one version to the next: every bit."""
    a, q, scales, zp, packed = integer_problem(M, 48, K, block)
    got = gpu_gemm(block, True, a.astype(np.float16), 48, packed.ravel(), scales.ravel(), zp.astype(np.uint8).ravel())
    assert (bits(got) == bits(sums_of_their_own(a, q, scales, zp, block))).all()


@pytest.mark.parametrize("block", [64, 128])
def test_two_rows_of_a_group(block):
    """Two matrices in one launch, the zero points' sums of the second row among them: every bit of their own calls."""
    import torch

    from gemmlib_b200 import capi
    from tests.test_gemm_gpu import to_cuda

    M, K = 2, 8192
    problems = [integer_problem(M, n, K, block, seed=n) for n in (32, 2416)]
    a = to_cuda(problems[0][0].astype(np.float16))
    q = [[to_cuda(p[4].ravel()), to_cuda(p[2].ravel()), to_cuda(p[3].astype(np.uint8).ravel())] for p in problems]
    out = [torch.full((M, n), float("nan"), dtype=torch.float16, device="cuda") for n in (32, 2416)]
    capi.gemm_group(block, True, M, K, a, [(n, *x, o, None) for n, x, o in zip((32, 2416), q, out)])
    torch.cuda.synchronize()
    for (_, w, scales, zp, packed), o in zip(problems, out):
        want = gpu_gemm(block, True, problems[0][0].astype(np.float16), w.shape[1], packed.ravel(), scales.ravel(),
                        zp.astype(np.uint8).ravel())
        assert (bits(o.cpu().numpy()) == bits(want)).all()
