"""Which groups of weight matrices one launch takes (host only)."""
import os
import subprocess
import sys

import pytest
import torch

from gemmlib_b200 import capi
from gemmlib_b200.ms_blkq4linear import BlkQ4Linear, can_share_launch


def test_supported_groups():
    assert capi.gemm_group_supported(64, True, 1, 4096, (4096, 4096, 4096))
    assert capi.gemm_group_supported(128, True, 8, 2048, (16, 28672))
    assert capi.gemm_group_supported(32, False, 17, 64, (32, 4096))   # the tensor-core kernels: any blocking
    assert capi.gemm_group_supported(16, True, 4096, 4096, (11008, 11008))
    for args in ((64, True, 9, 4096, (4096, 4096)),      # more rows than the decode kernel takes
                 (32, True, 1, 4096, (4096, 4096)),      # another kernel's blocking
                 (64, False, 1, 4096, (4096, 4096)),
                 (64, True, 1, 1984, (4096, 4096)),      # K too short, and not in groups of 256
                 (64, True, 1, 2112, (4096, 4096)),
                 (64, True, 1, 4096, (4096,)),
                 (64, True, 1, 4096, (16,) * 5),
                 (64, True, 1, 4096, (4096, 24)),
                 (64, True, 1, 4096, (4096, 0)),
                 (48, True, 1, 4096, (4096, 4096)),
                 (64, True, 0, 4096, (4096, 4096)),
                 (64, True, 64, 4064, (4096, 4096)),
                 (32, False, 64, 4096, (4096, 48))):
        assert not capi.gemm_group_supported(*args), args


@pytest.mark.parametrize("parts,message", [([], "2 to 4"), ([(64, (16, 1), (16, 1), None, (16, 1), None)] * 2, "Unexpected weight")])
def test_refused_groups(parts, message):
    with pytest.raises(capi.BlkQ4Error, match=message):
        capi.gemm_group(64, True, 1, 2048, (16, 4096), parts)


def test_workspace_of_a_group():
    """That of one matrix with the columns of all."""
    for m, k, widths in ((64, 8192, (14336, 14336)), (512, 4096, (4096, 4096, 4096)), (512, 4096, (11008, 11008)), (64, 4096, (1024, 1024))):
        assert capi.gemm_group_workspace_size(64, True, m, k, widths) == capi.gemm_workspace_size(m, sum(widths), k) > 0
    assert capi.gemm_group_workspace_size(64, True, 8, 4096, (4096, 4096)) == 0


def test_layers_with_calls_of_their_own_stay_apart():
    def layer(cls=BlkQ4Linear):
        n, k = 64, 2048
        return cls.from_packed(64, True, k, n, torch.zeros(n * k // 2, dtype=torch.uint8), torch.zeros(n * k // 64, dtype=torch.float16))

    class OwnCall(BlkQ4Linear):
        def __call__(self, *args, **kwargs):
            return super().__call__(*args, **kwargs)

    class OwnForward(BlkQ4Linear):
        def forward(self, input, out=None):
            return super().forward(input, out)

    class Plain(BlkQ4Linear):
        pass

    compiled, hooked, patched = layer(), layer(), layer()
    compiled.compile(backend="eager")
    hooked.register_forward_pre_hook(lambda *_: None)
    patched.forward = lambda x, out=None: x
    for other in (layer(), layer(Plain)):
        assert can_share_launch([layer(), other], 1)
    for other in (layer(OwnCall), layer(OwnForward), compiled, hooked, patched):
        assert not can_share_launch([layer(), other], 1) and not can_share_launch([other, layer()], 1)


@pytest.mark.parametrize("switch", ["BLKQ4_GEMV_NO_STREAM", "BLKQ4_GEMV_GENERIC"])
def test_no_decode_groups_where_the_decode_kernel_is_off(switch):
    """Its layers' own calls take another kernel there, with other bits."""
    code = ("from gemmlib_b200 import capi; w = (4096, 4096)\n"
            "print(*[int(capi.gemm_group_supported(64, True, m, 4096, w)) for m in (1, 8, 17, 512)])")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    for value, want in (("0", "1 1 1 1"), ("1", "0 0 1 1")):
        r = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True, timeout=300,
                           env={**os.environ, switch: value})
        assert r.returncode == 0 and r.stdout.split("\n")[0] == want, (r.stdout, r.stderr[-1000:])


def test_groups_that_keep_every_bit():
    """Those whose launch cuts K where the parts' own launches do (148 SMs without a device)."""
    for m, k, widths, keeps in ((8, 4096, (4096, 4096), True),           # the decode kernel
                                (512, 512, (4096, 4096, 4096), True),    # K too short to split
                                (40, 1024, (1024, 1024, 1024), True),    # two parts, one or three matrices
                                (40, 1024, (1024, 2816), True),          # of any widths
                                (64, 4096, (1024, 1024), True),          # eight parts of 16 tiles too
                                (64, 8192, (1024, 2048), True),          # eight parts each, six of 24 tiles
                                (512, 4096, (4096, 4096, 4096), False),  # two parts of 64 tiles, ranges of 96 pair tiles
                                (512, 4096, (11008, 11008), False),      # other ranges of 86 and of 172 pair tiles
                                (2048, 4096, (4096, 4096), True)):       # whole rounds of pair tiles
        plans = [capi.gemm_plan(m, n, k, 1 << 30) for n in widths + (sum(widths),)]
        same = m <= 16 or len({p["split"] for p in plans}) == 1 and not any(p["balanced"] for p in plans)
        assert capi.gemm_group_keeps_bits(64, True, m, k, widths) == same, (m, k, widths, plans)
    assert not capi.gemm_group_keeps_bits(64, True, 64, 4096, (4096,))
    assert not capi.gemm_group_keeps_bits(32, True, 1, 4096, (4096, 4096))
