"""Where an eager BlkQ4Linear call takes its split-K workspace from: the device and stream's buffer, grown on demand, or the
owner's; and what the native call refuses."""
import os
import subprocess
import sys

import pytest
import torch

from gemmlib_b200 import ms_blkq4linear as L

pytestmark = pytest.mark.gpu


def test_eager_workspaces_grow_and_owned_ones_are_used():
    small = L.BlkQ4Linear(64, True, False, (torch.randn(1024, 1024, device="cuda") * 0.02).half())
    large = L.BlkQ4Linear(64, True, False, (torch.randn(11008, 1024, device="cuda") * 0.02).half())
    xs, xl = torch.randn(64, 1024, device="cuda").half(), torch.randn(512, 1024, device="cuda").half()
    stream = torch.cuda.Stream()
    key = (torch.cuda.current_device(), stream.cuda_stream)
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        want = small(xs), large(xl)
        assert 0 < small.workspace_bytes(64) < large.workspace_bytes(512) <= L._WORKSPACES[key].numel()
        buffer = L._WORKSPACES[key]
        again = small(xs), large(xl)
        assert L._WORKSPACES[key] is buffer
        L._WORKSPACES[key] = torch.zeros(256, dtype=torch.uint8, device="cuda")  # too small: replaced
        third = small(xs), large(xl)
        assert L._WORKSPACES[key].numel() >= large.workspace_bytes(512)
        buffer = L._WORKSPACES[key]
        owned = {}
        with L.workspaces_owned_by(owned):
            fourth = small(xs), large(xl)
        assert [len(v) for v in owned.values()] == [2] and list(owned) == [key] and L._WORKSPACES[key] is buffer
    torch.cuda.synchronize()
    for got in (again, third, fourth):
        for a, b in zip(want, got):
            assert torch.equal(a.view(torch.int16), b.view(torch.int16))


def test_what_the_native_call_refuses():
    layer = L.BlkQ4Linear(64, True, False, (torch.randn(128, 256, device="cuda") * 0.02).half())
    with pytest.raises(TypeError):
        layer(None)
    with pytest.raises(TypeError):
        L._linear(64, True, 256)
    with pytest.raises(TypeError):
        L._linear(64, True, "256", 128, *[torch.zeros(1, 256, dtype=torch.float16, device="cuda")] * 4, None, 0, True, None)
    for x in (torch.zeros(1, 256, device="cuda"), torch.zeros(1, 256, dtype=torch.float16), torch.zeros(1, 255, dtype=torch.float16, device="cuda")):
        with pytest.raises(RuntimeError):
            layer(x)
    with pytest.raises(RuntimeError):
        layer(torch.zeros(20, 256, dtype=torch.float16, device="cuda"), out=torch.zeros(20, 128, device="cuda"))
    x = torch.randn(3, 256, device="cuda").half()
    assert torch.equal(layer(x), layer(x, out=torch.empty(3, 128, dtype=torch.float16, device="cuda")))


def test_native_call_without_the_module():
    """The extension alone, in a process of its own: no source of workspaces, so a shape that would split K runs whole."""
    code = """
import torch
from gemmlib_b200 import ms_blkq4linear_ext as ext
q = ext.quant(64, True, True, (torch.randn(1024, 1024, device="cuda") * 0.02).half())
x = torch.randn(64, 1024, device="cuda").half()
assert ext.gemm_workspace_size_blocked(64, True, 64, 1024, 1024) > 0
got = ext.linear(64, True, 1024, 1024, x, *q, None, 0, True, None)
assert torch.equal(got.view(torch.int16), ext.forward(64, True, 1024, 1024, x, *q).view(torch.int16))
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


def test_native_call_with_the_callers_workspace():
    layer = L.BlkQ4Linear(64, True, False, (torch.randn(1024, 1024, device="cuda") * 0.02).half())
    x = torch.randn(64, 1024, device="cuda").half()
    ws = torch.zeros(layer.workspace_bytes(64), dtype=torch.uint8, device="cuda")
    got = L._linear(block_size=64, col_wise=True, in_features=1024, out_features=1024, input=x, q_weights=layer.q_weights,
                    q_scales=layer.q_scales, q_zp=layer.q_zp, bias=None, flags=0, workspace=ws, out=None)
    assert torch.equal(got.view(torch.int16), layer(x).view(torch.int16))
