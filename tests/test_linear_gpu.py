"""GPU tests of the PyTorch surface (ms_blkq4linear_ext + BlkQ4Linear), the mirror of
the reference's python/ms_blkq4linear.py and python/ms_blkq4linear_ext."""
import numpy as np
import pytest

from oracle import blkq4_oracle as O
from tests._util import bits, gaussian_act, gaussian_weight

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def test_ext_quant_matches_oracle_and_returns_empty_zp_when_scale_only():
    from gemmlib_b200 import ms_blkq4linear_ext as ext

    w = gaussian_weight(96, 128, seed=2)
    for has_zp in (True, False):
        qw, qs, qz = ext.quant(32, False, has_zp, w.cuda())
        pw, ps, pz = O.quant_prepack(32, False, w.numpy(), has_zp)
        assert qw.dtype == torch.uint8 and qs.dtype == torch.float16 and qz.dtype == torch.uint8
        assert (qw.cpu().numpy() == pw).all() and (bits(qs.cpu().numpy()) == bits(ps)).all()
        assert qz.numel() == (pz.size if has_zp else 0)
        if has_zp:
            assert (qz.cpu().numpy() == pz).all()


def test_reference_usage_script_flow():
    """The flow of the reference's python/blkq4linear_test.py: known-answer weights for a
    64 -> 32 layer, row-wise block 32 with offsets; the module must hold the prepacked
    originals.  (The reference script only prints q_weights; here they are compared.)"""
    from gemmlib_b200.ms_blkq4linear import BlkQ4Linear

    K, N, block, colwise = 64, 32, 32, False
    q, s, z = O.kat_generate(block, colwise, K, N, True)
    w = torch.from_numpy(O.dequant_plain(block, colwise, K, N, q, s, z)).cuda()
    m = BlkQ4Linear(block, colwise, False, w)
    assert (m.in_features, m.out_features, m.has_offsets) == (K, N, True)
    assert (m.q_weights.cpu().numpy() == O.prepack_weights(K, N, q)).all()
    ps, pz = O.prepack_meta(block, colwise, K, N, s, z)
    assert (bits(m.q_scales.cpu().numpy()) == bits(ps)).all() and (m.q_zp.cpu().numpy() == pz).all()
    a = O.kat_activations(8, K)
    want = O.dequant_gemm(block, colwise, a, N, m.q_weights.cpu().numpy(), ps, pz)
    got = m(torch.from_numpy(a).cuda()).cpu().numpy()
    assert (bits(got) == bits(want)).all()


@pytest.mark.parametrize("scale_only", [True, False])
@pytest.mark.parametrize("M", [1, 24])
def test_forward_with_bias_batch_dims_and_state_dict(scale_only, M):
    from gemmlib_b200.ms_blkq4linear import BlkQ4Linear

    K, N = 256, 160
    w = gaussian_weight(N, K, seed=4)
    bias = torch.linspace(-1, 1, N).to(torch.float16).cuda()
    m = BlkQ4Linear(64, True, scale_only, w.cuda(), bias)
    x = gaussian_act(2 * M, K, seed=5).view(2, M, K)
    y = m(x.cuda())
    assert y.shape == (2, M, N)
    pw, ps, pz = O.quant_prepack(64, True, w.numpy(), not scale_only)
    want = O.dequant_gemm(64, True, x.view(-1, K).numpy(), N, pw, ps, pz).astype(np.float32) + bias.cpu().numpy().astype(np.float32)
    assert np.abs(y.view(-1, N).cpu().numpy().astype(np.float32) - want).max() <= 1e-2
    # packed tensors are buffers: they survive a state_dict round trip into a fresh module
    sd = {k: v.clone() for k, v in m.state_dict().items()}
    assert set(sd) == {"q_weights", "q_scales", "q_zp"}
    m2 = BlkQ4Linear.from_packed(64, True, K, N, sd["q_weights"], sd["q_scales"], sd["q_zp"], bias)
    assert torch.equal(m2(x.cuda()), y)


def test_forward_rejects_bad_inputs():
    from gemmlib_b200.ms_blkq4linear import BlkQ4Linear

    m = BlkQ4Linear(32, True, True, gaussian_weight(64, 128).cuda())
    with pytest.raises(RuntimeError, match="float16"):
        m(torch.zeros(2, 128, device="cuda"))
    with pytest.raises(RuntimeError):
        m(torch.zeros(2, 64, dtype=torch.float16, device="cuda"))
    with pytest.raises(RuntimeError, match="CUDA"):
        m(torch.zeros(2, 128, dtype=torch.float16))
    with pytest.raises(RuntimeError, match="Cannot block quantize"):
        BlkQ4Linear(32, True, True, torch.zeros(48, 128, dtype=torch.float16, device="cuda"))


def test_forward_in_cuda_graph_on_side_stream():
    """Calls go to PyTorch's current stream, so a forward can be captured and replayed."""
    from gemmlib_b200.ms_blkq4linear import BlkQ4Linear

    m = BlkQ4Linear(64, True, True, gaussian_weight(352, 512, seed=9).cuda())
    for M in (1, 40):
        x = gaussian_act(M, 512, seed=M).cuda()
        eager = m(x)
        out = torch.zeros_like(eager)
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            m(x, out=out)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            m(x, out=out)
        out.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, eager)


def test_save_load_packed_round_trip(tmp_path):
    """serialization.save_packed / load_packed: the reloaded layer computes the same bits."""
    from gemmlib_b200 import serialization as S
    from gemmlib_b200.ms_blkq4linear import BlkQ4Linear

    K, N = 512, 384
    w = gaussian_weight(N, K, seed=21)
    bias = torch.linspace(-1, 1, N).to(torch.float16).cuda()
    layers = {"a": BlkQ4Linear(64, True, False, w.cuda(), bias), "b": BlkQ4Linear(32, False, True, w.cuda())}
    S.save_packed(tmp_path / "m.blkq4", layers)
    back = S.load_packed(tmp_path / "m.blkq4")
    x = gaussian_act(7, K, seed=22).cuda()
    for name in layers:
        assert torch.equal(layers[name](x).view(torch.int16), back[name](x).view(torch.int16))


def test_linear_stack_graph_replay_matches_eager():
    """stack.LinearStack: a chain of layers with real dependencies, replayed from one CUDA graph
    (skinny kernels launched with the early weight fetch), equals the eager layer-by-layer pass."""
    from gemmlib_b200.stack import llama_like_stack

    st = llama_like_stack(1024, 2560, 3, 64, True, True, "cuda", sigma=0.03, seed=5)
    assert st.num_linears == 21
    for M in (1, 4, 40):  # 40 rows: tensor-core kernel, split-K through the per-stream workspace
        x = gaussian_act(M, 1024, seed=30 + M).cuda()
        got = st.forward(x, "h0").clone()
        got2 = st.forward(x, "h0").clone()   # second replay: same workspace, same graph
        # eager reference pass with fresh buffers
        bufs = {"x": x}
        for lyr, src, dst in st.steps:
            bufs[dst] = lyr(bufs[src])
        torch.cuda.synchronize()
        assert torch.equal(got.view(torch.int16), got2.view(torch.int16))
        want = bufs["h0"]
        assert torch.allclose(got.float(), want.float(), rtol=0, atol=2.0 ** -7 * max(1.0, float(want.abs().max())))


@pytest.mark.parametrize("M", [1, 16, 24])
def test_forward_takes_every_input_form(M):
    """One native call does the flattening, the allocation and the view: strided and batched inputs,
    a caller's output, a bias that cannot be fused, and a packed tensor that is no longer a buffer."""
    from gemmlib_b200.ms_blkq4linear import BlkQ4Linear

    K, N = 256, 160
    w = gaussian_weight(N, K, seed=4).cuda()
    m = BlkQ4Linear(32, True, False, w)
    x = gaussian_act(M, K, seed=5).cuda()
    want = m(x)
    assert want.shape == (M, N) and not want.requires_grad
    strided = torch.empty(M, 2 * K, dtype=torch.float16, device="cuda")[:, ::2].copy_(x)
    with pytest.raises(RuntimeError, match="contiguous"):  # two dimensions: taken as they are
        m(strided)
    turned = torch.stack([x, x]).transpose(0, 1)  # [M, 2, K], strided: flattening copies
    assert torch.equal(m(turned), torch.stack([want, want]).transpose(0, 1))
    assert torch.equal(m(x.view(1, M, 1, K)), want.view(1, M, 1, N))
    if M == 1:
        assert torch.equal(m(x.view(K)), want.view(N))
    out = torch.zeros(M, 1, N, dtype=torch.float16, device="cuda")
    got = m(x.view(M, 1, K), out=out)
    assert got.data_ptr() == out.data_ptr() and torch.equal(out.view(M, N), want)
    wide = torch.linspace(-1, 1, N).cuda()  # float32: added outside the kernel
    m.bias = wide
    assert torch.equal(m(x), want.clone().add_(wide))
    m.bias = None
    q = m.q_weights
    del m.q_weights
    m.q_weights = torch.nn.Parameter(q, requires_grad=False)
    assert torch.equal(m(x), want)
    for bad in (x.float(), x[:, :-64], x[:0]):
        with pytest.raises(RuntimeError):
            m(bad)


def _balanced_layer():
    """224 output tiles on 148 SMs: every row count cuts balanced ranges through a workspace."""
    from gemmlib_b200.ms_blkq4linear import BlkQ4Linear

    g = torch.Generator(device="cuda").manual_seed(3)
    w = (torch.randn(28672, 1216, generator=g, device="cuda") * 0.02).half()
    return BlkQ4Linear(32, True, False, w)


def test_stack_graphs_own_their_workspaces():
    """A graph's workspace outlives the capture of a row count that needs a larger one, is no other graph's and not
    the eager calls', so a replay reads and writes only its own memory."""
    from gemmlib_b200 import ms_blkq4linear as L
    from gemmlib_b200.stack import LinearStack

    layer = _balanced_layer()
    st = LinearStack([(layer, "x", "y")])
    x = gaussian_act(16, 1216, seed=8).cuda()
    want = layer(x)  # the eager workspace
    first = st.forward(x, "y").clone()
    held = {M: [b for buffers in st._split_k[M].values() for b in buffers] for M in (16,)}
    ptrs = [b.data_ptr() for b in held[16]]
    for M in (8, 512):
        st.buffers(M)
        held[M] = [b for buffers in st._split_k[M].values() for b in buffers]
    assert all(len(b) == 1 for b in held.values()) and held[512][0].numel() > 16 << 20 > held[16][0].numel()
    assert [b.data_ptr() for buffers in st._split_k[16].values() for b in buffers] == ptrs
    spans = sorted((b.data_ptr(), b.data_ptr() + b.numel()) for b in
                   [b for buffers in held.values() for b in buffers] + list(L._WORKSPACES.values()))
    assert all(a[1] <= b[0] for a, b in zip(spans, spans[1:]))
    del held
    torch.cuda.empty_cache()
    others = [torch.full((n,), 0xFF, dtype=torch.uint8, device="cuda") for n in (1 << 20, 1213184, 16 << 20, 20 << 20)]
    st.buffers(16)["y"].fill_(float("nan"))
    assert torch.equal(st.forward(x, "y"), first) and torch.equal(first, want)
    assert all(bool((o == 0xFF).all()) for o in others)


def test_captured_call_takes_a_workspace_that_its_graph_owns():
    """torch.cuda.graph around a layer: every graph holds a workspace of its own, zeroed by a node of its own, until it
    is destroyed; the eager calls' buffer is not used."""
    import gc
    import time

    from gemmlib_b200 import ms_blkq4linear as L
    from gemmlib_b200 import ms_blkq4linear_ext as ext

    layer = _balanced_layer()
    eager = dict(L._WORKSPACES)
    for M in (16, 40):
        x = gaussian_act(M, 1216, seed=M).cuda()
        want, out = layer(x), [torch.empty(M, 28672, dtype=torch.float16, device="cuda") for _ in range(2)]
        before, eager, allocated = ext.graph_workspaces(), dict(L._WORKSPACES), torch.cuda.memory_allocated()
        graphs = []
        for o in out:
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g):
                layer(x, out=o)
                layer(x, out=o)  # the same buffer again
            graphs.append(g)
        assert ext.graph_workspaces() == before + 2
        assert {k: v.data_ptr() for k, v in L._WORKSPACES.items()} == {k: v.data_ptr() for k, v in eager.items()}
        for g, o in list(zip(graphs, out))[::-1]:  # the later graph first
            o.fill_(float("nan"))
            g.replay()
            assert torch.equal(o, want)
        torch.cuda.synchronize()
        del g, graphs
        gc.collect()
        deadline = time.time() + 10  # user objects may be released a little later
        def left():  # buffers still held, MB not given back (two buffers are 2.4 MB and more)
            return ext.graph_workspaces() - before, max(0, torch.cuda.memory_allocated() - allocated) >> 20

        while left() != (0, 0) and time.time() < deadline:
            time.sleep(0.05)
        assert left() == (0, 0)
    assert torch.equal(layer(x), want)


def test_bias_broadcasts_against_flattened_rows():
    """A bias that cannot be fused is added to the [rows, out_features] result, as in the reference's two-dimensional
    `output += bias`: its shape has nothing to do with the leading dimensions of the input."""
    from gemmlib_b200.ms_blkq4linear import BlkQ4Linear

    K, N = 256, 160
    m = BlkQ4Linear(64, True, False, gaussian_weight(N, K, seed=4).cuda())
    x = gaussian_act(6, K, seed=5).cuda()
    plain = m(x)
    g = torch.Generator().manual_seed(6)
    for shape in [(1, N), (6, N), (6, 1), (1,), (N,)]:
        m.bias = torch.randn(shape, generator=g).cuda()  # float32: not fused
        want = plain.clone().add_(m.bias)
        assert torch.equal(m(x), want)
        assert torch.equal(m(x.view(2, 3, K)), want.view(2, 3, N))
        out = torch.empty(3, 2, N, dtype=torch.float16, device="cuda")
        assert m(x.view(3, 2, K), out=out).data_ptr() == out.data_ptr() and torch.equal(out.view(6, N), want)
    m.bias = torch.randn((1, N), generator=g).cuda()
    assert torch.equal(m(x[0]), plain[:1].clone().add_(m.bias).view(N))
    m.bias = torch.randn((3, N), generator=g).cuda()
    with pytest.raises(RuntimeError):
        m(x.view(2, 3, K))  # three rows against six
