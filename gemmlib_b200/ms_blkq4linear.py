"""``BlkQ4Linear``: blockwise-int4 weight-only linear layer.

Mirror of the reference module python/ms_blkq4linear.py:10-28: same class name,
constructor arguments ``(block_size, col_wise, scale_only, weights,
bias_tensor=None)``, attributes and ``forward(input)``.  Quantization and prepack
happen in the constructor (on the device the weights live on); ``forward`` runs the
W4A16 GEMM/GEMV and adds the bias.

Additive differences: the packed tensors are registered as buffers, so they travel
with ``state_dict()`` / ``.to()``; the constructor's diagnostic prints are gone;
``from_packed`` rebuilds a layer from already-quantized tensors; inputs with leading
batch dimensions are flattened to 2-D and restored; ``forward(input, out=...)`` writes
into a caller's tensor; a float16 bias on the layer's device is added inside the kernel's
epilogue (bit-identical to the reference's separate ``output += bias``, one pass over the
output less); and, from the second call on, the skinny kernel is launched with
``BLKQ4_GEMM_EARLY_WEIGHT_FETCH`` (set ``early_weight_fetch = False`` on a layer whose
packed tensors are rewritten by work queued on the same stream as ``forward``); prefill
shapes with too few output tiles to fill the GPU split K through a workspace that eager calls share
per (device, stream) and that a CUDA graph owns (``split_k = False`` turns that off).
"""
from __future__ import annotations

import contextlib
import threading

import torch
from torch import nn

from . import ms_blkq4linear_ext

_EARLY = ms_blkq4linear_ext.EARLY_WEIGHT_FETCH
_linear = ms_blkq4linear_ext.linear
_linear_group = ms_blkq4linear_ext.linear_group
_group_supported = ms_blkq4linear_ext.linear_group_supported
_group_workspace_size = ms_blkq4linear_ext.linear_group_workspace_size
_group_keeps_bits = ms_blkq4linear_ext.linear_group_keeps_bits
_gemm_plan = ms_blkq4linear_ext.gemm_plan
_graph_workspace = ms_blkq4linear_ext.graph_workspace
_workspace_size = ms_blkq4linear_ext.gemm_workspace_size_blocked

# Split-K workspaces.  Eager calls: one zero-initialised buffer per (device, stream), shared by all layers (calls
# on one stream run one at a time; the kernel leaves the buffer's flags zeroed).  Grown on demand, the smaller
# buffer going back to the allocator, which orders its reuse behind the stream's work.
# A CUDA graph keeps the address it was captured with and replays on any stream, so it never sees these: its
# buffers belong to the graph (``graph_workspace``) or to whoever captures it (``workspaces_owned_by``).
_WORKSPACES = {}
_owner = threading.local()


@contextlib.contextmanager
def workspaces_owned_by(workspaces: dict):
    """Within the block this thread's calls take their split-K workspaces from ``workspaces``
    ((device, stream) -> buffers, the last one in use).  The caller keeps the dict as long as a graph captured
    in the block may replay; unlike a graph's own workspace these need no zeroing node."""
    before = getattr(_owner, "workspaces", None)
    _owner.workspaces = workspaces
    ms_blkq4linear_ext.workspace_owners(1)
    try:
        yield workspaces
    finally:
        ms_blkq4linear_ext.workspace_owners(-1)
        _owner.workspaces = before


def split_k_workspace(device, nbytes: int):
    if nbytes <= 0:
        return None
    index = device.index if device.index is not None else torch.cuda.current_device()
    key = (index, torch.cuda.current_stream(device).cuda_stream)
    owned = getattr(_owner, "workspaces", None)
    if owned is not None:
        buffers = owned.setdefault(key, [])  # a captured call keeps the buffer it got: none is dropped here
        if not buffers or buffers[-1].numel() < nbytes:
            buffers.append(torch.zeros(nbytes, dtype=torch.uint8, device=device))
        return buffers[-1]
    ws = _graph_workspace(*key, nbytes)
    if ws is not None:
        return ws
    ws = _WORKSPACES.get(key)
    if ws is None or ws.numel() < nbytes:
        ws = torch.zeros(max(nbytes, 16 << 20), dtype=torch.uint8, device=device)
        _WORKSPACES[key] = ws
    return ws


ms_blkq4linear_ext.workspace_source(_WORKSPACES, lambda index, nbytes: split_k_workspace(torch.device("cuda", index), nbytes))

MAX_GROUP = 4  # layers of one launch
_PAIR_KERNEL = 2  # of blkq4_gemm_plan


def can_share_launch(layers, rows) -> bool:
    """Whether one launch can compute all ``layers`` (two to four) from the same ``rows`` activation rows: layers of one
    shape of blocks, with nothing of the user's in their calls (hooks, another ``forward`` or ``__call__``, ``compile``)."""
    first = layers[0]
    for l in layers:
        if not isinstance(l, BlkQ4Linear):
            return False
        q = l.q_weights
        if (type(l).forward is not BlkQ4Linear.forward or "forward" in l.__dict__
                or type(l).__call__ is not nn.Module.__call__ or getattr(l, "_compiled_call_impl", None) is not None
                or l._forward_hooks or l._forward_pre_hooks or nn.modules.module._has_any_global_hook()
                or (l.block_size, l.col_wise, l.in_features) != (first.block_size, first.col_wise, first.in_features)
                or (l.q_zp.numel() > 0) != (first.q_zp.numel() > 0) or q.device != first.q_weights.device
                or (l.bias is not None and l._fusable_bias(q) is None)
                or l.q_scales.data_ptr() % 16 or l.q_zp.data_ptr() % 16):
            return False
    return _group_supported(first.block_size, first.col_wise, rows, first.in_features, [l.out_features for l in layers])


def group_workspace_bytes(layers, rows):
    """Split-K workspace with which one launch for layers that ``can_share_launch`` gives every bit of their ``forward`` calls;
    None where it would not.  Up to 16 rows, and where no layer splits K alone, it does without any.  Otherwise the layers' own
    fp32 sums are added in the order of their splits, and a launch over the tiles of all layers has to cut K in the same
    places."""
    if rows <= 16 or all(l.workspace_bytes(rows) == 0 for l in layers):
        return 0
    first = layers[0]
    shape = first.block_size, first.col_wise, rows, first.in_features, [l.out_features for l in layers]
    if all(l.split_k for l in layers) and _group_keeps_bits(*shape):
        return _group_workspace_size(*shape)
    return None


def one_launch_is_faster(layers, rows) -> bool:
    """Whether layers that can share a launch are at least as fast in one.  They are, by up to half, but where
    layers that fill the one-CTA kernel alone become tiles of the CTA-pair kernel of fewer than 256 rows: that kernel's
    step does not get shorter with its rows as the other's does.  Only fewer rounds make up for it.  Measured on B200, blocks
    of 64 with zero points, separate / together, us: two layers of 5632 columns (two rounds either way), K = 4096: M = 300
    40.9 / 44.6, M = 400 42.4 / 45.8, M = 512 49.8 / 48.4; K = 11008, M = 333 93.9 / 105.0; K = 2048, M = 333 27.2 / 27.7; K = 1024,
    M = 333 19.2 / 19.2; four of them (four rounds / three), K = 3072, M = 300 62.2 / 50.3; three of 9472 (pairs alone too),
    K = 4096, M = 300 74.4 / 64.2."""
    first = layers[0]
    k = first.in_features
    if not 256 < rows < 512 or k <= 1024:
        return True
    alone = [_gemm_plan(rows, l.out_features, k) for l in layers]
    kernel, tiles = _gemm_plan(rows, sum(-(-l.out_features // 256) * 256 for l in layers), k)  # whole pairs of tiles, as in a group
    if kernel != _PAIR_KERNEL or any(kern == _PAIR_KERNEL for kern, _ in alone):
        return True
    sms = torch.cuda.get_device_properties(first.q_weights.device).multi_processor_count
    return -(-tiles // (sms // 2)) < sum(-(-t // sms) for _, t in alone)


def shares_launch(layers, rows) -> bool:
    """Whether one launch for layers that ``can_share_launch`` keeps every bit of their calls and is not slower."""
    return group_workspace_bytes(layers, rows) is not None and one_launch_is_faster(layers, rows)


def run_as_one(layers, input, outputs):
    """One launch for layers that ``shares_launch``: ``outputs[i] = layers[i](input)``, bit for bit."""
    first = layers[0]
    ws = split_k_workspace(input.device, group_workspace_bytes(layers, input.size(0)))
    early = all(l._settled and l.early_weight_fetch for l in layers)
    _linear_group(first.block_size, first.col_wise, first.in_features, input, [l.q_weights for l in layers],
                  [l.q_scales for l in layers], [l.q_zp for l in layers], [l.bias for l in layers], list(outputs),
                  _EARLY if early else 0, ws)
    for l in layers:
        l._settled = True


class BlkQ4Linear(nn.Module):
    def __init__(self, block_size, col_wise, scale_only, weights, bias_tensor=None):
        super().__init__()
        self.block_size = int(block_size)
        self.col_wise = bool(col_wise)
        self.has_offsets = not scale_only
        self.in_features = weights.size(1)
        self.out_features = weights.size(0)
        q_weights, q_scales, q_zp = ms_blkq4linear_ext.quant(
            self.block_size, self.col_wise, self.has_offsets, weights
        )
        self.register_buffer("q_weights", q_weights)
        self.register_buffer("q_scales", q_scales)
        self.register_buffer("q_zp", q_zp)
        self.bias = bias_tensor
        self.early_weight_fetch = True
        self.split_k = True  # prefill shapes with few output tiles split K through a shared workspace
        # The first forward is a plain launch.  It may run on another stream than the quantizer: no launch starts before
        # the CTAs of a quantizer ahead of it in its own stream have left.
        self._settled = False

    @classmethod
    def from_packed(cls, block_size, col_wise, in_features, out_features, q_weights, q_scales, q_zp=None,
                    bias_tensor=None):
        """Build a layer from tensors produced earlier by ``quant`` (no requantization)."""
        self = cls.__new__(cls)
        nn.Module.__init__(self)
        self.block_size, self.col_wise = int(block_size), bool(col_wise)
        self.in_features, self.out_features = int(in_features), int(out_features)
        if q_zp is None:
            q_zp = torch.empty(0, dtype=torch.uint8, device=q_weights.device)
        self.has_offsets = q_zp.numel() > 0
        self.register_buffer("q_weights", q_weights)
        self.register_buffer("q_scales", q_scales)
        self.register_buffer("q_zp", q_zp)
        self.bias = bias_tensor
        self.early_weight_fetch = True
        self.split_k = True  # prefill shapes with few output tiles split K through a shared workspace
        self._settled = False
        return self

    def _load_from_state_dict(self, *args, **kwargs):
        self._settled = False  # the buffers are about to be overwritten by a copy on some stream
        return super()._load_from_state_dict(*args, **kwargs)

    def _fusable_bias(self, x):
        b = self.bias
        if (b is not None and b.dtype == torch.float16 and b.device == x.device and b.dim() == 1
                and b.numel() == self.out_features and b.is_contiguous()):
            return b
        return None

    def workspace_bytes(self, rows):
        """Split-K workspace that ``forward`` uses for ``rows`` activation rows (0: none)."""
        if not self.split_k:
            return 0
        return _workspace_size(self.block_size, self.col_wise, rows, self.out_features, self.in_features)

    def forward(self, input, out=None):
        # Few and plain lookups: at decode sizes the host's time per call is what a caller sees.
        bias = self.bias
        fused = None if bias is None else self._fusable_bias(input)
        settled = self._settled
        buf = self._buffers
        if "q_weights" in buf and "q_scales" in buf and "q_zp" in buf:
            w, s, z = buf["q_weights"], buf["q_scales"], buf["q_zp"]
        else:  # replaced on the module by something other than a buffer
            w, s, z = self.q_weights, self.q_scales, self.q_zp
        output = _linear(self.block_size, self.col_wise, self.in_features, self.out_features, input, w, s, z, fused,
                         _EARLY if settled and self.early_weight_fetch else 0, self.split_k, out)
        if not settled:
            self._settled = True
        if bias is not None and fused is None:
            rows = output.view(-1, self.out_features)
            rows += bias  # broadcast against [rows, out_features], whatever the input's leading dimensions
        return output

    def extra_repr(self):
        return (f"in_features={self.in_features}, out_features={self.out_features}, block_size={self.block_size}, "
                f"col_wise={self.col_wise}, has_offsets={self.has_offsets}, bias={self.bias is not None}")
