"""Stack-level runner: a whole stack of quantized linears replayed as ONE CUDA graph.

Decode-time (M <= 16) layers take 3-25 us each on a B200, so launch gaps and per-call
allocations dominate a Python loop over ``BlkQ4Linear.forward`` (the reference module
allocates its output per call and launches on the legacy default stream,
python/ms_blkq4linear_ext/ms_blkq4linear.cpp:58,107).  ``LinearStack`` owns a
persistent workspace (one buffer per named activation), wires each layer to an input and
an output buffer, captures the whole pass once per row count M on its own stream, and
replays it.  Inside the graph the skinny kernels are launched with
``BLKQ4_GEMM_EARLY_WEIGHT_FETCH``: the weights of layer i+1 stream in while layer i
drains.  Consecutive layers that read the same buffer (q, k and v; gate and up) are one launch where a kernel
takes them together with every bit of their own calls' results.

It runs the linears only: what sits between them in a model (attention, activation
functions, norms) is the caller's and can be captured into the same graph by passing
``between`` hooks.
"""
from __future__ import annotations

from typing import Callable, Dict, List, Optional, Sequence, Tuple

import torch

from .ms_blkq4linear import MAX_GROUP, BlkQ4Linear, can_share_launch, group_workspace_bytes, run_as_one, shares_launch, workspaces_owned_by


class LinearStack:
    """``steps`` = [(layer, input buffer name, output buffer name), ...] executed in order.

    Buffer ``"x"`` is the stack's input ([M, in_features of the first reader]); every other
    name is created on first use as an output and can be read by later steps.
    """

    def __init__(self, steps: Sequence[Tuple[BlkQ4Linear, str, str]],
                 between: Optional[Dict[int, Callable[[Dict[str, torch.Tensor]], None]]] = None):
        self.steps = list(steps)
        self.between = dict(between or {})
        self._graphs: Dict[int, Tuple[torch.cuda.CUDAGraph, Dict[str, torch.Tensor]]] = {}
        self._split_k: Dict[int, dict] = {}  # row count -> split-K workspaces of its graph
        self.device = self.steps[0][0].q_weights.device
        self.stream = torch.cuda.Stream(self.device)
        written = {"x"}
        for lyr, src, dst in self.steps:
            if src not in written:
                raise ValueError(f"step reads buffer {src!r} before anything wrote it")
            written.add(dst)

    # ---- workspace ----
    def _workspace(self, M: int) -> Dict[str, torch.Tensor]:
        bufs: Dict[str, torch.Tensor] = {}
        for lyr, src, dst in self.steps:
            if src not in bufs:
                bufs[src] = torch.zeros(M, lyr.in_features, dtype=torch.float16, device=self.device)
            elif bufs[src].size(1) != lyr.in_features:
                raise ValueError(f"buffer {src!r} has width {bufs[src].size(1)}, layer wants {lyr.in_features}")
            if dst not in bufs:
                bufs[dst] = torch.zeros(M, lyr.out_features, dtype=torch.float16, device=self.device)
            elif bufs[dst].size(1) != lyr.out_features:
                raise ValueError(f"buffer {dst!r} has width {bufs[dst].size(1)}, layer writes {lyr.out_features}")
        return bufs

    def _groups(self, M: int) -> List[range]:
        """The steps in runs that one launch can take at this row count: up to four that follow one another, read the same
        buffer, write others, and have no hook between them."""
        runs: List[range] = []
        for i, (lyr, src, dst) in enumerate(self.steps):
            if runs and len(runs[-1]) < MAX_GROUP and (i - 1) not in self.between:
                run = runs[-1]
                members = [self.steps[j] for j in run] + [(lyr, src, dst)]
                outputs = [d for _, _, d in members]
                if (all(s == src for _, s, _ in members) and src not in outputs and len(set(outputs)) == len(outputs)
                        and can_share_launch([m for m, _, _ in members], M)):
                    runs[-1] = range(run.start, i + 1)
                    continue
            runs.append(range(i, i + 1))
        return runs

    def _launches(self, M: int) -> List[range]:
        """The steps of each launch: the runs that share one, every other step by itself."""
        launches: List[range] = []
        for run in self._groups(M):
            together = len(run) > 1 and shares_launch([self.steps[i][0] for i in run], M)
            launches += [run] if together else [range(i, i + 1) for i in run]
        return launches

    def _run_eager(self, bufs, launches):
        for run in launches:
            members = [self.steps[i] for i in run]
            if len(members) > 1:
                run_as_one([lyr for lyr, _, _ in members], bufs[members[0][1]], [bufs[dst] for _, _, dst in members])
            else:
                lyr, src, dst = members[0]
                lyr(bufs[src], out=bufs[dst])
            hook = self.between.get(run[-1])
            if hook is not None:
                hook(bufs)

    def _capture(self, M: int):
        bufs = self._workspace(M)
        launches = self._launches(M)
        # The layers' split-K workspace, like the buffers, from the caller's stream: its allocator pool has the blocks of
        # stacks that are gone, a new stream's is empty.  The largest at once, so that the layers do not outgrow it.
        need = max((group_workspace_bytes(layers, M) if len(layers) > 1 else layers[0].workspace_bytes(M)
                    for layers in ([self.steps[i][0] for i in run] for run in launches)
                    if isinstance(layers[0], BlkQ4Linear)), default=0)
        split_k = {}
        if need > 0:
            split_k[self.device.index, self.stream.cuda_stream] = [
                torch.zeros(need, dtype=torch.uint8, device=self.device)]
        self.stream.wait_stream(torch.cuda.current_stream(self.device))
        with workspaces_owned_by(split_k):
            with torch.cuda.stream(self.stream):
                for _ in range(2):  # the first pass settles every layer (plain launches), the second warms up
                    self._run_eager(bufs, launches)
            self.stream.synchronize()
            for buffers in split_k.values():
                del buffers[:-1]  # outgrown in the first pass
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=self.stream):
                self._run_eager(bufs, launches)
        self._split_k[M] = split_k
        self._graphs[M] = (graph, bufs)
        return self._graphs[M]

    # ---- public ----
    def buffers(self, M: int) -> Dict[str, torch.Tensor]:
        """The persistent workspace for row count M (captures the graph on first use)."""
        return (self._graphs.get(M) or self._capture(M))[1]

    def replay(self, M: int):
        """One pass over the stack on the current stream; reads ``buffers(M)["x"]``."""
        graph, _ = self._graphs.get(M) or self._capture(M)
        graph.replay()

    def forward(self, x: torch.Tensor, result: str) -> torch.Tensor:
        """Copy ``x`` into the input buffer, replay, return the buffer named ``result``."""
        M = x.size(0)
        _, bufs = self._graphs.get(M) or self._capture(M)
        bufs["x"].copy_(x)
        self.replay(M)
        return bufs[result]

    @property
    def num_linears(self) -> int:
        return len(self.steps)

    def weight_bytes(self) -> int:
        return sum(l.q_weights.numel() + 2 * l.q_scales.numel() + l.q_zp.numel() for l, _, _ in self.steps)


def llama_like_stack(hidden: int, ffn: int, blocks: int, block_size: int, col_wise: bool, scale_only: bool,
                     device, sigma: float = 0.02, seed: int = 0, weight_fn=None) -> LinearStack:
    """The seven linears of a Llama-style decoder block, ``blocks`` times, with random weights:
    q, k, v, o (hidden -> hidden), gate, up (hidden -> ffn), down (ffn -> hidden).  Shapes only:
    q/k/v/gate/up read the block input, o reads q's output and down reads gate's output, so every
    buffer a layer reads was produced inside the graph (true stream-order dependencies), and the
    block's output ("h") is o's and down's sum stand-in: down writes it."""
    steps: List[Tuple[BlkQ4Linear, str, str]] = []
    g = torch.Generator().manual_seed(seed)

    def make(n, k):
        w = weight_fn(n, k) if weight_fn else (torch.randn(n, k, generator=g) * sigma).to(torch.float16)
        return BlkQ4Linear(block_size, col_wise, scale_only, w.to(device))

    src = "x"
    for b in range(blocks):
        steps += [(make(hidden, hidden), src, "q"), (make(hidden, hidden), src, "k"), (make(hidden, hidden), src, "v"),
                  (make(hidden, hidden), "q", "o"), (make(ffn, hidden), "o", "gate"), (make(ffn, hidden), "o", "up"),
                  (make(hidden, ffn), "gate", f"h{b % 2}")]
        src = f"h{b % 2}"
    return LinearStack(steps)
