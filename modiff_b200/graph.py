"""CUDA-graph replay of the modulated UNet step.

From the third call after a `reset_cache()` every step launches the same kernels on the same
buffers (the first call is the unquantised step that creates the caches, the second is the
first quantised one and allocates the code buffers): that launch sequence - several hundred
small kernels - is captured once per input shape and replayed, which removes the per-launch
host cost.  In later passes the buffers are there from the start, so the second call launches
that sequence too and is replayed as well; the first call always runs eagerly, and a weight or
buffer that it finds changed bumps the generation and so ends the replays.  The reference has no counterpart (it runs eager PyTorch, with host synchronisations
in every quantiser call, qdiff/quant_layer.py:197-213).

The tensor returned by a replayed call is a static buffer that the next call overwrites.

A captured graph holds raw device addresses (each layer's caches, code planes, scale words and
packed weights).  Layers replace those buffers when they meet another input shape, when their
weights are repacked, or when a flag is set on a single layer; every such event bumps
`_lib.GENERATION`, and a graph captured under another generation is dropped and captured again
instead of being replayed.
"""
import torch

from . import _lib
from ._lib import ModiffError

EAGER_STEPS = 2


class GraphedModel:
    def __init__(self, qnn):
        self.qnn = qnn
        self._epoch = None
        self._config = None
        self._calls = 0
        self._graphs = {}       # (shape, context shape, device) -> dict(graph, x, t, c, out, kernels)

    def __call__(self, x, t=None, context=None):
        qnn = self.qnn
        config = getattr(qnn, "_config_epoch", 0)
        if config != self._config:          # flags changed: the captured launch lists are stale
            self._config = config
            self._graphs = {}
            self._calls = 0
        epoch = getattr(qnn, "_cache_epoch", 0)
        if epoch != self._epoch:
            self._epoch = epoch
            self._calls = 0
        self._calls += 1
        if self._calls == 1 or _lib.TIMER is not None:
            return qnn(x, t, context)
        _lib.require_cuda(x, "model input")
        key = (tuple(x.shape), None if context is None else tuple(context.shape), str(x.device))
        entry = self._graphs.get(key)
        if self._calls <= EAGER_STEPS and (entry is None or
                                           entry["generation"] != _lib.GENERATION[0]):
            return qnn(x, t, context)
        if entry is not None and entry["generation"] != _lib.GENERATION[0]:
            # some layer moved a buffer since the capture (another input shape in between, a
            # repacked weight, a flag set on one layer): the recorded addresses are stale
            del self._graphs[key]
            entry = None
        if entry is None:
            entry = self._capture(x, t, context)
            self._graphs[key] = entry
        entry["x"].copy_(x)
        entry["t"].copy_(t)
        if context is not None:
            entry["c"].copy_(context)
        entry["graph"].replay()
        _lib.LAUNCHES[0] += entry["kernels"]
        return entry["out"]

    def _capture(self, x, t, context=None):
        sx = x.clone()
        st = t.clone().float()
        sc = None if context is None else context.clone()
        graph = torch.cuda.CUDAGraph()
        before = _lib.LAUNCHES[0]
        torch.cuda.synchronize()
        try:
            with torch.cuda.graph(graph):
                out = self.qnn(sx, st, sc) if sc is not None else self.qnn(sx, st)
        except Exception as e:   # a capture that failed leaves no usable graph: report loudly
            raise ModiffError(f"CUDA graph capture of the UNet step failed: {e}") from e
        kernels = _lib.LAUNCHES[0] - before
        _lib.LAUNCHES[0] = before       # nothing ran during capture
        return dict(graph=graph, x=sx, t=st, c=sc, out=out, kernels=kernels,
                    generation=_lib.GENERATION[0])
