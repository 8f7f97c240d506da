"""PyTorch front-end of the aggregation layer: autograd over the C ABI, no PyTorch arithmetic.

    layer = TorchLayer(row_ptr, col_idx, vals, M, N, max_K)   # CUDA tensors, int32 / int32 / float32
    C = layer(H)                                              # C = A·H, differentiable in H and in vals
    C.sum().backward()                                        # dH = Aᵀ·dC (SpMM), dvals = SDDMM(dC, H)

Four operators are registered under the namespace ``hpspmm`` (``layer_forward``,
``layer_backward_features``, ``layer_backward_weights``, and ``layer_backward`` for both gradients at
once) by csrc/torch_binding.cpp, with an autograd formula that chains them; the shape functions for tracing are below, so the layer can sit inside a
compiled or exported module.  Every operator calls ``hpspmm_layer_*`` of libhpspmm.so on the current
CUDA stream of the input's device; a CPU tensor is rejected (there is no fallback).  PyTorch supplies
memory, streams and the autograd tape only.

The reference has no framework binding; this is the caller either side of its products
(test/test_all.cpp:63-107 issues them one at a time from a C++ driver).
"""
import itertools
import os

import torch
from torch.overrides import has_torch_function_variadic

from . import PKG_DIR, Context, Layer, load_extension

_layers = {}      # what a layer id stands for: the shapes, and what has to stay alive
_ids = itertools.count(1)

_C = load_extension("_hpspmm_torch", os.path.join(PKG_DIR, "lib", "_hpspmm_torch.so"))

layer_forward = torch.ops.hpspmm.layer_forward.default
layer_backward_features = torch.ops.hpspmm.layer_backward_features.default
layer_backward_weights = torch.ops.hpspmm.layer_backward_weights.default
layer_backward = torch.ops.hpspmm.layer_backward.default


def _entry(layer_id):
    try:
        return _layers[layer_id]
    except KeyError:
        raise RuntimeError("hpspmm: unknown or closed layer id %d" % layer_id) from None


@torch.library.register_fake("hpspmm::layer_forward")
def _(H, vals, layer_id):
    return H.new_empty((_entry(layer_id)["M"], H.shape[1]))


@torch.library.register_fake("hpspmm::layer_backward_features")
def _(dC, vals, layer_id):
    return dC.new_empty((_entry(layer_id)["N"], dC.shape[1]))


@torch.library.register_fake("hpspmm::layer_backward_weights")
def _(dC, H, layer_id):
    return dC.new_empty((_entry(layer_id)["nnz"],))


@torch.library.register_fake("hpspmm::layer_backward")
def _(dC, H, vals, layer_id):
    e = _entry(layer_id)
    return dC.new_empty((e["N"], dC.shape[1])), dC.new_empty((e["nnz"],))


class TorchLayer:
    """A sparse operand A (CSR on one GPU) as a differentiable map H -> A·H."""

    def __init__(self, row_ptr, col_idx, vals, M, N, max_K):
        for t, dt, what in ((row_ptr, torch.int32, "row_ptr"), (col_idx, torch.int32, "col_idx"),
                            (vals, torch.float32, "vals")):
            if not t.is_cuda or t.dtype != dt or not t.is_contiguous():
                raise RuntimeError("hpspmm: %s must be a contiguous CUDA %s tensor" % (what, dt))
        if row_ptr.numel() != M + 1 or col_idx.numel() != vals.numel():
            raise RuntimeError("hpspmm: CSR arrays disagree with M or with each other")
        self.M, self.N, self.nnz, self.max_K = int(M), int(N), int(vals.numel()), int(max_K)
        self.row_ptr, self.col_idx, self.vals = row_ptr, col_idx, vals
        dev = row_ptr.device
        # One context per layer.  A context owns scratch and a flag that plan building uses (also lazily, on
        # the first product of a new width class), and calls that share a context must not overlap on the
        # GPU: with a context of their own, two layers driven from different streams or threads cannot meet
        # there.  Products of ONE layer still must not overlap with each other.
        ctx = Context(dev.index if dev.index is not None else torch.cuda.current_device())
        with torch.cuda.device(dev):
            v = vals.detach()
            layer = Layer(ctx, self.M, self.N, self.nnz, row_ptr.data_ptr(), col_idx.data_ptr(), v.data_ptr(),
                          self.max_K, torch.cuda.current_stream().cuda_stream)
        self.layer_id = next(_ids)
        _layers[self.layer_id] = {"layer": layer, "ctx": ctx, "M": self.M, "N": self.N, "nnz": self.nnz,
                                  "keep": (row_ptr, col_idx)}
        _C.register_layer(self.layer_id, ctx.handle.value, layer.handle.value, self.M, self.N, self.nnz, v)

    def __call__(self, H, vals=None):
        if vals is None:
            vals = self.vals
        # tracers, tensor subclasses and function modes see the call through __torch_function__
        if (torch.compiler.is_compiling() or not isinstance(H, torch.Tensor) or not isinstance(vals, torch.Tensor)
                or has_torch_function_variadic(H, vals)):
            return layer_forward(H, vals, self.layer_id)
        return _C.layer_forward(H, vals, self.layer_id)    # the same operator without the Python dispatcher's share

    def close(self):
        e = _layers.pop(self.layer_id, None)
        if e:
            _C.forget_layer(self.layer_id)
            e["layer"].close()
            e["ctx"].close()

    def __del__(self):
        try:
            self.close()
        except Exception:
            pass
