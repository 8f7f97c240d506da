"""The PyTorch front-end of the layer beyond one forward and backward: second derivatives, tracing, subclasses, weights
of the wrong kind, several threads (needs a B200)."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class _Layer:
    def __init__(self, pkg, K=16, seed=31):
        import torch
        g = pkg.gen_rmat(9, 8, seed=seed)
        self.M, self.N, self.nnz, self.K = g["M"], g["N"], g["nnz"], K
        self.rp, self.ci, self.v = (torch.from_numpy(g[k]).cuda() for k in ("row_ptr", "col_idx", "vals"))
        self.ops = importlib.import_module(pkg.__name__ + ".torch_ops")
        self.layer = self.ops.TorchLayer(self.rp, self.ci, self.v, self.M, self.N, 64)
        self.H = torch.from_numpy(pkg.host_fill_uniform(self.N * K, seed, 1, -1.0, 1.0).reshape(self.N, K)).cuda()
        rows = torch.repeat_interleave(torch.arange(self.M, device="cuda"), (self.rp[1:] - self.rp[:-1]).long())
        self.index = torch.stack([rows, self.ci.long()])

    def dense(self, vals):
        import torch
        return torch.zeros((self.M, self.N), device="cuda", dtype=torch.float64).index_put(tuple(self.index), vals.double())

    def product(self, vals, H):
        return self.dense(vals) @ H.double()


def _close(got, want):
    # sums of up to a few hundred products in 32 bits: 1e-5 of the largest element leaves a factor of ten
    return bool((got.double() - want).abs().max() <= 1e-5 * want.abs().max())


@pytest.fixture
def work(pkg):
    pytest.importorskip("torch")
    w = _Layer(pkg)
    yield w
    w.layer.close()


def test_second_derivatives_are_refused(work):
    import torch
    H, W = work.H.clone().requires_grad_(), work.v.clone().requires_grad_()
    C = work.layer(H, W)
    dH, dW = torch.autograd.grad((C ** 2).sum(), (H, W), create_graph=True)
    assert _close(dH.detach(), 2 * work.dense(work.v).T @ work.product(work.v, work.H))
    for first in (dH, dW):
        with pytest.raises(RuntimeError, match="no derivative"):
            torch.autograd.grad((first ** 2).sum(), (H, W), retain_graph=True, allow_unused=True)
    # the operators by themselves
    dC = torch.ones((work.M, work.K), device="cuda", requires_grad=True)
    for op, other in ((work.ops.layer_backward_features, work.v), (work.ops.layer_backward_weights, work.H)):
        out = op(dC, other, work.layer.layer_id)
        assert out.requires_grad
        with pytest.raises(RuntimeError, match="no derivative"):
            out.sum().backward()
        with torch.no_grad():
            assert not op(dC, other, work.layer.layer_id).requires_grad
        assert not op(dC.detach(), other, work.layer.layer_id).requires_grad
