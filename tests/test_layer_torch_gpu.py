"""The PyTorch front-end of the layer beyond one forward and backward: second derivatives, tracing, subclasses, weights
of the wrong kind, several threads (needs a B200)."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class _Layer:
    def __init__(self, pkg, K=16, seed=31, max_K=64):
        import torch
        g = pkg.gen_rmat(9, 8, seed=seed)
        self.M, self.N, self.nnz, self.K = g["M"], g["N"], g["nnz"], K
        self.rp, self.ci, self.v = (torch.from_numpy(g[k]).cuda() for k in ("row_ptr", "col_idx", "vals"))
        self.ops = importlib.import_module(pkg.__name__ + ".torch_ops")
        self.layer = self.ops.TorchLayer(self.rp, self.ci, self.v, self.M, self.N, max_K)
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
    for out in work.ops.layer_backward(dC, work.H, work.v, work.layer.layer_id):
        assert out.requires_grad
        with pytest.raises(RuntimeError, match="no derivative"):
            out.sum().backward()


def test_weights_that_cannot_be_used_are_refused_every_time(work):
    import torch
    bad = [work.v.double(), work.v.cpu(), work.v[:-1].clone()]
    for vals in bad:
        for attempt in range(2):            # a refused tensor is not remembered as the one in use
            with pytest.raises(RuntimeError):
                work.layer(work.H, vals)
            with pytest.raises(RuntimeError):
                work.ops.layer_backward_features(torch.ones((work.M, work.K), device="cuda"), vals, work.layer.layer_id)
    assert _close(work.layer(work.H), work.product(work.v, work.H))
    two = torch.stack([work.v, work.v * 2], 1)
    assert _close(work.layer(work.H, two[:, 1]), work.product(work.v * 2, work.H))      # strided
    assert _close(work.layer(work.H, (work.v * 3)[None]), work.product(work.v * 3, work.H))


@pytest.mark.parametrize("K", [16, 129])
def test_threads_meet_on_one_layer(pkg, K):
    """Three threads on one stream, each with weights of its own that change in every step, beside the engine's; both
    gradients in one pass, and through the transpose's copy of the weights, which the threads overwrite for each other."""
    import threading

    import torch
    work = _Layer(pkg, K=K, max_K=K)
    want, errors = [work.product(work.v * (t + 1), work.H) for t in range(3)], []
    want_dH = [work.dense(work.v * (t + 1)).T @ torch.ones((work.M, work.K), device="cuda", dtype=torch.float64)
               for t in range(3)]
    torch.cuda.synchronize()

    def steps(t):
        try:
            for i in range(60):
                H = work.H.clone().requires_grad_()
                W = (work.v * (t + 1)).requires_grad_()
                C = work.layer(H, W)
                C.sum().backward()
                if i % 6 == 0:
                    assert _close(C.detach(), want[t]) and _close(H.grad, want_dH[t])
        except BaseException as e:      # noqa: B902 -- a thread's failure is the test's
            errors.append(e)

    threads = [threading.Thread(target=steps, args=(t,)) for t in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
    work.layer.close()


@pytest.mark.parametrize("K", [16, 129])
def test_feature_gradients_alone_follow_the_weights(pkg, K):
    """Only H asks for a gradient: the transpose's copy of the weights is filled again when they change in place, when others
    take their place, and not kept over a step with both gradients."""
    import torch
    w = _Layer(pkg, K=K, max_K=K)
    dC = torch.randn((w.M, K), device="cuda")
    W, other = w.v.clone(), w.v * 0.25

    def step(vals, learned=False):
        H = w.H.clone().requires_grad_()
        vals = vals.clone().requires_grad_() if learned else vals
        w.layer(H, vals).backward(dC)
        assert _close(H.grad, w.dense(vals.detach()).T @ dC.double())

    for turn in range(3):
        step(W)
        W.mul_(-2)
        step(W)
        step(other)
        step(W, learned=True)
        step(other)
        W[:: turn + 2] = 0.5
        step(W)
    w.layer.close()


def test_closing_under_calls(pkg):
    """close() waits for the call in flight; later calls find the layer closed."""
    import threading
    w = _Layer(pkg)
    ends = []

    def calls():
        try:
            for _ in range(2000):
                w.layer(w.H)
        except RuntimeError as e:
            ends.append(str(e))

    threads = [threading.Thread(target=calls) for _ in range(2)]
    for t in threads:
        t.start()
    w.layer.close()
    for t in threads:
        t.join()
    assert all("unknown or closed" in e for e in ends)
    with pytest.raises(RuntimeError, match="unknown or closed"):
        w.layer(w.H)


def test_tracers_modes_and_subclasses_see_the_operator(work):
    import torch
    from torch.overrides import TorchFunctionMode

    class Net(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.w = torch.nn.Parameter(work.v.clone())

        def forward(self, h):
            return work.layer(h * 2, self.w)

    traced = torch.fx.symbolic_trace(Net())
    assert any("layer_forward" in str(n.target) for n in traced.graph.nodes)
    assert _close(traced(work.H).detach(), 2 * work.product(work.v, work.H))

    seen = []

    class Mode(TorchFunctionMode):
        def __torch_function__(self, f, types, args=(), kwargs=None):
            seen.append(str(f))
            return f(*args, **(kwargs or {}))

    with Mode():
        work.layer(work.H)
    assert any("layer_forward" in s for s in seen)

    class Sub(torch.Tensor):
        pass

    assert type(work.layer(work.H.as_subclass(Sub))) is Sub
    assert type(work.layer(work.H, work.v.as_subclass(Sub))) is Sub
    assert type(work.layer(torch.nn.Parameter(work.H))) is torch.Tensor
    with pytest.raises(RuntimeError):
        work.layer(work.H.cpu().numpy())


# widths that one pass does not cover: rows of 4-byte vectors beyond 128 columns, and more than 256 columns
@pytest.mark.parametrize("K", [129, 260])
def test_both_gradients_where_one_pass_is_refused(pkg, K):
    """The product and the SDDMM instead, with the transpose's copy of the weights filled again after an in-place step;
    nothing is allocated but the two results."""
    import torch
    w = _Layer(pkg, K=K, max_K=K)
    dC = torch.randn((w.M, K), device="cuda")
    W = w.v.clone().requires_grad_()
    rows, cols = w.index
    for scale in (1.0, -0.5, 3.0):
        with torch.no_grad():
            W.mul_(scale)
        H = w.H.clone().requires_grad_()
        W.grad = None
        C = w.layer(H, W)
        C.backward(dC)
        assert _close(C.detach(), w.product(W.detach(), w.H))
        assert _close(H.grad, w.dense(W.detach()).T @ dC.double())
        assert _close(W.grad, (dC.double()[rows] * w.H.double()[cols]).sum(1))
    before = torch.cuda.memory_stats()["allocation.all.allocated"]
    out = w.ops.layer_backward(dC, w.H, W.detach(), w.layer.layer_id)
    assert torch.cuda.memory_stats()["allocation.all.allocated"] - before == 2
    assert _close(out[0], H.grad.double()) and _close(out[1], W.grad.double())
    w.layer.close()


def test_weights_of_the_transpose_around_a_capture(work):
    """Feature gradients alone, captured and eager in turn: a replay uses its weights as they are then, and an eager call
    never the weights that a recording or a replay has left or not yet left in the transpose."""
    import torch
    op, id_ = work.ops.layer_backward_features, work.layer.layer_id
    dC = torch.randn((work.M, work.K), device="cuda")

    def want(W):
        return work.dense(W).T @ dC.double()

    W, other, late = work.v.clone(), work.v * -3, work.v * 5
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        assert _close(op(dC, W, id_), want(W))
        torch.cuda.synchronize()
        graph, recorded_only = torch.cuda.CUDAGraph(), torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            out = op(dC, W, id_)
        graph.replay()
        assert _close(out, want(W))
        W.mul_(2)
        graph.replay()
        assert _close(out, want(W))
        for _ in range(2):
            assert _close(op(dC, other, id_), want(other))
            graph.replay()
            assert _close(out, want(W))
        with torch.cuda.graph(recorded_only, stream=side):
            op(dC, late, id_)
        assert _close(op(dC, late, id_), want(late))
        torch.cuda.synchronize()
        del graph, recorded_only, out
