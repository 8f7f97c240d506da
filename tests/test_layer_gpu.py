"""The aggregation layer (forward SpMM, transposed SpMM, SDDMM behind one handle) against the CPU oracle,
through the C ABI and through the PyTorch autograd front-end (needs a B200)."""
import ctypes
import importlib

import numpy as np
import pytest

from helpers import check_against_f64, guarded_output

pytestmark = pytest.mark.gpu


def _rect_graph(pkg, M, N, seed):
    """Rectangular CSR with a few heavy rows, empty rows and unreferenced columns."""
    g = pkg.gen_uniform_degree(M, N, 0, 24, seed=seed, vals_kind=pkg.VALS_UPM1)
    return g


@pytest.mark.parametrize("K", [32, 64, 128, 20])
@pytest.mark.parametrize("kind", ["rmat", "rect"])
def test_layer_products_match_oracle(gpu_ctx, pkg, oracle, K, kind):
    ctx = gpu_ctx
    g = pkg.gen_rmat(12, 16, seed=11) if kind == "rmat" else _rect_graph(pkg, 3000, 1777, 12)
    M, N, nnz = g["M"], g["N"], g["nnz"]
    H = pkg.host_fill_uniform(N * K, 11, 1, -1.0, 1.0).reshape(N, K)
    dC = pkg.host_fill_uniform(M * K, 11, 2, -1.0, 1.0).reshape(M, K)
    d_rp, d_ci, d_v = ctx.upload(g["row_ptr"]), ctx.upload(g["col_idx"]), ctx.upload(g["vals"])
    d_H, d_dC = ctx.upload(H), ctx.upload(dC)
    d_C, d_dH, d_dA = ctx.alloc((M, K), np.float32), ctx.alloc((N, K), np.float32), ctx.alloc((nnz,), np.float32)
    layer = pkg.Layer(ctx, M, N, nnz, d_rp, d_ci, d_v, 128)
    info = layer.info()
    assert (info["M"], info["N"], info["nnz"], info["max_K"]) == (M, N, nnz, 128) and info["owned_bytes"] > 0

    # the transpose the layer owns is the oracle's, bit for bit
    rpt, cit, vt, perm = oracle.csr_transpose(M, N, g["row_ptr"], g["col_idx"], g["vals"])
    p_rpt, p_cit, p_vt, p_perm = layer.transposed()

    def read(ptr, count, dtype):
        out = np.empty(count, dtype=dtype)
        ctx.memcpy_d2h(out, ptr)
        ctx.stream_sync()
        return out

    assert np.array_equal(read(p_rpt, N + 1, np.int32), rpt)
    assert np.array_equal(read(p_cit, nnz, np.int32), cit)
    assert np.array_equal(read(p_vt, nnz, np.float32), vt)
    assert np.array_equal(read(p_perm, nnz, np.int32), perm)

    layer.forward(K, d_H, d_C)
    ref, abs_sum = oracle.spmm_f64(g["row_ptr"], g["col_idx"], g["vals"], H)
    check_against_f64(d_C.to_host(), ref, abs_sum, "layer forward")

    layer.backward_features(K, d_dC, d_dH)
    ref, abs_sum = oracle.spmm_f64(rpt, cit, vt, dC)
    check_against_f64(d_dH.to_host(), ref, abs_sum, "layer backward (features)")

    layer.backward_weights(K, d_dC, d_H, d_dA)
    ref, abs_sum = oracle.sddmm_f64(g["row_ptr"], g["col_idx"], dC, H)
    check_against_f64(d_dA.to_host(), ref, abs_sum, "layer backward (weights)")

    # new edge weights reach both A and its transpose
    v2 = pkg.host_fill_uniform(nnz, 11, 3, -2.0, 2.0)
    d_v2 = ctx.upload(v2)
    layer.update_values(d_v2)
    layer.forward(K, d_H, d_C)
    ref, abs_sum = oracle.spmm_f64(g["row_ptr"], g["col_idx"], v2, H)
    check_against_f64(d_C.to_host(), ref, abs_sum, "layer forward, new weights")
    layer.backward_features(K, d_dC, d_dH)
    ref, abs_sum = oracle.spmm_f64(rpt, cit, v2[perm], dC)
    check_against_f64(d_dH.to_host(), ref, abs_sum, "layer backward, new weights")

    layer.close()
    for b in (d_rp, d_ci, d_v, d_v2, d_H, d_dC, d_C, d_dH, d_dA):
        b.free()


def test_layer_argument_errors(gpu_ctx, pkg):
    ctx = gpu_ctx
    g = pkg.gen_uniform_degree(64, 64, 1, 4, seed=3)
    d_rp, d_ci, d_v = ctx.upload(g["row_ptr"]), ctx.upload(g["col_idx"]), ctx.upload(g["vals"])
    layer = pkg.Layer(ctx, 64, 64, g["nnz"], d_rp, d_ci, d_v, 32)
    d_H, d_C = ctx.alloc((64, 64), np.float32), ctx.alloc((64, 64), np.float32)
    with pytest.raises(pkg.HpspmmError) as ei:
        layer.forward(64, d_H, d_C)             # wider than max_K
    assert ei.value.status == pkg.ERR_INVALID
    with pytest.raises(pkg.HpspmmError):
        pkg.Layer(ctx, 64, 64, g["nnz"], None, d_ci, d_v, 32)
    lib = ctx.lib
    assert lib.hpspmm_layer_forward(ctx.handle, None, 32, ctypes.c_void_p(d_H.ptr), ctypes.c_void_p(d_C.ptr),
                                    None) == pkg.ERR_INVALID
    assert lib.hpspmm_layer_destroy(ctx.handle, None) == 0
    layer.close()
    for b in (d_rp, d_ci, d_v, d_H, d_C):
        b.free()


def test_empty_layer(gpu_ctx, pkg):
    ctx = gpu_ctx
    rp = np.zeros(9, dtype=np.int32)
    d_rp = ctx.upload(rp)
    layer = pkg.Layer(ctx, 8, 5, 0, d_rp, None, None, 32)
    d_H, d_C, d_dH = ctx.alloc((5, 32), np.float32), ctx.alloc((8, 32), np.float32), ctx.alloc((5, 32), np.float32)
    ctx.fill(d_C, 8 * 32, 7.0)
    ctx.fill(d_dH, 5 * 32, 7.0)
    layer.forward(32, d_H, d_C)
    layer.backward_features(32, d_C, d_dH)
    assert not d_C.to_host().any() and not d_dH.to_host().any()
    layer.close()
    for b in (d_rp, d_H, d_C, d_dH):
        b.free()


# every instance of the one-pass kernel: full and ragged widths of 16-, 8- and 4-byte vectors, and the first widths it refuses
@pytest.mark.parametrize("K", [4, 16, 28, 32, 52, 64, 96, 116, 128, 160, 196, 256, 2, 6, 14, 30, 46, 62, 94, 126, 190, 254,
                               1, 3, 7, 15, 23, 31, 47, 63, 95, 127, 129, 260])
def test_both_gradients_in_one_pass(gpu_ctx, pkg, oracle, K):
    """hpspmm_layer_backward against the oracle, rows split over several carry groups and empty rows among them."""
    ctx = gpu_ctx
    for g in (pkg.gen_rmat(10, 24, seed=41), _rect_graph(pkg, 700, 333, 42)):
        M, N, nnz = g["M"], g["N"], g["nnz"]
        H = pkg.host_fill_uniform(N * K, 41, 1, -1.0, 1.0).reshape(N, K)
        dC = pkg.host_fill_uniform(M * K, 41, 2, -1.0, 1.0).reshape(M, K)
        v2 = pkg.host_fill_uniform(nnz, 41, 3, -2.0, 2.0)
        bufs = [ctx.upload(a) for a in (g["row_ptr"], g["col_idx"], g["vals"], H, dC, v2)]
        d_rp, d_ci, d_v, d_H, d_dC, d_v2 = bufs
        layer = pkg.Layer(ctx, M, N, nnz, d_rp, d_ci, d_v, 260)
        out_H, p_H, read_H = guarded_output(ctx, (N, K))
        out_A, p_A, read_A = guarded_output(ctx, (nnz,))

        def call(width=K, a=p_A):
            return ctx.lib.hpspmm_layer_backward(ctx.handle, layer.handle, width, d_v2.ptr, d_dC.ptr, d_H.ptr, p_H, a, None)

        if K in (129, 260):
            assert call() == pkg.ERR_UNSUPPORTED
        else:
            for _ in range(2):                  # the counters of split rows are zero again afterwards
                assert call() == 0
                ctx.stream_sync()
                rpt, cit, vt, _ = oracle.csr_transpose(M, N, g["row_ptr"], g["col_idx"], v2)
                ref, abs_sum = oracle.spmm_f64(rpt, cit, vt, dC)
                check_against_f64(read_H(), ref, abs_sum, "dH")
                ref, abs_sum = oracle.sddmm_f64(g["row_ptr"], g["col_idx"], dC, H)
                check_against_f64(read_A(), ref, abs_sum, "dA")
            assert call(width=261) == pkg.ERR_INVALID and call(a=None) == pkg.ERR_INVALID
        layer.close()
        for b in bufs + [out_H, out_A]:
            b.free()


@pytest.mark.parametrize("K", [30, 62, 126, 128, 130, 254])
def test_both_gradients_of_rows_on_4_byte_boundaries(gpu_ctx, pkg, oracle, K):
    """Even widths whose operands allow only 4-byte vectors: up to 128 columns then."""
    ctx = gpu_ctx
    g = pkg.gen_rmat(10, 24, seed=44)
    M, N, nnz = g["M"], g["N"], g["nnz"]
    H = pkg.host_fill_uniform(N * K, 44, 1, -1.0, 1.0).reshape(N, K)
    dC = pkg.host_fill_uniform(M * K, 44, 2, -1.0, 1.0).reshape(M, K)
    shifted = [np.concatenate([np.zeros(1, np.float32), x.ravel()]) for x in (H, dC)]
    d_rp, d_ci, d_v, d_H, d_dC = bufs = [ctx.upload(a) for a in (g["row_ptr"], g["col_idx"], g["vals"], *shifted)]
    layer = pkg.Layer(ctx, M, N, nnz, d_rp, d_ci, d_v, 256)
    out_H, out_A = ctx.alloc((N * K + 1,), np.float32), ctx.alloc((nnz,), np.float32)
    rpt, cit, vt, _ = oracle.csr_transpose(M, N, g["row_ptr"], g["col_idx"], g["vals"])
    for off_C, off_H, off_dH in ((4, 4, 4), (4, 0, 0), (0, 4, 0), (0, 0, 4)):
        at = [d_dC.ptr + off_C, d_H.ptr + off_H, out_H.ptr + off_dH]
        st = ctx.lib.hpspmm_layer_backward(ctx.handle, layer.handle, K, d_v.ptr, *at, out_A.ptr, None)
        if K == 128:
            assert st == pkg.ERR_INVALID             # a multiple of 4 is refused unless the rows are 16-byte aligned
        elif K > 128:
            assert st == pkg.ERR_UNSUPPORTED
        else:
            assert st == 0
            ctx.stream_sync()
            dC_seen, H_seen = (x[1:] if o else x[:-1] for x, o in ((shifted[1], off_C), (shifted[0], off_H)))
            ref, abs_sum = oracle.spmm_f64(rpt, cit, vt, dC_seen.reshape(M, K))
            got = out_H.to_host()
            check_against_f64((got[1:] if off_dH else got[:-1]).reshape(N, K), ref, abs_sum, "dH")
            ref, abs_sum = oracle.sddmm_f64(g["row_ptr"], g["col_idx"], dC_seen.reshape(M, K), H_seen.reshape(N, K))
            check_against_f64(out_A.to_host(), ref, abs_sum, "dA")
    layer.close()
    for b in bufs + [out_H, out_A]:
        b.free()


def test_both_gradients_refused_before_anything_is_built(gpu_ctx, pkg):
    """Weights that fill the L2 cache: no plan can change the answer, so none is built for it."""
    import torch
    ctx = gpu_ctx
    M, per_row = 700_000, 16
    nnz = M * per_row
    assert 8 * nnz > ctx.lib.hpspmm_ctx_l2_bytes(ctx.handle) * 5 // 8
    rp = torch.arange(0, nnz + 1, per_row, dtype=torch.int32, device="cuda")
    ci = torch.randint(M, (nnz,), dtype=torch.int32, device="cuda")
    v, x = torch.rand(nnz, device="cuda"), torch.empty((M, 32), device="cuda")
    torch.cuda.synchronize()
    layer = pkg.Layer(ctx, M, M, nnz, rp.data_ptr(), ci.data_ptr(), v.data_ptr(), 64)
    owned = layer.info()["owned_bytes"]
    st = ctx.lib.hpspmm_layer_backward(ctx.handle, layer.handle, 32, v.data_ptr(), x.data_ptr(), x.data_ptr(), x.data_ptr(),
                                       v.data_ptr(), None)
    assert st == pkg.ERR_UNSUPPORTED and layer.info()["owned_bytes"] == owned
    layer.close()


def test_a_layer_is_refused_by_the_context_of_another_device(gpu_ctx, pkg):
    """Every product of the handle, also of a width whose plans are still to be built.  (One GPU is enough: the handle
    begins with its device's ordinal, which is set to another one here.)"""
    ctx, K = gpu_ctx, 32
    g = pkg.gen_rmat(8, 8, seed=43)
    M, N, nnz = g["M"], g["N"], g["nnz"]
    bufs = [ctx.upload(a) for a in (g["row_ptr"], g["col_idx"], g["vals"])]
    x, dA = ctx.alloc((M, 64), np.float32), ctx.alloc((nnz,), np.float32)
    layer = pkg.Layer(ctx, M, N, nnz, *bufs, 64)
    device = ctypes.c_int.from_address(layer.handle.value)
    assert device.value == 0
    lib, h = ctx.lib, ctx.handle
    device.value = 1
    try:
        for width in (64, K):
            assert lib.hpspmm_layer_backward(h, layer.handle, width, bufs[2].ptr, x.ptr, x.ptr, x.ptr, dA.ptr,
                                             None) == pkg.ERR_INVALID
            assert lib.hpspmm_layer_forward(h, layer.handle, width, x.ptr, x.ptr, None) == pkg.ERR_INVALID
            assert lib.hpspmm_layer_forward_values(h, layer.handle, width, bufs[2].ptr, x.ptr, x.ptr, None) == pkg.ERR_INVALID
            assert lib.hpspmm_layer_backward_features(h, layer.handle, width, x.ptr, x.ptr, None) == pkg.ERR_INVALID
            assert lib.hpspmm_layer_backward_weights(h, layer.handle, width, x.ptr, x.ptr, dA.ptr, None) == pkg.ERR_INVALID
    finally:
        device.value = 0
    layer.close()
    for b in bufs + [x, dA]:
        b.free()


@pytest.mark.parametrize("K", [64, 48])
def test_torch_autograd_front_end(pkg, oracle, K):
    torch = pytest.importorskip("torch")
    ops = importlib.import_module(pkg.__name__ + ".torch_ops")
    dev = torch.device("cuda", 0)
    g = pkg.gen_rmat(11, 16, seed=21)
    M, N, nnz = g["M"], g["N"], g["nnz"]
    H_h = pkg.host_fill_uniform(N * K, 21, 1, -1.0, 1.0).reshape(N, K)
    G_h = pkg.host_fill_uniform(M * K, 21, 2, -1.0, 1.0).reshape(M, K)
    rp, ci = torch.from_numpy(g["row_ptr"]).to(dev), torch.from_numpy(g["col_idx"]).to(dev)
    vals = torch.from_numpy(g["vals"]).to(dev).requires_grad_(True)
    H = torch.from_numpy(H_h).to(dev).requires_grad_(True)
    G = torch.from_numpy(G_h).to(dev)
    layer = ops.TorchLayer(rp, ci, vals, M, N, max_K=128)

    C = layer(H)
    ref, abs_sum = oracle.spmm_f64(g["row_ptr"], g["col_idx"], g["vals"], H_h)
    check_against_f64(C.detach().cpu().numpy(), ref, abs_sum, "torch forward")
    (C * G).sum().backward()
    rpt, cit, vt, perm = oracle.csr_transpose(M, N, g["row_ptr"], g["col_idx"], g["vals"])
    ref, abs_sum = oracle.spmm_f64(rpt, cit, vt, G_h)
    check_against_f64(H.grad.cpu().numpy(), ref, abs_sum, "torch dH")
    ref, abs_sum = oracle.sddmm_f64(g["row_ptr"], g["col_idx"], G_h, H_h)
    check_against_f64(vals.grad.cpu().numpy(), ref, abs_sum, "torch dvals")

    # an in-place step on the weights (what an optimiser does) reaches the next forward and backward
    with torch.no_grad():
        vals.mul_(-0.5)
    H.grad = None
    C2 = layer(H)
    v2 = (g["vals"] * np.float32(-0.5)).astype(np.float32)
    ref, abs_sum = oracle.spmm_f64(g["row_ptr"], g["col_idx"], v2, H_h)
    check_against_f64(C2.detach().cpu().numpy(), ref, abs_sum, "torch forward after step")
    (C2 * G).sum().backward()
    ref, abs_sum = oracle.spmm_f64(rpt, cit, v2[perm], G_h)
    check_against_f64(H.grad.cpu().numpy(), ref, abs_sum, "torch dH after step")

    # registration: schema and shape function agree with the real operator
    torch.library.opcheck(ops.layer_forward, (H.detach(), vals.detach(), layer.layer_id),
                          test_utils=("test_schema", "test_faketensor"))

    torch.library.opcheck(ops.layer_backward, (G, H.detach(), vals.detach(), layer.layer_id),
                          test_utils=("test_schema", "test_faketensor"))

    # no CPU path
    with pytest.raises(RuntimeError, match="CUDA"):
        layer(H.detach().cpu())
    layer.close()
    with pytest.raises(RuntimeError, match="unknown or closed"):
        layer(H)
