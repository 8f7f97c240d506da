"""Rules that choose a kernel by the number of chunks, the evenness of the rows and the width: both sides of every line,
with a plan of rows of even length, a plan of rows longer than a chunk, and without a plan (needs a B200)."""
import numpy as np
import pytest

from helpers import check_against_f64, guarded_output, random_csr

pytestmark = pytest.mark.gpu

CHUNK = 32
SMS = 148     # the lines lie at multiples of the number of SMs


def _matrix(n_chunks, even, N=4000, seed=0):
    """CSR of about n_chunks chunks of 32 entries: rows of 4 to 28 entries and empty ones, or some of them far longer
    than a chunk (every chunk of those begins inside a row)."""
    rng = np.random.default_rng(seed + n_chunks)
    nnz = n_chunks * CHUNK - 5
    degrees = []
    if not even:
        degrees = [900] * max(1, nnz // 1800) + [0, 33, 64]
    left = nnz - sum(degrees)
    while left > 0:
        d = int(rng.integers(4, 29)) if rng.random() > 0.05 else 0
        d = min(d, left)
        degrees.append(d)
        left -= d
    order = rng.permutation(len(degrees))
    return random_csr(len(degrees), N, [degrees[i] for i in order], seed=seed)


def _operands(pkg, rp, K, N=4000):
    M = len(rp) - 1
    X = pkg.host_fill_uniform(M * K, 7, 1, -1.0, 1.0).reshape(M, K)
    Y = pkg.host_fill_uniform(N * K, 7, 2, -1.0, 1.0).reshape(N, K)
    return M, X, Y


@pytest.mark.parametrize("K", [32, 64, 128])
@pytest.mark.parametrize("even", [True, False])
@pytest.mark.parametrize("per_sm", [12, 20, 30, 48, 80])
def test_sddmm_of_fixed_widths_with_few_chunks(gpu_ctx, pkg, oracle, K, even, per_sm):
    ctx, N = gpu_ctx, 4000
    assert ctx.lib.hpspmm_ctx_sm_count(ctx.handle) == SMS
    opts = pkg.Opts(chunk_nnz=CHUNK)
    for n_chunks in (per_sm * SMS, per_sm * SMS + 1):
        rp, ci, _ = _matrix(n_chunks, even)
        M, X, Y = _operands(pkg, rp, K)
        nnz = len(ci)
        ref, abs_sum = oracle.sddmm_f64(rp, ci, X, Y)
        d_rp, d_ci, d_X, d_Y = (ctx.upload(x) for x in (rp, ci, X, Y))
        d_out = ctx.alloc((nnz,), np.float32)
        plan = ctx.plan_create(M, nnz, d_rp, K, opts, N=N, col_idx=d_ci)
        info = ctx.plan_info(plan)
        assert info["n_chunks"] == n_chunks and (info["n_split_chunks"] * 8 < n_chunks) == even
        for p in (plan, None):
            ctx.fill(d_out, nnz, 7.0)
            ctx.sddmm_csr(M, N, K, nnz, d_rp, d_ci, d_X, d_Y, d_out, plan=p, opts=opts)
            check_against_f64(d_out.to_host(), ref, abs_sum, "sddmm K=%d chunks=%d plan=%s" % (K, n_chunks, p is not None))
        ctx.plan_destroy(plan)
        for b in (d_rp, d_ci, d_X, d_Y, d_out):
            b.free()


@pytest.mark.parametrize("even", [True, False])
@pytest.mark.parametrize("K", [252, 256, 260, 288, 384, 388, 448, 512, 640])
def test_wide_products_in_one_pass_and_in_several(gpu_ctx, pkg, oracle, K, even):
    """Passes of 128 columns beyond 384 columns, and from 256 on where the rows are even: the last pass is as narrow as
    the width leaves it."""
    ctx, N = gpu_ctx, 4000
    opts = pkg.Opts(chunk_nnz=CHUNK)
    for per_sm in (48, 64):
        for n_chunks in (per_sm * SMS, per_sm * SMS + 1):
            rp, ci, v = _matrix(n_chunks, even)
            M, nnz = len(rp) - 1, len(ci)
            B = pkg.host_fill_uniform(N * K, 8, 1, -1.0, 1.0).reshape(N, K)
            ref, abs_sum = oracle.spmm_f64(rp, ci, v, B)
            d_rp, d_ci, d_v, d_B = (ctx.upload(x) for x in (rp, ci, v, B))
            buf, c_ptr, read = guarded_output(ctx, (M, K))
            plan = ctx.plan_create(M, nnz, d_rp, K, opts, N=N, col_idx=d_ci)
            assert ctx.plan_info(plan)["n_chunks"] == n_chunks
            for p in (plan, None):
                passes = (K > 384 and n_chunks > 48 * SMS) or (K >= 256 and even and p is not None and n_chunks > 64 * SMS)
                before = ctx.launch_count()
                ctx.spmm_csr(M, N, K, nnz, d_rp, d_ci, d_v, d_B, c_ptr, plan=p, opts=opts)
                launches = ctx.launch_count() - before - (0 if p is not None else 2 if n_chunks > 40 * SMS else 0)
                widest = 128 if passes else 512
                assert launches == (K >= widest) + (K % widest > 0)
                ctx.stream_sync()
                check_against_f64(read(), ref, abs_sum, "K=%d chunks=%d plan=%s" % (K, n_chunks, p is not None))
            ctx.plan_destroy(plan)
            for b in (d_rp, d_ci, d_v, d_B, buf):
                b.free()


@pytest.mark.parametrize("even", [True, False])
@pytest.mark.parametrize("K", [256, 260, 288, 292, 320, 448, 512, 516])
def test_wide_sddmm_in_one_pass_and_in_several(gpu_ctx, pkg, oracle, K, even):
    """Passes of 256 columns where they are ahead; the second adds to what the first has written."""
    ctx = gpu_ctx
    opts = pkg.Opts(chunk_nnz=CHUNK)
    l2 = ctx.lib.hpspmm_ctx_l2_bytes(ctx.handle)
    for per_sm, N in ((48, 4000), (80, 4000), (48, 140000)):
        for n_chunks in (per_sm * SMS, per_sm * SMS + 1):
            rp, ci, _ = _matrix(n_chunks, even, N=N)
            M, X, Y = _operands(pkg, rp, K, N)
            nnz = len(ci)
            ref, abs_sum = oracle.sddmm_f64(rp, ci, X, Y)
            d_rp, d_ci, d_X, d_Y = (ctx.upload(x) for x in (rp, ci, X, Y))
            d_out = ctx.alloc((nnz,), np.float32)
            plan = ctx.plan_create(M, nnz, d_rp, K, opts, N=N, col_idx=d_ci)
            for p in (plan, None):
                two = 256 < K <= 288 and n_chunks > 48 * SMS
                if 320 <= K <= 512 and even and p is not None:
                    two = n_chunks > 80 * SMS or (n_chunks > 48 * SMS and 4 * N * K > l2)
                before = ctx.launch_count()
                ctx.fill(d_out, nnz, 7.0)
                ctx.sddmm_csr(M, N, K, nnz, d_rp, d_ci, d_X, d_Y, d_out, plan=p, opts=opts)
                launches = ctx.launch_count() - before - 1 - (0 if p is not None else 2)
                assert launches == (2 if two else -(-K // 512))
                check_against_f64(d_out.to_host(), ref, abs_sum, "K=%d chunks=%d plan=%s" % (K, n_chunks, p is not None))
            ctx.plan_destroy(plan)
            for b in (d_rp, d_ci, d_X, d_Y, d_out):
                b.free()


@pytest.mark.parametrize("K", [68, 96, 100, 132, 164, 196])
def test_sddmm_on_both_sides_of_the_row_length_lines(gpu_ctx, pkg, oracle, K):
    """Average row lengths of just under and just over 4, 5 and 10 entries, with enough chunks for the shapes of many."""
    ctx, N = gpu_ctx, 3000
    opts = pkg.Opts(chunk_nnz=CHUNK)
    n_chunks = 80 * SMS + 40
    for length in (4, 5, 10):
        for rows_more in (0, 1):      # nnz = length * M, and one row too many for that
            M = n_chunks * CHUNK // length
            nnz = length * M
            rng = np.random.default_rng(length)
            degrees = np.full(M, length)
            move = rng.integers(0, length - 1, M // 2)
            degrees[:M // 2] -= move
            degrees[M - M // 2:] += move[::-1]
            degrees = np.concatenate([rng.permutation(degrees), np.zeros(rows_more, int)])
            M += rows_more
            rp = np.concatenate([[0], np.cumsum(degrees)]).astype(np.int32)
            first = rng.integers(0, N - 64, M)
            within = np.arange(nnz) - np.repeat(rp[:-1], degrees)
            ci = (np.repeat(first, degrees) + within * 3 % 64).astype(np.int32)
            assert (nnz >= length * M) == (rows_more == 0)
            M_, X, Y = _operands(pkg, rp, K, N)
            ref, abs_sum = oracle.sddmm_f64(rp, ci, X, Y)
            d_rp, d_ci, d_X, d_Y = (ctx.upload(x) for x in (rp, ci, X, Y))
            d_out = ctx.alloc((nnz,), np.float32)
            plan = ctx.plan_create(M, nnz, d_rp, K, opts, N=N, col_idx=d_ci)
            for p in (plan, None):
                ctx.fill(d_out, nnz, 7.0)
                ctx.sddmm_csr(M, N, K, nnz, d_rp, d_ci, d_X, d_Y, d_out, plan=p, opts=opts)
                check_against_f64(d_out.to_host(), ref, abs_sum, "K=%d rows of %d plan=%s" % (K, length, p is not None))
            ctx.plan_destroy(plan)
            for b in (d_rp, d_ci, d_X, d_Y, d_out):
                b.free()


def test_the_signature_names_the_shape_that_is_launched(gpu_ctx, pkg):
    ctx, N = gpu_ctx, 4000
    opts = pkg.Opts(chunk_nnz=CHUNK)

    def signature(n_chunks, K, even=True):
        rp, ci, _ = _matrix(n_chunks, even)
        d_rp, d_ci = ctx.upload(rp), ctx.upload(ci)
        plan = ctx.plan_create(len(rp) - 1, len(ci), d_rp, K, opts, N=N, col_idx=d_ci)
        try:
            return ctx.kernel_signature(plan, K)
        finally:
            ctx.plan_destroy(plan)
            d_rp.free()
            d_ci.free()

    for K, few, many, line in ((128, "<4,32,1>", "<4,32,1>", 16), (96, "<4,32,1>", "<4,8,3>", 24),
                               (160, "<4,32,2>", "<4,16,3>", 16), (32, "<4,8,1>", "<4,8,1>", 24)):
        assert few in signature(line * SMS, K) and "few=1" in signature(line * SMS, K)
        assert many in signature(line * SMS + 1, K) and "few=0" in signature(line * SMS + 1, K)
    assert "<4,32,3>" in signature(64 * SMS, 384) and "<4,32,3>" in signature(64 * SMS + 1, 384, even=False)
    assert "<4,32,1>" in signature(64 * SMS + 1, 384)
    # twice the gathers in flight from 16 to 24 and from 36 to 48 chunks per SM, over 97 to 128 and 193 to 256 columns
    for K in (100, 128, 196, 256):
        for line, below, above in ((16, "few=1 hint", "few=0 mid=1 hint"), (24, "few=0 mid=1 hint", "few=0 hint"),
                                   (36, "few=0 hint", "few=0 mid=1 hint"), (48, "few=0 mid=1 hint", "few=0 hint")):
            assert below in signature(line * SMS, K) and above in signature(line * SMS + 1, K)
    for K in (64, 96, 98, 132, 192, 260):
        assert "mid" not in signature(17 * SMS, K) and "mid" not in signature(48 * SMS, K)


def _layer_graph(nnz, even, M=None):
    """Square CSR on the GPU with rows of nearly the same length; its columns, the rows of the transpose, likewise, or half
    of the entries in columns of about 900."""
    import torch
    M = M or nnz // (16 if even else 8)
    rp = torch.arange(M + 1, device="cuda", dtype=torch.int64) * nnz // M
    ci = torch.randint(M, (nnz,), dtype=torch.int32, device="cuda")
    if not even:
        ci[::2] %= nnz // 1800
    return M, rp.int(), ci


def _one_pass(ctx, pkg, nnz, even, Ks, M=None):
    """For every width whether hpspmm_layer_backward takes the call, captured and not."""
    import torch
    M, rp, ci = _layer_graph(nnz, even, M)
    v, dA = torch.rand(nnz, device="cuda"), torch.empty(nnz, device="cuda")
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    taken = {}
    with torch.cuda.stream(side):
        s = side.cuda_stream
        layer = pkg.Layer(ctx, M, M, nnz, rp.data_ptr(), ci.data_ptr(), v.data_ptr(), max(Ks), s)
        for K in Ks:
            dC, H, dH = (torch.rand((M, K), device="cuda") for _ in range(3))
            layer.forward(K, H.data_ptr(), dH.data_ptr(), s)       # builds the plans of the class

            def call():
                st = ctx.lib.hpspmm_layer_backward(ctx.handle, layer.handle, K, v.data_ptr(), dC.data_ptr(), H.data_ptr(),
                                                   dH.data_ptr(), dA.data_ptr(), s)
                assert st in (0, pkg.ERR_UNSUPPORTED)
                return st == 0

            eager = call()
            torch.cuda.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=side):
                dA.zero_()
                captured = call()
            del graph
            taken[K] = (captured, eager)
        torch.cuda.synchronize()
        layer.close()
    return taken


@pytest.mark.parametrize("line,even,K", [(100, False, 16), (72, False, 20), (72, False, 30), (48, False, 32), (36, False, 48),
                                         (36, False, 126), (24, False, 128), (24, False, 256), (36, True, 68), (24, True, 100),
                                         (36, True, 132), (15, True, 256)])
def test_one_pass_gradients_of_few_entries(gpu_ctx, pkg, line, even, K):
    nnz = line * 128 * gpu_ctx.lib.hpspmm_ctx_sm_count(gpu_ctx.handle)
    small = nnz * K < (80_000_000 if even and K == 256 else 40_000_000)
    assert _one_pass(gpu_ctx, pkg, nnz, even, [K]) == {K: (False, small)}
    assert _one_pass(gpu_ctx, pkg, nnz + 1, even, [K]) == {K: (True, True)}


def test_one_pass_gradients_of_few_entries_at_other_widths(gpu_ctx, pkg):
    assert all(c and e for c, e in _one_pass(gpu_ctx, pkg, 20_000, False, [31, 47, 64, 127]).values())
    assert all(c and e for c, e in _one_pass(gpu_ctx, pkg, 20_000, True, [1, 16, 31, 62, 64, 126, 127]).values())
    assert all(e and not c for c, e in _one_pass(gpu_ctx, pkg, 20_000, False, [1, 16, 32, 48, 62, 96, 128, 254]).values())
    for nnz, eager in ((312_499, True), (312_501, False)):
        assert _one_pass(gpu_ctx, pkg, nnz, False, [128]) == {128: (False, eager)}
        assert _one_pass(gpu_ctx, pkg, nnz, True, [256], M=8000) == {256: (False, eager)}        # long rows
    nnz = 24 * 128 * gpu_ctx.lib.hpspmm_ctx_sm_count(gpu_ctx.handle)
    assert _one_pass(gpu_ctx, pkg, nnz, True, [256], M=8000) == {256: (False, False)}
    assert _one_pass(gpu_ctx, pkg, nnz + 1, True, [256], M=8000) == {256: (True, True)}


def test_one_pass_gradients_of_many_entries(gpu_ctx, pkg):
    l2 = gpu_ctx.lib.hpspmm_ctx_l2_bytes(gpu_ctx.handle)
    both, none = (True, True), (False, False)
    for even, part, M, inside, beyond in (
            (True, 5 / 16, l2 // 400, {32: both, 100: both}, {32: both, 100: both}),      # 16 entries per row
            (True, 5 / 16, l2 // 2000, {64: both, 68: both, 192: both}, {64: both, 68: none, 127: both, 192: none, 196: both}),
            (True, 3 / 8, l2 // 400, {8: both, 32: both}, {8: both, 32: none}),           # rows of dC: 0.08 and 0.32 of the cache
            (True, 3 / 8, l2 // 50, {8: both, 16: both}, {8: none, 16: both}),            # 0.64 and 1.28
            (True, 7 / 16, l2 // 400, {8: both}, {8: none}),
            (False, 1 / 2, l2 // 64, {32: both, 100: both}, {32: none, 100: both}),
            (False, 1 / 2, l2 // 400, {32: both}, {32: both}),
            (False, 5 / 8, l2 // 400, {32: both, 100: both}, {32: none, 100: none})):
        nnz = int(l2 * part) // 8
        assert _one_pass(gpu_ctx, pkg, nnz, even, list(inside), M) == inside
        assert _one_pass(gpu_ctx, pkg, nnz + 1, even, list(beyond), M) == beyond


@pytest.mark.parametrize("K", [1, 31, 32, 100, 256])
def test_planless_products_on_both_sides_of_the_search_line(gpu_ctx, pkg, oracle, K):
    """One launch that searches row_ptr for its chunks, or three that build records first: up to 40 chunks per SM of fewer
    than 128 entries or below 32 columns, else up to 32."""
    ctx, N = gpu_ctx, 2000
    sms = ctx.lib.hpspmm_ctx_sm_count(ctx.handle)
    for S, line in ((32, 40), (96, 40), (128, 32), (160, 32)):
        line = 40 if K < 32 else line
        for n_chunks in (17 * sms, line * sms, line * sms + 1):
            rng = np.random.default_rng(S)
            nnz = n_chunks * S - 5
            degrees = rng.choice([0, 3, 40, 31, S + 1, 5 * S], size=8 * nnz // S)
            rp = np.minimum(np.concatenate([[0], np.cumsum(degrees)]), nnz).astype(np.int32)
            rp[-1] = nnz
            ci = rng.integers(0, N, nnz).astype(np.int32)
            v = rng.uniform(-1, 1, nnz).astype(np.float32)
            M = len(rp) - 1
            B = pkg.host_fill_uniform(N * K, 9, 1, -1.0, 1.0).reshape(N, K)
            bufs = [ctx.upload(x) for x in (rp, ci, v, B)]
            buf, c_ptr, read = guarded_output(ctx, (M, K))
            before = ctx.launch_count()
            ctx.spmm_csr(M, N, K, nnz, *bufs, c_ptr, opts=pkg.Opts(chunk_nnz=S))
            assert ctx.launch_count() - before == (1 if n_chunks <= line * sms else 3), (S, n_chunks)
            ctx.stream_sync()
            ref, abs_sum = oracle.spmm_f64(rp, ci, v, B)
            check_against_f64(read(), ref, abs_sum, "K=%d S=%d chunks=%d" % (K, S, n_chunks))
            for b in bufs + [buf]:
                b.free()
