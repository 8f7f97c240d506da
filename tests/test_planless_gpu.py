"""Products without a plan between other users of the context: the counters of split rows start at zero in every call
(needs a B200)."""
import numpy as np
import pytest

from helpers import check_against_f64, random_csr

pytestmark = pytest.mark.gpu


class _Work:
    """Operands of one plan-less product whose rows are longer than a chunk, with its reference."""

    def __init__(self, pkg, oracle, degrees, N, K, seed):
        import torch
        self.rp_h, self.ci_h, self.v_h = random_csr(len(degrees), N, degrees, seed=seed)
        self.M, self.N, self.K, self.nnz = len(degrees), N, K, len(self.ci_h)
        B = pkg.host_fill_uniform(N * K, seed, 1, -1.0, 1.0).reshape(N, K)
        self.ref, self.abs_sum = oracle.spmm_f64(self.rp_h, self.ci_h, self.v_h, B)
        self.rp, self.ci, self.v, self.B = (torch.from_numpy(x).cuda() for x in (self.rp_h, self.ci_h, self.v_h, B))
        self.C = torch.empty((self.M, K), device="cuda")

    def call(self, ctx, stream, opts=None):
        self.C.fill_(7.0)
        ctx.spmm_csr(self.M, self.N, self.K, self.nnz, self.rp.data_ptr(), self.ci.data_ptr(), self.v.data_ptr(),
                     self.B.data_ptr(), self.C.data_ptr(), opts=opts, stream=stream)

    def check(self, what):
        import torch
        torch.cuda.synchronize()
        check_against_f64(self.C.cpu().numpy(), self.ref, self.abs_sum, what)


def _dirty_scratch(ctx, w, stream):
    """A transpose keeps its own tables where plan-less products keep theirs."""
    import torch
    rpt = torch.empty(w.N + 1, dtype=torch.int32, device="cuda")
    cit, vt = torch.empty_like(w.ci), torch.empty_like(w.v)
    ctx.csr_transpose(w.M, w.N, w.nnz, w.rp.data_ptr(), w.ci.data_ptr(), w.v.data_ptr(), rpt.data_ptr(), cit.data_ptr(),
                      vt.data_ptr(), stream=stream)
    return rpt, cit, vt


DEGREES = [5000, 1, 700, 0, 33, 9000, 64, 65, 2, 3000] * 3


@pytest.mark.parametrize("chunk", [0, 32])
def test_eager_products_around_a_capture(pkg, oracle, chunk):
    """Eager products before the first replay, between replays of narrower and wider captured ones, and beside a
    captured SDDMM and transpose: a replay writes the scratch without the host knowing."""
    import torch
    opts = pkg.Opts(chunk_nnz=chunk)
    N = 20000
    small = _Work(pkg, oracle, DEGREES[:10], N, 32, 101)
    wide = _Work(pkg, oracle, DEGREES, N, 128, 102)
    with pkg.Context(0) as ctx:
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            s = side.cuda_stream
            out = torch.empty(wide.nnz, device="cuda")
            X = torch.rand((wide.M, 32), device="cuda")

            def sddmm():
                ctx.sddmm_csr(wide.M, N, 32, wide.nnz, wide.rp.data_ptr(), wide.ci.data_ptr(), X.data_ptr(),
                              wide.B.data_ptr(), out.data_ptr(), opts=opts, stream=s)

            keep = _dirty_scratch(ctx, wide, s)
            for w in (wide, small):                       # sizes the scratch for every call below
                w.call(ctx, s, opts)
                w.check("warm-up")
            sddmm()
            keep = _dirty_scratch(ctx, wide, s)           # the counters' old place now holds sort keys
            side.synchronize()
            g_small, g_sddmm, g_wide = (torch.cuda.CUDAGraph() for _ in range(3))
            with torch.cuda.graph(g_small, stream=side):
                small.call(ctx, s, opts)
            small.call(ctx, s, opts)                      # before the first replay: only recorded so far
            small.check("eager product after a capture")
            with torch.cuda.graph(g_sddmm, stream=side):
                sddmm()
            with torch.cuda.graph(g_wide, stream=side):
                wide.call(ctx, s, opts)
            for turn in range(3):
                wide.call(ctx, s, opts)
                wide.check("wide, eager, turn %d" % turn)
                g_small.replay()
                small.check("small, replayed, turn %d" % turn)
                wide.call(ctx, s, opts)
                wide.check("wide after a replay of small, turn %d" % turn)
                g_sddmm.replay()
                wide.call(ctx, s, opts)
                wide.check("wide after a replayed SDDMM, turn %d" % turn)
                small.call(ctx, s, opts)
                small.check("small, eager, turn %d" % turn)
                keep = _dirty_scratch(ctx, wide, s)
                g_wide.replay()
                wide.check("wide, replayed, turn %d" % turn)
                g_wide.replay()
                wide.check("wide, replayed twice, turn %d" % turn)
            del g_small, g_sddmm, g_wide, keep


def test_products_of_changing_sizes_without_a_plan(pkg, oracle):
    """One launch per product, then with the structure built first (many empty rows), in turn: each kind keeps its
    counters elsewhere, and the sets grow between calls."""
    import torch
    N = 20000
    works = [_Work(pkg, oracle, DEGREES[:10], N, 32, 103), _Work(pkg, oracle, DEGREES, N, 96, 104),
             _Work(pkg, oracle, ([0] * 30000 + [900]) * 3, N, 64, 105), _Work(pkg, oracle, DEGREES, N, 600, 106),
             _Work(pkg, oracle, [4000], N, 5, 107)]
    assert works[2].M > 8 * works[2].nnz                 # this one has its structure built
    with pkg.Context(0) as ctx:
        s = torch.cuda.current_stream().cuda_stream
        for turn in range(3):
            for i, w in enumerate(works):
                for rep in range(2):
                    w.call(ctx, s)
                    w.check("product %d, turn %d, call %d" % (i, turn, rep))


@pytest.mark.parametrize("chunk", [1 << 20, (1 << 31) - 64, (1 << 31) - 32])
def test_chunks_larger_than_any_matrix(pkg, oracle, chunk):
    """One chunk for the whole matrix, up to the largest size that can be asked for, with the structure built."""
    import torch
    opts = pkg.Opts(chunk_nnz=chunk)
    w = _Work(pkg, oracle, [40, 0, 1, 700, 33, 5000], 8000, 32, 110)
    sparse = _Work(pkg, oracle, ([0] * 30000 + [900]) * 3, 8000, 64, 111)
    with pkg.Context(0) as ctx:
        s = torch.cuda.current_stream().cuda_stream
        for x in (w, sparse):
            x.call(ctx, s, opts)
            x.check("without a plan, chunk %d" % chunk)
            plan = ctx.plan_create(x.M, x.nnz, x.rp.data_ptr(), x.K, opts, N=x.N, col_idx=x.ci.data_ptr(), stream=s)
            assert ctx.plan_info(plan)["n_chunks"] == 1
            x.C.fill_(7.0)
            ctx.spmm_csr(x.M, x.N, x.K, x.nnz, x.rp.data_ptr(), x.ci.data_ptr(), x.v.data_ptr(), x.B.data_ptr(),
                         x.C.data_ptr(), plan=plan, stream=s)
            x.check("with a plan, chunk %d" % chunk)
            X = torch.rand((x.M, x.K), device="cuda")
            out = torch.empty(x.nnz, device="cuda")
            rows = torch.repeat_interleave(torch.arange(x.M, device="cuda"), (x.rp[1:] - x.rp[:-1]).long())
            want = (X[rows].double() * x.B[x.ci.long()].double()).sum(1)
            for p in (plan, None):
                out.fill_(7.0)
                ctx.sddmm_csr(x.M, x.N, x.K, x.nnz, x.rp.data_ptr(), x.ci.data_ptr(), X.data_ptr(), x.B.data_ptr(),
                              out.data_ptr(), plan=p, opts=opts, stream=s)
                assert float((out.double() - want).abs().max()) <= 2e-5      # 64 terms of at most 1, in 32 bits
            ctx.plan_destroy(plan)


@pytest.mark.parametrize("mode", ["thread_local", "relaxed"])
def test_plans_come_and_go_beside_a_capture_in_another_thread(pkg, oracle, mode):
    """A plan destroyed and another built here while a thread records a graph of its own: neither disturbs the other."""
    import threading

    import torch
    w = _Work(pkg, oracle, [3000] * 40, 20000, 64, 112)     # the plan's block is well over 256 KB
    with pkg.Context(0) as ctx:
        s = torch.cuda.current_stream().cuda_stream

        def build():
            return ctx.plan_create(w.M, w.nnz, w.rp.data_ptr(), w.K, pkg.Opts(chunk_nnz=32), N=w.N,
                                   col_idx=w.ci.data_ptr(), stream=s)

        plan = build()
        x = torch.zeros(1000, device="cuda")
        torch.cuda.synchronize()
        begun, go_on, result = threading.Event(), threading.Event(), []

        def record():
            try:
                graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
                with torch.cuda.stream(side):
                    graph.capture_begin(capture_error_mode=mode)
                    x.add_(1)
                    begun.set()
                    go_on.wait(30)
                    x.add_(1)
                    graph.capture_end()
                graph.replay()
                torch.cuda.synchronize()
                result.append(float(x[0]))
            except BaseException as e:      # noqa: B902 -- a thread's failure is the test's
                result.append(e)
            finally:
                begun.set()

        t = threading.Thread(target=record)
        t.start()
        begun.wait(30)
        try:
            ctx.plan_destroy(plan)
            plan = build()
        finally:
            go_on.set()
            t.join()
        assert result == [2.0]
        w.C.fill_(7.0)
        ctx.spmm_csr(w.M, w.N, w.K, w.nnz, w.rp.data_ptr(), w.ci.data_ptr(), w.v.data_ptr(), w.B.data_ptr(),
                     w.C.data_ptr(), plan=plan, stream=s)
        w.check("product with the plan built meanwhile")
        ctx.plan_destroy(plan)


def test_only_the_first_product_of_a_width_allocates(pkg, oracle):
    """After a large product without a plan, smaller ones of up to its width find all they need."""
    import torch
    lib = pkg.load_library()
    N = 20000
    large = _Work(pkg, oracle, [300] * 3000, N, 96, 120)                        # has its structure built
    works = [_Work(pkg, oracle, DEGREES, N, K, 121) for K in (96, 64, 5)]      # one launch each
    with pkg.Context(0) as ctx:
        s = torch.cuda.current_stream().cuda_stream
        large.call(ctx, s)
        large.check("large")
        lib.hpspmm_debug_fail_device_alloc(1, 1000)
        try:
            for w in works + [large]:
                w.call(ctx, s)
                w.check("K=%d, no allocation possible" % w.K)
        finally:
            lib.hpspmm_debug_fail_device_alloc(0, 0)


@pytest.mark.parametrize("seed", [0, 1, 2])
def test_pieces_of_long_rows_come_last(gpu_ctx, pkg, oracle, seed):
    """The records of a call without a plan: rows that end on, just before and just after a cut, rows of one to many
    pieces side by side and across the builder's tiles of rows, the first and last row among them."""
    ctx, S, K, M, N = gpu_ctx, 32, 20, 9000, 600
    rng = np.random.default_rng(seed)
    n = rng.choice([0, 1, 3, 31, 32, 33, 64, 65, 96, 130, 500], size=M)
    n[[0, -1]] = [(700, 0), (0, 321), (64, 64)][seed]
    row_ptr = np.concatenate([[0], np.cumsum(n)]).astype(np.int32)
    nnz = int(row_ptr[-1])
    col_idx = rng.integers(0, N, size=nnz).astype(np.int32)
    vals = rng.uniform(-1, 1, size=nnz).astype(np.float32)
    B = rng.uniform(-1, 1, size=(N, K)).astype(np.float32)
    X = rng.uniform(-1, 1, size=(M, K)).astype(np.float32)
    bufs = [ctx.upload(a) for a in (row_ptr, col_idx, vals, B, X)]
    d_C, d_o = ctx.alloc((M, K), np.float32), ctx.alloc((nnz,), np.float32)
    opts = pkg.Opts(chunk_nnz=S)
    assert nnz > 40 * 160 * S           # more chunks than the warps of the GPU search for by themselves
    for _ in range(2):
        ctx.spmm_csr(M, N, K, nnz, bufs[0], bufs[1], bufs[2], bufs[3], d_C, opts=opts)
        ref, abs_sum = oracle.spmm_f64(row_ptr, col_idx, vals, B)
        check_against_f64(d_C.to_host(), ref, abs_sum, "product without a plan")
    ctx.sddmm_csr(M, N, K, nnz, bufs[0], bufs[1], bufs[4], bufs[3], d_o, opts=opts)
    ref, abs_sum = oracle.sddmm_f64(row_ptr, col_idx, X, B)
    check_against_f64(d_o.to_host(), ref, abs_sum, "SDDMM without a plan")
    for b in bufs + [d_C, d_o]:
        b.free()


class _ManyRows(_Work):
    """36 chunks per SM in three million rows: the records need 24 MB more than a search does."""

    def __init__(self, pkg, oracle, K):
        import torch
        rng = np.random.default_rng(130)
        self.M, self.N, self.K, self.nnz = 3_000_000, 20000, K, 36 * 148 * 128 - 9
        degrees = np.bincount(rng.integers(0, self.M, self.nnz - 30 * 2000), minlength=self.M)
        degrees[rng.integers(0, self.M, 30)] += 1
        degrees[np.arange(30) * 90_000 + 5] += (self.nnz - degrees.sum()) // 30
        degrees[-1] += self.nnz - degrees.sum()
        self.rp_h = np.concatenate([[0], np.cumsum(degrees)]).astype(np.int32)
        self.ci_h = rng.integers(0, self.N, self.nnz).astype(np.int32)
        self.v_h = rng.uniform(-1, 1, self.nnz).astype(np.float32)
        self.B_h = pkg.host_fill_uniform(self.N * K, 130, 1, -1.0, 1.0).reshape(self.N, K)
        self.ref, self.abs_sum = oracle.spmm_f64(self.rp_h, self.ci_h, self.v_h, self.B_h)
        self.rp, self.ci, self.v, self.B = (torch.from_numpy(x).cuda() for x in (self.rp_h, self.ci_h, self.v_h, self.B_h))
        self.C = torch.empty((self.M, K), device="cuda")


def test_no_room_for_the_records(pkg, oracle):
    """A product of 33 to 40 chunks per SM searches for them where the scratch has no room for records and cannot grow:
    under capture, with the device full, and in the host pipeline."""
    import torch
    lib = pkg.load_library()
    before = _Work(pkg, oracle, [300] * 300, 20000, 96, 131)       # sizes the scratch for a search
    w = _ManyRows(pkg, oracle, 32)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with pkg.Context(0) as ctx, torch.cuda.stream(side):
        s = side.cuda_stream
        before.call(ctx, s)
        before.check("warm-up")
        opts = pkg.Opts(chunk_nnz=128)
        before.call(ctx, s, pkg.Opts(chunk_nnz=32))
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            w.call(ctx, s, opts)
        for turn in range(2):
            graph.replay()
            w.check("replay %d" % turn)
        launches = ctx.launch_count()
        lib.hpspmm_debug_fail_device_alloc(1, 1000)
        try:
            w.call(ctx, s, opts)
            w.check("device full")
        finally:
            lib.hpspmm_debug_fail_device_alloc(0, 0)
        assert ctx.launch_count() - launches == 1
        del graph
        w.call(ctx, s, opts)
        w.check("room again")
        assert ctx.launch_count() - launches == 1 + 3
    with pkg.Context(0) as ctx:
        C = np.full((w.M, w.K), 7.0, np.float32)
        lib.hpspmm_debug_fail_device_alloc(2, 2)                    # the first one is for the operands
        try:
            ctx.spmm_csr_host_multi(w.M, w.N, w.nnz, w.rp_h, w.ci_h, w.v_h, [w.K], [w.B_h], [C], opts=opts)
        finally:
            lib.hpspmm_debug_fail_device_alloc(0, 0)
        check_against_f64(C, w.ref, w.abs_sum, "host pipeline")


@pytest.mark.parametrize("chunk,per_sm", [(32, 30), (32, 60), (128, 30), (128, 60)])
def test_operands_written_by_the_kernel_in_front(pkg, oracle, chunk, per_sm):
    """Two matrices in turn in the same buffers, row_ptr last, each product right behind the copy that brings it and never
    a synchronisation between: the first loads of a kernel wait for the kernel in front."""
    import torch
    rng = np.random.default_rng(chunk)
    nnz, K, N = per_sm * 148 * chunk - 3, 32, 3000
    M = nnz // 12
    works = []
    for i in range(2):
        rp = np.sort(rng.integers(0, nnz + 1, M - 1 - 40 * i))
        rp = np.concatenate([[0], np.zeros(40 * i, np.int64), rp, [nnz]]).astype(np.int32)
        ci, v = rng.integers(0, N, nnz).astype(np.int32), rng.uniform(-1, 1, nnz).astype(np.float32)
        B, X = (pkg.host_fill_uniform(n * K, 140 + i, j, -1.0, 1.0).reshape(n, K) for j, n in ((1, N), (2, M)))
        works.append((oracle.spmm_f64(rp, ci, v, B), oracle.sddmm_f64(rp, ci, X, B),
                      [torch.from_numpy(a).cuda() for a in (B, X, v, ci, rp)]))
    now = [torch.empty_like(t) for t in works[0][2]]
    B, X, v, ci, rp = (t.data_ptr() for t in now)
    opts = pkg.Opts(chunk_nnz=chunk)
    with pkg.Context(0) as ctx:
        s = torch.cuda.current_stream().cuda_stream
        got = []
        for turn in range(12):
            C, out = torch.full((M, K), 7.0, device="cuda"), torch.full((nnz,), 7.0, device="cuda")
            for dst, src in zip(now, works[turn % 2][2]):
                dst.copy_(src)
            ctx.spmm_csr(M, N, K, nnz, rp, ci, v, B, C.data_ptr(), opts=opts, stream=s)
            now[4].copy_(works[1 - turn % 2][2][4])
            now[4].copy_(works[turn % 2][2][4])
            ctx.sddmm_csr(M, N, K, nnz, rp, ci, X, B, out.data_ptr(), opts=opts, stream=s)
            got.append((C, out))
        torch.cuda.synchronize()
        for turn, (C, out) in enumerate(got):
            (ref_C, sum_C), (ref_out, sum_out), _ = works[turn % 2]
            check_against_f64(C.cpu().numpy(), ref_C, sum_C, "product, turn %d" % turn)
            check_against_f64(out.cpu().numpy(), ref_out, sum_out, "SDDMM, turn %d" % turn)


@pytest.mark.parametrize("captured", [True, False])
def test_products_behind_an_event_join(pkg, oracle, captured):
    """Products whose launch follows work of two streams: one kernel of their own stream and one, or a copy, of another, with
    nothing between the join and the launch; also as the first work of a stream that forks."""
    import torch
    N = 20000
    works = [_Work(pkg, oracle, DEGREES, N, K, 150) for K in (32, 100)]
    plans = []
    with pkg.Context(0) as ctx:
        main, other = torch.cuda.Stream(), torch.cuda.Stream()
        main.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(main):
            for w in works:
                plans.append(ctx.plan_create(w.M, w.nnz, w.rp.data_ptr(), w.K, N=N, col_idx=w.ci.data_ptr(),
                                             stream=main.cuda_stream))
                w.call(ctx, main.cuda_stream)          # sizes the scratch
            keep = [(w.rp.clone(), w.v.clone(), w.B.clone()) for w in works]
            pinned = [w.v.cpu().pin_memory() for w in works]
            big = torch.rand(1 << 25, device="cuda")
            main.synchronize()

            def joined(w, i, plan):
                """row_ptr and B arrive late on the other stream, the weights by a copy there; C is filled on this one."""
                fork = torch.cuda.Event()
                fork.record(main)
                other.wait_event(fork)
                with torch.cuda.stream(other):
                    for _ in range(4):
                        big.mul_(1.0)
                    w.rp.copy_(keep[i][0])
                    w.v.copy_(pinned[i], non_blocking=True)
                    w.B.copy_(keep[i][2])
                    done = torch.cuda.Event()
                    done.record(other)
                w.C.fill_(7.0)
                main.wait_event(done)
                ctx.spmm_csr(w.M, w.N, w.K, w.nnz, w.rp.data_ptr(), w.ci.data_ptr(), w.v.data_ptr(), w.B.data_ptr(),
                             w.C.data_ptr(), plan=plan, stream=main.cuda_stream)

            def steps():
                for i, w in enumerate(works):
                    joined(w, i, plans[i])
                    joined(w, i, None)
                # the first work of a stream that was forked, its predecessor a product
                fork = torch.cuda.Event()
                fork.record(main)
                other.wait_event(fork)
                with torch.cuda.stream(other):
                    ctx.spmm_csr(w.M, w.N, w.K, w.nnz, w.rp.data_ptr(), w.ci.data_ptr(), w.v.data_ptr(), w.B.data_ptr(),
                                 w.C.data_ptr(), plan=plans[1], stream=other.cuda_stream)
                    done = torch.cuda.Event()
                    done.record(other)
                main.wait_event(done)

            graph = None
            if captured:
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph, stream=main):
                    steps()
            for turn in range(3):
                for i, w in enumerate(works):           # what a launch before the join would use
                    w.B.fill_(float("nan"))
                    w.v.fill_(3.0)
                    w.rp.copy_(keep[i][0])
                graph.replay() if captured else steps()
                for w in works:
                    w.check("K=%d, turn %d" % (w.K, turn))
            del graph
        for p in plans:
            ctx.plan_destroy(p)


@pytest.mark.parametrize("M", [262_145, 900_001])
@pytest.mark.parametrize("chunk", [32, 160])
def test_tiles_of_several_passes(gpu_ctx, pkg, oracle, M, chunk):
    """Matrices whose tiles of rows the builder walks in several passes: passes with rows longer than two chunks, with
    shorter ones only, and with none that holds entries, in turn; records with and without a plan."""
    ctx, K, N = gpu_ctx, 4, 500
    rng = np.random.default_rng(M + chunk)
    degrees = rng.integers(0, 4 if chunk == 32 else 12, M)
    zone = np.arange(M) // 256
    degrees[zone % 5 == 2] = 0
    at = np.flatnonzero((zone % 5 == 4) & (np.arange(M) % 64 == 7))[::23]
    degrees[at] = rng.choice([2 * chunk, 2 * chunk + 1, 3 * chunk, 7 * chunk - 1], size=len(at))
    at = np.flatnonzero((zone % 5 == 1) & (np.arange(M) % 32 == 3))
    degrees[at] = rng.integers(1, 2 * chunk + 1, size=len(at))[: len(at)] // 4
    rp = np.concatenate([[0], np.cumsum(degrees)]).astype(np.int32)
    nnz = int(rp[-1])
    assert nnz > 40 * 160 * chunk           # records also without a plan
    ci, v = rng.integers(0, N, nnz).astype(np.int32), rng.uniform(-1, 1, nnz).astype(np.float32)
    B, X = (pkg.host_fill_uniform(n * K, M % 1000, j, -1.0, 1.0).reshape(n, K) for j, n in ((1, N), (2, M)))
    bufs = [ctx.upload(a) for a in (rp, ci, v, B, X)]
    d_C, d_o = ctx.alloc((M, K), np.float32), ctx.alloc((nnz,), np.float32)
    opts = pkg.Opts(chunk_nnz=chunk)
    plan = ctx.plan_create(M, nnz, bufs[0], K, opts, N=N, col_idx=bufs[1])
    for p in (None, plan):
        ctx.fill(d_C, M * K, 7.0)
        ctx.spmm_csr(M, N, K, nnz, *bufs[:4], d_C, plan=p, opts=opts)
        check_against_f64(d_C.to_host(), *oracle.spmm_f64(rp, ci, v, B), "product, plan=%s" % (p is not None))
        ctx.fill(d_o, nnz, 7.0)
        ctx.sddmm_csr(M, N, K, nnz, bufs[0], bufs[1], bufs[4], bufs[3], d_o, plan=p, opts=opts)
        check_against_f64(d_o.to_host(), *oracle.sddmm_f64(rp, ci, X, B), "SDDMM, plan=%s" % (p is not None))
    ctx.plan_destroy(plan)
    for b in bufs + [d_C, d_o]:
        b.free()
