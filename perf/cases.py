"""The work that users of this library time: products of a sparse matrix with a dense one, and what goes with them.

listed() names twelve calls over the real range of sizes, draw() gives more of the same ranges, prepare() makes what a
program holds before the call (device arrays, plan, layer handle), run() is one pass through the public entry points.

The operations:
  spmm       C = A * B, one plan for the structure, reused from call to call (GNN inference; the benchmark's product)
  spmm_once  the same call without a plan: the structure is new each time (sampled blocks of a graph, one-off products)
  sddmm      out[j] = dot(X[row(j)], Y[col[j]]) over the pattern of A (attention scores, weight gradients), with a plan
  coo        C = 0, then C += A * B from padded (row, col, value) triples: the arrays of the LBSpMM call
  train      one training step of an aggregation layer through PyTorch: forward, gradient of the features and, where
             the edge weights are learned, gradient of the weights, whose values are new in every step
  host       three products that share A (K = k, 2k, 4k), operands and results in page-locked host memory

Graphs: "powerlaw" is R-MAT (0.57, 0.19, 0.19, 0.05) with both directions of every draw kept, duplicates removed and
rows sorted; "random" has columns spread uniformly (Poisson row lengths), rows sorted.  Values lie in (0, 1), dense
operands in (-1, 1).
"""
import importlib.util
import math
import os
import sys

import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NAME = "hp_spmm_sddmm_b200"
PADDING = 32          # COO triples are padded to whole warps, as LBSpMM's callers pad them


def _package(sub=None):
    """The package lies in a directory whose name has hyphens, so it is imported by path (from the working folder)."""
    if NAME not in sys.modules:
        init = os.path.join(os.getcwd(), "hp-spmm-sddmm_b200", "__init__.py")
        if not os.path.exists(init):
            init = os.path.join(ROOT, "hp-spmm-sddmm_b200", "__init__.py")
        spec = importlib.util.spec_from_file_location(NAME, init)
        mod = importlib.util.module_from_spec(spec)
        sys.modules[NAME] = mod
        spec.loader.exec_module(mod)
    return importlib.import_module(NAME + "." + sub) if sub else sys.modules[NAME]


_ctx = None


def _context():
    """One context for the process, as a program keeps one per device."""
    global _ctx
    if _ctx is None:
        _ctx = _package().Context(0)
    return _ctx


def _case(name, op, graph, rows, cols, nnz, k, learned=False):
    c = {"op": op, "graph": graph, "rows": rows, "cols": cols, "nnz": nnz, "k": k, "learned": learned}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest configuration of the benchmark plan: launches and host time are all of it
        _case("spmm-4k-k32", "spmm", "random", 4096, 4096, 67_600, 32),
        # the benchmark's graph (R-MAT scale 20) at its narrowest and widest product
        _case("spmm-powerlaw-1m-k32", "spmm", "powerlaw", 1 << 20, 1 << 20, 16_000_000, 32),
        _case("spmm-powerlaw-1m-k128", "spmm", "powerlaw", 1 << 20, 1 << 20, 16_000_000, 128),
        # the largest: uniformly sparse, the dense operand far larger than the L2 cache
        _case("spmm-random-2450k-k64", "spmm", "random", 2_450_000, 2_450_000, 122_500_000, 64),
        # the last layer of a classifier: as many columns as classes, on a mid-sized graph
        _case("spmm-powerlaw-170k-k47", "spmm", "powerlaw", 169_999, 169_999, 2_330_001, 47),
        # a sampled block of a mini-batch: rectangular, its structure seen once, input features 100 wide
        _case("block-20k-k100", "spmm_once", "random", 20_011, 150_001, 300_007, 100),
        # a one-off product on a mid-sized graph at a common hidden width
        _case("once-powerlaw-250k-k64", "spmm_once", "powerlaw", 250_000, 250_000, 4_000_003, 64),
        # scores of every edge of the benchmark's graph
        _case("sddmm-powerlaw-1m-k64", "sddmm", "powerlaw", 1 << 20, 1 << 20, 16_000_000, 64),
        # the reference's own call on its own arrays
        _case("coo-powerlaw-250k-k64", "coo", "powerlaw", 250_000, 250_000, 4_000_003, 64),
        # a training step with learned edge weights, and one on a citation-sized graph where the host sets the pace
        _case("train-powerlaw-250k-k64", "train", "powerlaw", 250_000, 250_000, 4_000_003, 64, learned=True),
        _case("train-3k-k16", "train", "powerlaw", 2_999, 2_999, 11_111, 16),
        # operands on the host: everything crosses the bus
        _case("host-powerlaw-130k-k32", "host", "powerlaw", 131_072, 131_072, 2_000_000, 32),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(("spmm", "spmm", "spmm", "spmm_once", "spmm_once", "sddmm", "sddmm", "coo", "train", "train",
                     "host"))
    graph = rng.choice(("powerlaw", "powerlaw", "random"))
    # widths: the three the library is built around, other multiples of 32, and whatever a model happens to have
    k = rng.choice((32, 64, 128, 32, 64, 128, 96, 160, 256, None, None, None)) or log_int(3, 300)
    top = 60_000_000 if op == "spmm" else 16_000_000
    nnz = log_int(10_000, top)
    nnz = max(10_000, min(nnz, int(2.0e9) // k))
    degree = math.exp(rng.uniform(math.log(4), math.log(64)))
    rows = max(500, int(nnz / degree))
    cols = rows
    if op in ("spmm_once", "sddmm") and rng.random() < 0.5:   # blocks of a graph are rectangular
        cols = max(500, int(rows * math.exp(rng.uniform(math.log(0.2), math.log(8)))))
    limit = int(1.2e9) // (4 * k)                                          # dense operands of about a gigabyte
    if op == "host":
        k = rng.choice((16, 32, 64))
        nnz, limit = min(nnz, 8_000_000), int(1.5e8) // (28 * k)
    rows, cols = min(rows, limit), min(cols, limit)
    nnz = min(nnz, rows * cols // 8, 100 * rows)
    return _case(None, op, graph, rows, cols, nnz, k, learned=op == "train" and rng.random() < 0.5)


# ---- inputs --------------------------------------------------------------------------------------------------

def _keys(graph, rows, cols, count, gen):
    """`count` draws of row * cols + col."""
    dev = gen.device
    if graph == "random":
        r = torch.randint(rows, (count,), device=dev, generator=gen)
        return r * cols + torch.randint(cols, (count,), device=dev, generator=gen)
    bits = max(1, (max(rows, cols) - 1).bit_length())
    half = (count + 1) // 2
    r = torch.zeros(half, dtype=torch.int64, device=dev)
    c = torch.zeros(half, dtype=torch.int64, device=dev)
    for _ in range(bits):                       # one quadrant per bit: a = 0.57, b = 0.19, c = 0.19, d = 0.05
        u = torch.rand(half, device=dev, generator=gen)
        r = (r << 1) | (u >= 0.76)
        c = (c << 1) | (((u >= 0.57) & (u < 0.76)) | (u >= 0.95))
    span = 1 << bits
    return torch.cat((r * rows // span * cols + c * cols // span, c * rows // span * cols + r * cols // span))


def _csr(case, gen):
    """row_ptr, col_idx (int32) of `nnz` distinct entries, rows and columns ascending."""
    rows, cols, nnz = case["rows"], case["cols"], case["nnz"]
    have = _keys(case["graph"], rows, cols, nnz + nnz // 20 + 64, gen).unique()
    tries = 0
    while have.numel() < nnz:                   # duplicates were removed: draw what is missing
        tries += 1
        graph = case["graph"] if tries < 12 else "random"
        more = _keys(graph, rows, cols, 2 * (nnz - have.numel()) + nnz // 20 + 64, gen)
        have = torch.cat((have, more)).unique()
    if have.numel() > nnz:                      # leave surplus entries out, evenly
        at = torch.linspace(0, have.numel() - 1, have.numel() - nnz, device=gen.device, dtype=torch.float64).long()
        keep = torch.ones(have.numel(), dtype=torch.bool, device=gen.device)
        keep[at] = False
        have = have[keep]
        if have.numel() != nnz:
            raise RuntimeError("surplus entries coincide")
    r = have // cols
    row_ptr = torch.zeros(rows + 1, dtype=torch.int32, device=gen.device)
    row_ptr[1:] = torch.bincount(r, minlength=rows).cumsum(0)
    return row_ptr, (have - r * cols).int(), r.int()


class _Plan:
    """A plan that is given back with the state that holds it."""

    def __init__(self, ctx, rows, cols, nnz, row_ptr, col_idx, k):
        self.ctx = ctx
        self.handle = ctx.plan_create(rows, nnz, row_ptr.data_ptr(), k, N=cols, col_idx=col_idx.data_ptr(),
                                      stream=torch.cuda.current_stream().cuda_stream)

    def __del__(self):
        self.ctx.plan_destroy(self.handle)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    op, rows, cols, nnz, k = (case[x] for x in ("op", "rows", "cols", "nnz", "k"))

    def dense(n, width):
        return torch.rand((n, width), device="cuda", generator=gen) * 2 - 1

    row_ptr, col_idx, row_idx = _csr(case, gen)
    vals = torch.rand(nnz, device="cuda", generator=gen)
    st = {"op": op, "rows": rows, "cols": cols, "nnz": nnz, "k": k, "row_ptr": row_ptr, "col_idx": col_idx,
          "vals": vals}
    if op in ("spmm", "spmm_once"):
        st["B"] = dense(cols, k)
        st["C"] = torch.empty((rows, k), device="cuda")
    elif op == "sddmm":
        st["X"], st["Y"] = dense(rows, k), dense(cols, k)
        st["out"] = torch.empty(nnz, device="cuda")
    elif op == "coo":
        padded = -(-nnz // PADDING) * PADDING
        st["padded"] = padded
        for name, src in (("row", row_idx), ("col", col_idx), ("val", vals)):
            st[name] = torch.zeros(padded, dtype=src.dtype, device="cuda")
            st[name][:nnz] = src
        st["B"] = dense(cols, k)
        st["C"] = torch.empty((rows, k), device="cuda")
    elif op == "train":
        st["H"] = dense(cols, k).requires_grad_()
        st["dC"] = dense(rows, k)
        st["scores"] = (dense(1, nnz)[0] * 2).requires_grad_() if case["learned"] else None
        st["layer"] = _package("torch_ops").TorchLayer(row_ptr, col_idx, vals, rows, cols, k)
    elif op == "host":
        def pinned(t):
            h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
            h.copy_(t)
            return h

        for name in ("row_ptr", "col_idx", "vals"):
            st[name] = pinned(st[name])
        st["Ks"] = [k, 2 * k, 4 * k]
        st["Bs"] = [pinned(dense(cols, w)) for w in st["Ks"]]
        st["Cs"] = [torch.empty((rows, w), pin_memory=True) for w in st["Ks"]]
    if op in ("spmm", "sddmm"):
        st["plan"] = _Plan(_context(), rows, cols, nnz, row_ptr, col_idx, k)
    return st


# ---- one pass ------------------------------------------------------------------------------------------------

def run(st):
    op, rows, cols, nnz, k = st["op"], st["rows"], st["cols"], st["nnz"], st["k"]
    if op == "train":
        st["H"].grad = None
        if st["scores"] is None:                        # fixed weights: the values the layer was built with
            C = st["layer"](st["H"])
            C.backward(st["dC"])
            return C.detach(), st["H"].grad
        st["scores"].grad = None
        C = st["layer"](st["H"], torch.sigmoid(st["scores"]))
        C.backward(st["dC"])
        return C.detach(), st["H"].grad, st["scores"].grad
    ctx = _context()
    if op == "host":
        ctx.spmm_csr_host_multi(rows, cols, nnz, st["row_ptr"].data_ptr(), st["col_idx"].data_ptr(),
                                st["vals"].data_ptr(), st["Ks"], [b.data_ptr() for b in st["Bs"]],
                                [c.data_ptr() for c in st["Cs"]])
        return st["Cs"]
    stream = torch.cuda.current_stream().cuda_stream
    if op == "coo":
        ctx.fill(st["C"].data_ptr(), rows * k, 0.0, stream=stream)
        ctx.spmm_coo(rows, cols, k, st["padded"], st["row"].data_ptr(), st["col"].data_ptr(), st["val"].data_ptr(),
                     st["B"].data_ptr(), st["C"].data_ptr(), stream=stream)
        return st["C"]
    row_ptr, col_idx = st["row_ptr"].data_ptr(), st["col_idx"].data_ptr()
    if op in ("spmm", "spmm_once"):
        ctx.spmm_csr(rows, cols, k, nnz, row_ptr, col_idx, st["vals"].data_ptr(), st["B"].data_ptr(),
                     st["C"].data_ptr(), plan=st["plan"].handle if op == "spmm" else None, stream=stream)
        return st["C"]
    ctx.sddmm_csr(rows, cols, k, nnz, row_ptr, col_idx, st["X"].data_ptr(), st["Y"].data_ptr(), st["out"].data_ptr(),
                  plan=st["plan"].handle, stream=stream)
    return st["out"]


def work(case):
    """Bytes and operations that a pass cannot do without: each input read once, each output written once."""
    op, rows, cols, nnz, k = (case[x] for x in ("op", "rows", "cols", "nnz", "k"))
    a = 4 * (rows + 1) + 8 * nnz
    product = 2 * nnz * k
    if op == "sddmm":
        return {"bytes": a + 4 * k * (rows + cols), "flops": product}
    if op == "coo":
        return {"bytes": 12 * nnz + 4 * k * (rows + cols), "flops": product}
    if op == "train":
        step = a + 4 * k * (2 * rows + 2 * cols)        # H and dC in, C and dH out
        if not case["learned"]:
            return {"bytes": step, "flops": 2 * product}
        return {"bytes": step + 4 * nnz, "flops": 3 * product}   # scores are the values read; their gradient comes out
    if op == "host":
        return {"bytes": a + 28 * k * (rows + cols), "flops": 7 * product}
    return {"bytes": a + 4 * k * (rows + cols), "flops": product}


def tolerance(case):
    return {"rel": 1e-5, "max": 4e-4}         # sums of 32-bit products in another order
