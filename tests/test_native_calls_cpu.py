"""The hot calls take their arguments as ctypes takes them for the same prototypes: both are pointed at a function that
records what arrives, no GPU needed."""
import ctypes

import numpy as np
import pytest

FUNCTIONS = ("spmm_csr_f32", "spmm_coo_f32", "sddmm_csr_f32", "fill_f32", "layer_forward", "layer_backward_features",
             "layer_backward_weights")
# per call: what each argument is
KINDS = {"spmm_csr_f32": "hhiiiipppppoh", "sddmm_csr_f32": "hhiiiipppppoh", "spmm_coo_f32": "hiiiipppppoh",
         "fill_f32": "hpifh", "layer_forward": "hhipph", "layer_backward_features": "hhipph",
         "layer_backward_weights": "hhippph"}
NATIVE = {"spmm_csr_f32": "spmm_csr", "spmm_coo_f32": "spmm_coo", "sddmm_csr_f32": "sddmm_csr", "fill_f32": "fill"}


class _Parameter:
    def __init__(self, v):
        self._as_parameter_ = v


@pytest.fixture(scope="module")
def recorded(pkg):
    """(native, seen, through_ctypes): the extension bound to recording functions, and the same through ctypes."""
    lib = pkg.load_library()
    native = pkg.load_native()
    seen = {}

    def recorder(name, argtypes):
        def f(*args):
            def plain(a):
                if not isinstance(a, ctypes.POINTER(pkg.Opts)):
                    return a
                return (a.contents.algo, a.contents.chunk_nnz, a.contents.b_l2_hint) if a else None
            seen[name] = tuple(plain(a) for a in args)
            return 0
        c = ctypes.CFUNCTYPE(ctypes.c_int, *argtypes)(f)
        c.argtypes = argtypes
        return c

    fns = {n: recorder(n, pkg.PROTOTYPES["hpspmm_" + n][1]) for n in FUNCTIONS}
    real = [ctypes.cast(getattr(lib, "hpspmm_" + n), ctypes.c_void_p).value for n in FUNCTIONS]
    types = (np.ndarray, pkg.DeviceBuffer, pkg.Opts)
    native.bind(*[ctypes.cast(fns[n], ctypes.c_void_p).value for n in FUNCTIONS], *types)

    def through_ctypes(name, args):
        out = []
        for kind, a in zip(KINDS[name], args):
            out.append(pkg._ptr(a) if kind == "p" else (ctypes.byref(a) if a else None) if kind == "o" else a)
        return fns[name](*out)

    yield native, seen, through_ctypes
    native.bind(*real, *types)


def _values(pkg, kind):
    """Values for one argument: (accepted ones, refused ones)."""
    buf = object.__new__(pkg.DeviceBuffer)
    buf.ptr = 0x7f0012345600
    freed = object.__new__(pkg.DeviceBuffer)
    freed.ptr = 0
    sub = type("Sub", (pkg.Opts,), {"_fields_": [("more", ctypes.c_int)]})
    arr = np.arange(6, dtype=np.float32)

    class Array(np.ndarray):
        ptr = 1
        value = 2

    if kind == "p":
        return ([None, 0, 1 << 45, (1 << 64) + 5, True, buf, freed, arr, arr[1:], arr.view(Array), np.int64(77), 12.0, "34",
                 np.float64(8.0)], [object(), "x", ctypes.c_void_p(9), [1], _Parameter(3)])
    if kind == "h":
        return ([None, 0, 7, False, 1 << 45, ctypes.c_void_p(1 << 45), ctypes.c_void_p(None), _Parameter(9),
                 _Parameter(ctypes.c_void_p(11)), _Parameter(_Parameter(None))], [object(), 2.0, [1], arr])
    if kind == "i":
        return ([5, 0, -1, True, 1 << 40, 1 << 63, 1 << 70, (1 << 64) + 3, np.int64(6), np.int32(-2), ctypes.c_int64(8),
                 _Parameter(4)], [None, 5.0, "5", object(), ctypes.c_void_p(None)])
    if kind == "f":
        return [2, 1.5, np.float32(0.25), True, -1.0], ["1", None, object()]
    return ([None, 0, False, (), {}, "", pkg.Opts(1, 64, 2, 0), sub(2, 96, 1, 0)], [bytes(16), object(), 1, np.zeros(4, np.int32)])


PLAIN = {"h": 3, "i": 4, "p": 0x1000, "f": 1.0, "o": None}


@pytest.mark.parametrize("name", FUNCTIONS)
def test_arguments_arrive_as_through_ctypes(pkg, recorded, name):
    native, seen, through_ctypes = recorded
    call = getattr(native, NATIVE.get(name, name))
    kinds = KINDS[name]
    for at, kind in enumerate(kinds):
        accepted, refused = _values(pkg, kind)
        for v in accepted:
            args = [PLAIN[k] for k in kinds]
            args[at] = v
            seen.clear()
            assert through_ctypes(name, args) == 0
            want = seen.pop(name)
            assert call(*args) == 0
            assert seen.pop(name) == want, (name, at, kind, v)
        for v in refused:
            args = [PLAIN[k] for k in kinds]
            args[at] = v
            with pytest.raises(Exception):
                through_ctypes(name, args)
            with pytest.raises(Exception):
                call(*args)
            assert not seen, (name, at, kind, v)
    with pytest.raises(TypeError):
        call(*[PLAIN[k] for k in kinds][:-1])
