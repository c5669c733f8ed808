"""ctypes binding of libb200jt.so (declared in include/b200jt.h).

The library is the only compute path of this package: if it is missing the import fails with
instructions to build it, and a call without a CUDA device raises -- there is no CPU fallback.
"""
import ctypes
import importlib.util
import os
import threading

import torch
from torch.multiprocessing.reductions import StorageWeakRef

_HERE = os.path.dirname(os.path.abspath(__file__))
LIB_PATH = os.path.join(_HERE, "csrc", "libb200jt.so")
HOST_PATH = os.path.join(_HERE, "csrc", "_b200jt_host.so")

MAX_DIMS = 10

DTYPE_CODES = {"bool": 0, "int8": 1, "int16": 2, "int32": 3, "int64": 4, "uint8": 5,
               "float16": 6, "bfloat16": 7, "float32": 8, "float64": 9}
TORCH_DTYPES = {"bool": torch.bool, "int8": torch.int8, "int16": torch.int16, "int32": torch.int32,
                "int64": torch.int64, "uint8": torch.uint8, "float16": torch.float16,
                "bfloat16": torch.bfloat16, "float32": torch.float32, "float64": torch.float64}
DTYPE_NAMES = {v: k for k, v in TORCH_DTYPES.items()}


class Tensor(ctypes.Structure):
    """struct b200jt_tensor"""
    _fields_ = [("ptr", ctypes.c_void_p), ("dtype", ctypes.c_int32), ("ndim", ctypes.c_int32),
                ("shape", ctypes.c_int64 * MAX_DIMS)]


def _load():
    if not os.path.exists(LIB_PATH):
        raise ImportError(
            f"{LIB_PATH} not found: build the CUDA library first "
            f"(`make -C {os.path.join(_HERE, 'csrc')}` or `python -c 'import __graft_entry__ as g; g.build()'`). "
            "jittor_b200 has no CPU fallback.")
    return ctypes.CDLL(LIB_PATH)


def _load_host():
    if not os.path.exists(HOST_PATH):
        raise ImportError(f"{HOST_PATH} not found: build it with `make -C {os.path.join(_HERE, 'csrc')}`")
    spec = importlib.util.spec_from_file_location("_b200jt_host", HOST_PATH)
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


lib = _load()
host = _load_host()

_TP = ctypes.POINTER(Tensor)
_SP = ctypes.POINTER(ctypes.c_char_p)
_vp, _i, _d, _u32, _sz = ctypes.c_void_p, ctypes.c_int, ctypes.c_double, ctypes.c_uint32, ctypes.c_size_t
_FP = ctypes.c_void_p   # float* device pointers are passed as raw addresses

# every symbol of include/b200jt.h: (name, restype, argtypes)
SIGNATURES = [
    ("b200jt_last_error", ctypes.c_char_p, []),
    ("b200jt_version", _i, []),
    ("b200jt_index_affine", _i, [ctypes.POINTER(ctypes.c_int64), _i, ctypes.POINTER(ctypes.c_int64), _i, _SP, _i,
                                 ctypes.POINTER(ctypes.c_int64), ctypes.POINTER(ctypes.c_int64)]),
    ("b200jt_reindex", _i, [_TP, _TP, _SP, _i, _d, _SP, _i, _TP, _i, _vp]),
    ("b200jt_reindex_source", _i, [_TP, _TP, _SP, _i, _d, _SP, _i, _TP, _i, ctypes.c_char_p, ctypes.c_int64,
                                   ctypes.POINTER(ctypes.c_int64), ctypes.POINTER(_i)]),
    ("b200jt_reindex_reduce_workspace", _sz, [_TP, _TP, ctypes.c_char_p, _SP, _i, _SP, _i, _TP, _i]),
    ("b200jt_reindex_reduce", _i, [_TP, _TP, ctypes.c_char_p, _SP, _i, _SP, _i, _TP, _i, _vp, _sz, _vp]),
    ("b200jt_reindex_reduce_noalloc_max_scratch", _sz, []),
    ("b200jt_reindex_reduce_noalloc", _i, [_TP, _TP, ctypes.c_char_p, _SP, _i, _SP, _i, _TP, _i, _vp]),
    ("b200jt_setitem", _i, [_TP, _TP, _TP, ctypes.c_char_p, _SP, _i, _TP, _i, _vp]),
    ("b200jt_broadcast_to", _i, [_TP, _TP, _u32, _vp]),
    ("b200jt_reduce_workspace", _sz, [_TP, _TP, ctypes.c_char_p, _u32]),
    ("b200jt_reduce", _i, [_TP, _TP, ctypes.c_char_p, _u32, _vp, _sz, _vp]),
    ("b200jt_binary", _i, [_TP, _TP, _TP, ctypes.c_char_p, _vp]),
    ("b200jt_unary", _i, [_TP, _TP, ctypes.c_char_p, _vp]),
    ("b200jt_ternary", _i, [_TP, _TP, _TP, _TP, _vp]),
    ("b200jt_fused_chain", _i, [_TP, _i, ctypes.POINTER(ctypes.c_int64), _i, _i, ctypes.POINTER(ctypes.c_int32), _i, _TP, _vp]),
    ("b200jt_fused_chain_source", _i, [_TP, _i, ctypes.POINTER(ctypes.c_int64), _i, _i, ctypes.POINTER(ctypes.c_int32), _i, _TP,
                                       ctypes.c_char_p, ctypes.c_int64, ctypes.POINTER(ctypes.c_int64), ctypes.POINTER(_i)]),
    ("b200jt_chain_jit_stats", _i, [ctypes.POINTER(_i), ctypes.POINTER(_i), ctypes.POINTER(_i)]),
    ("b200jt_softmax", _i, [_TP, _TP, _i, _vp]),
    ("b200jt_softmax_backward", _i, [_TP, _TP, _TP, _i, _vp]),
    ("b200jt_layer_norm", _i, [_TP, _TP, _TP, _TP, _d, _vp]),
    ("b200jt_layer_norm_backward_workspace", _sz, [_TP, _i]),
    ("b200jt_layer_norm_backward", _i, [_TP, _TP, _TP, _TP, _FP, _d, _vp, _sz, _vp]),
    ("b200jt_bn_backward_sums", _i, [_TP, _TP, _FP, _d, _FP, _FP, _d, _i, _FP, _vp]),
    ("b200jt_bn_backward_dx", _i, [_TP, _TP, _FP, _d, _FP, _FP, _d, _i, _FP, _TP, _vp]),
    ("b200jt_bn_backward", _i, [_TP, _TP, _FP, _d, _FP, _FP, _d, _i, _FP, _TP, _vp]),
    ("b200jt_optim_step", _i, [ctypes.c_char_p, _i, ctypes.POINTER(ctypes.c_int64)] + [ctypes.POINTER(_vp)] * 7
     + [ctypes.POINTER(_d), _i, _i, _vp]),
    ("b200jt_matmul_workspace", _sz, [_TP, _TP, _TP, _i, _i]),
    ("b200jt_matmul_least_workspace", _sz, [_TP, _TP, _TP, _i, _i]),
    ("b200jt_matmul", _i, [_TP, _TP, _TP, _i, _i, _vp, _sz, _vp]),
    ("b200jt_batched_matmul", _i, [_TP, _TP, _TP, _i, _i, _vp]),
    ("b200jt_device_status", _i, []),
    ("b200jt_conv2d_workspace", _sz, [_TP, _TP, _TP, _i, _i, _i, _i, _i, _i, _i]),
    ("b200jt_conv2d", _i, [_TP, _TP, _TP, _i, _i, _i, _i, _i, _i, _i, _FP, _vp, _sz, _vp]),
    ("b200jt_conv2d_formats_workspace", _sz, [_TP, _TP, _TP, _i, _i, _i, _i, _i, _i, ctypes.c_char_p, ctypes.c_char_p, ctypes.c_char_p]),
    ("b200jt_conv2d_formats", _i, [_TP, _TP, _TP, _i, _i, _i, _i, _i, _i, ctypes.c_char_p, ctypes.c_char_p, ctypes.c_char_p,
                                   _FP, _vp, _sz, _vp]),
    ("b200jt_conv2d_transpose", _i, [_TP, _TP, _TP, _i, _i, _i, _i, _i, _i, _i, _vp]),
    ("b200jt_conv2d_backward_w", _i, [_TP, _TP, _TP, _i, _i, _i, _i, _i, _i, _vp]),
    ("b200jt_conv2d_backward_w_workspace", _sz, [_TP, _TP, _TP, _i, _i, _i, _i, _i, _i]),
    ("b200jt_conv2d_backward_w_tc", _i, [_TP, _TP, _TP, _i, _i, _i, _i, _i, _i, _vp, _sz, _vp]),
    ("b200jt_conv2d_backward_w_formats_workspace", _sz, [_TP, _TP, _TP, _i, _i, _i, _i, _i, _i, ctypes.c_char_p, ctypes.c_char_p, ctypes.c_char_p]),
    ("b200jt_conv2d_backward_w_formats", _i, [_TP, _TP, _TP, _i, _i, _i, _i, _i, _i, ctypes.c_char_p, ctypes.c_char_p, ctypes.c_char_p,
                                              _vp, _sz, _vp]),
    ("b200jt_bn_stats", _i, [_TP, _FP, _vp]),
    ("b200jt_bn_apply", _i, [_TP, _FP, _d, _FP, _FP, _d, _i, _TP, _FP, _FP, _d, _vp]),
    ("b200jt_pool2d", _i, [_TP, _TP, _vp, ctypes.c_char_p, _i, _i, _i, _i, _i, _i, _i, _vp]),
    ("b200jt_pool2d_backward", _i, [_TP, _TP, _TP, _TP, ctypes.c_char_p, _i, _i, _i, _i, _i, _i, _i, _vp]),
    ("b200jt_conv2d_backward_x_workspace", _sz, [_TP, _TP, _TP, _i, _i, _i, _i, _i, _i]),
    ("b200jt_conv2d_backward_x", _i, [_TP, _TP, _TP, _i, _i, _i, _i, _i, _i, _vp, _sz, _vp]),
    ("b200jt_pool2d_taps", _i, [_TP, _TP, _vp, ctypes.c_char_p, _i, _i, _i, _i, _i, _i, _vp]),
    ("b200jt_pool2d_backward_taps", _i, [_vp, _TP, _TP, _i, _i, _i, _i, _i, _i, _vp]),
    ("b200jt_pool2d_backward_indices", _i, [_TP, _TP, _vp, _TP, _TP, _i, _i, _i, _i, _i, _i, _vp]),
    ("b200jt_peer_segment_bytes", _sz, [_sz]),
    ("b200jt_peer_segment_create", _i, [_sz, ctypes.POINTER(_vp), ctypes.c_char_p]),
    ("b200jt_peer_segment_destroy", _i, [_vp]),
    ("b200jt_peer_comm_create", _i, [_i, _i, _vp, ctypes.c_char_p, _sz, _d, ctypes.POINTER(_vp)]),
    ("b200jt_peer_comm_destroy", _i, [_vp]),
    ("b200jt_peer_max_bytes", _sz, [_vp]),
    ("b200jt_peer_comm_set_max_blocks", _i, [_vp, _i]),
    ("b200jt_set_sm_reserve", _i, [_i]),
    ("b200jt_probe_rate", _i, [ctypes.c_char_p, _i, _vp, ctypes.c_int64, ctypes.POINTER(ctypes.c_double)]),
    ("b200jt_peer_all_reduce", _i, [_vp, _vp, _vp, ctypes.c_int64, _i, ctypes.c_char_p, _vp]),
    ("b200jt_peer_comm_create_local", _i, [_i, _sz, _d, ctypes.POINTER(_vp)]),
    ("b200jt_peer_all_reduce_local", _i, [ctypes.POINTER(_vp), _i, ctypes.POINTER(_vp), ctypes.POINTER(_vp),
                                          ctypes.c_int64, _i, ctypes.c_char_p, _vp]),
]
for _name, _res, _args in SIGNATURES:
    _fn = getattr(lib, _name)
    _fn.restype = _res
    _fn.argtypes = _args


class B200Error(RuntimeError):
    pass


def check(rc, what=""):
    if rc != 0:
        msg = lib.b200jt_last_error().decode(errors="replace")
        raise B200Error(f"{what}: {msg} (status {rc})" if what else f"{msg} (status {rc})")


def require_cuda():
    if not torch.cuda.is_available():
        raise B200Error("jittor_b200 needs a CUDA device (sm_100a); there is no CPU fallback")


def desc(t, shape=None):
    """b200jt_tensor for a contiguous torch tensor, optionally viewed with another shape of equal size."""
    if not t.is_contiguous():
        raise B200Error("internal: non-contiguous tensor passed to the C ABI")
    shp = list(t.shape) if shape is None else list(shape)
    if len(shp) == 0:
        shp = [1]
    if len(shp) > MAX_DIMS:
        raise B200Error(f"tensors have at most {MAX_DIMS} dims, got {len(shp)}")
    d = Tensor()
    d.ptr = t.data_ptr() if t.numel() else None
    d.dtype = DTYPE_CODES[DTYPE_NAMES[t.dtype]]
    d.ndim = len(shp)
    for i, s in enumerate(shp):
        d.shape[i] = int(s)
    return d


def strings(items):
    arr = (ctypes.c_char_p * max(len(items), 1))()
    for i, s in enumerate(items):
        arr[i] = s.encode()
    return arr


def descs(tensors):
    arr = (Tensor * max(len(tensors), 1))()
    for i, t in enumerate(tensors):
        arr[i] = desc(t)
    return arr


def stream_ptr():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


# ---- allocations and launches of a plan -----------------------------------------------------------------------------
# Plans allocate and launch through the functions below. While a graph is run for the first time, `recorder` writes each of
# them down with its pointers as (buffer number, offset); csrc/host.cpp replays that tape when a graph of the same structure
# is synced again.
ARGTYPES = {name: args for name, _, args in SIGNATURES}
recorder = None
SCALAR_TYPES = {torch.uint8: 0, torch.int8: 1, torch.int16: 2, torch.int32: 3, torch.int64: 4, torch.float16: 5,
                torch.float32: 6, torch.float64: 7, torch.bool: 11, torch.bfloat16: 15}


class _NotReplayable(Exception):
    pass


def recording():
    return recorder is not None and recorder.thread == threading.get_ident()


class Recorder:
    def __init__(self, leaves):
        self.ok = True
        self.thread = threading.get_ident()   # what other threads launch meanwhile is not part of this graph
        self.steps = []
        self.moves = []                       # (step, Var): the step moves the running statistics that Var was to move
        self.computed = {}                    # id of a Var -> steps after which it has its value
        self.spans = []                       # (base, bytes, dtype, storage) per buffer; of two with an address one is alive
        for t in leaves:
            self._add(t)

    def _add(self, t):
        self.spans.append((t.data_ptr(), t.numel() * t.element_size(), t.dtype, StorageWeakRef(t.untyped_storage())))
        return len(self.spans) - 1

    def locate(self, ptr):
        for k in range(len(self.spans) - 1, -1, -1):
            base, n, _, storage = self.spans[k]
            if n and base <= ptr < base + n and not storage.expired():
                return k, ptr - base
        raise _NotReplayable(f"pointer {ptr:#x} belongs to no buffer of the plan")

    def locate_result(self, t):
        """A buffer that holds all of t as elements of its dtype (leaves may share memory in part, or as another dtype)."""
        ptr, size = t.data_ptr(), t.numel() * t.element_size()
        for k in range(len(self.spans) - 1, -1, -1):
            base, n, dtype, storage = self.spans[k]
            if base <= ptr and ptr + size <= base + n and dtype == t.dtype and not storage.expired():
                return k, ptr - base
        raise _NotReplayable("a result in no buffer of the plan")

    def alloc(self, t):
        k = self._add(t)
        self.steps.append(("alloc", k, tuple(t.shape), SCALAR_TYPES[t.dtype]))
        return k

    def _tensor(self, d):
        buf, off = self.locate(d.ptr) if d.ptr else (-1, 0)
        return (d.dtype, tuple(d.shape[:d.ndim]), buf, off)

    def _args(self, name, args):
        out, last = [], -1
        for a, ty in zip(args, ARGTYPES[name]):
            if isinstance(a, Tensor):
                out.append(("T", [self._tensor(a)]))
            elif isinstance(a, ctypes.Array) and a._type_ is Tensor:
                out.append(("T", [self._tensor(d) for d in a]))
            elif isinstance(a, ctypes.Array) and a._type_ is ctypes.c_char_p:
                out.append(("S", [s for s in a if s is not None]))
            elif isinstance(a, ctypes.Array) and a._type_ in (ctypes.c_int64, ctypes.c_int32):
                out.append(("q" if a._type_ is ctypes.c_int64 else "w", list(a)))
            elif isinstance(a, bytes):
                out.append(("b", a))
            elif ty in (ctypes.c_double,):
                out.append(("d", float(a)))
            elif ty is ctypes.c_size_t:
                out.append(("n", last) if last >= 0 else ("i", int(a)))       # the size of the workspace passed before it
            elif ty is ctypes.c_void_p or a is None:
                v = a.value if isinstance(a, ctypes.c_void_p) else a
                if v:
                    last, off = self.locate(v)
                    out.append(("p", last, off))
                else:
                    last = -1
                    out.append(("0",))
            else:
                out.append(("i", int(a)))
        return out

    def note(self, fn, *args):
        if self.ok:
            try:
                fn(*args)
            except _NotReplayable:
                self.ok = False

    def call(self, name, args, what):
        self.note(lambda: self.steps.append(("call", -1, name, self._args(name, args) + [("z",)], what)))

    def moved(self, v):
        """The next step moves v's running statistics."""
        self.moves.append((len(self.steps), v))

    def workspace(self, name, args, t):
        k = self._add(t)
        self.note(lambda: self.steps.append(("workspace", k, name, self._args(name, args))))

    def fill(self, t, value):
        def write():
            if isinstance(value, int) and abs(value) >= 1 << 53:
                raise _NotReplayable("an integer a double does not hold")
            self.steps.append(("fill", self.locate(t.data_ptr())[0], float(value)))
        if t.numel():
            self.note(write)


def alloc(shape, dtype):
    """An uninitialised CUDA tensor of a plan; `dtype` is a torch dtype."""
    t = torch.empty(shape, dtype=dtype, device="cuda")
    if recording():
        recorder.alloc(t)
    return t


def full(shape, value, dtype):
    t = torch.full(shape, value, dtype=dtype, device="cuda")
    if recording():
        recorder.alloc(t)
        recorder.fill(t, value)
    return t


# entry points that also run, if slower, with less scratch memory than they ask for -> what they cannot do without (host.cpp knows it too)
LEAST = {"b200jt_matmul_workspace": "b200jt_matmul_least_workspace"}


def workspace(name, *args):
    """(bytes, pointer, tensor that owns it) of the scratch memory `name` asks for, or that it runs with where there is no room."""
    n = getattr(lib, name)(*args)
    if n == 0:
        return 0, None, None
    try:
        t = torch.empty(int(n), dtype=torch.uint8, device="cuda")
    except torch.OutOfMemoryError:
        if name not in LEAST:
            raise
        if recording():
            recorder.ok = False               # not the steps of the next run, which may find room
        n = getattr(lib, LEAST[name])(*args)
        if n == 0:
            return 0, None, None
        t = torch.empty(int(n), dtype=torch.uint8, device="cuda")
    if recording():
        recorder.workspace(name, args, t)
    return n, t.data_ptr(), t


def call(name, *args, what=None):
    """Launches entry point `name` on the current stream (its last argument)."""
    rc = getattr(lib, name)(*args, stream_ptr())
    if rc or recording():
        what = what() if callable(what) else what or name
        check(rc, what)
        recorder.call(name, args, what)
