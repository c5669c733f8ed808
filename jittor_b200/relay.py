"""Layers planned without their meta-operator graph: matmul, convolution, softmax, LayerNorm and training BatchNorm (+ ReLU),
forward and backward.

The reference's callers write these as meta-op graphs and its tuners look for them again (python/jittor/src/opt/tuner/
matmul_tuner.cc:21-102, conv_tuner.cc:218-411). Here the caller hands the executor a record (`Var._relay`) of what it
wrote; the graph itself is a builder that runs only when something reads `Var._op` -- another matcher, the fuser, or
jt.grad when it differentiates a gradient. First-order gradients come from `Var._vjp`: (inputs, rule), where
rule(y, dout, wanted) gives one gradient per input, again as records, whose builders derive the same gradient from the
graph by the per-op rules; a rule that takes two of the program's steps at once names the Var between them, and the graph
is followed when the gradient of that one is asked for or ends there. A record is only made for shapes, dtypes and flags whose graph the executor's matcher recognises
(`_recognised`), so a layer runs the same kernels with or without it."""
import weakref

import torch

from . import _capi as C
from . import dtypes
from . import var as V
from .flags import flags, flag_scope

_KNOWN = {}                 # (layer, dtypes, ranks, flags) -> dtype of the result, or None where the matcher does not take the graph


def _recognised(key, build, matcher):
    r = _KNOWN.get(key, False)
    if r is False:
        v = build()
        r = _KNOWN[key] = v.dtype if matcher(v) is not None else None
    return r


def lazy(shape, dtype, record, build):
    """A Var of a record; `build()` writes the graph (a Var of the same shape and dtype) when it is asked for."""
    v = V.Var(shape, dtype)
    v._relay = record
    if build is not None:
        amp = flags._v["amp_reg"]

        def op():
            with flag_scope(amp_reg=amp):
                g = build()
            return g._op if g._op is not None and g._data is None else V.Op("reshape", [g])
        v._builder = op
    return v


def _graph_grad(y, dout, x):
    """d(y . dout) / dx by the per-op rules of y's graph."""
    g = backprop(y, dout, [x], through_graph=y)[0]
    return g if g.dtype == x.dtype else g.cast(x.dtype)


def plan(v):
    """The Plan of a record, or None when its operands miss what the kernels take (the graph is used then)."""
    r = v._relay
    return _PLANS[r[0]](v, r)


def _plan(leaves, run):
    return E.Plan(leaves, run)


# ------------------------------------------------------------------------------------------------ matmul
_MM = (dtypes.DType("float32"), dtypes.DType("bfloat16"))


def matmul(a, b, ta, tb, dtype, build):
    m, n = a._shape[1 if ta else 0], b._shape[0 if tb else 1]
    y = lazy([m, n], dtype, ("matmul", a, b, ta, tb), build)

    def rule(y, dout, wanted):
        da = db = None
        if dout.dtype != a.dtype and wanted:
            dout = dout.cast(a.dtype)
        if wanted[0]:
            l, r, t0, t1 = (b, dout, tb, True) if ta else (dout, b, False, not tb)
            da = matmul(l, r, t0, t1, a.dtype, lambda: _graph_grad(y, dout, a))
        if wanted[1]:
            l, r, t0, t1 = (dout, a, True, ta) if tb else (a, dout, not ta, False)
            db = matmul(l, r, t0, t1, b.dtype, lambda: _graph_grad(y, dout, b))
        return da, db
    y._vjp = ((a, b), rule)
    return y


def _plan_matmul(v, r):
    _, a, b, ta, tb = r
    return _plan([a, b], lambda: E.run_matmul(a, b, ta, tb, v.dtype))


# ------------------------------------------------------------------------------------------------ convolution
def conv_vjp(y, x, w, geo):
    def rule(y, dout, wanted):
        if dout.dtype != x.dtype:
            dout = dout.cast(x.dtype)
        dx = lazy(x.shape, x.dtype, ("conv2d_dx", dout, w, geo, tuple(x.shape)), lambda: _graph_grad(y, dout, x)) if wanted[0] else None
        dw = lazy(w.shape, w.dtype, ("conv2d_dw", x, dout, geo, tuple(w.shape)), lambda: _graph_grad(y, dout, w)) if wanted[1] else None
        return dx, dw
    y._vjp = ((x, w), rule)


def _plan_conv(v, r):
    kind, x, w, geo, groups = r
    if x.dtype not in _MM or w.dtype not in _MM:
        return None
    if kind == "conv2d":
        return _plan([x, w], lambda: E.run_conv2d(x, w, geo, v.dtype, groups=groups))
    return _plan([x, w], lambda: E.run_conv2d_transpose(x, w, geo, groups, list(v.shape), v.dtype))


def _plan_conv_dx(v, r):
    return E.conv_dx_plan(v, r[1], r[2], r[3])


def _plan_conv_dw(v, r):
    _, x, dy, geo, wshape = r
    return _plan([x, dy], lambda: E.run_conv2d_backward_w(x, dy, geo, list(wshape), v.dtype))


# ------------------------------------------------------------------------------------------------ softmax
def softmax(x, log, rows, cols, build, backward):
    if x.dtype not in _MM or rows * cols == 0:
        return None
    if _recognised(("softmax", str(x.dtype), log, x.ndim, rows == 1 and x.ndim > 1, flags._v["amp_reg"]), build, E._match_softmax) != x.dtype:
        return None
    y = lazy(x.shape, x.dtype, ("softmax", x, log, rows, cols), build)
    y._vjp = ((x,), lambda y, dout, wanted: (backward(y, dout),))
    return y


def _plan_softmax(v, r):
    _, x, log, rows, cols = r

    def run():
        out = C.alloc([rows, cols], C.TORCH_DTYPES[x.dtype])
        C.call("b200jt_softmax", C.desc(x._data, [rows, cols]), C.desc(out), int(log), what="softmax")
        return out
    return _plan([x], run)


# ------------------------------------------------------------------------------------------------ mean pooling
def mean_pool_dx(x, y, dout, k, s, p):
    return lazy(x.shape, x.dtype, ("mean_pool_dx", dout, tuple(x.shape), tuple(k), tuple(s), tuple(p)), lambda: _graph_grad(y, dout, x))


def _plan_mean_pool_dx(v, r):
    _, dy, xshape, k, s, p = r

    def run():
        dx = C.alloc(list(xshape), C.TORCH_DTYPES[v.dtype])
        d = C.desc(dy._data, list(dy.shape))
        C.call("b200jt_pool2d_backward", C.desc(dx), d, d, C.desc(dx), b"mean", *k, *s, *p, 1, what="pool2d_backward")
        return dx
    return _plan([dy], run)


# ------------------------------------------------------------------------------------------------ parameters of the norms
def _param(p, shape, neutral):
    """A float32 Var of that shape, "const" for the neutral Python number, or None for what the records do not hold: other
    numbers, arrays, and shapes that the graph would stretch or refuse."""
    if isinstance(p, V.Var):
        return p if p.dtype == "float32" and p._const is None and list(p.shape) == list(shape) else None
    return "const" if isinstance(p, (int, float)) and p == neutral else None


def _var_or_none(p):
    return p if isinstance(p, V.Var) else None


def _desc_or_none(p, shape):
    return C.desc(p._data, shape) if p is not None else None


def _ptr_or_none(p):
    return p._data.data_ptr() if p is not None else None


def _part(whole, offset, shape, build):
    """A slice of a flat float32 Var, as the parameters' gradients come out of one buffer."""
    return lazy(shape, "float32", ("part", whole, offset), build)


def _plan_part(v, r):
    _, whole, offset = r
    n = v.numel()
    return _plan([whole], lambda: whole._data[offset:offset + n])


# ------------------------------------------------------------------------------------------------ LayerNorm
MAX_NORM_COLS = 8192        # rows the gradient kernel keeps in registers


def layer_norm(x, weight, bias, eps, k, build):
    """LayerNorm over the last k axes; None if the graph has to be written."""
    cols = 1
    for s in x._shape[x.ndim - k:]:
        cols *= s
    g, b = _param(weight, x._shape[x.ndim - k:], 1), _param(bias, x._shape[x.ndim - k:], 0)
    if g is None or b is None or x.dtype not in _MM or x.numel() == 0:
        return None
    key = ("layer_norm", str(x.dtype), x.ndim, k, isinstance(g, str), isinstance(b, str), flags._v["amp_reg"])
    if _recognised(key, build, E._match_layernorm) != x.dtype:
        return None
    g, b = _var_or_none(g), _var_or_none(b)
    rows = x.numel() // cols
    y = lazy(x.shape, x.dtype, ("layer_norm", x, g, b, float(eps), rows, cols), build)
    if cols > MAX_NORM_COLS:
        return y
    params = tuple(p for p in (g, b) if p is not None)

    def rule(y, dout, wanted):
        if dout.dtype != x.dtype:
            dout = dout.cast(x.dtype)
        if list(dout.shape) != list(x.shape):
            dout = dout.broadcast(x.shape)
        dx = lazy(x.shape, x.dtype, ("layer_norm_dx", x, g, dout, float(eps), rows, cols), lambda: _graph_grad(y, dout, x)) if wanted[0] else None
        out = [dx]
        if any(wanted[1:]):
            both = lazy([2 * cols], "float32", ("layer_norm_params", x, g, dout, float(eps), rows, cols, dx), None)
            for p, want in zip(params, wanted[1:]):
                out.append(_part(both, 0 if p is g else cols, p.shape, lambda p=p: _graph_grad(y, dout, p)) if want else None)
        return out + [None] * (1 + len(params) - len(out))
    y._vjp = ((x,) + params, rule)
    return y


def _plan_layer_norm(v, r):
    _, x, g, b, eps, rows, cols = r

    def run():
        out = C.alloc([rows, cols], C.TORCH_DTYPES[x.dtype])
        C.call("b200jt_layer_norm", C.desc(x._data, [rows, cols]), _desc_or_none(g, [cols]), _desc_or_none(b, [cols]), C.desc(out), eps,
               what="layer_norm")
        return out
    return _plan([x] + [p for p in (g, b) if p is not None], run)


def _run_layer_norm_backward(x, g, dy, eps, rows, cols, want_dx, want_params):
    xd = C.desc(x._data, [rows, cols])
    dx = C.alloc([rows, cols], C.TORCH_DTYPES[x.dtype]) if want_dx else None
    params = C.alloc([2 * cols], torch.float32) if want_params else None
    n, p, ws = C.workspace("b200jt_layer_norm_backward_workspace", xd, int(want_params))
    C.call("b200jt_layer_norm_backward", xd, _desc_or_none(g, [cols]), C.desc(dy._data, [rows, cols]), C.desc(dx) if want_dx else None,
           params.data_ptr() if want_params else None, eps, p, n, what="layer_norm_backward")
    return dx, params


def _plan_layer_norm_dx(v, r):
    _, x, g, dy, eps, rows, cols = r
    return _plan([x, dy] + ([g] if g is not None else []), lambda: _run_layer_norm_backward(x, g, dy, eps, rows, cols, True, False)[0])


def _plan_layer_norm_params(v, r):
    """The parameters' gradients; an x gradient that is still to be computed comes out of the same launch."""
    _, x, g, dy, eps, rows, cols, dx = r

    def run():
        with_dx = dx is not None and dx._data is None
        dxd, params = _run_layer_norm_backward(x, g, dy, eps, rows, cols, with_dx, True)
        if with_dx:
            dx._data = dxd.view(list(dx.shape))
        return params
    return _plan([x, dy] + ([g] if g is not None else []), run)


def ahead(roots):
    """Records whose launch also yields one of the roots: computed before the roots are taken in order."""
    first = []
    for v in roots:
        r = v._relay
        if r is not None and r[0] == "part" and r[1]._relay is not None and r[1]._relay[0] == "layer_norm_params" and r[1]._data is None:
            dx = r[1]._relay[7]
            if dx is not None and any(u is dx for u in roots) and not any(u is r[1] for u in first):
                first.append(r[1])
    return first


# ------------------------------------------------------------------------------------------------ BatchNorm (+ ReLU)
def batch_norm(module, x, weight, bias, eps, build):
    """Training BatchNorm of one process; None if the graph has to be written. build() returns (normalised x, batch mean,
    batch variance)."""
    if x.ndim < 3 or x.dtype not in _MM or x.numel() == 0:
        return None
    cn = x._shape[1]
    g, b = _param(weight, [cn], 1), _param(bias, [cn], 0)
    if g is None or b is None or cn > 2048:
        return None
    key = ("batch_norm", str(x.dtype), x.ndim, isinstance(g, str), isinstance(b, str), flags._v["amp_reg"])
    dtype = _recognised(key, lambda: build()[0], E._match_batchnorm)
    if dtype not in _MM:
        return None
    g, b = _var_or_none(g), _var_or_none(b)
    stats = V.Var([2 * cn], "float32", V.Op("custom", [x], fn=_run_bn_stats, name="bn_stats", sig=("bn_stats",)))

    def graph():
        norm, xmean, xvar = build()
        owner = me()                    # weak: a Var must not hold itself through its builder
        if owner is not None and owner._bn_running is not None:
            owner._bn_running = (module, xmean, xvar)
        return norm
    y = lazy(x.shape, dtype, ("batch_norm", x, g, b, float(eps), stats), graph)
    me = weakref.ref(y)
    y._bn_running = (module, None, None)
    _bn_vjp(y, y, False)
    return y


def relu_of(x, build):
    """relu of a BatchNorm record as one record; None for anything else."""
    r = x._relay
    if r is None or r[0] != "batch_norm" or x._data is not None:
        return None
    dtype = dtypes.binary_dtype_infer("add", x.dtype, "float32", False, True)
    if dtype not in _MM:
        return None
    y = lazy(x.shape, dtype, ("batch_norm_relu", x), build)
    _bn_vjp(y, x, True)
    return y


def _bn_vjp(y, root, relu):
    _, x, g, b, eps, stats = root._relay
    params = tuple(p for p in (g, b) if p is not None)
    cn = x._shape[1]

    def rule(y, dout, wanted):
        if dout.dtype not in _MM:
            dout = dout.cast(y.dtype)
        if list(dout.shape) != list(x.shape):
            dout = dout.broadcast(x.shape)
        rounding = 0 if x.dtype == "float32" else 4 if y.dtype == "bfloat16" else 2         # where the graph's dtypes round
        rest = (x, dout, stats, g, b, eps, int(relu) + rounding)
        sums = lazy([4 * cn], "float32", ("batch_norm_sums",) + rest, None)
        out = [lazy(x.shape, x.dtype, ("batch_norm_dx",) + rest + (sums,), lambda: _graph_grad(y, dout, x)) if wanted[0] else None]
        for p, want in zip(params, wanted[1:]):
            out.append(_part(sums, cn if p is g else 0, p.shape, lambda p=p: _graph_grad(y, dout, p)) if want else None)
        return out
    y._vjp = ((x,) + params, rule, root) if relu else ((x,) + params, rule)


def _run_bn_stats(xd):
    cn = xd.shape[1]
    stats = C.alloc([2 * cn], torch.float32)
    C.call("b200jt_bn_stats", C.desc(xd), stats.data_ptr(), what="bn_stats")
    return stats


def _plan_batch_norm(v, r):
    root = v if r[0] == "batch_norm" else r[1]
    if root._relay is None:                 # the normalised Var was assigned to: the ReLU is of its new value
        return None
    _, x, g, b, eps, stats = root._relay
    return E.batch_norm_plan(v, x, ("var", g) if g is not None else ("const", 1.0), ("var", b) if b is not None else ("const", 0.0),
                             eps, r[0] != "batch_norm", False, root, stats)


def _bn_operands(r):
    _, x, dy, stats, g, b, eps, relu = r[:8]
    cn = x._shape[1]
    count = float(x.numel() // cn)
    leaves = [stats, x, dy] + [p for p in (g, b) if p is not None]
    return leaves, lambda: (C.desc(x._data), C.desc(dy._data, list(x.shape)), stats._data.data_ptr(), count, _ptr_or_none(g), _ptr_or_none(b),
                            eps, relu)


def _plan_bn_sums(v, r):
    leaves, args = _bn_operands(r)

    def run():
        a = args()
        sums = C.alloc(list(v.shape), torch.float32)
        C.call("b200jt_bn_backward_sums", *a, sums.data_ptr(), what="bn_backward_sums")
        return sums
    return _plan(leaves, run)


def _plan_bn_dx(v, r):
    """The gradient of x; sums that are still to be computed come out of the same call."""
    leaves, args = _bn_operands(r)
    sums = r[8]

    def run():
        a = args()
        dx = C.alloc(list(v.shape), C.TORCH_DTYPES[v.dtype])
        if sums._data is not None:
            C.call("b200jt_bn_backward_dx", *a, sums._data.data_ptr(), C.desc(dx), what="bn_backward_dx")
            return dx
        both = C.alloc(list(sums.shape), torch.float32)
        C.call("b200jt_bn_backward", *a, both.data_ptr(), C.desc(dx), what="bn_backward")
        sums._data = both
        return dx
    return _plan(leaves, run)


_PLANS = {"matmul": _plan_matmul, "conv2d": _plan_conv, "conv2d_transpose": _plan_conv, "conv2d_dx": _plan_conv_dx, "conv2d_dw": _plan_conv_dw,
          "softmax": _plan_softmax, "mean_pool_dx": _plan_mean_pool_dx, "layer_norm": _plan_layer_norm, "layer_norm_dx": _plan_layer_norm_dx,
          "layer_norm_params": _plan_layer_norm_params, "part": _plan_part, "batch_norm": _plan_batch_norm,
          "batch_norm_relu": _plan_batch_norm, "batch_norm_sums": _plan_bn_sums, "batch_norm_dx": _plan_bn_dx}

from . import executor as E             # noqa: E402  (imports this module)
from .grad import backprop              # noqa: E402
