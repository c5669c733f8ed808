"""Reverse-mode differentiation over the lazy graph with the reference's per-op rules:
reindex <-> reindex_reduce(add) (python/jittor/src/ops/reindex_op.cc:76-80, reindex_reduce_op.cc:45-63),
broadcast_to <-> reduce(add) (broadcast_to_op.cc:112-117, reduce_op.cc:339-362), element-wise rules
(binary_op.cc:491-550, unary_op.cc:891-966), ternary, reshape and the all-reduce (its own adjoint,
python/jittor/extern/mpi/ops/mpi_all_reduce_op.cc:67-71).

`grad(loss, targets)` builds new lazy Vars; nothing runs until they are synced, and the backward graph goes through
the same executor (so e.g. the gradient of a max-pool written with reindex + reduce(max) lands on the injective
reindex_reduce kernel)."""
from . import var as V
from ._capi import host


def _bcast_like(x, ref, mask, keep):
    """broadcast_to with explicit masks (the constructor the reference's grad rules call)."""
    return V.Var(ref.shape, x.dtype, V.Op("broadcast_to", [x], bcast_mask=mask, keepdims_mask=keep))


def _zeros_like(v):
    return V.full(list(v.shape), 0, v.dtype)


def _op_grad(out, dout, k):
    """Gradient w.r.t. input k of the op that produced `out` (None: no gradient flows), for the kinds csrc/host.cpp does not
    write itself (its op_grad has add, subtract, multiply, divide, maximum / minimum, negative, log, exp, casts, ternary,
    reshape, broadcast_to and the add / mean reduces)."""
    op = out._op
    kind, a = op.kind, op.attrs
    x = op.inputs[k]
    if kind == "reindex":
        if k != 0:
            return None
        return V.reindex_reduce(dout, "add", list(x.shape), a["indexes"], a["overflow_conditions"], op.inputs[1:])
    if kind == "reindex_reduce":
        if k != 0:
            return None
        args = (list(x.shape), a["indexes"], 0, a["overflow_conditions"], op.inputs[1:])
        if a["op"] == "add":
            return V.reindex(dout, *args)
        if a["op"] == "multiply":
            return V.reindex(dout * out, *args) / x
        if a["op"] in ("maximum", "minimum"):
            cond = V.binary(x, V.reindex(out, *args), "equal")
            return V.ternary(cond, V.reindex(dout, *args), _zeros_like(x))
        return None
    if kind == "reduce":
        mask, keep, rop = a["reduce_mask"], a["keepdims_mask"], a["op"]
        if rop == "multiply":
            return _bcast_like(dout * out, x, mask, keep) / x
        if rop in ("maximum", "minimum"):
            cond = V.binary(x, _bcast_like(out, x, mask, keep), "equal")
            return V.ternary(cond, _bcast_like(dout, x, mask, keep), _zeros_like(x))
        return None
    if kind == "binary":
        p, q = op.inputs
        if a["op"] != "pow":
            return None
        g = dout * q * V.binary(p, q - 1, "pow") if k == 0 else dout * (out * V.unary(p, "log"))
        gs, shape = list(g.shape), list(x.shape)
        if gs != shape:                           # back over the axes the operand was stretched along
            pad = len(gs) - len(shape)
            dims = list(range(pad)) + [pad + i for i, s in enumerate(shape) if s == 1 and gs[pad + i] != 1]
            g = (V.reduce(g, "add", dims, True) if dims else g).reshape(shape)
        return g
    if kind == "unary":
        uop = a["op"]
        if uop == "abs":
            return V.ternary(V.binary(x, 0.0, "greater_equal"), dout, -dout)
        if uop == "sqrt":
            return dout / (out * 2.0)
        if uop == "sin":
            return dout * V.unary(x, "cos")
        if uop == "cos":
            return dout * (-V.unary(x, "sin"))
        if uop == "tanh":
            c = V.unary(x, "cosh")
            return dout / (c * c)
        if uop == "sigmoid":
            return dout * out * (1.0 - out)
        return None
    if kind == "custom":
        rule = a.get("grad")                      # relays bring their own backward (e.g. the pooling kernels)
        return rule(out, dout, k) if rule is not None else None
    if kind == "mpi_all_reduce":
        from . import dist
        return dist.mpi_all_reduce(dout, "add")
    return None


def backprop(loss, dout, targets, through_graph=None):
    """The gradients that reach `targets` when `dout` is the gradient at `loss`: nodes from which a target is reachable are
    walked in reverse topological order (csrc/host.cpp; the rules of rare op kinds are `_op_grad` above). A Var with its own
    backward (`_vjp` = inputs, rule) takes one step to its inputs; `through_graph` names one whose rule is passed over in
    favour of its graph's."""
    return [g if g is not None else _zeros_like(t) for g, t in zip(host.backprop(loss, dout, targets, through_graph), targets)]


def grad(loss, targets, retain_graph=True):
    """d(sum(loss)) / d(target) for every target; a list of Vars (a single Var if `targets` is one)."""
    single = isinstance(targets, V.Var)
    out = backprop(loss, V.full(list(loss.shape), 1, loss.dtype if loss.dtype.is_float() else "float32"), [targets] if single else list(targets))
    return out[0] if single else out
