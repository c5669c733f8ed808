"""What a Var holds besides its value: copies and pickles of it, assignment over it, which layers carry a record,
which Vars a gradient reaches, what a producer that fails raises. No GPU: the values are CPU tensors that nothing computes with."""
import copy
import pickle

import numpy as np
import pytest
import torch

import jittor_b200 as jt
from jittor_b200 import nn, pool
from jittor_b200 import var as V


def leaf(*shape, dtype=torch.float32):
    t = torch.arange(int(np.prod(shape)), dtype=torch.float32).reshape(shape).to(dtype)
    return V.Var(list(shape), str(dtype).split(".")[1], data=t)


def layers():
    x = leaf(2, 3, 8, 8)
    bn = nn.BatchNorm(3)
    return {"leaf": x, "expression": (x * 2.0 + x).sum(1), "constant": jt.array(2.5), "conv2d": nn.conv2d(x, leaf(4, 3, 3, 3), None, 1, 1),
            "matmul": nn.matmul(leaf(4, 5), leaf(5, 6)), "softmax": nn.softmax(x, -1), "layer_norm": nn.layer_norm(x, (8,), leaf(8), leaf(8)),
            "batch_norm_relu": nn.relu(bn(x)), "index": x[1], "mean_pool": pool.avg_pool2d(x, 2, 2)}


def same(a, b):
    assert list(a.shape) == list(b.shape) and a.dtype == b.dtype and a.is_scalar == b.is_scalar and a._const == b._const
    assert a.is_stop_grad() == b.is_stop_grad() and a.is_stop_fuse() == b.is_stop_fuse() and a.name() == b.name()
    assert (a._data is None) == (b._data is None) and (a._data is None or torch.equal(a._data, b._data))
    assert (a._op is None) == (b._op is None) and (a._op is None or (a._op.kind == b._op.kind and len(a._op.inputs) == len(b._op.inputs)))


@pytest.mark.parametrize("how", [copy.copy, copy.deepcopy, lambda v: pickle.loads(pickle.dumps(v))], ids=["copy", "deepcopy", "pickle"])
@pytest.mark.parametrize("kind", sorted(layers()))
def test_copies_of_a_var(kind, how):
    v = layers()[kind]
    v.name("v")
    v.stop_grad()
    v.stop_fuse()
    v.compile_options["G"] = 1
    v.note = "kept"
    c = how(v)
    same(v, c)
    assert c is not v and c.note == "kept" and c.compile_options == {"G": 1}
    c.start_grad()
    assert v.is_stop_grad()


def test_copies_share_or_own_their_memory():
    x = leaf(3, 4)
    assert copy.copy(x)._data is x._data
    assert copy.deepcopy(x)._data.data_ptr() != x._data.data_ptr()
    pair = copy.deepcopy([x, x * 2.0])
    assert pair[1]._op.inputs[0] is pair[0]


def reaches(y, x):
    """Whether a gradient of y reaches x (a Var that none reaches gets zeros)."""
    g = jt.grad(y, x)
    return g._op.kind != "fill"


class Net(nn.Module):
    def __init__(self):
        self.norms, self.table, self.head = [nn.BatchNorm(4), nn.LayerNorm(6)], {"a": leaf(5, 2)}, leaf(2, 3)


@pytest.mark.parametrize("how", [copy.deepcopy, lambda m: pickle.loads(pickle.dumps(m))], ids=["deepcopy", "pickle"])
def test_copies_of_a_module(how):
    net = Net()
    twin = how(net)
    assert len(twin.parameters()) == len(net.parameters()) == 8
    for a, b in zip(net.parameters(), twin.parameters()):
        assert a is not b
        same(a, b)


def test_gradients_flow_through_a_copied_graph():
    """A deep copy of a layer's result and its input is differentiated with respect to the copied input."""
    x = leaf(4, 6)
    y = nn.softmax(x, -1)
    x2, y2 = copy.deepcopy((x, y))
    assert reaches(y2.sum(), x2) and not reaches(y2.sum(), x)
    assert reaches(copy.copy(y).sum(), x)


@pytest.mark.parametrize("kind", ["softmax", "log_softmax", "layer_norm", "matmul", "conv2d", "batch_norm", "batch_norm_relu", "mean_pool"])
def test_an_assigned_var_is_a_leaf(kind):
    """assign() over a layer's result: no gradient reaches the layer's input, in whatever way it is looked for."""
    x = leaf(8, 8) if kind == "matmul" else leaf(2, 4, 8, 8)
    y = {"softmax": lambda: nn.softmax(x, -1), "log_softmax": lambda: nn.log_softmax(x, -1), "layer_norm": lambda: nn.layer_norm(x, (8,), leaf(8), leaf(8)),
         "matmul": lambda: nn.matmul(x, leaf(8, 3)), "conv2d": lambda: nn.conv2d(x, leaf(4, 4, 3, 3), None, 1, 1), "batch_norm": lambda: nn.BatchNorm(4)(x),
         "batch_norm_relu": lambda: nn.relu(nn.BatchNorm(4)(x)), "mean_pool": lambda: pool.avg_pool2d(x, 2, 2)}[kind]()
    assert reaches(y.sum(), x)
    y.assign(leaf(3, 5))
    assert y._op is None and y._relay is None and y._vjp is None and y._bn_running is None and list(y.shape) == [3, 5]
    assert not reaches((y * y).sum(), x)


def test_a_constant_that_was_assigned_is_no_constant():
    s = jt.array(0.0)
    s.assign(leaf(1))
    assert s._const is None


def test_relu_of_an_assigned_norm_is_of_the_new_value():
    h = nn.BatchNorm(4)(leaf(2, 4, 8, 8))
    y = nn.relu(h)
    h.assign(leaf(2, 4, 8, 8))
    from jittor_b200 import relay
    assert relay.plan(y) is None and y._op.kind == "ternary" and y._op.inputs[1] is h


@pytest.mark.parametrize("weight,bias,recorded", [(1.0, 0.0, True), (1, 0, True), (2.0, 0.0, False), (1.0, 0.5, False), (0, 0, False), ((4,), (4,), True),
                                                  ((4,), 0.0, True), (2.0, (4,), False), ((1, 1), 0.0, False)])
def test_norms_with_numbers_for_parameters(weight, bias, recorded):
    """A record holds float32 parameters of the layer's shape or none; any other weight or bias goes into the graph."""
    def par(p):
        return leaf(*p) if isinstance(p, tuple) else p
    bn = nn.BatchNorm(4)
    bn.weight, bn.bias = par(weight), par(bias)
    if weight != (1, 1):
        assert (bn(leaf(2, 4, 3, 3))._relay is not None) == recorded
    ln = nn.LayerNorm(4)
    ln.weight, ln.bias = par(weight), par(bias)
    assert (ln(leaf(6, 4))._relay is not None) == recorded


def test_a_norm_refuses_parameters_that_its_graph_refuses():
    ln = nn.LayerNorm((4, 6))
    assert ln(leaf(2, 4, 6))._relay is not None
    ln.weight = leaf(24)
    with pytest.raises(ValueError):
        ln(leaf(2, 4, 6))
    bn = nn.BatchNorm(4)
    assert bn(leaf(2, 4, 3, 3))._relay is not None
    bn.weight = leaf(2, 2)
    with pytest.raises(ValueError):
        bn(leaf(2, 4, 3, 3))


def test_a_gradient_reaches_the_norm_under_a_relu():
    """relu(batch_norm(x)) is one record; its gradient still reaches the normalised Var, and ends there when told to."""
    x = leaf(2, 4, 3, 3)
    h = nn.BatchNorm(4)(x)
    y = nn.relu(h)
    assert reaches(y.sum(), h) and reaches(y.sum(), x)
    gh, gx = jt.grad((y * y).sum(), [h, x])
    assert gh._op.kind != "fill" and gx._op.kind == "fill"            # a target takes the gradient: it does not go on from there
    h.stop_grad()
    assert not reaches(y.sum(), x)
    h.start_grad()
    assert jt.grad(y.sum(), x)._relay[0] == "batch_norm_dx"           # one step where nothing asks for h
    h.assign(leaf(2, 4, 3, 3))
    assert not reaches(y.sum(), x) and reaches(y.sum(), h)


def test_a_producer_that_fails_raises_its_own_error_each_time():
    def build():
        raise ValueError("no such graph")
    v = V.LazyVar([2], "float32", build)
    for _ in range(3):
        with pytest.raises(ValueError, match="no such graph"):
            v._op
    with pytest.raises(ValueError, match="no such graph"):
        jt.grad((v * v).sum(), leaf(2))


@pytest.mark.gpu
def test_sync_of_a_producer_that_fails_raises_its_own_error():
    def build():
        raise ValueError("no such graph")
    with pytest.raises(ValueError, match="no such graph"):
        (V.LazyVar([2], "float32", build) * 2.0).sync()
