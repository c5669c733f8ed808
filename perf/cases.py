"""Performance cases: what programs written against this package have it do, one case per kind of call and size.

A case is a dict of plain values; `kind` names the path, the rest its sizes, data type and options. `listed()` holds the
sizes of the benchmark configurations (config 0-4 and the callers of the path) with an ordinary or ragged size beside
them, `draw()` samples the same kinds over the ranges they stand for: small calls where the launch path counts, sizes
that are no multiple of any tile, both directions, float32 and bfloat16.

    conv        nn.conv2d, forward or with both gradients (data, weights)
    block       nn.conv2d -> BatchNorm (training statistics) -> relu, forward or with the gradients of x, w, gamma, beta
    linear      nn.matmul forward and both gradients (a dense layer's training step without the optimiser)
    softmax     nn.softmax / log_softmax over the last axis, forward and backward
    layernorm   nn.layer_norm with affine parameters, forward and the gradients of x, gamma, beta
    scatter     Var.reindex_reduce of a value list into bins by an index Var
    pool        pool.max_pool2d / avg_pool2d forward and backward
    embedding   table[idx] and the gradient of the table
    net         one optimiser step of a small convolutional classifier
"""
import math

import torch

import jittor_b200 as jt
from jittor_b200 import nn, optim, pool

_TORCH = {"f32": torch.float32, "bf16": torch.bfloat16, "int32": torch.int32}
_BYTES = {"f32": 4, "bf16": 2, "int32": 4}


def listed():
    return [
        # config 0: the convolution at the size the reference's CPU path runs; 1.6 MB, so launch latency counts
        dict(name="conv-f32-small", kind="conv", dtype="f32", n=4, c=32, h=32, w=32, co=64, k=3, stride=1, train=False),
        # config 4: a ResNet-50 stage layer with training BatchNorm and ReLU at the full batch
        dict(name="block-bf16-stage", kind="block", dtype="bf16", n=256, c=256, h=56, w=56, co=256, k=3, stride=1, train=False),
        # the training pass of an ordinary residual-network layer: forward, data and weight gradients, BatchNorm gradients
        dict(name="block-bf16-train", kind="block", dtype="bf16", n=64, c=128, h=28, w=28, co=128, k=3, stride=1, train=True),
        # config 3's second shape as a dense layer's training pass
        dict(name="linear-bf16-large", kind="linear", dtype="bf16", m=16384, k=4096, n=4096),
        # a ragged dense layer in the reference's default type (a classifier head over a batch)
        dict(name="linear-f32-ragged", kind="linear", dtype="f32", m=500, k=777, n=1000),
        # config 2: attention / classifier rows in bf16
        dict(name="softmax-bf16-large", kind="softmax", dtype="bf16", rows=32768, cols=4096, log=False),
        # rows of an ordinary ragged batch, with the parameter gradients
        dict(name="layernorm-f32-ragged", kind="layernorm", dtype="f32", rows=5000, cols=1001),
        # config 1 (a): integer counts into many bins
        dict(name="scatter-int-uniform", kind="scatter", dtype="int32", op="add", n=1 << 24, bins=1 << 20, zipf=False),
        # config 1 (b): float sums into few bins with a skewed index distribution
        dict(name="scatter-f32-zipf", kind="scatter", dtype="f32", op="add", n=1 << 24, bins=4096, zipf=True),
        # the stem pooling of a residual network, forward and backward
        dict(name="pool-f32-large", kind="pool", dtype="f32", op="maximum", n=64, c=128, h=112, w=112, k=3, stride=2, pad=1),
        # an embedding lookup of a batch of sequences and the table's gradient
        dict(name="embedding-f32", kind="embedding", vocab=50000, dim=256, picks=8192),
        # a whole training step where every call is small
        dict(name="net-step-small", kind="net", opt="sgd", batch=16, side=32, c1=16, c2=32, classes=10),
    ]


# ------------------------------------------------------------------------------------------------ drawn cases
def _log(rng, lo, hi):
    """A whole number spread over [lo, hi] by its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _size(rng, lo, hi):
    """Like _log; a third of them as they fall (odd ones among them), the rest multiples of 8 or 64 as layers have them."""
    v = _log(rng, lo, hi)
    step = rng.choice((1, 8, 64))
    return max(lo, min(hi, v // step * step)) if v >= step else v


def draw(rng):
    kind = rng.choice(("conv", "block", "linear", "softmax", "layernorm", "scatter", "pool", "embedding", "net"))
    dtype = rng.choice(("f32", "bf16"))
    if kind == "conv":
        while True:
            h = _log(rng, 7, 64)
            c = dict(kind=kind, dtype="f32", n=_log(rng, 1, 64), c=_size(rng, 3, 128), h=h, w=max(7, h + rng.choice((0, 0, 1, -3))),
                     co=_size(rng, 8, 128), k=rng.choice((1, 3, 3, 5)), stride=rng.choice((1, 1, 2)), train=rng.random() < 0.5)
            if work(c)["flops"] <= 2e10:
                return c
    if kind == "block":
        while True:
            h = rng.choice((7, 14, 28, 56, _log(rng, 7, 56)))
            c = dict(kind=kind, dtype=rng.choice(("bf16", "bf16", "f32")), n=_log(rng, 1, 256), c=_size(rng, 16, 512), h=h, w=h,
                     co=_size(rng, 16, 512), k=rng.choice((1, 3, 3)), stride=rng.choice((1, 1, 2)), train=rng.random() < 0.6)
            # float32 training is in `conv` and `net`: an activation whose last bit decides its sign would decide this comparison
            c["train"] = c["train"] and c["dtype"] == "bf16"
            if work(c)["flops"] <= (4e11 if c["dtype"] == "bf16" else 2e10):
                return c
    if kind == "linear":
        while True:
            c = dict(kind=kind, dtype=dtype, m=_size(rng, 16, 16384), k=_size(rng, 32, 4096), n=_size(rng, 10, 4096))
            if work(c)["flops"] <= (1.6e12 if dtype == "bf16" else 1e11):
                return c
    if kind in ("softmax", "layernorm"):
        while True:
            c = dict(kind=kind, dtype=dtype, rows=_size(rng, 16, 65536), cols=_size(rng, 16, 16384))
            if c["rows"] * c["cols"] <= 1 << 27:
                return dict(c, log=rng.random() < 0.5) if kind == "softmax" else c
    if kind == "scatter":
        return dict(kind=kind, dtype=rng.choice(("int32", "f32")), op=rng.choice(("add", "add", "maximum")), n=_log(rng, 1 << 10, 1 << 24),
                    bins=_log(rng, 16, 1 << 20), zipf=rng.random() < 0.5)
    if kind == "pool":
        k, stride, pad = rng.choice(((2, 2, 0), (3, 2, 1), (3, 1, 1)))
        while True:
            h = _log(rng, 8, 112)
            c = dict(kind=kind, dtype=dtype, op=rng.choice(("maximum", "maximum", "mean")), n=_log(rng, 1, 64), c=_size(rng, 16, 256),
                     h=h, w=max(8, h + rng.choice((0, 0, 1))), k=k, stride=stride, pad=pad)
            if c["n"] * c["c"] * c["h"] * c["w"] <= 64 * 128 * 112 * 112:
                return c
    if kind == "embedding":
        while True:
            c = dict(kind=kind, vocab=_log(rng, 1000, 1 << 18), dim=_size(rng, 16, 1024), picks=_log(rng, 64, 1 << 17))
            if max(c["vocab"], c["picks"]) * c["dim"] <= 1 << 26:
                return c
    return dict(kind="net", opt=rng.choice(("sgd", "adam")), batch=_log(rng, 4, 64), side=rng.choice((16, 24, 28, 32)), c1=_log(rng, 8, 32),
                c2=_log(rng, 16, 64), classes=rng.choice((2, 10, 100)))


# ------------------------------------------------------------------------------------------------ states
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _randn(g, shape, dtype="f32", scale=1.0):
    return jt.array((torch.randn(*shape, generator=g, device="cuda") * scale).to(_TORCH[dtype]))


def _indices(g, n, bins, zipf):
    """Bin numbers of n values: uniform, or skewed by Zipf(1.1) over a random order of the bins."""
    if not zipf:
        return torch.randint(0, bins, (n,), generator=g, device="cuda", dtype=torch.int32)
    cdf = torch.arange(1, bins + 1, device="cuda", dtype=torch.float64).pow_(-1.1).cumsum_(0)
    rank = torch.searchsorted(cdf, torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * cdf[-1]).clamp_(max=bins - 1)
    return torch.randperm(bins, generator=g, device="cuda")[rank].to(torch.int32)


def _out_side(side, k, stride, pad):
    return (side + 2 * pad - k) // stride + 1


class _Classifier(nn.Module):
    """conv 3x3 -> relu -> max-pool, twice, then a dense layer: the smallest network that uses every kind of layer."""

    def __init__(self, g, side, c1, c2, classes):
        self.conv1, self.conv2 = nn.Conv(3, c1, 3, padding=1), nn.Conv(c1, c2, 3, padding=1)
        self.conv1.weight, self.conv1.bias = _randn(g, (c1, 3, 3, 3), scale=27 ** -0.5), _randn(g, (c1,), scale=0.05)
        self.conv2.weight, self.conv2.bias = _randn(g, (c2, c1, 3, 3), scale=(9 * c1) ** -0.5), _randn(g, (c2,), scale=0.05)
        self.features = c2 * (side // 4) ** 2
        self.weight, self.bias = _randn(g, (self.features, classes), scale=self.features ** -0.5), _randn(g, (classes,), scale=0.05)

    def execute(self, x):
        x = pool.max_pool2d(nn.relu(self.conv1(x)), 2, 2)
        x = pool.max_pool2d(nn.relu(self.conv2(x)), 2, 2)
        return nn.matmul(x.reshape((-1, self.features)), self.weight) + self.bias


def prepare(case, seed):
    g, c = _gen(seed), case
    kind, s = c["kind"], {"case": case}
    if kind in ("conv", "block"):
        o = [_out_side(c[a], c["k"], c["stride"], c["k"] // 2) for a in ("h", "w")]
        s["x"] = _randn(g, (c["n"], c["c"], c["h"], c["w"]), c["dtype"])
        s["w"] = _randn(g, (c["co"], c["c"], c["k"], c["k"]), c["dtype"], (2 / (c["k"] ** 2 * c["c"])) ** 0.5)
        if c["train"]:
            s["dy"] = _randn(g, (c["n"], c["co"], *o), c["dtype"])
        if kind == "block":
            s["bn"] = nn.BatchNorm(c["co"], is_train=True, sync=True)
            s["bn"].weight = jt.array(1 + 0.02 * torch.randn(c["co"], generator=g, device="cuda"))
            s["bn"].bias = _randn(g, (c["co"],), scale=0.1)
    elif kind == "linear":
        s["x"], s["w"] = _randn(g, (c["m"], c["k"]), c["dtype"]), _randn(g, (c["k"], c["n"]), c["dtype"], c["k"] ** -0.5)
        s["dy"] = _randn(g, (c["m"], c["n"]), c["dtype"])
    elif kind in ("softmax", "layernorm"):
        s["x"], s["dy"] = _randn(g, (c["rows"], c["cols"]), c["dtype"]), _randn(g, (c["rows"], c["cols"]), c["dtype"])
        if kind == "layernorm":
            s["gamma"] = jt.array(1 + 0.02 * torch.randn(c["cols"], generator=g, device="cuda"))
            s["beta"] = _randn(g, (c["cols"],), scale=0.1)
    elif kind == "scatter":
        if c["dtype"] == "int32":
            s["x"] = jt.array(torch.randint(0, 100, (c["n"],), generator=g, device="cuda", dtype=torch.int32))
        else:
            s["x"] = _randn(g, (c["n"],))
        s["idx"] = jt.array(_indices(g, c["n"], c["bins"], c["zipf"]))
    elif kind == "pool":
        s["x"] = _randn(g, (c["n"], c["c"], c["h"], c["w"]), c["dtype"])
        s["dy"] = _randn(g, (c["n"], c["c"], *(_out_side(c[a], c["k"], c["stride"], c["pad"]) for a in ("h", "w"))), c["dtype"])
    elif kind == "embedding":
        s["table"] = _randn(g, (c["vocab"], c["dim"]))
        s["idx"] = jt.array(_indices(g, c["picks"], c["vocab"], True))
        s["dy"] = _randn(g, (c["picks"], c["dim"]))
    else:
        s["net"] = _Classifier(g, c["side"], c["c1"], c["c2"], c["classes"])
        params = s["net"].parameters()
        s["opt"] = optim.SGD(params, 0.01, momentum=0.9) if c["opt"] == "sgd" else optim.Adam(params, 1e-3)
        s["x"] = _randn(g, (c["batch"], 3, c["side"], c["side"]))
        label = torch.randint(0, c["classes"], (c["batch"],), generator=g, device="cuda")
        s["onehot"] = jt.array(torch.nn.functional.one_hot(label, c["classes"]).float())
    return s


def _results(*outs):
    jt.sync(outs)
    return [v.torch() for v in outs]


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "conv":
        y = nn.conv2d(s["x"], s["w"], None, c["stride"], c["k"] // 2)
        if not c["train"]:
            return _results(y)
        return _results(y, *jt.grad((y * s["dy"]).sum(), [s["x"], s["w"]]))
    if kind == "block":
        bn = s["bn"]
        with jt.flag_scope(amp_reg=2):                  # 16-bit activations stay 16-bit
            y = nn.relu(bn(nn.conv2d(s["x"], s["w"], None, c["stride"], c["k"] // 2)))
            outs = [y]
            if c["train"]:
                outs += jt.grad((y * s["dy"]).sum(), [s["x"], s["w"], bn.weight, bn.bias])
            return _results(*outs) + [bn.running_mean.torch(), bn.running_var.torch()]
    if kind == "linear":
        y = nn.matmul(s["x"], s["w"])
        return _results(y, *jt.grad((y * s["dy"]).sum(), [s["x"], s["w"]]))
    if kind == "softmax":
        y = nn.log_softmax(s["x"], -1) if c["log"] else nn.softmax(s["x"], -1)
        return _results(y, jt.grad((y * s["dy"]).sum(), s["x"]))
    if kind == "layernorm":
        y = nn.layer_norm(s["x"], (c["cols"],), s["gamma"], s["beta"])
        return _results(y, *jt.grad((y * s["dy"]).sum(), [s["x"], s["gamma"], s["beta"]]))
    if kind == "scatter":
        return _results(s["x"].reindex_reduce(c["op"], [c["bins"]], ["@e0(i0)"], extras=[s["idx"]]))
    if kind == "pool":
        f = pool.max_pool2d if c["op"] == "maximum" else pool.avg_pool2d
        y = f(s["x"], c["k"], c["stride"], c["pad"])
        return _results(y, jt.grad((y * s["dy"]).sum(), s["x"]))
    if kind == "embedding":
        rows = s["table"][s["idx"]]
        return _results(rows, jt.grad((rows * s["dy"]).sum(), s["table"]))
    loss = -(nn.log_softmax(s["net"](s["x"]), -1) * s["onehot"]).sum(1).mean()
    s["opt"].step(loss)
    return _results(loss, *s["net"].parameters())


# ------------------------------------------------------------------------------------------------ work and tolerance
def work(case):
    c = case
    kind, b = c["kind"], _BYTES[c.get("dtype", "f32")]
    if kind in ("conv", "block"):
        o = [_out_side(c[a], c["k"], c["stride"], c["k"] // 2) for a in ("h", "w")]
        x, w, y = c["n"] * c["c"] * c["h"] * c["w"], c["co"] * c["c"] * c["k"] ** 2, c["n"] * c["co"] * o[0] * o[1]
        flops = 2 * y * c["c"] * c["k"] ** 2
        small = 4 * 6 * c["co"] if kind == "block" else 0
        if not c["train"]:
            return {"bytes": b * (x + w + y) + small, "flops": flops}
        return {"bytes": b * 2 * (x + w + y) + small, "flops": 3 * flops}
    if kind == "linear":
        m, k, n = c["m"], c["k"], c["n"]
        return {"bytes": 2 * b * (m * k + k * n + m * n), "flops": 6 * m * k * n}
    if kind in ("softmax", "layernorm"):
        n = c["rows"] * c["cols"]
        return {"bytes": 4 * b * n + (16 * c["cols"] if kind == "layernorm" else 0), "flops": 16 * n}
    if kind == "scatter":
        return {"bytes": 8 * c["n"] + 4 * c["bins"], "flops": c["n"]}
    if kind == "pool":
        x = c["n"] * c["c"] * c["h"] * c["w"]
        y = c["n"] * c["c"] * _out_side(c["h"], c["k"], c["stride"], c["pad"]) * _out_side(c["w"], c["k"], c["stride"], c["pad"])
        return {"bytes": 2 * b * (x + y), "flops": 2 * y * c["k"] ** 2}
    if kind == "embedding":
        # distinct rows read at most once each, the picked rows written, dy read, the whole gradient table written
        rows = min(c["vocab"], c["picks"])
        return {"bytes": 4 * (c["dim"] * (rows + 2 * c["picks"] + c["vocab"]) + c["picks"]), "flops": c["picks"] * c["dim"]}
    p1, p2 = c["side"] ** 2, (c["side"] // 2) ** 2
    feat = c["c2"] * (c["side"] // 4) ** 2
    flops = 6 * c["batch"] * (p1 * 27 * c["c1"] + p2 * 9 * c["c1"] * c["c2"] + feat * c["classes"])
    params = 27 * c["c1"] + 9 * c["c1"] * c["c2"] + feat * c["classes"] + c["c1"] + c["c2"] + c["classes"]
    state = 4 if c["opt"] == "sgd" else 6
    return {"bytes": 4 * (params * state + c["batch"] * 3 * p1), "flops": flops}


def tolerance(case):
    c = case
    if c["kind"] == "scatter" and (c["dtype"] == "int32" or c["op"] == "maximum"):
        return "exact"
    if c.get("dtype") == "bf16":
        return {"rel": 1e-2}
    if c["kind"] == "net":
        return {"rel": 1e-5, "max": 1e-3}       # Adam's first steps turn a gradient's last bits into whole steps where it is nearly zero
    return {"rel": 1e-5}
