"""Replayed graphs (csrc/host.cpp): a graph synced for the second and third time, with other inputs, gives the bits the
planner's own run of it gives -- across shared sub-expressions, by-products, constants, in-place running statistics,
unaligned leaves, streams and threads."""
import threading

import pytest
import torch

import jittor_b200 as jt
from jittor_b200 import _capi as C, nn, pool
from jittor_b200 import var as V

pytestmark = pytest.mark.gpu


def data(seed, *shape, dtype=torch.float32, skew=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = 1
    for s in shape:
        n *= s
    return jt.array(torch.randn(n + skew, generator=g, device="cuda").to(dtype)[skew:].view(*shape))


def chain(s, skew):
    x, w = data(s, 33, 65, skew=skew), data(s + 1, 65)
    u = nn.relu(x * w + 0.5)
    return [u, (u * u).sum(1), u + u, x.reshape([65, 33])]


def softmax(s, skew):
    x, dy = data(s, 20, 300, skew=skew), data(s + 1, 20, 300)
    y = nn.softmax(x, -1)
    return [y, jt.grad((y * dy).sum(), x)]


def block(s, skew):
    x, w = data(s, 4, 64, 14, 14, dtype=torch.bfloat16, skew=skew), data(s + 1, 64, 64, 3, 3, dtype=torch.bfloat16)
    bn = nn.BatchNorm(64)
    with jt.flag_scope(amp_reg=2):
        y = nn.relu(bn(nn.conv2d(x, w, None, 1, 1)))
        return [y] + jt.grad((y * data(s + 2, 4, 64, 14, 14, dtype=torch.bfloat16)).sum(), [x, w, bn.weight, bn.bias]) + [bn.running_mean, bn.running_var]


def pooled(s, skew):
    x = data(s, 2, 3, 17, 18, skew=skew)
    y = pool.max_pool2d(x, 3, 2, 1)
    return [y, jt.grad((y * data(s + 1, 2, 3, 9, 9)).sum(), x)]


def rows(s, skew):
    t = data(s, 50, 24, skew=skew)
    r = t[jt.array(torch.arange(7, device="cuda", dtype=torch.int32) * 5)]
    return [r, jt.grad((r * data(s + 1, 7, 24)).sum(), t), t.setitem((slice(2, 9),), 1.5)]


def values(outs):
    jt.sync(outs)
    return [v.torch().clone() for v in outs]


@pytest.mark.parametrize("skew", [0, 1])
@pytest.mark.parametrize("graph", [chain, softmax, block, pooled, rows])
def test_replay_gives_the_planners_bits(graph, skew):
    want = []
    for s in (1, 5, 9):
        C.host.clear()                                        # planned
        want.append(values(graph(s, skew)))
    before = C.host.stats()["replayed"]
    C.host.clear()
    got = [values(graph(s, skew)) for s in (1, 5, 9)]         # planned once, replayed twice
    assert C.host.stats()["replayed"] >= before + 2
    for a, b in zip(want, got):
        for x, y in zip(a, b):
            if graph is block:                                # its statistics are summed with atomics
                assert (x.float() - y.float()).norm() <= 1e-3 * x.float().norm()
            else:
                assert torch.equal(x, y)


def pair(s, sharing):
    """Two leaves of one structure: of their own, or in one memory."""
    if sharing == "overlap":
        t = data(s, 80).torch()
        return jt.array(t[:64].view(4, 16)), jt.array(t[16:].view(4, 16))
    a = data(s, 4, 16)
    if sharing == "assign":
        return a, data(s + 1, 4, 16).assign(a)
    if sharing == "reshape":
        return a, a.reshape([64]).sync().reshape([4, 16]).sync()
    if sharing == "tensor":
        return a, jt.array(a.torch())
    return a, data(s + 1, 4, 16)


@pytest.mark.parametrize("first,second", [(k, "own") for k in ("assign", "reshape", "tensor", "overlap")]
                         + [("own", k) for k in ("assign", "reshape", "tensor", "overlap")] + [("overlap", "tensor"), ("tensor", "overlap")])
def test_leaves_that_share_memory_are_a_graph_of_their_own(first, second):
    def run(s, sharing):
        a, b = pair(s, sharing)
        return values([(a - b) * data(s + 2, 4, 16), a + a, b.sum(1), b.reshape([2, 32])])
    want = []
    for s, sharing in ((1, first), (5, second), (9, first)):
        C.host.clear()
        want.append(run(s, sharing))
    C.host.clear()
    for w, (s, sharing) in zip(want, ((1, first), (5, second), (9, first))):
        assert all(torch.equal(x, y) for x, y in zip(w, run(s, sharing)))


def test_threads_and_streams_share_the_tapes():
    want = {s: values(softmax(s, 0)) for s in range(4)}
    bad = []

    def work(s):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(20):
                got = values(softmax(s, 0))
                torch.cuda.current_stream().synchronize()
                if not all(torch.equal(a, b) for a, b in zip(want[s], got)):
                    bad.append(s)

    C.host.clear()
    ts = [threading.Thread(target=work, args=(s,)) for s in range(4)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not bad


class Handle:
    """Stands for a collective in flight: waiting for it lets another thread run."""
    def __init__(self, meanwhile):
        self.meanwhile = meanwhile

    def wait(self):
        t = threading.Thread(target=self.meanwhile)
        t.start()
        t.join()


@pytest.mark.parametrize("meanwhile", ["replay", "other", "clear"])
def test_a_wait_lets_other_threads_into_the_tapes(meanwhile):
    """A leaf that is still in flight is waited for before a tape is touched; what runs meanwhile does not disturb it."""
    want, other, seen = values(softmax(3, 0)), values(softmax(7, 0)), []

    def run():
        if meanwhile == "clear":
            C.host.clear()
        else:
            seen.append(values(softmax(7, 0) if meanwhile == "replay" else softmax(7, 1)))

    values(softmax(1, 0))                                     # recorded
    x, dy = data(3, 20, 300), data(4, 20, 300)
    x._pending, dy._pending = Handle(run), Handle(run)
    y = nn.softmax(x, -1)
    got = values([y, jt.grad((y * dy).sum(), x)])
    assert x._pending is None and dy._pending is None
    assert all(torch.equal(a, b) for a, b in zip(want, got))
    if meanwhile == "replay":
        assert len(seen) == 2 and all(torch.equal(a, b) for s in seen for a, b in zip(other, s))


class limited_memory:
    """Allocations beyond `spare` bytes fail, as on a GPU that is full."""
    def __init__(self, spare):
        self.spare = spare

    def __enter__(self):
        torch.cuda.empty_cache()
        total = torch.cuda.get_device_properties(0).total_memory
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + self.spare) / total)

    def __exit__(self, *exc):
        torch.cuda.set_per_process_memory_fraction(1.0)


def test_running_out_of_memory_is_the_same_error_from_planner_and_replay():
    x = data(1, 1, 1 << 20)
    graph = lambda: (x * 3.0).broadcast([64, 1 << 20]).reindex([64, 1 << 20], ["i0", f"{(1 << 20) - 1}-i1"])
    for prepared in (False, True):
        C.host.clear()
        if prepared:
            want = graph().sync().torch().clone()             # recorded
        with limited_memory(32 << 20), pytest.raises(torch.OutOfMemoryError):
            graph().sync()
        assert graph().sync().numel() == 64 << 20             # and it runs once there is room
    assert torch.equal(graph().torch(), want)


# float32: operands split into parts; bfloat16: partial sums of a split K; an odd K needs room for operands at TMA's pitch besides
@pytest.mark.parametrize("m,k,n,dtype,spare", [(2048, 2048, 2048, torch.float32, 20 << 20), (512, 16384, 512, torch.bfloat16, 4 << 20), (512, 16383, 512, torch.bfloat16, 22 << 20)])
def test_a_product_runs_where_there_is_no_room_for_all_its_scratch(m, k, n, dtype, spare):
    x, w = data(1, m, k, dtype=dtype), data(2, k, n, dtype=dtype)
    out = torch.empty(m, n, dtype=dtype, device="cuda")
    args = (C.desc(x.torch()), C.desc(w.torch()), C.desc(out), 0, 0)
    assert C.lib.b200jt_matmul_least_workspace(*args) < spare < C.lib.b200jt_matmul_workspace(*args) + out.numel() * out.element_size()
    want = x.torch().double() @ w.torch().double()
    del out
    for prepared in (False, True):
        C.host.clear()
        if prepared:
            nn.matmul(x, w).sync()                            # recorded
        with limited_memory(spare):
            y = nn.matmul(x, w).sync()
        assert (y.torch().double() - want).norm() <= (1e-5 if dtype == torch.float32 else 2.0 ** -8) * want.norm()
        for _ in range(2):                                    # and with its scratch once there is room
            assert (nn.matmul(x, w).torch().double() - want).norm() <= (1e-5 if dtype == torch.float32 else 2.0 ** -8) * want.norm()


@pytest.mark.parametrize("prepared", [False, True])
def test_running_statistics_move_once_when_a_later_step_fails(prepared):
    x = torch.randn(4, 16, 8, 8, device="cuda") + 0.3

    def graph():
        bn = nn.BatchNorm(16)
        y = nn.relu(bn(jt.array(x)))
        return bn, y, (y.reshape([1, 4096]) * 2.0).broadcast([1 << 14, 4096]).reindex([1 << 14, 4096], ["i0", "4095-i1"])
    C.host.clear()
    if prepared:
        jt.sync(list(graph()[1:]))
    bn, y, wide = graph()
    with limited_memory(32 << 20), pytest.raises(torch.OutOfMemoryError):
        jt.sync([y, wide])
    jt.sync([y, wide])
    want = 0.1 * x.double().mean((0, 2, 3))
    assert (bn.running_mean.torch().double() - want).abs().max() <= 1e-6


def test_recording_takes_no_more_memory_than_planning():
    """Temporaries and workspaces (here the channels-last copies) are freed as they are when nothing is recorded."""
    from jittor_b200 import executor
    w = [data(k, 64, 64, 3, 3, dtype=torch.bfloat16) for k in range(4)]

    def peak(run):
        x = data(9, 16, 64, 56, 56, dtype=torch.bfloat16)
        y = x
        for k in w:
            y = nn.conv2d(y, k, None, 1, 1)
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        base = torch.cuda.memory_allocated()
        run([y])
        return torch.cuda.max_memory_allocated() - base
    planned = peak(executor._realize)
    C.host.clear()
    assert peak(executor.realize) <= planned                  # recorded
    assert peak(executor.realize) <= planned                  # replayed


def test_a_number_that_changes_is_not_recorded_for_ever():
    x = data(1, 8, 32)
    C.host.clear()
    before = C.host.stats()
    for k in range(100):
        got = values([x * (1.0 + k) + 0.5, V.full([8, 32], k) * x])
        assert torch.equal(got[0], x.torch() * (1.0 + k) + 0.5) and torch.equal(got[1], x.torch() * k)
    after = C.host.stats()
    assert after["recorded"] - before["recorded"] <= 16 and after["tapes"] <= 16
    values([x * 3.0 + 0.5, V.full([8, 32], 2) * x])          # k = 2: one of the recorded ones
    assert C.host.stats()["replayed"] == after["replayed"] + 1


def test_a_graph_in_use_outlives_endless_shapes():
    x = data(1, 1, 5000)
    hot = lambda: (x * 2.0).sum(1).sync()
    C.host.clear()
    hot()
    before = C.host.stats()["recorded"]
    for n in range(1, 4301):
        jt.array(x.torch()[:, :n]).exp().sync()
        if n % 256 == 0:
            hot()
    stats = C.host.stats()
    assert stats["recorded"] == before + 4300 and stats["tapes"] <= 4096


def test_a_recorded_launch_keeps_what_its_error_is_called():
    t = torch.ones(8, device="cuda")
    C.recorder = C.Recorder([t])
    try:
        C.call("b200jt_unary", C.desc(t), C.desc(t), b"negative", what=lambda: "negative [8]")
        step = C.recorder.steps[-1]
    finally:
        C.recorder = None
    assert step[0] == "call" and step[4] == "negative [8]"


@pytest.mark.parametrize("kind", ["sgd", "nesterov", "adam", "adamw", "rmsprop"])
def test_many_tensor_update_has_the_bits_of_the_op_by_op_rule(kind):
    from jittor_b200 import optim

    def steps(together):
        make = {"sgd": lambda p: optim.SGD(p, 0.1, momentum=0.9, weight_decay=1e-3, dampening=0.2), "nesterov": lambda p: optim.SGD(p, 0.1, 0.9, nesterov=True),
                "adam": lambda p: optim.Adam(p, 1e-2, weight_decay=1e-3), "adamw": lambda p: optim.AdamW(p, 1e-2, weight_decay=1e-2),
                "rmsprop": lambda p: optim.RMSprop(p)}[kind]
        shapes = [(1,), (3,), (7, 5), (2048,), (2049,), (64, 100)] + [(k + 1,) for k in range(60)]         # more than one launch takes
        params = [data(k, *s) for k, s in enumerate(shapes)]
        opt = make(params)
        if not together:
            opt._step_together = lambda *a: False
        for k in range(3):
            loss = None
            for p in params:
                term = (p * p * p).sum()
                loss = term if loss is None else loss + term
            opt.step(loss)
        return [p.torch().clone() for p in params]
    for a, b in zip(steps(True), steps(False)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("kind", ["sgd", "adam"])
def test_a_parameter_kept_from_a_step_keeps_little_else(kind):
    from jittor_b200 import optim
    params = [data(1, 1024, 4096), data(2, 10), data(3, 300, 1000), data(4, 7)]
    opt = optim.SGD(params, 0.1, momentum=0.9) if kind == "sgd" else optim.Adam(params, 1e-3)
    kept = []

    def step():
        loss = None
        for p in params:
            loss = (p * p).sum() if loss is None else loss + (p * p).sum()
        opt.step(loss)
    step()
    step()
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    for _ in range(6):
        step()
        kept += [params[1].torch(), params[3].torch()]
    assert torch.cuda.memory_allocated() - before <= 12 << 20           # two buffers of at most 1 MB a step; the weights are 17 MB


@pytest.mark.parametrize("rows,dim,vocab,skew", [(1, 16, 5, 0), (3, 17, 2, 0), (127, 16, 3, 1), (129, 36, 40, 0), (1000, 64, 7, 0), (2500, 132, 900, 0), (40000, 20, 11, 0),
                                                 (90000, 128, 3000, 0)])
def test_row_gather_and_folded_row_scatter(rows, dim, vocab, skew):
    table, dy = data(1, vocab, dim, skew=skew), data(2, rows, dim, skew=skew)
    idx = jt.array(torch.randint(0, vocab, (rows,), device="cuda", dtype=torch.int32))
    r = table[idx]
    g = jt.grad((r * dy).sum(), table)
    jt.sync([r, g])
    at = idx.torch().long()
    assert torch.equal(r.torch(), table.torch()[at])
    want = torch.zeros(vocab, dim, device="cuda", dtype=torch.float64)
    want.index_add_(0, at, dy.torch().double())
    assert (g.torch().double() - want).norm() <= 1e-5 * want.norm()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("k,s,p", [(2, 2, 0), (3, 2, 1), (3, 2, 0), (3, 1, 1), (3, 1, 0), (5, 3, 2)])
@pytest.mark.parametrize("h,w", [(6, 7), (8, 8), (9, 16), (17, 12), (33, 20)])
def test_pool_tiles_against_torch(h, w, k, s, p, dtype):
    x = (torch.randint(-9, 9, (2, 3, h, w), device="cuda").float() / 4).to(dtype)              # ties: the first element wins
    vx = jt.array(x)
    for op, ref in (("maximum", torch.nn.functional.max_pool2d), ("minimum", lambda t, *a: -torch.nn.functional.max_pool2d(-t, *a)),
                    ("mean", torch.nn.functional.avg_pool2d)):
        y = pool.Pool(k, s, p, op=op)(vx)
        xt = x.double().requires_grad_()
        yt = ref(xt, k, s, p)
        dy = torch.randn(yt.shape, device="cuda").to(dtype)
        dx = jt.grad((y * jt.array(dy)).sum(), vx)
        jt.sync([y, dx])
        yt.backward(dy.double())
        tol = 1e-6 if dtype == torch.float32 else 1e-2
        assert (y.torch().double() - yt.detach()).abs().max() <= tol * (1 + yt.detach().abs().max())
        assert (dx.torch().double() - xt.grad).abs().max() <= tol * (1 + xt.grad.abs().max())
