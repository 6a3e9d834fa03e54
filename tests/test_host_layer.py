"""CPU: tape, deferral and buffer bookkeeping of the host layer over a device in host memory
(fake_device.py), whose fresh memory is full of junk."""
import numpy as np
import pytest

import litenn_b200 as nn
from fake_device import fake_device


@pytest.fixture
def fake():
    with fake_device() as f:
        yield f
    assert not f.errors, f.errors


def _rand(*shape, seed=0):
    return np.random.default_rng(seed).standard_normal(shape).astype(np.float32)


# ---- a tensor that one call reads and overwrites is initialised first ----------------------------
@pytest.mark.parametrize("seed", [2.0, [1.0, 2.0, 3.0], np.full((4, 3), 2.0, np.float32)], ids=["number", "row", "full"])
def test_seeds_of_every_shape(fake, seed):
    w = nn.Tensor_from_value(_rand(4, 3))
    opt = nn.optimizer.SGD([w])
    y = w * 3.0
    for k in (1, 2):
        nn.backward({y: seed})
        np.testing.assert_array_equal(w.get_grad().np(), np.broadcast_to(np.float32(k * 3) * np.float32(seed), (4, 3)))
    del opt


@pytest.mark.parametrize("shape,call,want", [
    ((3, 4), lambda t, u: nn.op.mul_const_op(t, 3.0, output_t=t), lambda t, u: t * 3),
    ((3, 4), lambda t, u: nn.op.add_op(t, u, output_t=t), lambda t, u: t + u),
    ((3, 4), lambda t, u: nn.op.mul_op(u, t, output_t=t), lambda t, u: u * t),
    ((3, 4), lambda t, u: nn.op.add_op(t.reshape((6, 2)), u.reshape((6, 2)), output_t=t), lambda t, u: t + u),
    ((1, 2, 16), lambda t, u: nn.op.add_const_op(t * u[:, :, :1], 1.0, output_t=t), lambda t, u: t * u[:, :, :1] + 1),
], ids=["eltwise", "binary_a", "binary_b", "reference", "deferred"])
def test_output_that_is_an_input_too(fake, shape, call, want):
    t, u = nn.Tensor(shape, init=nn.initializer.Scalar(2.0)), nn.Tensor_from_value(_rand(*shape))
    call(t, u)
    np.testing.assert_array_equal(t.np(), want(np.full(shape, 2, np.float32), u.np()))


def test_output_that_a_deferred_convolution_reads(fake):
    x, kernel = nn.Tensor((1, 2, 8, 8)), nn.Tensor_from_value(_rand(2, 2, 3, 3))
    nn.op.add_const_op(nn.conv2D(x, kernel), 1.0, output_t=x)
    assert fake.calls.index("lnn_fill_f32") < fake.calls.index("lnn_conv2d_fwd_packed")


def test_overwritten_tensors_draw_their_random_numbers_in_order(fake):
    """An initializer that draws from np.random runs even where its values are lost, outputs first."""
    order = []

    class Drawn(nn.initializer.Initializer):
        def __init__(self, name):
            self.name = name

        def initialize_buffer(self, buf, shape):
            order.append(self.name)
            buf.fill(1.0)

    a, b, out = (nn.Tensor((3,), init=Drawn(n)) for n in ("a", "b", "out"))
    nn.op.add_op(a, b, output_t=out)
    assert order == ["out", "a", "b"]


# ---- gradients own what their launches point to ---------------------------------------------------
def test_more_slices_than_the_plan_cache_holds(fake):
    rows = nn.ops._slice_plan.cache_info().maxsize + 200
    x = nn.Tensor_from_value(_rand(rows + 1, 2))
    opt = nn.optimizer.SGD([x])
    parts = [x[i:i + 1] for i in range(rows)]
    nn.backward({p: float(i) for i, p in enumerate(parts)})
    got = x.get_grad().np()
    np.testing.assert_array_equal(got[:-1], np.repeat(np.arange(rows, dtype=np.float32)[:, None], 2, 1))
    assert not got[-1].any()
    del opt


# ---- kept gradients of a chain's intermediates, as the separate operators keep them ----------------
def _branches(n, hold, passes, keep, drop_at=None):
    """Gradients of x, g, b after `passes` over n activations of one x * g + b, in two lists as they are asked for."""
    x, g, b = (nn.Tensor_from_value(_rand(*s, seed=k)) for k, s in enumerate([(2, 3, 4, 4), (1, 3, 1, 1), (1, 3, 1, 1)]))
    opt = nn.optimizer.SGD([x, g, b])
    u = x * g + b
    ys = [nn.leaky_relu(u, 0.1 * (k + 1)) for k in range(n)]
    held = u if hold else None
    del u
    for which in passes:
        if drop_at is not None and which == drop_at:
            held = None
        nn.backward([ys[k] for k in which], **keep)
    if held is not None and keep:
        assert held.has_grad()
    return [t.get_grad().np() for t in (x, g, b)], opt


@pytest.mark.parametrize("keep", [{"keep_gradient_for_non_trainables": True}, {"grad_for_non_trainables": True}, {}],
                         ids=["keep", "non_trainables", "plain"])
@pytest.mark.parametrize("hold", [False, True], ids=["dropped", "held"])
@pytest.mark.parametrize("n,passes,drop_at", [
    (2, [(0, 1)], None), (3, [(0, 1, 2)], None), (2, [(0,), (1,)], None), (2, [(0,), (0, 1)], None),
    (2, [(0,), (1,)], (1,)), (1, [(0,), (0,)], None),
], ids=["two", "three", "one_by_one", "overlapping", "dropped_between", "twice"])
def test_gradients_of_branches(fake, n, passes, drop_at, hold, keep):
    with nn.deferred.disabled():
        want, _ = _branches(n, hold, passes, keep, drop_at)
    got, _ = _branches(n, hold, passes, keep, drop_at)
    for a, r, name in zip(got, want, ("dx", "dg", "db")):
        np.testing.assert_allclose(a, r, rtol=0, atol=1e-5 * np.abs(r).max(), err_msg=name)


def test_kept_gradient_lives_as_long_as_a_branch(fake):
    """The intermediate and what a pass kept for it go with the last tensor computed from it."""
    import gc
    gc.disable()
    try:
        before = nn._lib._native.tensor_count()
        grads = []
        for disabled in (True, False):
            with nn.deferred.disabled() if disabled else _nothing():
                x, g, b = (nn.Tensor_from_value(_rand(*s)) for s in [(1, 2, 16), (1, 2, 1), (1, 2, 1)])
                opt = nn.optimizer.SGD([x, g, b])
                u = x * g + b
                y1, y2 = nn.leaky_relu(u, 0.1), nn.leaky_relu(u, 0.2)
                nn.backward(y1, keep_gradient_for_non_trainables=True)
                del u, y1
                nn.backward(y2, keep_gradient_for_non_trainables=True)
                grads.append(x.get_grad().np())
                del x, g, b, y2, opt
        np.testing.assert_allclose(grads[1], grads[0], rtol=1e-6)
        assert nn._lib._native.tensor_count() == before, "no reference cycle keeps a tensor"
    finally:
        gc.enable()


def _nothing():
    import contextlib
    return contextlib.nullcontext()


# ---- a gradient tensor is the same object for as long as the gradient lives ------------------------
@pytest.mark.parametrize("seed", [None, "tensor", "array"])
@pytest.mark.parametrize("form", ["add", "sub", "leaf", "mul"])
def test_gradient_taken_before_the_pass(fake, form, seed):
    w, u = nn.Tensor_from_value(_rand(4, 3)), nn.Tensor_from_value(_rand(4, 3, seed=1))
    opt = nn.optimizer.SGD([w])
    g = w.get_grad()
    y = {"add": lambda: w + u, "sub": lambda: w - u, "leaf": lambda: w, "mul": lambda: w * u}[form]()
    gy = y.get_grad()
    dy = np.ones((4, 3), np.float32) if seed is None else _rand(4, 3, seed=2)
    value = nn.Tensor_from_value(dy) if seed == "tensor" else dy
    nn.backward(y if seed is None else {y: value})
    want = dy * u.np() if form == "mul" else dy
    assert w.get_grad() is g
    np.testing.assert_array_equal(g.np(), want)
    np.testing.assert_array_equal(gy.np(), dy)                # (held, so it outlives the pass)
    if seed == "tensor":
        value.fill(9.0)                                       # the caller's tensor stays the caller's
        np.testing.assert_array_equal(g.np(), want)
        np.testing.assert_array_equal(gy.np(), dy)
    del opt


def test_seeds_in_shallow_mode(fake):
    with nn.devices._shallow_mode():
        w = nn.Tensor((4, 3))
        opt = nn.optimizer.SGD([w])
        nn.backward({w + nn.Tensor((4, 3)): nn.Tensor((4, 3))})
        assert w.has_grad() and not fake.calls, "no kernel, no memory"
        del opt


# ---- deep graphs -----------------------------------------------------------------------------------
@pytest.mark.parametrize("end", ["pool", "convolution", "crossentropy"])
def test_operators_behind_a_deep_graph(fake, end):
    """An operator that asks whether anything upstream is trained finds out without recursion."""
    depth = 3000
    x = nn.Tensor((1, 1, 4, 4))
    opt = nn.optimizer.SGD([x])
    y = x
    for _ in range(depth):
        y = nn.mul_const(y, 1.0)
    if end == "pool":
        y = nn.max_pool2D(y)
    elif end == "convolution":
        y = nn.conv2D(y, nn.Tensor((1, 1, 3, 3)))
        assert not nn.deferred.is_deferred(y)
    else:
        y = nn.categorical_crossentropy(nn.Tensor((4, 4)), y.reshape((4, 4)))
        assert fake.calls[-1] == "lnn_reduce", "a target that needs a gradient takes the composition"
    nn.backward(y)
    assert x.has_grad()
    assert fake.calls.count("lnn_eltwise_bwd_acc") >= depth
    del opt


def test_pool_looks_at_a_bounded_part_of_the_graph(fake, monkeypatch):
    """Whether to keep the map of winners is not worth a walk of the whole graph from every pool."""
    visited = []
    inputs = nn.Tensor._tape_inputs
    monkeypatch.setattr(nn.Tensor, "_tape_inputs", lambda t: visited.append(t) or inputs(t))
    y = nn.Tensor((1, 1, 64, 64))
    for _ in range(400):
        y = nn.max_pool2D(nn.mul_const(y, 1.0), 3, 1)
    assert len(visited) <= 400 * 256
    w = nn.Tensor((1, 1, 1, 1))
    opt = nn.optimizer.SGD([w])
    y = nn.add(y, w)
    del visited[:]
    nn.max_pool2D(y)
    assert len(visited) == 1, "the operands that were added last are looked at first"
    del opt


# ---- work that has been put off sees the values of its time ----------------------------------------
def test_allreduce_of_a_gradient_that_a_chain_reads(fake, monkeypatch):
    monkeypatch.setitem(nn.parallel._state, "mode", "all")
    w, s = nn.Tensor_from_value(_rand(1, 2, 16)), nn.Tensor_from_value(_rand(1, 2, 1))
    w.get_grad().set(_rand(1, 2, 16, seed=1))
    y = w.get_grad() * s
    nn.parallel.allreduce_grads([w])
    np.testing.assert_array_equal(w.get_grad().np(), 2 * _rand(1, 2, 16, seed=1))
    np.testing.assert_array_equal(y.np(), _rand(1, 2, 16, seed=1) * s.np())


@pytest.mark.parametrize("kind", ["chain", "convolution"])
def test_launch_that_fails_can_be_repeated(fake, kind):
    x, s = nn.Tensor_from_value(_rand(1, 2, 8, 8)), nn.Tensor_from_value(_rand(1, 2, 1, 1))
    if kind == "chain":
        y, entry = x * s, "lnn_channel_chain_fwd"
    else:
        y, entry = nn.conv2D(x, nn.Tensor((2, 2, 3, 3))), "lnn_conv2d_fwd_packed"
    for failing in ("lnn_alloc", entry):
        fake.fail[failing] = nn._lib.E_NOMEM
        with pytest.raises(nn.LnnError):
            y.np()
    fake.fail[entry] = nn._lib.E_NOMEM
    if kind == "chain":
        with pytest.raises(nn.LnnError):
            x.fill(5.0)                                   # the chain has to run first, and cannot
        x.fill(5.0)
        np.testing.assert_array_equal(y.np(), _rand(1, 2, 8, 8) * s.np())
    else:
        with pytest.raises(nn.LnnError):
            y.np()
        del fake.calls[:]
        y.np()
        assert fake.calls == [entry]


def test_nothing_runs_in_shallow_mode(fake):
    x, s = nn.Tensor_from_value(_rand(1, 2, 16)), nn.Tensor_from_value(_rand(1, 2, 1))
    opt = nn.optimizer.SGD([x, s])
    t = x * s
    y, z = nn.leaky_relu(t + s, 0.1), nn.leaky_relu(x + s, 0.1)
    del t
    del fake.calls[:]
    with nn.devices._shallow_mode():
        nn.backward(y)
        y.np()
        x.fill(3.0)
        opt.step()
    assert set(fake.calls) <= {"lnn_alloc"}
    u = x.np() * s.np() + s.np()
    np.testing.assert_array_equal(y.np(), u * np.where(u >= 0, np.float32(1), np.float32(0.1)))
    assert z._chain.changed is False
    del opt


def test_joint_gradient_adds_to_one_that_only_one_device_has_touched():
    """Each device has its own memory: a gradient touched on one of them starts from zero on the other."""
    with fake_device(2) as fake:
        x, g, b = (nn.Tensor_from_value(_rand(*s)) for s in [(1, 2, 16), (1, 2, 1), (1, 2, 1)])
        opt = nn.optimizer.SGD([x, g, b])
        for t in (x, g, b):
            t.get_grad().fill(1.0, device_id=0)
        nn.backward(nn.leaky_relu(x * g + b, 0.1))
        for t in (x, g, b):
            np.testing.assert_allclose(t.get_grad().np(0), t.get_grad().np(1) + 1, rtol=1e-6)
        assert not fake.errors
        del opt, x, g, b, t


def test_edge_added_to_a_chain_keeps_its_own(fake):
    """A grad function registered on an operator's result joins those it has."""
    x, g, w = (nn.Tensor_from_value(_rand(*s)) for s in [(1, 2, 16), (1, 2, 1), (1, 2, 16)])
    opt = nn.optimizer.SGD([x, g, w])
    y = nn.leaky_relu(x * g, 0.1)
    seen = []
    y._assign_gradfn(w, lambda O_t, dO_t: seen.append(w.get_grad()))
    nn.backward(y)
    assert len(seen) == 1 and x.has_grad() and g.has_grad()
    dz = np.where(x.np() * g.np() >= 0, np.float32(1), np.float32(0.1))
    np.testing.assert_allclose(x.get_grad().np(), dz * g.np(), rtol=1e-6)
    np.testing.assert_allclose(g.get_grad().np(), (dz * x.np()).sum((0, 2), keepdims=True), rtol=1e-5)
    del opt


@pytest.mark.parametrize("when", ["before", "after"])
def test_edge_added_to_an_intermediate(fake, when):
    """The same on an intermediate that a longer chain was grown from, and that nobody holds any more."""
    x, g, w = (nn.Tensor_from_value(_rand(*s)) for s in [(1, 2, 16), (1, 2, 1), (1, 2, 16)])
    opt = nn.optimizer.SGD([x, g, w])
    seen = []
    y = x * g
    z = nn.leaky_relu(y, 0.1) if when == "after" else None
    y._assign_gradfn(w, lambda O_t, dO_t: seen.append(dO_t.np()))
    z = nn.leaky_relu(y, 0.1) if when == "before" else z
    del y
    nn.backward(z)
    dz = np.where(x.np() * g.np() >= 0, np.float32(1), np.float32(0.1))
    np.testing.assert_allclose(seen[0], dz, rtol=1e-6)
    np.testing.assert_allclose(x.get_grad().np(), dz * g.np(), rtol=1e-6)
    del opt


# ---- plans that are kept by their arguments ----------------------------------------------------------
@pytest.mark.parametrize("padding", [1.0, np.int64(1)])
def test_padding_that_equals_an_accepted_one(fake, padding):
    """A plan is not found under an argument that has never been accepted."""
    x, kernel = nn.Tensor((1, 2, 8, 8)), nn.Tensor((2, 2, 3, 3))
    nn.conv2D(x, kernel, padding=1)
    with pytest.raises(ValueError):
        nn.conv2D(x, kernel, padding=padding)


# ---- a deferred convolution runs before one of its sources is written to ---------------------------
@pytest.mark.parametrize("source", ["x", "kernel", "bias", "fused_bias"])
@pytest.mark.parametrize("write", ["fill", "set", "output", "optimizer"])
def test_write_to_a_source_of_a_deferred_convolution(fake, source, write):
    t = {"x": nn.Tensor((1, 2, 8, 8)), "kernel": nn.Tensor((2, 2, 3, 3)), "bias": nn.Tensor((1, 2, 1, 1)), "fused_bias": nn.Tensor((2,))}
    opt = nn.optimizer.SGD([t[source]])
    t[source].get_grad().fill(1.0)
    with nn.optimizer.freeze():
        y = nn.conv2D(t["x"], t["kernel"], bias_t=t["fused_bias"] if source == "fused_bias" else None)
        y = y if source == "fused_bias" else y + t["bias"]
        y = nn.max_pool2D(nn.leaky_relu(y, 0.1))
        dropped = nn.conv2D(t["x"], t["kernel"])
    del dropped
    assert nn.deferred.is_deferred(y)
    for s in t.values():
        s._ptr(0)
    del fake.calls[:]
    {"fill": lambda s: s.fill(2.0), "set": lambda s: s.set(np.ones(s.shape.shape, np.float32)),
     "output": lambda s: nn.op.add_const_op(s, 1.0, output_t=s), "optimizer": lambda s: opt.step()}[write](t[source])
    calls = [c for c in fake.calls if c not in ("lnn_alloc", "lnn_fill_f32") or write == "fill"]
    assert calls.count("lnn_conv2d_fwd_packed") == 1, "once, and not for the one nobody holds"
    assert calls.index("lnn_conv2d_fwd_packed") < len(calls) - 1, "before the write"
    assert not nn.deferred.is_deferred(y)
    del fake.calls[:]
    y.np()
    assert not fake.calls


def test_write_under_a_deferred_network(fake):
    """Only what reads the written tensor itself has to run; what follows takes its values."""
    x, k = nn.Tensor((1, 2, 8, 8)), nn.Tensor((2, 2, 3, 3))
    with nn.optimizer.freeze():
        y = nn.conv2D(nn.leaky_relu(nn.conv2D(x, k), 0.1), nn.Tensor((2, 2, 3, 3)))
    x._ptr(0)
    del fake.calls[:]
    x.fill(1.0)
    assert fake.calls.count("lnn_conv2d_fwd_packed") == 1 and nn.deferred.is_deferred(y)
    y.np()
    assert fake.calls.count("lnn_conv2d_fwd_packed") == 2


def test_sources_forget_what_has_been_dropped(fake):
    x, k, s = nn.Tensor((1, 2, 8, 8)), nn.Tensor((2, 2, 3, 3)), nn.Tensor((1, 2, 1, 1))
    for _ in range(100):
        nn.conv2D(x, k)
        x * s
    assert len(x._deps) <= 8 and len(k._deps) <= 8 and len(s._deps) <= 8
    held = [nn.conv2D(x, k) for _ in range(100)] + [x * s for _ in range(100)]
    assert len(x._deps) <= 208
    x.fill(1.0)
    assert not any(nn.deferred.is_deferred(t) or t._pending is not None and not t._pending.done for t in held)
    assert x._deps is None


@pytest.mark.parametrize("op", ["bias", "act", "pool"])
def test_gradient_stops_at_a_frozen_convolution(fake, op):
    """What follows a deferred convolution outside freeze() does not take its place on the tape."""
    x, kernel, bias = nn.Tensor((1, 2, 8, 8)), nn.Tensor((2, 2, 3, 3)), nn.Tensor((1, 2, 1, 1))
    opt = nn.optimizer.SGD([x, kernel])
    with nn.optimizer.freeze():
        frozen = nn.conv2D(x, kernel)
    y = {"bias": lambda: frozen + bias, "act": lambda: nn.leaky_relu(frozen, 0.1), "pool": lambda: nn.max_pool2D(frozen)}[op]()
    nn.backward(y, keep_gradient_for_non_trainables=True)
    assert frozen.has_grad() and not x.has_grad() and not kernel.has_grad()
    del opt
