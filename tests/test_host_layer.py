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
