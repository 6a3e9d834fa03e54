"""x * g, + b and leaky_relu with per-channel g and b run as one kernel forward and one backward; values
equal the separate operators bit for bit, gradients up to the order of the channel sums, whatever the
user does with the intermediates or the sources in between."""
import numpy as np
import pytest

from conftest import assert_bit_exact

pytestmark = pytest.mark.gpu

SHAPES = [(2, 3, 4, 4), (1, 1, 16), (3, 8, 6, 10), (5, 7, 3, 9), (2, 1300, 4, 8), (40, 16, 28, 28), (300, 2, 33),
          (1, 3, 257, 259), (1, 2, 512, 512), (16385, 3, 16)]


def _inputs(shape, seed=0):
    rng = np.random.default_rng(seed)
    per = (1, shape[1]) + (1,) * (len(shape) - 2)
    return (rng.standard_normal(shape).astype(np.float32), rng.uniform(0.5, 1.5, per).astype(np.float32),
            rng.uniform(-0.5, 0.5, per).astype(np.float32), rng.standard_normal(shape).astype(np.float32))


def _sum_bound(terms, shape):
    """|error| of a float32 sum of n terms in any order, twice (two orders are compared)."""
    axes = (0,) + tuple(range(2, len(shape)))
    n = terms.size // shape[1]
    return 2 * n * 2.0 ** -24 * np.abs(terms).sum(axes, keepdims=True) + 1e-30


@pytest.mark.parametrize("form", ["mul_add_act", "mul_add", "add_act", "mul_act"])
@pytest.mark.parametrize("shape", SHAPES)
def test_chain_equals_separate_operators(nn_gpu, shape, form):
    nn = nn_gpu
    x, g, b, dy = _inputs(shape)

    def run():
        xt, gt, bt = (nn.Tensor_from_value(a) for a in (x, g, b))
        opt = nn.optimizer.SGD([xt, gt, bt])
        for _ in range(2):                                   # the second pass adds into the gradients
            y = xt * gt if "mul" in form else xt
            y = y + bt if "add" in form else y
            y = nn.leaky_relu(y, 0.1) if "act" in form else y
            nn.backward({y: nn.Tensor_from_value(dy)})
        return y.np(), [t.get_grad().np() if t.has_grad() else None for t in (xt, gt, bt)], opt

    with nn.deferred.disabled():
        want = run()
    got = run()
    assert_bit_exact(got[0], want[0], "values")
    assert_bit_exact(got[1][0], want[1][0], "dx")
    t = x.astype(np.float64) * (g if "mul" in form else 1) + (b if "add" in form else 0)
    dz = dy * (np.where(t >= 0, 1.0, 0.1) if "act" in form else 1.0)
    for k, terms, name in ((1, dz * x, "dg"), (2, dz, "db")):
        if want[1][k] is None:
            assert got[1][k] is None
            continue
        assert (np.abs(got[1][k] - want[1][k]) <= 2 * _sum_bound(terms, shape)).all(), name


def test_intermediates_and_sources_that_change(nn_gpu):
    nn = nn_gpu
    shape = (4, 8, 6, 6)
    x, g, b, dy = _inputs(shape, 1)
    xt, gt, bt = (nn.Tensor_from_value(a) for a in (x, g, b))
    opt = nn.optimizer.SGD([xt, gt, bt])
    m = xt * gt
    s = m + bt
    y = nn.leaky_relu(s, 0.1)
    gt.fill(3.0)                                             # everything put off still sees the old values
    assert_bit_exact(m.np(), x * g, "product")
    assert_bit_exact(s.np(), x * g + b, "sum")
    t = x * g + b
    assert_bit_exact(y.np(), t * (t >= 0) + (np.float32(0.1) * t) * (t < 0), "activation")
    nn.backward({y: nn.Tensor_from_value(dy)}, keep_gradient_for_non_trainables=True)
    assert s.has_grad() and m.has_grad(), "intermediates that are held get gradients"
    dz = dy * np.where(t >= 0, np.float32(1), np.float32(0.1))
    assert_bit_exact(s.get_grad().np(), dz, "gradient of the sum")
    # dropped intermediates: the gradient goes to the sources at once, with the signs of the forward pass
    for tensor, value in ((xt, x), (gt, g), (bt, b)):
        tensor.zero_grad()
        tensor.set(value)
    y2 = nn.leaky_relu(xt * gt + bt, 0.1)
    y2.np()
    bt.fill(-100.0)                                          # would flip every sign if t were computed again
    nn.backward({y2: nn.Tensor_from_value(dy)})
    assert_bit_exact(xt.get_grad().np(), dz * g, "dx after the shift changed")
    # a gradient stopped at an intermediate goes no further
    xt.zero_grad()
    m = xt * gt
    y3 = nn.leaky_relu(m + bt, 0.1)
    nn.backward({y3: nn.Tensor_from_value(dy)}, stop_grad=m)
    assert not xt.has_grad()
    # a chain that reads a chain, launched from its end
    z = nn.leaky_relu(nn.leaky_relu(xt * gt, 0.1) + bt, 0.2)
    u = x * g
    u = u * (u >= 0) + (np.float32(0.1) * u) * (u < 0) + np.float32(-100.0)
    assert_bit_exact(z.np(), u * (u >= 0) + (np.float32(0.2) * u) * (u < 0), "chain of chains")
    assert opt.get_iteration() == 0


def test_kept_gradients_of_dropped_intermediates(nn_gpu):
    """Passes that keep gradients add to those of the intermediates too, held or not."""
    nn = nn_gpu
    x, g, b, dy = _inputs((3, 5, 8, 12), 3)

    def run():
        xt, gt, bt = (nn.Tensor_from_value(a) for a in (x, g, b))
        y = nn.leaky_relu(xt * gt + bt, 0.1)
        for k in range(3):
            nn.backward({y: nn.Tensor_from_value(dy)}, grad_for_non_trainables=k < 2,
                        keep_gradient_for_non_trainables=k == 2)
            if k == 1:
                bt.fill(-100.0)                              # the signs of the forward pass still hold
        return [t.get_grad().np() for t in (xt, gt, bt)]

    with nn.deferred.disabled():
        want = run()
    for got, ref, name in zip(run(), want, ("dx", "dg", "db")):
        bound = 2 * 288 * 2.0 ** -24 * 4 * np.abs(ref).max() * 288 if name != "dx" else 4 * 2.0 ** -24 * np.abs(ref).max()
        assert np.abs(got - ref).max() <= bound, name


def test_stock_convolution_with_separate_bias_trains(nn_gpu):
    nn = nn_gpu
    rng = np.random.default_rng(2)
    x, w = rng.standard_normal((2, 6, 12, 12)).astype(np.float32), (rng.standard_normal((8, 6, 3, 3)) * 0.2).astype(np.float32)
    b, dy = rng.standard_normal((8,)).astype(np.float32), rng.standard_normal((2, 8, 12, 12)).astype(np.float32)

    def run():
        xt, wt, bt = (nn.Tensor_from_value(a) for a in (x, w, b))
        opt = nn.optimizer.SGD([xt, wt, bt])
        y = nn.leaky_relu(nn.conv2D(xt, wt) + bt.reshape((1, -1, 1, 1)), 0.1)
        nn.backward({y: nn.Tensor_from_value(dy)})
        return y.np(), xt.get_grad().np(), wt.get_grad().np(), bt.get_grad().np(), opt

    with nn.deferred.disabled():
        want = run()
    got = run()
    for k, name in enumerate(("values", "dx", "dw")):
        assert_bit_exact(got[k], want[k], name)
    np.testing.assert_allclose(got[3], want[3], rtol=0, atol=2 * 288 * 2.0 ** -24 * np.abs(dy).sum((0, 2, 3)).max())


def test_channel_of_a_billion_elements(nn_gpu):
    """A channel of 2^30 elements is put off like any other, and its gradient takes it."""
    nn = nn_gpu
    shape = (1, 2, 32768, 32768)
    x, dy = nn.Tensor(shape, init=nn.initializer.Scalar(0.5)), nn.Tensor(shape, init=nn.initializer.Scalar(1.0))
    g, b = nn.Tensor_from_value(np.array([2.0, -4.0], np.float32).reshape(1, 2, 1, 1)), nn.Tensor((1, 2, 1, 1))
    opt = nn.optimizer.SGD([x, g, b])
    nn.backward({nn.leaky_relu(x * g + b, 0.25): dy})
    factor = np.array([1.0, 0.25])                            # sums of powers of two: exact
    assert_bit_exact(g.get_grad().np().ravel(), factor * 2.0 ** 29, "dg")
    assert_bit_exact(b.get_grad().np().ravel(), factor * 2.0 ** 30, "db")
    for op in (nn.reduce_min, nn.reduce_max):
        assert_bit_exact(op(x.get_grad(), (2, 3)).np().ravel(), factor * [2.0, -4.0], "dx")
    assert opt.get_iteration() == 0
