"""Pooling that keeps the map of winning positions for its gradient (trainable inputs) against the form that
looks at the input again (inputs nothing trainable depends on): same values and gradients bit for bit,
with ties, infinities and NaN, at sizes that take the four-wide, the two-wide and the generic kernels."""
import numpy as np
import pytest

from conftest import assert_bit_exact

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("op", ["max", "min", "avg"])
@pytest.mark.parametrize("shape,pool,stride,padding", [
    ((2, 3, 8, 8), 2, 2, "same"), ((2, 3, 7, 12), 2, 2, "same"), ((1, 5, 6, 10), 2, 2, "same"), ((3, 2, 5, 6), 2, 2, "same"),
    ((2, 4, 9, 7), 2, 2, "same"), ((2, 3, 11, 13), 3, 2, "same"), ((2, 3, 12, 9), 3, 3, "same"), ((1, 2, 9, 9), 4, 1, "same"),
    ((2, 2, 16, 15), 15, 4, "same"), ((1, 1, 20, 20), 16, 5, "same"), ((2, 3, 8, 8), 2, 2, 1), ((2, 2, 10, 10), 3, 2, "valid")])
def test_winner_map_equals_second_look(nn_gpu, op, shape, pool, stride, padding):
    nn = nn_gpu
    rng = np.random.default_rng(sum(shape) + pool)
    x = np.round(rng.standard_normal(shape) * 2).astype(np.float32) / 2        # many ties
    x[0, 0, :2] = np.nan
    x[0, 0, 2, :3] = [np.inf, -np.inf, -np.inf]
    x[-1, -1, :, :2] = -np.inf if op == "max" else np.inf
    f = getattr(nn, op + "_pool2D")
    res = []
    for trainable in (False, True):
        xt = nn.Tensor_from_value(x)
        opt = nn.optimizer.SGD([xt]) if trainable else None
        y = f(xt, pool, stride, padding)
        dy = np.random.default_rng(5).standard_normal(tuple(y.shape)).astype(np.float32)
        nn.backward({y: dy}, grad_for_non_trainables=True)
        first = xt.get_grad().np()
        y2 = f(xt, pool, stride, padding)
        nn.backward({y2: dy}, grad_for_non_trainables=True)
        res.append((y.np(), first, xt.get_grad().np(), opt))
    for k, name in enumerate(("values", "gradient, written", "gradient, added")):
        assert_bit_exact(res[1][k], res[0][k], name)
