"""Reductions at the sizes where the planner changes kernel and where stages of odd length leave
columns without a partner: bit-exact against the reference's ceil-halving tree in numpy, and their
gradients written into untouched tensors and added to touched ones."""
import numpy as np
import pytest

from conftest import assert_bit_exact

pytestmark = pytest.mark.gpu


def _tree(x, op):
    """x[c] = x[c] (+) x[c + ceil(n/2)] along the last axis until one column is left (reduce.py:279-293)."""
    comb = np.maximum if op == "max" else (lambda a, b: (a + b).astype(np.float32))
    while x.shape[-1] > 1:
        h = (x.shape[-1] + 1) // 2
        y = x[..., :h].copy()
        y[..., :x.shape[-1] - h] = comb(x[..., :x.shape[-1] - h], x[..., h:])
        x = y
    return x[..., 0]


SHAPES = [
    ((5, 1), (1,)), ((3, 7), (1,)), ((300, 31), (1,)), ((70, 33), (1,)), ((5000, 225), (1,)),      # a warp per row
    ((9000, 128), (1,)), ((4100, 1024), (1,)), ((40, 4096), (1,)),                                 # 128-bit warps
    ((2400, 3001), (1,)), ((33, 5000), (1,)), ((2, 600), (1,)),                                    # a block per row
    ((3, 40001), (1,)), ((2, 9, 65536), (2,)), ((1, 20000), None), ((1 << 14,), None), ((100003,), None),   # split rows
    ((37, 32, 9, 15), (0, 2, 3)), ((64, 24, 14, 14), (0, 2, 3)), ((129, 3, 50, 20), (0, 2, 3)),    # two reduced groups
    ((1, 64), (0,)), ((64, 512), (0,)), ((257, 60), (0,)), ((9, 31), (0,)), ((5000, 36), (0,)),    # inner axis kept
    ((8, 100, 1024), (1,)), ((6, 3, 40000), (1,)), ((4, 1000, 129), (1,)), ((16, 7, 5), (1,)),
]


@pytest.mark.parametrize("op", ["sum", "mean", "max"])
@pytest.mark.parametrize("shape,axes", SHAPES)
def test_reduce_tree_and_gradient(nn_gpu, shape, axes, op):
    nn = nn_gpu
    rng = np.random.default_rng(abs(hash((shape, axes))) % 1000)
    x = rng.standard_normal(shape).astype(np.float32)
    red = tuple(range(len(shape))) if axes is None else axes
    kept = tuple(a for a in range(len(shape)) if a not in red)
    moved = x.transpose(kept + red).reshape([shape[a] for a in kept] + [-1])
    want = _tree(moved, "max" if op == "max" else "sum")
    cols = moved.shape[-1]
    if op == "mean":
        want = (want / np.float32(cols)).astype(np.float32)
    want = np.asarray(want, np.float32).reshape([shape[a] for a in kept] or (1,))
    xt = nn.Tensor_from_value(x)
    y = getattr(nn, "reduce_" + op)(xt, axes)
    assert_bit_exact(y.np(), want, f"{op} {shape} {axes}")
    dy = rng.standard_normal(want.shape).astype(np.float32)
    up = dy.reshape([shape[a] if a in kept else 1 for a in range(len(shape))])
    if op == "max":
        first = np.zeros_like(moved)
        np.put_along_axis(first, np.argmax(moved, -1)[..., None], 1.0, -1)
        back = first.reshape([shape[a] for a in kept + red]).transpose(np.argsort(kept + red))
        grad = up * back
    else:
        grad = np.broadcast_to(up if op == "sum" else (up / np.float32(cols)).astype(np.float32), shape).astype(np.float32)
    nn.backward({y: nn.Tensor_from_value(dy)}, grad_for_non_trainables=True)
    assert_bit_exact(xt.get_grad().np(), grad, "gradient, written")
    y2 = getattr(nn, "reduce_" + op)(xt, axes)
    nn.backward({y2: nn.Tensor_from_value(dy)}, grad_for_non_trainables=True)
    assert_bit_exact(xt.get_grad().np(), (grad + grad).astype(np.float32), "gradient, added")


@pytest.mark.parametrize("op", ["sum", "max"])
@pytest.mark.parametrize("cols", [1, 2, 3, 4, 5, 7, 8, 9, 15, 16, 17, 24, 31, 32, 33, 63, 64, 65, 100, 127, 129, 255, 256, 257])
def test_short_rows(nn_gpu, cols, op):
    """The row kernel's lanes per row and stages per lane, a last row that fills no warp, and the limits of the
    thread-per-row kernels over a kept inner axis (enough rows to cover the chip, and few)."""
    nn = nn_gpu
    rng = np.random.default_rng(cols)
    for shape in ((1003, cols), (7, cols), (6001, cols, 7), (5, cols, 3), (3, 40, cols)):
        x = rng.standard_normal(shape).astype(np.float32)
        axis = 2 if shape[:2] == (3, 40) else 1
        want = _tree(np.moveaxis(x, axis, -1), op)
        xt = nn.Tensor_from_value(x)
        assert_bit_exact(getattr(nn, "reduce_" + op)(xt, axis).np(), want, f"{op} {shape}")
        out = nn.Tensor_from_value(np.ones(want.shape, np.float32))
        getattr(nn.op, f"reduce_{op}_op")(xt, axis, output_t=out, is_add_to_output=True)
        assert_bit_exact(out.np(), (np.float32(1) + want).astype(np.float32), f"{op} {shape}, added")


def test_gradients_that_share_memory_stay_separate(nn_gpu):
    """z = x + y hands its gradient on without copies; afterwards every tensor owns its own."""
    nn = nn_gpu
    rng = np.random.default_rng(3)
    a, b, d = (rng.standard_normal((6, 50)).astype(np.float32) for _ in range(3))
    x, y, dz = nn.Tensor_from_value(a), nn.Tensor_from_value(b), nn.Tensor_from_value(d)
    opt = nn.optimizer.SGD([x, y])
    w = x + y                                 # w is used twice, so its gradient is added to after it was taken over
    z = (w + y) + (w - x)
    nn.backward({z: dz})
    assert_bit_exact(dz.np(), d, "the given gradient is not written to")
    assert_bit_exact(x.get_grad().np(), (d + d) - d, "dx")
    assert_bit_exact(y.get_grad().np(), (d + d) + d, "dy")
    dz.fill(7.0)
    x.get_grad().fill(1.0)
    assert_bit_exact(y.get_grad().np(), (d + d) + d, "dy after dx and dz changed")
    x.zero_grad(); y.zero_grad()
    s = x + y
    nn.backward({s: dz})
    dz.fill(0.0)
    assert_bit_exact(x.get_grad().np(), np.full_like(d, 7.0), "dx keeps the values of the pass")
    x.get_grad().fill(2.0)
    assert_bit_exact(y.get_grad().np(), np.full_like(d, 7.0), "dy is not dx")
    assert opt.get_trainable_tensors() == [x, y]
