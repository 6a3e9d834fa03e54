"""Gradients of a convolution at the sizes where their dispatch changes: input channels up to 32 and about
64 (hi and lo rows of the kernel in one instruction), output channels and column groups that leave a last
tile short, strides whose residue classes are written by separate launches, added to and written anew."""
import numpy as np
import pytest

import oracle as o

pytestmark = pytest.mark.gpu

CASES = [(ic, 24, 3, 1, 13) for ic in (5, 8, 16, 31, 32, 33, 56, 57, 63, 64, 65)] + \
        [(32, 64, 3, 2, 15), (64, 8, 1, 2, 9), (24, 48, 5, 1, 11), (64, 136, 2, 3, 16), (96, 160, 3, 1, 12)]


@pytest.mark.parametrize("ic,oc,k,stride,size", CASES)
def test_gradients_against_oracle(nn_gpu, ic, oc, k, stride, size):
    nn = nn_gpu
    rng = np.random.default_rng(ic * 1000 + oc)
    n = 5
    x = rng.standard_normal((n, ic, size, size)).astype(np.float32)
    w = (rng.standard_normal((oc, ic, k, k)) * (ic * k * k) ** -0.5).astype(np.float32)
    xt, wt = nn.Tensor_from_value(x), nn.Tensor_from_value(w)
    opt = nn.optimizer.SGD([xt, wt])
    y = nn.conv2D(xt, wt, stride)
    dy = rng.standard_normal(y.shape.shape).astype(np.float32)
    info = nn.info.InfoConv2D(size, size, k, k, stride, 1, "same")
    kw = dict(stride=stride, accum64=True)
    for turn in (1, 2):                                  # written, then added to
        nn.backward({y: nn.Tensor_from_value(dy)})
        for got, ref, bound, terms in (
                (xt, o.conv2d_dx(np.zeros_like(x), dy, w, x.shape, **kw),
                 o.conv2d_dx(np.zeros_like(x), np.abs(dy), np.abs(w), x.shape, **kw), oc * k * k),
                (wt, o.conv2d_dw(np.zeros_like(w), dy, x, **kw),
                 o.conv2d_dw(np.zeros_like(w), np.abs(dy), np.abs(x), **kw), n * info.OH * info.OW)):
            # operands keep 22 bits each, sums of `terms` products in 32 bits, one more addition per turn
            limit = turn * (2.0 ** -20 + terms * 2.0 ** -23) * bound + 1e-6
            assert (np.abs(got.get_grad().np().astype(np.float64) - turn * ref) <= limit).all()
    assert opt.get_iteration() == 0


@pytest.mark.parametrize("ic,oc,k,stride,size", [(300, 260, 3, 1, 5), (520, 300, 1, 1, 4), (70, 900, 2, 1, 6), (256, 290, 3, 2, 7),
                                                 (33, 700, 4, 1, 5), (5, 1200, 3, 1, 4), (129, 300, 5, 1, 4), (48, 96, 5, 1, 20)])
def test_kernel_gradients_with_few_splits(nn_gpu, ic, oc, k, stride, size):
    """Few pixels and many channels: the partial sums of whole channel groups with all their taps."""
    test_gradients_against_oracle(nn_gpu, ic, oc, k, stride, size)


@pytest.mark.parametrize("ic,oc,k,size", [(260, 200, 3, 4), (6, 5, 3, 9), (40, 900, 2, 3)])
def test_kernel_gradient_of_the_transposed_convolution(nn_gpu, ic, oc, k, size):
    """It is that of a convolution with the roles swapped, stored [output][input channel]."""
    nn = nn_gpu
    rng = np.random.default_rng(ic)
    x = rng.standard_normal((2, ic, size, size)).astype(np.float32)
    xt, kt = nn.Tensor_from_value(x), nn.Tensor_from_value(rng.standard_normal((oc, ic, k, k)).astype(np.float32))
    opt = nn.optimizer.SGD([xt, kt])
    y = nn.conv2DTranspose(xt, kt, 2)
    dy = rng.standard_normal(y.shape.shape).astype(np.float32)
    zero, kw = np.zeros((ic, oc, k, k), np.float32), dict(stride=2, accum64=True)
    ref, bound = (o.conv2d_dw(zero, a, b, **kw).swapaxes(0, 1) for a, b in ((x, dy), (np.abs(x), np.abs(dy))))
    for turn in (1, 2):
        nn.backward({y: nn.Tensor_from_value(dy)})
        limit = turn * (2.0 ** -20 + 2 * size * size * 2.0 ** -23) * bound + 1e-6
        assert (np.abs(kt.get_grad().np().astype(np.float64) - turn * ref) <= limit).all()
    assert opt.get_iteration() == 0


@pytest.mark.parametrize("ic,oc,k,stride", [(24, 5, 3, 2), (24, 32, 3, 2), (40, 33, 3, 2), (16, 56, 2, 2), (16, 57, 3, 2), (24, 64, 3, 1),
                                            (24, 65, 3, 2), (136, 16, 3, 3)])
def test_transposed_convolution_forward(nn_gpu, ic, oc, k, stride):
    """It is the input gradient of a convolution with the roles swapped and takes the same kernels."""
    nn = nn_gpu
    rng = np.random.default_rng(ic + oc)
    x = rng.standard_normal((3, ic, 7, 9)).astype(np.float32)
    w = (rng.standard_normal((oc, ic, k, k)) * (ic * k * k) ** -0.5).astype(np.float32)
    y = nn.conv2DTranspose(nn.Tensor_from_value(x), nn.Tensor_from_value(w), stride).np()
    ref, bound = (o.conv2d_dx(np.zeros_like(y), a, b.swapaxes(0, 1), y.shape, stride=stride, accum64=True)
                  for a, b in ((x, w), (np.abs(x), np.abs(w))))
    assert (np.abs(y.astype(np.float64) - ref) <= (2.0 ** -20 + ic * k * k * 2.0 ** -23) * bound + 1e-6).all()
