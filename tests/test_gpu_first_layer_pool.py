"""The pooled first layer (at most four input channels) gives the bits of the separate operators whatever
part of a tile, of a 32-channel chunk or of a group of four pooled columns its result ends in; with its map
of winners (training) and without, channel-innermost and as NCHW."""
import numpy as np
import pytest

from conftest import assert_bit_exact

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("alpha", [0.1, -0.5])
@pytest.mark.parametrize("ic,oc,h,w", [(3, 8, 16, 16), (3, 32, 34, 20), (1, 40, 18, 12), (4, 70, 6, 36), (2, 96, 2, 2),
                                       (3, 200, 10, 72), (3, 64, 48, 130), (3, 256, 20, 28)])
def test_pooled_first_layer(nn_gpu, ic, oc, h, w, alpha):
    nn = nn_gpu
    rng = np.random.default_rng(oc)
    x = rng.standard_normal((3, ic, h, w)).astype(np.float32)
    k = (rng.standard_normal((oc, ic, 3, 3)) * 0.3).astype(np.float32)
    b = rng.standard_normal((oc,)).astype(np.float32)
    xt, kt, bt = (nn.Tensor_from_value(a) for a in (x, k, b))
    with nn.deferred.disabled():
        y = nn.leaky_relu(nn.conv2D(xt, kt) + bt.reshape((1, -1, 1, 1)), alpha)
        want = nn.max_pool2D(y).np()
    assert_bit_exact(nn.ops.conv2D_pool(xt, kt, bias_t=bt, activation="leaky_relu", alpha=alpha).np(), want, "pooled")
    packed = nn.ops.conv2D_pool(xt, kt, bias_t=bt, activation="leaky_relu", alpha=alpha, packed_output=True).np()
    assert np.abs(packed - want).max() <= 2.0 ** -20 * np.abs(want).max()
    if alpha > 0.0:
        opt = nn.optimizer.SGD([xt, kt, bt])
        dy = rng.standard_normal(want.shape).astype(np.float32)
        t = nn.conv2D_block(xt, kt, bias_t=bt, activation="leaky_relu", alpha=alpha)
        assert_bit_exact(t.np(), want, "block")
        nn.backward({t: nn.Tensor_from_value(dy)})
        got = [v.get_grad().np() for v in (xt, kt, bt)]
        opt.zero_grad()
        with nn.deferred.disabled():
            t = nn.max_pool2D(nn.leaky_relu(nn.conv2D(xt, kt) + bt.reshape((1, -1, 1, 1)), alpha))
        nn.backward({t: nn.Tensor_from_value(dy)})
        assert_bit_exact(got[0], xt.get_grad().np(), "dx")
        for g, v in ((got[1], kt), (got[2], bt)):          # the same terms in another order
            r = v.get_grad().np()
            assert np.abs(g - r).max() <= 2.0 ** -23 * x.shape[0] * h * w * np.abs(r).max() + 1e-5
