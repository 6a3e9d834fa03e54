"""Matrix products around the edges of the small-product kernel (32 x 32 and 64 x 64 tiles, K slabs of 16,
four thread groups, clusters of up to eight blocks) and past its limit, where the operands are
prepared in one or in several launches.  A float32 sum of k products in any order is off by at most
gamma_k * sum |a||b| with gamma_k = k u / (1 - k u), u = 2**-24; the split-FP16 engine adds 2**-21 of that
sum for the dropped lo * lo terms and the truncation of its accumulator."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(1, 1, 1, 1), (1, 31, 33, 15), (1, 32, 32, 16), (1, 33, 5, 65), (1, 64, 64, 1024), (1, 7, 130, 4097), (3, 40, 36, 100),
         (1, 96, 1030, 129), (1, 1200, 1100, 60), (2, 700, 900, 50), (5, 17, 19, 23), (1, 512, 515, 516),
         (1, 1003, 650, 777), (2, 300, 260, 1700)]


@pytest.mark.parametrize("batch,m,n,k", SIZES)
def test_gemm_sizes(nn_gpu, batch, m, n, k):
    nn = nn_gpu
    rng = np.random.default_rng(m * 7 + n * 3 + k)
    lead = () if batch == 1 else (batch,)
    a = rng.standard_normal(lead + (m, k)).astype(np.float32)
    b = rng.standard_normal(lead + (k, n)).astype(np.float32)
    d = rng.standard_normal(lead + (m, n)).astype(np.float32)
    a64, b64, d64 = a.astype(np.float64), b.astype(np.float64), d.astype(np.float64)
    at, bt = nn.Tensor_from_value(a), nn.Tensor_from_value(b)
    y = nn.matmul(at, bt)
    nn.backward({y: nn.Tensor_from_value(d)}, grad_for_non_trainables=True)

    def check(got, x, z, terms, what, times=1):
        want, size = x @ z, np.abs(x) @ np.abs(z)
        u = 2.0 ** -24
        bound = times * size * (terms * u / (1 - terms * u) + 2.0 ** -21) + (times - 1) * np.abs(want) * u
        err = np.abs(got - times * want)
        assert (err <= bound).all(), f"{what}: {float((err / bound).max())} of the bound"

    t = lambda v: np.swapaxes(v, -1, -2)     # noqa: E731
    check(y.np(), a64, b64, k, "product")
    check(at.get_grad().np(), d64, t(b64), n, "dA")
    check(bt.get_grad().np(), t(a64), d64, m, "dB")
    y2 = nn.matmul(at, bt)
    nn.backward({y2: nn.Tensor_from_value(d)}, grad_for_non_trainables=True)
    check(at.get_grad().np(), d64, t(b64), n, "dA, added to", 2)
    check(bt.get_grad().np(), t(a64), d64, m, "dB, added to", 2)
    nn.devices.check_status()


@pytest.mark.parametrize("batch,m,n,k", [(1, 1, 20000, 64), (1, 20000, 3, 70), (1, 2, 19000, 63), (1, 33, 20000, 65),
                                         (400, 16, 16, 16), (400, 20, 9, 130), (300, 33, 33, 64), (150, 30, 100, 20)])
def test_half_empty_tiles(nn_gpu, batch, m, n, k):
    """Enough products to cover the chip whose 64 x 64 tiles would be half or three quarters empty."""
    test_gemm_sizes(nn_gpu, batch, m, n, k)


def test_dense_bias_small_and_large(nn_gpu):
    nn = nn_gpu
    rng = np.random.default_rng(9)
    for rows, cin, cout in ((5, 40, 10), (64, 256, 513), (700, 600, 650)):
        x, w = rng.standard_normal((rows, cin)).astype(np.float32), rng.standard_normal((cin, cout)).astype(np.float32)
        b = rng.standard_normal(cout).astype(np.float32)
        y = nn.dense(nn.Tensor_from_value(x), nn.Tensor_from_value(w), nn.Tensor_from_value(b)).np()
        want = x.astype(np.float64) @ w.astype(np.float64) + b
        size = np.abs(x).astype(np.float64) @ np.abs(w) + np.abs(b)
        assert (np.abs(y - want) <= size * ((cin + 1) * 2.0 ** -24 * 1.01 + 2.0 ** -21)).all()
