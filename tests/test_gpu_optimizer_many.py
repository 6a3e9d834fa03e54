"""One optimizer launch for many tensors: sizes around the chunk of a block, more tensors than one
launch takes, and the same values as one call per tensor."""
import ctypes

import numpy as np
import pytest

from conftest import assert_bit_exact

pytestmark = pytest.mark.gpu

SIZES = [1, 3, 4, 1023, 1024, 1025, 4096, 5000] + [7] * 30


@pytest.mark.parametrize("kind,dropout", [("SGD", 0.0), ("SGD", 0.3), ("RMSprop", 0.0), ("RMSprop", 0.3), ("Adam", 0.0), ("Adam", 0.3)])
def test_many_tensors_equal_one_by_one(nn_gpu, kind, dropout):
    nn = nn_gpu
    from litenn_b200 import _lib, optimizer
    rng = np.random.default_rng(17)
    values = [rng.standard_normal(n).astype(np.float32) for n in SIZES]
    grads = [rng.standard_normal(n).astype(np.float32) for n in SIZES]
    tensors = [nn.Tensor_from_value(v) for v in values]
    kw = {"SGD": {"momentum": 0.9, "nesterov": True}, "RMSprop": {"rho": 0.9}, "Adam": {}}[kind]
    opt = getattr(nn.optimizer, kind)(tensors, lr=0.01, lr_decay=0.1, lr_dropout=dropout, **kw)
    for t, g in zip(tensors, grads):
        t.get_grad().set(g)
    np.random.seed(3)
    opt.step()
    after = np.random.randint(1 << 30)
    np.random.seed(3)
    lib, dev = _lib.get_lib(), nn.devices.get_current()[0].index
    number = {"SGD": optimizer.SGD_KIND, "RMSprop": optimizer.RMSPROP_KIND, "Adam": optimizer.ADAM_KIND}[kind]
    betas = {"SGD": (0.9, 0.0), "RMSprop": (0.9, 0.0), "Adam": (0.9, 0.999)}[kind]
    for t, v, g in zip(tensors, values, grads):
        seed_a = int(np.random.randint(2147483648))
        seed_b = int(np.random.randint(2147483648)) if kind == "SGD" else seed_a
        vt, gt, s1, s2 = (nn.Tensor_from_value(a) for a in (v, g, np.zeros_like(v), np.zeros_like(v)))
        p = optimizer.OptParams(0.01, 0.1, dropout, 1.0, *betas, 0, seed_a, seed_b, 1 if kind == "SGD" else 0)
        lib.lnn_optimizer_step(dev, number, vt._ptr(0), gt._ptr(0), s1._ptr(0), s2._ptr(0), v.size, ctypes.byref(p))
        assert_bit_exact(t.np(), vt.np(), f"{kind} size {v.size}")
    assert after == np.random.randint(1 << 30), "the host's random stream is where one draw per kernel leaves it"


def test_calls_check_their_arguments(nn_gpu):
    nn = nn_gpu
    from litenn_b200 import _lib
    t = nn.Tensor((4,))
    dev = nn.devices.get_current()[0].index
    with pytest.raises(TypeError):
        _lib.call.lnn_reduce(0, dev)
    with pytest.raises(TypeError):
        _lib.call.lnn_reduce(0, dev, 0, t, "x", 1, 1, 1, 4, 1, 0)
    with pytest.raises(IndexError):
        _lib.call.lnn_reduce(7, dev, 0, t, t, 1, 1, 1, 4, 1, 0)
    with pytest.raises(_lib.LnnError) as e:
        _lib.call.lnn_reduce(0, dev, 99, t, t, 1, 1, 1, 4, 1, 0)
    assert e.value.code == _lib.E_INVALID and "reduce" in str(e.value)
