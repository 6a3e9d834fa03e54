"""A device in host memory under the host layer (litenn_b200's Python and its extension module): the tests of
tape, deferral and buffer bookkeeping run without a GPU.  Memory comes from the fake pool full of `JUNK`, so a
tensor whose initializer was skipped shows; a kernel that is not among those below does nothing."""
import contextlib
import ctypes
import gc
import importlib

import numpy as np

from litenn_b200 import _lib

devices_module = importlib.import_module("litenn_b200.devices")      # (the package's attribute of that name is the class)
devices = devices_module.devices
JUNK = 777.0
_EW = {v: k for k, v in _lib.EW.items()}
_BIN = {v: k for k, v in _lib.BIN.items()}
_keep = []          # the callbacks of every fake: a buffer that outlives its test is still freed through them


def floats(address, shape):
    n = int(np.prod(shape))
    return np.frombuffer((ctypes.c_float * n).from_address(address), np.float32).reshape(shape)


def _words(address, n):
    return [int(x) for x in (ctypes.c_int64 * n).from_address(address)]


def _put(target, value, acc):
    target[...] = target + value if acc else value


def _act_grad(t, alpha):
    return np.where(t >= 0, np.float32(1), np.float32(alpha))


class Kernels:
    """The entries of the C library that compute something here, with their C arguments."""

    def lnn_fill_f32(self, dev, p, n, v):
        floats(p, n)[:] = v

    def lnn_h2d(self, dev, dst, src, size):
        ctypes.memmove(dst, src, size)

    def lnn_d2d(self, dev, dst, src, size):
        ctypes.memmove(dst, src, size)

    def lnn_eltwise_fwd(self, dev, op, o, i, n, p0, p1, flag, acc):
        x = floats(i, n)
        f = {"add_const": lambda: x + np.float32(p0), "mul_const": lambda: x * np.float32(p0), "square": lambda: x * x,
             "clip": lambda: np.clip(x, np.float32(p0), np.float32(p1)), "log": lambda: np.log(x),
             "leaky_relu": lambda: x * _act_grad(x, p0)}[_EW[op]]
        _put(floats(o, n), f(), acc)

    def lnn_eltwise_bwd_acc(self, dev, op, di, i, o, do, n, p0, p1, flag, acc):
        x, d = floats(i, n), floats(do, n)
        f = {"add_const": lambda: d, "mul_const": lambda: d * np.float32(p0), "square": lambda: 2 * x * d,
             "clip": lambda: d * ((x >= np.float32(p0)) & (x <= np.float32(p1)) if not flag else 1), "log": lambda: d / x,
             "leaky_relu": lambda: d * _act_grad(x, p0)}[_EW[op]]
        _put(floats(di, n), f(), acc)

    def lnn_binary_fwd(self, dev, op, o, a, b, rank, so, sa, sb, acc):
        x, y = floats(a, _words(sa, rank)), floats(b, _words(sb, rank))
        _put(floats(o, _words(so, rank)), {"add": np.add, "sub": np.subtract, "mul": np.multiply}[_BIN[op]](x, y), acc)

    def lnn_binary_bwd_acc(self, dev, op, which, dx, a, b, o, do, rank, so, sa, sb, acc):
        shape = _words(so, rank)
        other = floats(b, _words(sb, rank)) if which == 0 else floats(a, _words(sa, rank))
        f = {"add": lambda: 1.0, "sub": lambda: 1.0 if which == 0 else -1.0, "mul": lambda: other}[_BIN[op]]
        _put(floats(dx, shape), floats(do, shape) * np.float32(f()) if _BIN[op] != "mul" else floats(do, shape) * f(), acc)

    def lnn_reduce(self, dev, op, o, i, outer, r0, mid, r1, inner, acc):
        x = floats(i, (outer, r0, mid, r1, inner))
        v = x.sum((1, 3)) if op < 2 else (x.max((1, 3)) if op == 2 else x.min((1, 3)))
        _put(floats(o, (outer, mid, inner)), v / np.float32(r0 * r1) if op == 1 else v, acc)

    def lnn_slice_fwd(self, dev, o, i, rank, si, so, begin, step, acc):
        _put(floats(o, _words(so, rank)), floats(i, _words(si, rank))[_index(rank, so, begin, step)], acc)

    def lnn_slice_bwd(self, dev, di, do, rank, si, so, begin, step):
        floats(di, _words(si, rank))[_index(rank, so, begin, step)] += floats(do, _words(so, rank))

    def lnn_channel_chain_fwd(self, dev, y, x, g, b, outer, ch, inner, act, alpha):
        floats(y, (outer, ch, inner))[...] = self._chain(x, g, b, outer, ch, inner, act, alpha)

    def lnn_channel_chain_bwd(self, dev, dx, dg, db, dy, x, g, b, s, outer, ch, inner, act, alpha, acc_x, acc_g, acc_b):
        shape = (outer, ch, inner)
        dz = floats(dy, shape)
        if act:
            dz = dz * _act_grad(floats(s, shape) if s else self._chain(x, g, b, outer, ch, inner, 0, 0.0), alpha)
        if dx:
            _put(floats(dx, shape), dz * floats(g, (ch, 1)) if g else dz, acc_x)
        if dg:
            _put(floats(dg, ch), (dz * floats(x, shape)).sum((0, 2)), acc_g)
        if db:
            _put(floats(db, ch), dz.sum((0, 2)), acc_b)

    @staticmethod
    def _chain(x, g, b, outer, ch, inner, act, alpha):
        t = floats(x, (outer, ch, inner))
        t = t * floats(g, (ch, 1)) if g else t
        t = t + floats(b, (ch, 1)) if b else t
        return t * _act_grad(t, alpha) if act else t


def _index(rank, so, begin, step):
    return np.ix_(*[[b + k * s for k in range(n)] for n, b, s in zip(_words(so, rank), _words(begin, rank), _words(step, rank))])


class FakeDevice:
    """The library object and, through `calls` (names in order) and `fail` (name -> status of the next call),
    what a test sees and breaks."""

    def __init__(self, count):
        self.calls, self.fail, self.errors = [], {}, []
        self.memory = {}
        self._kernels = Kernels()
        self.devices = []
        for i in range(count):
            d = devices_module.Device(i, f"fake {i}", 1 << 30, 148, (10, 0))
            d._inited = True
            self.devices.append(d)

    # -- what the host layer asks of the ctypes library object
    def lnn_last_error(self):
        return b"fake device"

    def lnn_sync(self, dev):
        return 0

    def lnn_shutdown(self, dev):
        return 0

    def lnn_d2h(self, dev, dst, src, size):
        ctypes.memmove(dst, src, size)

    def lnn_nccl_group_start(self):
        return 0

    lnn_nccl_group_end = lnn_nccl_group_start

    def lnn_nccl_allreduce_sum(self, dev, p, n):
        floats(p, n)[:] *= 2                      # (every replica has the same values)

    # -- the pool
    def _alloc(self, dev, size, out):
        self.calls.append("lnn_alloc")
        if self.fail.get("lnn_alloc"):
            return self.fail.pop("lnn_alloc")
        a = np.full((size + 3) // 4, JUNK, np.float32)
        self.memory[a.ctypes.data] = a
        out[0] = a.ctypes.data
        return 0

    def _free(self, dev, p, size):
        self.memory.pop(p, None)
        return 0

    # -- kernels
    def _entry(self, name):
        kernel = getattr(self._kernels, name, None)

        def entry(*args):
            self.calls.append(name)
            if self.fail.get(name):
                return self.fail.pop(name)
            try:
                if kernel is not None:
                    kernel(*args)
            except Exception as e:                # (an exception may not pass through the C caller)
                self.errors.append(e)
                return _lib.E_INVALID
            return 0
        return entry


@contextlib.contextmanager
def fake_device(count=1):
    """Put the fake under the host layer; the library and the devices of before come back at the end."""
    fake = FakeDevice(count)
    saved = _lib._lib, dict(vars(_lib.call)), devices._all_devices, devices._current_devices, devices._pairs
    alloc = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_int, ctypes.c_uint64, ctypes.POINTER(ctypes.c_uint64))(fake._alloc)
    free = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_int, ctypes.c_uint64, ctypes.c_uint64)(fake._free)
    _keep.append((fake, alloc, free))
    address = lambda f: ctypes.cast(f, ctypes.c_void_p).value      # noqa: E731
    _lib._native.bind(address(alloc), address(free), _lib._raise_status)
    for name, letters in _lib._CALLS.items():
        f = ctypes.CFUNCTYPE(ctypes.c_int, *[ctypes.c_float if c == "f" else ctypes.c_int64 for c in letters])(fake._entry(name))
        _keep.append(f)
        setattr(_lib.call, name, _lib._native.Function(address(f), name, letters))
    _lib._lib = fake
    devices._all_devices, devices._current_devices = fake.devices, tuple(fake.devices)
    devices._pairs = [(i, d.index) for i, d in enumerate(fake.devices)]
    try:
        yield fake
    finally:
        gc.collect()
        _lib._lib, calls, devices._all_devices, devices._current_devices, devices._pairs = saved
        vars(_lib.call).clear()
        vars(_lib.call).update(calls)
        if _lib._lib is not None:
            real = lambda name: ctypes.cast(getattr(_lib._lib, name), ctypes.c_void_p).value      # noqa: E731
            _lib._native.bind(real("lnn_alloc"), real("lnn_free"), _lib._raise_status)
