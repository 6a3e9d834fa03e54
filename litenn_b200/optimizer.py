"""Optimizer base, SGD (momentum, nesterov), RMSprop, Adam and `freeze`
(litenn/core/optimizer/Optimizer.py:36-203, SGD.py:28-83, RMSprop.py:26-69, Adam.py:28-84,
optimizer/__init__.py:9-25).  An optimizer is a saveable module: `iteration` and its state
tensors (`_accs`, or `_ms` / `_vs`) appear in checkpoints under the reference's keys.

All tensors of an optimizer are updated by ONE fused kernel (the reference launches two or three per
tensor), with the same operations in the same order.  The multi-device step all-reduces the GRADIENTS over NCCL and
folds 1/replicas into the update, so replicas stay identical; for plain SGD started from
identical weights that equals the reference's host-side weight averaging
(Optimizer.py:149-153)."""
import ctypes

import numpy as np

from . import _lib
from . import ops
from . import parallel
from .devices import devices
from .module import ModuleBase
from .tensor import Tensor, Tensor_zeros_like


class freeze:
    """with nn.optimizer.freeze(): tensors produced inside do not pass gradient to
    trainable inputs (backward.py:135-137)."""

    def __enter__(self):
        Tensor._freeze_stack += 1
        return self

    def __exit__(self, *exc):
        Tensor._freeze_stack -= 1
        if Tensor._freeze_stack < 0:
            raise ValueError("Wrong _freeze_stack")


class OptParams(ctypes.Structure):
    """Mirror of struct lnn_opt_params."""
    _fields_ = [("lr", ctypes.c_float), ("lr_decay", ctypes.c_float), ("lr_dropout", ctypes.c_float),
                ("gscale", ctypes.c_float), ("beta1", ctypes.c_float), ("beta2", ctypes.c_float),
                ("iteration", ctypes.c_uint32), ("seed_a", ctypes.c_uint32), ("seed_b", ctypes.c_uint32),
                ("nesterov", ctypes.c_int)]


SGD_KIND, RMSPROP_KIND, ADAM_KIND = 0, 1, 2


class Optimizer(ModuleBase):
    """Base class: Optimizer(tensors_list, lr, lr_decay, lr_dropout, clipnorm, saveables)."""

    def __init__(self, _tensors_list, lr=0.001, lr_decay=0.0, lr_dropout=0.0, clipnorm=0.0, saveables=None):
        if _tensors_list is None:
            raise ValueError("_tensors_list must be specified.")
        _tensors_list = list(_tensors_list)
        seen, names = set(), {}
        for i, t in enumerate(_tensors_list):
            if id(t) in seen:
                raise ValueError(f"Tensor {t.get_name()} has duplicate in a list.")
            seen.add(id(t))
            name = t.get_name()
            if name in names:
                raise ValueError(f"Different tensors with the same name '{name}' indexes {names[name]} {i}. "
                                 f"If the same module class is used twice, subclass it under two names.")
            names[name] = i
        for t in _tensors_list:
            if t._is_reference():
                raise ValueError(f"Tensor {t.get_name()} is reference, and cannot be trained in optimizer.")
            if t._is_grad():
                raise ValueError(f"Tensor {t.get_name()} is gradient tensor, and cannot be trained in optimizer.")
            if t._is_trainable():
                raise ValueError(f"Tensor {t.get_name()} is already used by another optimizer.")
            if t._get_gradfns() is not None:
                raise Exception(f"Tensor {t.get_name()} is produced by operator and cannot be trained in optimizer.")
            t._set_trainable(True)
        self._tensors_list = _tensors_list
        self.lr = lr
        self.lr_decay = lr_decay
        self.lr_dropout = lr_dropout
        self.clipnorm = clipnorm
        self.iteration = 0
        super().__init__((saveables or []) + ["iteration"])

    def get_trainable_tensors(self):
        return self._tensors_list

    def get_iteration(self):
        return self.iteration

    def set_iteration(self, iteration):
        self.iteration = iteration

    def zero_grad(self):
        for t in self._tensors_list:
            t.zero_grad()

    def print_no_grad(self):
        for t in self.get_trainable_tensors():
            if not t.has_grad():
                print(f"Tensor has no gradient : {t.get_name()}")

    def step(self, multi_gpu_step=False):
        """Apply one update.  multi_gpu_step=True keeps the replicas in step: gradients are summed
        over all devices / ranks with one group of NCCL all-reduces and the update uses their mean.
        With several current devices and no communicator yet, the single-process communicator is
        created here (the reference averages whenever more than one device is current,
        Optimizer.py:149-153)."""
        tensors = [t for t in self._tensors_list if t.has_grad()]
        gscale = 1.0
        if multi_gpu_step and devices._shallow == 0:
            if parallel.world_size() == 1 and len(devices.get_current()) > 1:
                parallel.init_single_process()
            if parallel.world_size() > 1:
                parallel.allreduce_grads(tensors)
                gscale = 1.0 / parallel.world_size()
        if self.clipnorm != 0.0:
            sums = [ops.square(t.get_grad()).sum().np()[0] for t in tensors]
            l2 = float(np.sqrt(np.sum(sums))) * gscale
            if l2 > self.clipnorm:
                gscale *= self.clipnorm / l2
        self._on_step(tensors, gscale)
        self.iteration += 1

    def _state_tensors(self):
        """{tensor name at construction: zero tensor}, the reference's accumulator dicts."""
        return {t.get_name(): Tensor_zeros_like(t) for t in self.get_trainable_tensors()}

    def _step_all(self, kind, tensors, s1, s2, gscale, beta1, beta2, nesterov, draws):
        """One launch for all tensors.  `draws` seeds per tensor are taken from the host's random stream,
        as the reference does for every kernel that takes the learning rate (Optimizer.py:176-180),
        so that the stream stays in step with a run on the reference."""
        n = len(tensors)
        if n == 0:
            return
        drawn = np.random.randint(2147483648, size=draws * n)
        if devices._shallow > 0:
            return
        seeds = None
        if self.lr_dropout != 0.0:
            seeds = np.repeat(drawn, 2 // draws).astype(np.uint32)
        p = OptParams(float(self.lr), float(self.lr_decay), float(self.lr_dropout), float(gscale), float(beta1), float(beta2),
                      int(self.iteration) & 0xFFFFFFFF, 0, 0, 1 if nesterov else 0)
        sizes = (ctypes.c_int64 * n)(*[t.shape.size for t in tensors])
        grads = [t.get_grad() for t in tensors]
        for i, dev in devices._pairs:
            _lib.call.lnn_optimizer_step_many(i, dev, kind, n, tensors, grads, s1, s2 if s2 is not None else s1,
                                              ctypes.addressof(sizes), seeds.ctypes.data if seeds is not None else 0,
                                              ctypes.addressof(p))

    def _on_step(self, tensors, gscale):
        raise NotImplementedError()


class SGD(Optimizer):
    """SGD(tensors_list, momentum=0.0, nesterov=False, lr=0.001, lr_decay=0.0, lr_dropout=0.0,
    clipnorm=0.0): A = momentum*A - lr*G; V += A (nesterov: V += momentum*A - lr*G)."""

    def __init__(self, tensors_list, momentum=0.0, nesterov=False, lr=0.001, lr_decay=0.0, lr_dropout=0.0, clipnorm=0.0):
        super().__init__(tensors_list, lr=lr, lr_decay=lr_decay, lr_dropout=lr_dropout, clipnorm=clipnorm,
                         saveables=["_accs"])
        self.momentum = momentum
        self.nesterov = nesterov
        self._accs = self._state_tensors()
        self._names = {id(t): t.get_name() for t in self.get_trainable_tensors()}

    def _on_step(self, tensors, gscale):
        names = self._names
        self._step_all(SGD_KIND, tensors, [self._accs[names[id(t)]] for t in tensors], None, gscale, self.momentum, 0.0,
                       self.nesterov, 2)


class RMSprop(Optimizer):
    """RMSprop(tensors_list, rho=0.9, lr=0.001, ...): A = rho*A + (1-rho)*G*G;
    V += -lr*G / (sqrt(A) + 1e-7)."""

    def __init__(self, tensors_list, rho=0.9, lr=0.001, lr_decay=0.0, lr_dropout=0.0, clipnorm=0.0):
        super().__init__(tensors_list, lr=lr, lr_decay=lr_decay, lr_dropout=lr_dropout, clipnorm=clipnorm,
                         saveables=["_accs"])
        self._accs = self._state_tensors()
        self._names = {id(t): t.get_name() for t in self.get_trainable_tensors()}
        self.rho = rho

    def _on_step(self, tensors, gscale):
        names = self._names
        self._step_all(RMSPROP_KIND, tensors, [self._accs[names[id(t)]] for t in tensors], None, gscale, self.rho, 0.0,
                       False, 1)


class Adam(Optimizer):
    """Adam(tensors_list, beta_1=0.9, beta_2=0.999, lr=0.001, ...) without bias correction, as the
    reference: M = b1*M + (1-b1)*G; U = b2*U + (1-b2)*G*G; V += -lr*M / (sqrt(U) + 1e-7)."""

    def __init__(self, tensors_list, beta_1=0.9, beta_2=0.999, lr=0.001, lr_decay=0.0, lr_dropout=0.0, clipnorm=0.0):
        super().__init__(tensors_list, lr=lr, lr_decay=lr_decay, lr_dropout=lr_dropout, clipnorm=clipnorm,
                         saveables=["_ms", "_vs"])
        self.beta_1 = beta_1
        self.beta_2 = beta_2
        self._ms = self._state_tensors()
        self._vs = self._state_tensors()
        self._names = {id(t): t.get_name() for t in self.get_trainable_tensors()}

    def _on_step(self, tensors, gscale):
        keys = [self._names[id(t)] for t in tensors]
        self._step_all(ADAM_KIND, tensors, [self._ms[k] for k in keys], [self._vs[k] for k in keys], gscale, self.beta_1,
                       self.beta_2, False, 1)
