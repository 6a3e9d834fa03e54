"""Deferred operators: how the stock operator chain reaches the fused kernels.

A model written the way LiteNN's user guide writes it -- `nn.Conv2D` (conv2D, then `+ bias`),
`nn.leaky_relu`, `nn.max_pool2D`, the next `nn.Conv2D` -- asks for four kernels and three
intermediate tensors per block (litenn/core/module/Conv2D.py:58-62, op/element_wise_op.py:207-221,
op/pool2D.py:47-146).  The library has one kernel for the whole block and an operand format that lets
the next convolution start from it without an NCHW tensor in between, but it can only use them if it
knows what follows a convolution.  So `conv2D` does not launch: it returns a tensor that carries a
record of the work (a `Pending`).  `add` with a per-channel bias, `leaky_relu` and
`max_pool2D(2, 2, 'same')` on such a tensor return a new tensor with the extended record; a
convolution whose input is such a tensor chains to it.  The launch happens when somebody needs the
values: any other operator, `np()`, `set()` (through `Tensor._get_buffers`).  A convolution that
consumes a deferred tensor asks for it in the packed operand format, so the activation between two
convolutions is never written as NCHW.  Values are those of the separate kernels, bit for bit (the
fused epilogues apply the same roundings in the same order).

Intermediate tensors stay valid: each carries its own record and launches its own (shorter) chain if
its values are ever asked for.

Convolutions are only put off in graphs that need no gradient (no trainable tensor upstream, or inside
`optimizer.freeze()`): in a training step they take the eager path with their grad functions.  If a
gradient is asked for anyway (`backward(..., grad_for_non_trainables=True)`), the tape edges of a deferred
convolution are built at that moment by running the trainable form of the same block once.

Per-channel scale, shift and activation (`Chain`) are put off in training too, with one kernel for the gradient.

What has been put off reads its sources when it is launched, so it is launched before one of them is written to.
"""
import contextlib
import functools
import os
import weakref

from . import _lib, ops
from .devices import DeviceBuffer, devices
from .shape import TensorShape
from .tensor import Tensor

_observe = _lib._native.observe           # observe(tensor, watch): the tensor's `_deps` refer weakly to the watch
_enabled = [os.environ.get("LNN_EAGER", "0") != "1"]      # LNN_EAGER=1: every operator launches at once


composed_softmax = [False]      # True: softmax / categorical_crossentropy run as the reference's compositions


@contextlib.contextmanager
def disabled():
    """Inside this context every operator is the reference's own composition, one kernel per
    operator: conv2D launches eagerly, softmax and categorical_crossentropy are built from exp,
    reduce_sum, div, clip, log, mul."""
    old = _enabled[0], composed_softmax[0]
    _enabled[0], composed_softmax[0] = False, True
    try:
        yield
    finally:
        _enabled[0], composed_softmax[0] = old


class _Watch:
    """The tensors of one convolution or chain that may still have to read its sources.  Their records hold it, the
    sources refer to it weakly (`Tensor._deps`)."""
    __slots__ = ("members", "__weakref__")

    def __init__(self):
        self.members = []           # weak references

    def before_write(self):
        for r in self.members:
            t = r()
            if t is not None:
                if t._pending is not None:
                    materialize(t)
                if t._chain is not None:
                    t._chain.changed = True


class _Conv(_Watch):
    """conv2D(x, kernel): what the records of a convolution with more or less behind it have in common."""
    __slots__ = ("x", "kernel", "stride", "dilation", "padding", "geom", "shape")      # shape: of the un-pooled result

    def __init__(self, x, kernel, stride, dilation, padding, geom, shape):
        self.members = []
        self.x, self.kernel = x, kernel
        self.stride, self.dilation, self.padding = stride, dilation, padding
        self.geom, self.shape = geom, shape


class Pending:
    """conv2D(x, kernel) [+ bias] [leaky_relu] [max_pool2D(2, 2, 'same')] not yet launched."""
    __slots__ = ("conv", "bias", "act", "alpha", "pool", "done")

    def __init__(self, conv, bias, act, alpha, pool):
        self.conv, self.bias, self.act, self.alpha, self.pool, self.done = conv, bias, act, alpha, pool, False

    def out_shape(self):
        return _pooled_shape(self.conv.shape.shape) if self.pool else self.conv.shape


@functools.lru_cache(maxsize=4096)
def _pooled_shape(shape):
    n, oc, oh, ow = shape
    return TensorShape((n, oc, (oh + 1) // 2, (ow + 1) // 2))


def before_write(t):
    """The memory of t is about to change: whatever still has to read it does so now."""
    for r in t._deps:
        w = r()
        if w is not None:
            w.before_write()
    t._deps = None                # (kept where one of them could not run)


def _source(t):
    return t._get_top_reference_source()


def reaches_trainable(t, limit=None):
    """True when a gradient could have to flow through t to a trainable tensor, or when `limit` tensors have
    been looked at without an answer.  The last inputs come first: they are the weights."""
    t = _source(t)
    if t._trainable:
        return True
    seen, stack = set(), [t]
    while stack:
        t = stack.pop()
        if t._trainable:
            return True
        if t not in seen:
            if len(seen) == limit:
                return True
            seen.add(t)
            stack.extend([_source(i) for i in t._tape_inputs()])
    return False


def is_deferred(t):
    """t is a tensor whose convolution has not been launched."""
    return _record(_source(t)) is not None


def _record(t):
    """The record of a convolution that has not been launched; None for anything else, references too."""
    p = t._pending
    return p if type(p) is Pending and not p.done else None


def _growing(t):
    """The record that the next operator may extend: not one from the other side of freeze(), which decides
    where gradients stop."""
    p = t._pending
    return p if type(p) is Pending and not p.done and t._freezed == (Tensor._freeze_stack != 0) else None


def _no_tape_needed(*tensors):
    if Tensor._freeze_stack != 0:
        return True
    for t in tensors:
        if t is not None and reaches_trainable(t):
            return False
    return True


def _new(p, op_name):
    return _lib._native.new_tensor(Tensor, DeviceBuffer, devices._current_devices or devices.get_current(), p.out_shape(),
                                   Tensor._freeze_stack, op_name, p, p.conv.members)


def start(input_t, kernel_t, stride, dilation, padding, geom, conv_shape, bias_t=None, act=0, alpha=0.0):
    """The deferred result of conv2D, or None when the call has to run eagerly."""
    if not _enabled[0] or devices._shallow > 0 or not _no_tape_needed(kernel_t, bias_t, input_t):
        return None
    c = _Conv(input_t, kernel_t, stride, dilation, padding, geom, conv_shape)
    _observe(input_t, c)
    _observe(kernel_t, c)
    if bias_t is not None:
        _observe(bias_t, c)
    if _record(input_t) is not None:
        input_t._packed_users = getattr(input_t, "_packed_users", 0) + 1     # its packed copy is wanted once more
    return _new(Pending(c, bias_t, act, float(alpha), False), "conv2D")


def try_bias(a_t, b_t):
    """a + b where a is a deferred convolution without epilogue and b a per-channel bias."""
    p = _growing(a_t)
    if p is None:
        return None
    oc = p.conv.shape.shape[1]
    if p.bias is not None or p.act or p.pool or is_deferred(b_t):
        return None
    if b_t.shape.shape != (1, oc, 1, 1) or not _no_tape_needed(b_t):
        return None
    _observe(b_t, p.conv)
    return _new(Pending(p.conv, b_t, 0, 0.0, False), "add")


def try_act(t, alpha):
    if t._chain is not None:
        return extend_chain(t, act=1, alpha=float(alpha))
    p = _growing(t)
    if p is None or p.act or p.pool or not _no_tape_needed():
        return None
    return _new(Pending(p.conv, p.bias, 1, float(alpha), False), "leaky_relu")


def try_pool(op_type, t, pool_size, stride, padding):
    if op_type != "max" or pool_size != 2 or stride != 2 or padding != "same":
        return None
    p = _growing(t)
    if p is None or p.pool or not _no_tape_needed():
        return None
    return _new(Pending(p.conv, p.bias, p.act, p.alpha, True), "max_pool2D")


def _launch(p, y, y_lo, out_packed, precision):
    """One lnn_conv2d_fwd_packed per device.  A deferred input is taken in the packed format."""
    c = p.conv
    x = c.x
    packed_in = None
    if isinstance(x, ops.PackedActivation):
        packed_in = x
    elif _record(x) is not None:
        packed_in = materialize_packed(x)
    xp, xl = (packed_in.hi, packed_in.lo) if packed_in is not None else (x, None)
    for i, dev in devices._pairs:
        _lib.call.lnn_conv2d_fwd_packed(i, dev, c.geom.address, y, y_lo, xp, xl, c.kernel, p.bias, p.act, p.alpha, p.pool,
                                        packed_in is not None, out_packed, precision)
    if packed_in is not None and packed_in is not x:
        x._packed_users = getattr(x, "_packed_users", 1) - 1
        if x._packed_users <= 0:
            x._packed = None      # the packed copy of the intermediate has served its last consumer


def materialize(t):
    """Launch the work of a deferred tensor into its own (NCHW) buffers.  (In shallow mode it keeps waiting.)"""
    p = t._pending
    if p is None or p.done or devices._shallow > 0:
        return
    p.done = True                 # before the launch: the buffers are about to be requested
    deps, t._deps = t._deps, None     # work that waits for t's values is not disturbed by their arrival
    try:
        if type(p) is Chain:
            t._pending = None
            for i, dev in devices._pairs:
                _lib.call.lnn_channel_chain_fwd(i, dev, t, p.x, p.g, p.b, *p.view, p.act, p.alpha)
        else:
            _launch(p, t, None, False, _lib.precision())
    except BaseException:
        p.done, t._pending = False, p     # (out of memory, say) t still has no values
        raise
    finally:
        t._deps = deps


def materialize_packed(t):
    """The values of a deferred tensor in the packed operand format (no NCHW tensor is written)."""
    cached = getattr(t, "_packed", None)
    if cached is not None:
        return cached
    p = t._pending
    n, oc, oh, ow = p.out_shape().shape
    out = ops._packed_like(n, oc, oh, ow)
    _launch(p, out.hi, out.lo, True, out.precision)
    t._packed = out
    return out


def tape_inputs(t):
    """The tensors a deferred tensor was computed from (what reachability walks need)."""
    p = t._chain
    if p is not None:
        return chain_inputs(p) + list(t._gradfns or ())
    p = t._pending
    ins = [p.conv.kernel]
    if not isinstance(p.conv.x, ops.PackedActivation):
        ins.insert(0, p.conv.x)
    if p.bias is not None:
        ins.append(p.bias)
    return ins


def build_gradfns(t):
    """Tape edges of a deferred tensor, built on demand: the trainable form of the same block runs
    once (its values equal the deferred ones) and its grad functions become t's."""
    p = t._pending
    c = p.conv
    if isinstance(c.x, ops.PackedActivation):
        return None
    _enabled[0] = False
    try:
        bias_1d = None
        if p.bias is not None:
            bias_1d = p.bias if p.bias.shape.rank == 1 else p.bias.reshape((c.shape.shape[1],))
        act = "leaky_relu" if p.act else None
        if p.pool:
            r = ops.conv2D_block(c.x, c.kernel, c.stride, c.dilation, c.padding, bias_t=bias_1d, activation=act,
                                 alpha=p.alpha if p.act else 0.1)
        else:
            r = ops.conv2D(c.x, c.kernel, c.stride, c.dilation, c.padding, bias_t=bias_1d, activation=act,
                           alpha=p.alpha if p.act else 0.1)
    finally:
        _enabled[0] = True
    return r._get_gradfns()


# ---- per-channel scale, shift and activation ------------------------------------------------------
# x * g, + b, leaky_relu with g and b of one element per channel are three passes over a large tensor
# forward and seven backward as separate operators.  They are put off the same way, trainable or not:
# the tensor that is asked for its values launches the whole chain as one kernel, and its gradient is
# one kernel too.  Intermediates cost nothing once nobody holds them; while somebody does, they can be
# asked for values or gradients, so the gradient then goes through them one operator at a time.  A pass
# that keeps the gradients of what is not trainable keeps theirs too (the next pass adds to them), so
# it brings back those that nobody holds.
class Chain:
    """[leaky_relu](x [* g] [+ b]), not launched while the tensor's `_pending` is set."""
    __slots__ = ("x", "g", "b", "act", "alpha", "view", "ancestors", "info", "watch", "changed", "done",
                 "own_link")

    def __init__(self, x, view, watch):
        self.x, self.view, self.watch = x, view, watch
        self.g = self.b = None
        self.act, self.alpha = 0, 0.0
        self.ancestors = ()         # _Links of the shorter chains this one grew from, nearest first
        self.own_link = None        # weak reference to the _Link that the chains grown from this one share
        self.info = None            # broadcast plan of the last mul / add
        self.changed = False        # x, g or b have been written to since the launch
        self.done = False


class _Link:
    """An intermediate of longer chains, as all of them see it.  They hold the link and the intermediate's own
    chain only knows it weakly, so that a tensor kept here goes with the last chain that grew from it."""
    __slots__ = ("tensor", "seq_id", "chain", "kept", "__weakref__")

    def __init__(self, t):
        self.tensor, self.seq_id, self.chain = weakref.ref(t), t._seq_id, t._chain
        self.kept = None            # that tensor, or one in its place, once a pass has kept its gradient

    @staticmethod
    def of(t):
        link = t._chain.own_link and t._chain.own_link()
        if link is None:
            link = _Link(t)
            t._chain.own_link = weakref.ref(link)
        return link


def _chain_tensor(c, shape, op_name):
    t = _lib._native.new_tensor(Tensor, DeviceBuffer, devices._current_devices or devices.get_current(), shape,
                                Tensor._freeze_stack, op_name, c, c.watch.members)
    t._chain = c
    return t


def try_channel(name, a_t, b_t, info):
    """a * b or a + b with one operand per channel, put off; None when it has to run at once."""
    if not _enabled[0] or devices._shallow > 0:
        return None
    full, view = info.channel
    x, v = (a_t, b_t) if full == 0 else (b_t, a_t)
    c = x._chain
    if (name == "add" and c is not None and c.b is None and not c.act and c.view == view and not c.done and
            v._get_top_reference_source() is not c.g._get_top_reference_source() and
            x._freezed == (Tensor._freeze_stack != 0)):
        return extend_chain(x, b=v, info=info)
    if x._get_top_reference_source() is v._get_top_reference_source():
        return None
    c = Chain(x, view, _Watch())
    if name == "mul":
        c.g = v
    else:
        c.b = v
    c.info = info
    _observe(x, c.watch)
    _observe(v, c.watch)
    return _chain_tensor(c, info.output_shape, name)


def extend_chain(t, b=None, info=None, act=0, alpha=0.0):
    """The chain of t with one more operator, or None when it cannot grow."""
    p = t._chain
    if p.act or p.done or t._gradfns is not None or not _enabled[0] or devices._shallow > 0 or t._is_reference() or \
            t._freezed != (Tensor._freeze_stack != 0) or (act and alpha <= 0.0):
        return None
    c = Chain(p.x, p.view, p.watch)
    c.g, c.b, c.info, c.ancestors = p.g, p.b, p.info, (_Link.of(t),) + p.ancestors
    if b is not None:
        c.b, c.info = b, info
        _observe(b, c.watch)
    c.act, c.alpha = act, alpha
    return _chain_tensor(c, t.shape, "leaky_relu" if act else "add")


def _revive(c, link):
    """A tensor in the place of an ancestor of chain c, with its place in the order of the tape."""
    p = link.chain
    a = Chain(p.x, p.view, p.watch)
    a.g, a.b, a.info, a.ancestors, a.changed = p.g, p.b, p.info, p.ancestors, c.changed
    t = _chain_tensor(a, p.info.output_shape, "add" if p.b is not None else "mul")
    t._seq_id = link.seq_id
    return t


def keep_in_chains(t):
    """t is more than its chain says: the chains that have been grown from it hold on to it."""
    link = t._chain.own_link and t._chain.own_link()
    if link is not None:
        link.kept = t


def _from_held(c):
    """(x, g, b): what the gradient of a chain goes through when it starts from the nearest
    intermediate that somebody still holds, or whose gradient a pass has kept."""
    for link in c.ancestors:
        t = link.kept
        if t is None:
            t = link.tensor()
            if ops.backward_pass.keep:
                if t is None:
                    t = _revive(c, link)
                link.kept = t           # as the tape of the separate operators holds it
        if t is not None:
            return t, None, None if t._chain.b is not None else c.b
    return c.x, c.g, c.b


def chain_inputs(c):
    """The tensors the gradient of a chain's end goes to."""
    return [s for s in _from_held(c) if s is not None]


class JointGrad(dict):
    """Grad functions per input, as every tensor has them, and `joint(O_t, dO_t, inputs)`, which adds
    into the gradients of several inputs in one pass."""
    joint = None


def _act_grad(c, t, O_t, dO_t):
    """dt of leaky_relu(t).  A revived t whose sources have changed has lost its values: O has their signs."""
    g, acc = t._grad_to_write()
    signs = O_t if c.changed and any(t is l.kept and t is not l.tensor() for l in c.ancestors) else t
    for i, dev in ops._each_device():
        _lib.call.lnn_eltwise_bwd_acc(i, dev, _lib.EW["leaky_relu"], g, signs, O_t, dO_t, t.shape.size, c.alpha, 0.0, 0, acc)


def chain_gradfns(c, more=None):
    """The grad functions of a chain's end; `more`: those somebody has registered besides."""
    if more is not None:
        fns = {s: list(f) for s, f in chain_gradfns(c).items()}
        for s, f in more.items():
            fns.setdefault(s, []).extend(f)
        return fns
    x, g, b = _from_held(c)
    if g is None and b is None:
        return {x: [lambda O_t, dO_t: _act_grad(c, x, O_t, dO_t)]}
    if not c.act and (g is None or b is None):
        # one operator: the reference's two steps, with its summation order
        name, v = ("add", b) if b is not None else ("mul", g)
        a_t, b_t = (x, v) if c.info.channel[0] == 0 else (v, x)
        return {a_t: [lambda O_t, dO_t: ops._bin_grad(name, c.info, 0, a_t, b_t, O_t, dO_t)],
                b_t: [lambda O_t, dO_t: ops._bin_grad(name, c.info, 1, a_t, b_t, O_t, dO_t)]}

    def joint(O_t, dO_t, inputs):
        targets, flags = [], []
        for s in (x, g, b):
            target, acc = s._grad_to_write() if s is not None and s in inputs else (None, 0)
            targets.append(target)
            flags.append(acc)
        signs = O_t if c.act and c.changed else None        # alpha > 0: the output has the signs of the input
        for i, dev in ops._each_device():
            for target, acc in zip(targets, flags):
                if acc:
                    target._ptr(i)              # (zero-filled where only another device's memory has been touched)
            _lib.call.lnn_channel_chain_bwd(i, dev, *targets, dO_t, x, g, b, signs, *c.view, c.act, c.alpha, *flags)

    fns = JointGrad((s, [lambda O_t, dO_t, s=s: joint(O_t, dO_t, (s,))]) for s in (x, g, b) if s is not None)
    fns.joint = joint
    return fns
