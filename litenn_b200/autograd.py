"""Reverse pass over the dynamic tape (the contract of litenn/core/backward.py:8-158).

Tensors are processed in descending creation order; each grad function adds into the
lazily created zero gradient of its input; branches that cannot reach a trainable tensor
are pruned unless grad_for_non_trainables; gradients of non-trainable intermediates are
released as soon as they have been consumed.
"""
import heapq

from . import ops
from .tensor import Tensor, Tensor_from_value


def backward(loss, stop_grad=None, grad_for_non_trainables=False, keep_gradient_for_non_trainables=False):
    state = ops.backward_pass
    outer_keep = state.keep
    state.keep = bool(grad_for_non_trainables or keep_gradient_for_non_trainables)
    try:
        _backward(state, loss, stop_grad, grad_for_non_trainables, state.keep)
    finally:
        state.keep = outer_keep


def _backward(state, loss, stop_grad, grad_for_non_trainables, keep):
    loss_gradients = {}
    if isinstance(loss, dict):
        loss_gradients = loss
        loss = list(loss.keys())
    elif not isinstance(loss, (tuple, list)):
        loss = [loss]
    if stop_grad is None:
        stop_grad = []
    elif not isinstance(stop_grad, (tuple, list)):
        stop_grad = [stop_grad]
    user_stop = set(t._get_seq_id() for t in stop_grad)

    # ---- which tensors lead to a trainable leaf? ----------------------------------------
    # `blocked` holds sequence ids through which no gradient has to flow.
    blocked = user_stop
    if not grad_for_non_trainables:
        reaches = {}            # seq id -> True if a trainable tensor is reachable (in user_stop too: it is blocked below)
        stack = [t._get_top_reference_source() for t in loss]
        while stack:
            t = stack[-1]
            sid = t._seq_id
            if reaches.get(sid) is not None:
                stack.pop()
                continue
            if t._trainable:
                reaches[sid] = True
                stack.pop()
                continue
            inputs = t._tape_inputs()
            if sid not in reaches:
                reaches[sid] = None                     # its inputs first
                todo = [s for s in (i._get_top_reference_source() for i in inputs) if s._seq_id not in reaches]
                if todo:
                    stack.extend(todo)
                    continue
            r = False
            for i in inputs:
                if reaches.get(i._get_top_reference_source()._seq_id):
                    r = True
                    break
            reaches[sid] = r
            stack.pop()
        blocked = {sid for sid, r in reaches.items() if not r} | user_stop

    loss_list = [t for t in loss if t._get_seq_id() not in blocked]

    state.depth += 1
    try:
        # ---- seed -------------------------------------------------------------------------
        for t in loss_list:
            if t not in loss_gradients:
                g, acc = t._grad_to_write()
                if acc:
                    ops.add_const_op(g, 1.0, output_t=g)
                else:
                    g.fill(1.0)
                continue
            value = loss_gradients[t]
            if not isinstance(value, Tensor):
                value = Tensor_from_value(value)
            # a gradient that does not exist yet takes the given one's memory; get_grad() copies it before a write
            if value.shape != t.shape or not ops.share_grad(t, value):
                g, acc = t._grad_to_write()
                if acc or value.shape != t.shape:
                    ops.add_op(g, value, output_t=g)
                else:
                    g.set(value)

        # ---- walk: max-heap on sequence id ------------------------------------------------
        heap, queued = [], set()
        for t in loss_list:
            t = t._get_top_reference_source()
            if t._seq_id not in queued:
                queued.add(t._seq_id)
                heapq.heappush(heap, (-t._seq_id, t))

        while heap:
            t = heapq.heappop(heap)[1]
            fns = t._get_gradfns()
            if fns is not None:
                freezed = t._freezed
                joint = getattr(fns, "joint", None)
                together = []
                for input_t, funcs in fns.items():
                    source = input_t._get_top_reference_source()
                    sid = source._seq_id
                    if sid in blocked or (freezed and source._trainable):
                        continue
                    if joint is not None:
                        together.append(input_t)
                    else:
                        for func in funcs:
                            func(t, t._grad_t or t.get_grad())
                    if sid not in queued:
                        queued.add(sid)
                        heapq.heappush(heap, (-sid, source))
                if together:
                    joint(t, t._grad_t or t.get_grad(), together)
            if not keep and not t._trainable:
                t._grad_t = None
    finally:
        state.depth -= 1
        # gradients that outlive the pass get memory of their own
        if state.depth == 0:
            shared, state.shared = state.shared, []
            for t in shared:
                if t._grad_t is not None:
                    t.get_grad()
