"""ctypes binding of liblitenn_b200.so (declared in include/litenn_b200.h).

Plays the part litenn/core/minicl/api/OpenCL/OpenCL.py plays in the reference: every
entry point gets argtypes, and a non-zero return code raises LnnError carrying
lnn_last_error() (the reference raises CLException from its errcheck hook,
OpenCL.py:175-198).  There is no fallback: if the shared library is missing the first
device call fails loudly.
"""
import ctypes
import os
from ctypes import (POINTER, c_char_p, c_float, c_int, c_int64, c_uint64, c_void_p)

_HERE = os.path.dirname(os.path.abspath(__file__))
if not os.path.exists(os.path.join(_HERE, "_native.so")):
    # the host layer's extension module: the package itself cannot be imported without it, so a fresh
    # source tree compiles it here (a few seconds)
    from .csrc.build import build_native
    build_native()
from . import _native       # noqa: E402
LIB_PATH = os.environ.get("LNN_LIB") or os.path.join(_HERE, "liblitenn_b200.so")

OK, E_INVALID, E_CUDA, E_NOMEM, E_NOTINIT, E_UNSUPPORTED, E_NCCL, E_TIMEOUT = 0, -1, -2, -3, -4, -5, -6, -7
MAX_DIMS = 6

EW = {name: i for i, name in enumerate(
    ["abs", "add_const", "clip", "cos", "exp", "leaky_relu", "log", "mul_const", "rdiv_const",
     "rsub_const", "relu", "sigmoid", "sin", "sqrt", "square", "tanh"])}
BIN = {name: i for i, name in enumerate(["add", "sub", "mul", "div", "max", "min", "binary_crossentropy"])}
POOL = {"avg": 0, "max": 1, "min": 2}
RED = {"sum": 0, "mean": 1, "max": 2, "min": 3}


class LnnError(Exception):
    """A C-ABI call returned a negative status."""

    def __init__(self, code, message, func=None):
        self.code = code
        self.func = func
        super().__init__(f"{func or 'lnn'}: [{code}] {message}")


class ConvGeom(ctypes.Structure):
    """Mirror of struct lnn_conv_geom."""
    _fields_ = [(n, c_int) for n in
                ("n", "ic", "ih", "iw", "oc", "kh", "kw", "oh", "ow", "stride", "dilation", "padl", "padt")]

    def __init__(self, *values):
        super().__init__(*values)
        self.address = ctypes.addressof(self)


_I64P = POINTER(c_int64)
_SIGNATURES = {
    "lnn_version": (c_int, []),
    "lnn_last_error": (c_char_p, []),
    "lnn_device_count": (c_int, [POINTER(c_int)]),
    "lnn_device_info": (c_int, [c_int, c_char_p, c_int, POINTER(c_uint64), POINTER(c_int), POINTER(c_int), POINTER(c_int)]),
    "lnn_init": (c_int, [c_int]),
    "lnn_shutdown": (c_int, [c_int]),
    "lnn_alloc": (c_int, [c_int, c_uint64, POINTER(c_uint64)]),
    "lnn_free": (c_int, [c_int, c_uint64, c_uint64]),
    "lnn_mem_stats": (c_int, [c_int, POINTER(c_uint64), POINTER(c_uint64)]),
    "lnn_pool_trim": (c_int, [c_int]),
    "lnn_h2d": (c_int, [c_int, c_uint64, c_void_p, c_uint64]),
    "lnn_d2h": (c_int, [c_int, c_void_p, c_uint64, c_uint64]),
    "lnn_d2d": (c_int, [c_int, c_uint64, c_uint64, c_uint64]),
    "lnn_fill_f32": (c_int, [c_int, c_uint64, c_int64, c_float]),
    "lnn_init_uniform": (c_int, [c_int, c_uint64, c_int64, ctypes.c_uint32, c_float, c_float]),
    "lnn_init_normal": (c_int, [c_int, c_uint64, c_int64, ctypes.c_uint32, c_float, c_float]),
    "lnn_sync": (c_int, [c_int]),
    "lnn_h2d_async": (c_int, [c_int, c_uint64, c_void_p, c_uint64]),
    "lnn_d2h_async": (c_int, [c_int, c_void_p, c_uint64, c_uint64]),
    "lnn_h2d_prefetch": (c_int, [c_int, c_uint64, c_void_p, c_uint64, c_uint64]),
    "lnn_wait_prefetch": (c_int, [c_int]),
    "lnn_d2h_readback": (c_int, [c_int, c_void_p, c_uint64, c_uint64]),
    "lnn_wait_readback": (c_int, [c_int]),
    "lnn_host_alloc": (c_int, [c_uint64, POINTER(c_void_p)]),
    "lnn_host_free": (c_int, [c_void_p]),
    "lnn_launch_count": (c_int, [c_int, POINTER(c_uint64)]),
    "lnn_device_status": (c_int, [c_int, POINTER(c_int)]),
    "lnn_debug_set_status": (c_int, [c_int, c_int, c_int, c_int, c_int]),
    "lnn_event_create": (c_int, [c_int, POINTER(c_uint64)]),
    "lnn_event_record": (c_int, [c_int, c_uint64]),
    "lnn_event_elapsed_ms": (c_int, [c_int, c_uint64, c_uint64, POINTER(c_float)]),
    "lnn_event_destroy": (c_int, [c_int, c_uint64]),
    "lnn_profile_enable": (c_int, [c_int, c_int]),
    "lnn_profile_read": (c_int, [c_int, c_int, POINTER(c_uint64), POINTER(c_float)]),
    "lnn_eltwise_fwd": (c_int, [c_int, c_int, c_uint64, c_uint64, c_int64, c_float, c_float, c_int, c_int]),
    "lnn_eltwise_bwd": (c_int, [c_int, c_int, c_uint64, c_uint64, c_uint64, c_uint64, c_int64, c_float, c_float, c_int]),
    "lnn_binary_fwd": (c_int, [c_int, c_int, c_uint64, c_uint64, c_uint64, c_int, _I64P, _I64P, _I64P, c_int]),
    "lnn_binary_bwd": (c_int, [c_int, c_int, c_int, c_uint64, c_uint64, c_uint64, c_uint64, c_uint64, c_int, _I64P, _I64P, _I64P]),
    "lnn_softmax_fwd": (c_int, [c_int, c_uint64, c_uint64, c_int64, c_int64]),
    "lnn_softmax_bwd": (c_int, [c_int, c_uint64, c_uint64, c_uint64, c_int64, c_int64]),
    "lnn_cce_fwd": (c_int, [c_int, c_uint64, c_uint64, c_uint64, c_int64, c_int64, c_int64]),
    "lnn_cce_bwd": (c_int, [c_int, c_uint64, c_uint64, c_uint64, c_uint64, c_int64, c_int64, c_int64]),
    "lnn_scale_bias_lrelu": (c_int, [c_int, c_uint64, c_uint64, c_uint64, c_uint64, c_int64, c_int64, c_int64, c_float, c_int]),
    "lnn_channel_chain_fwd": (c_int, [c_int, c_uint64, c_uint64, c_uint64, c_uint64, c_int64, c_int64, c_int64, c_int, c_float]),
    "lnn_channel_chain_bwd": (c_int, [c_int] + [c_uint64] * 8 + [c_int64, c_int64, c_int64, c_int, c_float, c_int, c_int, c_int]),
    "lnn_pool2d_fwd": (c_int, [c_int, c_int, c_uint64, c_uint64, c_int64, c_int64] + [c_int] * 8),
    "lnn_pool2d_bwd": (c_int, [c_int, c_int, c_uint64, c_uint64, c_uint64, c_uint64, c_int64, c_int64] + [c_int] * 8),
    "lnn_pool2x2_lrelu_bwd": (c_int, [c_int, c_uint64, c_uint64, c_uint64, c_uint64, c_int64, c_int64, c_int, c_int, c_float, c_int]),
    "lnn_pool2x2_idx_lrelu_bwd": (c_int, [c_int, c_uint64, c_uint64, c_uint64, c_uint64, c_uint64, c_int64, c_int64, c_int, c_int, c_float, c_int]),
    "lnn_pool2x2_winner_grad": (c_int, [c_int, c_uint64, c_uint64, c_uint64, c_uint64, c_int64, c_int64, c_int, c_int, c_float, c_int]),
    "lnn_conv2d_dw_winners": (c_int, [c_int, POINTER(ConvGeom), c_uint64, c_uint64, c_uint64, c_uint64]),
    "lnn_pool2x2_idx_lrelu_bwd_packed": (c_int, [c_int, c_uint64, c_uint64, c_uint64, c_uint64, c_uint64, c_uint64, c_int64, c_int64, c_int, c_int, c_float, c_int]),
    "lnn_reduce": (c_int, [c_int, c_int, c_uint64, c_uint64] + [c_int64] * 5 + [c_int]),
    "lnn_reduce_noalloc": (c_int, [c_int, c_int, c_uint64, c_uint64] + [c_int64] * 5 + [c_int]),
    "lnn_reduce_bwd": (c_int, [c_int, c_int, c_uint64, c_uint64, c_uint64, c_uint64] + [c_int64] * 5),
    "lnn_transpose": (c_int, [c_int, c_uint64, c_uint64, c_int, _I64P, POINTER(c_int), c_int]),
    "lnn_slice_fwd": (c_int, [c_int, c_uint64, c_uint64, c_int, _I64P, _I64P, _I64P, _I64P, c_int]),
    "lnn_slice_bwd": (c_int, [c_int, c_uint64, c_uint64, c_int, _I64P, _I64P, _I64P, _I64P]),
    "lnn_gemm_f32": (c_int, [c_int, c_uint64, c_uint64, c_uint64, c_uint64, c_int64, c_int64, c_int64, c_int64, c_int, c_int, c_int, c_int]),
    "lnn_conv2d_fwd": (c_int, [c_int, POINTER(ConvGeom), c_uint64, c_uint64, c_uint64, c_uint64, c_int, c_float, c_int, c_int]),
    "lnn_conv2d_pool_fwd": (c_int, [c_int, POINTER(ConvGeom), c_uint64, c_uint64, c_uint64, c_uint64, c_int, c_float, c_int]),
    "lnn_packed_bytes": (c_int, [c_int64, c_int64, c_int64, c_int64, c_int, POINTER(c_uint64), POINTER(c_uint64)]),
    "lnn_nhwc_split": (c_int, [c_int, c_uint64, c_uint64, c_uint64, c_int, c_int, c_int, c_int, c_int]),
    "lnn_conv2d_fwd_packed": (c_int, [c_int, POINTER(ConvGeom), c_uint64, c_uint64, c_uint64, c_uint64, c_uint64, c_uint64,
                                      c_int, c_float, c_int, c_int, c_int, c_int]),
    "lnn_conv2d_dx": (c_int, [c_int, POINTER(ConvGeom), c_uint64, c_uint64, c_uint64, c_int]),
    "lnn_conv2d_dw": (c_int, [c_int, POINTER(ConvGeom), c_uint64, c_uint64, c_uint64, c_int]),
    "lnn_conv2d_dx_packed": (c_int, [c_int, POINTER(ConvGeom), c_uint64, c_uint64, c_uint64, c_uint64, c_int]),
    "lnn_conv2d_dw_packed": (c_int, [c_int, POINTER(ConvGeom), c_uint64, c_uint64, c_uint64, c_uint64, c_uint64, c_int]),
    "lnn_conv2d_transpose_fwd": (c_int, [c_int, POINTER(ConvGeom), c_uint64, c_uint64, c_uint64, c_int, c_int]),
    "lnn_conv2d_transpose_dx": (c_int, [c_int, POINTER(ConvGeom), c_uint64, c_uint64, c_uint64, c_int]),
    "lnn_conv2d_transpose_dk": (c_int, [c_int, POINTER(ConvGeom), c_uint64, c_uint64, c_uint64, c_int]),
    "lnn_depthwise_conv2d_fwd": (c_int, [c_int, POINTER(ConvGeom), c_uint64, c_uint64, c_uint64, c_int]),
    "lnn_depthwise_conv2d_dx": (c_int, [c_int, POINTER(ConvGeom), c_uint64, c_uint64, c_uint64]),
    "lnn_depthwise_conv2d_dk": (c_int, [c_int, POINTER(ConvGeom), c_uint64, c_uint64, c_uint64]),
    "lnn_eltwise_bwd_acc": (c_int, [c_int, c_int, c_uint64, c_uint64, c_uint64, c_uint64, c_int64, c_float, c_float, c_int, c_int]),
    "lnn_binary_bwd_acc": (c_int, [c_int, c_int, c_int, c_uint64, c_uint64, c_uint64, c_uint64, c_uint64, c_int, _I64P, _I64P, _I64P, c_int]),
    "lnn_softmax_bwd_acc": (c_int, [c_int, c_uint64, c_uint64, c_uint64, c_int64, c_int64, c_int]),
    "lnn_cce_bwd_acc": (c_int, [c_int, c_uint64, c_uint64, c_uint64, c_uint64, c_int64, c_int64, c_int64, c_int]),
    "lnn_pool2d_fwd_idx": (c_int, [c_int, c_int, c_uint64, c_uint64, c_uint64, c_int64, c_int64] + [c_int] * 8),
    "lnn_pool2d_bwd_idx": (c_int, [c_int, c_int, c_uint64, c_uint64, c_uint64, c_int64, c_int64] + [c_int] * 9),
    "lnn_pool2d_bwd_acc": (c_int, [c_int, c_int, c_uint64, c_uint64, c_uint64, c_uint64, c_int64, c_int64] + [c_int] * 9),
    "lnn_reduce_bwd_acc": (c_int, [c_int, c_int, c_uint64, c_uint64, c_uint64, c_uint64] + [c_int64] * 5 + [c_int]),
    "lnn_conv2d_dx_acc": (c_int, [c_int, POINTER(ConvGeom), c_uint64, c_uint64, c_uint64, c_int, c_uint64, c_int, c_int]),
    "lnn_conv2d_dw_acc": (c_int, [c_int, POINTER(ConvGeom), c_uint64, c_uint64, c_uint64, c_uint64, c_uint64, c_int, c_int, c_int]),
    "lnn_conv2d_dw_winners_acc": (c_int, [c_int, POINTER(ConvGeom), c_uint64, c_uint64, c_uint64, c_uint64, c_int]),
    "lnn_sgd_step": (c_int, [c_int, c_uint64, c_uint64, c_int64, c_float, c_float]),
    "lnn_optimizer_step": (c_int, [c_int, c_int, c_uint64, c_uint64, c_uint64, c_uint64, c_int64, c_void_p]),
    "lnn_optimizer_step_many": (c_int, [c_int, c_int, c_int] + [POINTER(c_uint64)] * 4 + [_I64P, POINTER(ctypes.c_uint32), c_void_p]),
    "lnn_nccl_unique_id": (c_int, [c_void_p]),
    "lnn_nccl_init_rank": (c_int, [c_int, c_int, c_int, c_void_p]),
    "lnn_nccl_init_all": (c_int, [POINTER(c_int), c_int]),
    "lnn_nccl_allreduce_sum": (c_int, [c_int, c_uint64, c_int64]),
    "lnn_nccl_group_start": (c_int, []),
    "lnn_nccl_group_end": (c_int, []),
    "lnn_nccl_destroy": (c_int, [c_int]),
}
# How the host layer calls the compute entries: call.<name>(i, ...) for current device number i, with tensors
# in place of device pointers (_native.Function explains the letters).
_CALLS = {
    "lnn_fill_f32": "nwnf",
    "lnn_h2d": "nwnn",
    "lnn_d2d": "nwpn",
    "lnn_eltwise_fwd": "nnopnffna",
    "lnn_eltwise_bwd_acc": "nnopppnffna",
    "lnn_binary_fwd": "nnoppnnnna",
    "lnn_binary_bwd_acc": "nnnoppppnnnna",
    "lnn_softmax_fwd": "nwpnn",
    "lnn_softmax_bwd_acc": "noppnna",
    "lnn_cce_fwd": "nwppnnn",
    "lnn_cce_bwd_acc": "nopppnnna",
    "lnn_scale_bias_lrelu": "nopppnnnfa",
    "lnn_channel_chain_fwd": "nwpppnnnnf",
    "lnn_channel_chain_bwd": "nwwwpppppnnnnfnnn",
    "lnn_pool2d_fwd_idx": "nnwwpnnnnnnnnnn",
    "lnn_pool2d_bwd_idx": "nnoppnnnnnnnnnna",
    "lnn_pool2d_bwd_acc": "nnopppnnnnnnnnnna",
    "lnn_pool2x2_idx_lrelu_bwd": "nwwpppnnnnfn",
    "lnn_pool2x2_winner_grad": "nwpppnnnnfn",
    "lnn_pool2x2_idx_lrelu_bwd_packed": "nwwwpppnnnnfn",
    "lnn_reduce": "nnopnnnnna",
    "lnn_reduce_bwd_acc": "nnopppnnnnna",
    "lnn_transpose": "nopnnna",
    "lnn_slice_fwd": "nopnnnnna",
    "lnn_slice_bwd": "nmpnnnnn",
    "lnn_gemm_f32": "nopppnnnnnnan",
    "lnn_nhwc_split": "nwwpnnnnn",
    "lnn_conv2d_fwd": "nnopppnfan",
    "lnn_conv2d_fwd_packed": "nnwwppppnfnnnn",
    "lnn_conv2d_dx_acc": "nnoppnpna",
    "lnn_conv2d_dw_acc": "nnoppppnna",
    "lnn_conv2d_dw_winners_acc": "nnopppa",
    "lnn_conv2d_transpose_fwd": "nnoppan",
    "lnn_conv2d_transpose_dx": "nnmppn",
    "lnn_conv2d_transpose_dk": "nnmppn",
    "lnn_depthwise_conv2d_fwd": "nnoppa",
    "lnn_depthwise_conv2d_dx": "nnmpp",
    "lnn_depthwise_conv2d_dk": "nnmpp",
    "lnn_optimizer_step_many": "nnnLlLLnnn",
}


class _Calls:
    """Filled when the library is loaded."""


call = _Calls()

# entry points that report status through their return value
_NO_ERRCHECK = {"lnn_version", "lnn_last_error"}

EXPORTS = tuple(_SIGNATURES)

_lib = None


def _make_errcheck(name):
    def errcheck(result, func, args):
        if result != 0:
            _raise_status(result, name)
        return result
    return errcheck


def _raise_status(code, name):
    msg = _lib.lnn_last_error()
    raise LnnError(code, msg.decode("utf-8", "replace") if msg else "", name)


def get_lib():
    """Load the shared library once and type every export.  Raises if it is missing."""
    global _lib
    if _lib is not None:
        return _lib
    if not os.path.exists(LIB_PATH):
        raise LnnError(E_NOTINIT,
                       f"{LIB_PATH} not found: build it with `python -m litenn_b200.csrc.build` "
                       f"(there is no CPU fallback)", "get_lib")
    lib = ctypes.CDLL(LIB_PATH)
    for name, (restype, argtypes) in _SIGNATURES.items():
        fn = getattr(lib, name)     # AttributeError if the library lacks a declared symbol
        fn.restype = restype
        fn.argtypes = argtypes
    _lib = lib
    address = lambda name: ctypes.cast(getattr(lib, name), c_void_p).value      # noqa: E731
    _native.bind(address("lnn_alloc"), address("lnn_free"), _raise_status)
    for name, letters in _CALLS.items():
        setattr(call, name, _native.Function(address(name), name, letters))
    for name in _SIGNATURES:
        if name not in _NO_ERRCHECK:
            getattr(lib, name).errcheck = _make_errcheck(name)
    return lib


def i64_array(values, pad_to=None, pad_value=1):
    vals = [int(v) for v in values]
    if pad_to is not None:
        vals = vals + [pad_value] * (pad_to - len(vals))
    return (c_int64 * len(vals))(*vals)


# the dict behind os.environ, whose own get() encodes and decodes on every call (1 us)
_ENV = getattr(os.environ, "_data", None) if os.name == "posix" else None


def precision():
    """Operand split of the tensor-core contractions (the `precision` argument of the C entries):
    2 = split FP16 (default), 3 = split TF32, 1 = plain TF32.  LNN_PRECISION overrides it."""
    v = os.environ.get("LNN_PRECISION") if _ENV is None else _ENV.get(b"LNN_PRECISION")
    if v is None:
        return 2
    v = int(v)
    if v not in (1, 2, 3):
        raise ValueError("LNN_PRECISION must be 1, 2 or 3")
    return v


# older name of the same setting
tf32_passes = precision
