"""ctypes signatures of the compute kernels in libtb200_cuda.so."""

import ctypes
import functools
import warnings

import torch

from ..parallel.symm import check_rc, cuda_lib  # noqa: F401


@functools.cache
def lib():
    L = cuda_lib()
    vp, i, f = ctypes.c_void_p, ctypes.c_int, ctypes.c_float
    sig = {
        "tb_gemm_error": ([], i),
        "tb_gemm_last_error": ([], ctypes.c_char_p),
        "tb_gemm_force_tile": ([i], None),
        "tb_gemm_tma_store": ([i], None),
        "tb_gemm_gathered": ([vp, vp, i, i, i, i, i, i, vp, vp, vp, ctypes.POINTER(vp), ctypes.POINTER(ctypes.c_longlong),
                              ctypes.POINTER(ctypes.c_longlong), i, vp, ctypes.c_longlong, ctypes.c_longlong, vp, ctypes.c_uint, i, i, vp], i),
        "tb_gemm_bf16": ([vp, vp, vp, i, i, i, i, i, i, i, i, i, vp, vp, vp, i, vp, ctypes.c_longlong, vp], i),
        "tb_gemm_workspace_bytes": ([i, i, i], ctypes.c_longlong),
        "tb_gemm_plan": ([i, i, i, ctypes.POINTER(ctypes.c_int)], None),
        "tb_gemm_force_splits": ([i], None),
        "tb_gemm_reciprocals": ([vp, vp, ctypes.c_longlong, vp], i),
        "tb_layernorm_fwd": ([vp, vp, vp, vp, vp, vp, i, i, f, vp], i),
        "tb_layernorm_bwd_blocks": ([i], i),
        "tb_layernorm_bwd": ([vp, vp, vp, vp, vp, vp, vp, vp, vp, i, i, vp], i),
        "tb_layernorm_bwd_add": ([vp, vp, vp, vp, vp, vp, vp, vp, vp, vp, i, i, vp], i),
        "tb_col_sum": ([vp, i, i, i, vp, vp, vp], i),
        "tb_xent_fwd": ([vp, vp, vp, vp, vp, i, i, i, vp], i),
        "tb_xent_bwd": ([vp, vp, vp, vp, i, i, i, i, vp], i),
        "tb_stream_wait": ([vp, vp], i),
        "tb_stream_wait_events": ([], i),
        "tb_embed_fwd": ([vp, vp, vp, vp, i, i, i, vp], i),
        "tb_embed_bwd": ([vp, vp, vp, vp, vp, i, i, i, i, vp], i),
    }
    for name, (argtypes, restype) in sig.items():
        if not hasattr(L, name):
            continue
        fn = getattr(L, name)
        fn.argtypes, fn.restype = argtypes, restype
    return L


def stream(t):
    """The raw handle of the current stream of t's device (building a torch.cuda.Stream object for it costs 2 us a launch).
    A CPU tensor is refused, as torch.cuda.current_stream does: its device number, -1, would get the current GPU's stream,
    and a kernel host pointers."""
    if not t.is_cuda:
        raise ValueError(f"Expected a cuda device, but got: {t.device}")
    return _raw_stream(t.get_device())


# Two shortcuts of the host path rest on names that torch does not document: the raw stream query, and whether a functorch
# transform or a tracer is active.  A torch without one of them takes the documented, slower way.
_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None) or (lambda device: torch.cuda.current_stream(device).cuda_stream)
_functorch_level = getattr(getattr(torch._C, "_functorch", None), "peek_interpreter_stack", None)
_tracing_state = getattr(torch._C, "_get_tracing_state", None)
_can_tell = _functorch_level is not None and _tracing_state is not None and hasattr(torch.autograd.forward_ad, "_current_level")


@functools.cache
def native():
    """The natively issued operators (csrc/ops.cpp) bound to the kernel library; None, with a warning, where they are not built
    for this torch: the Python functions then do the same more slowly."""
    try:
        from .. import _ops
    except ImportError as e:
        warnings.warn(f"tandem_b200._ops cannot be imported ({e}); eager operators are issued from Python. Build it with "
                      "python -m tandem_b200.utils.build", stacklevel=3)
        return None
    from ..utils.build import CUDA_LIB

    cuda_lib()  # with its message if the library is missing
    _ops.bind(CUDA_LIB)
    return _ops


def direct(*tensors):
    """The native operators if they may answer this call, else None: a functorch transform, a forward-mode level, a tracer or a
    tensor with a __torch_function__ of its own (or a mode with one) has to meet the Python function."""
    if (not _can_tell or torch.autograd.forward_ad._current_level >= 0 or _functorch_level() is not None or _tracing_state() is not None
            or torch.overrides.has_torch_function(tensors)):
        return None
    return native()


class _Untracked:
    """Stands in for the context of an autograd function whose backward cannot be asked for."""

    def save_for_backward(self, *tensors):
        pass


def run(function, *args):
    """function.apply(*args), or its forward alone (5 us less a call) where nothing can want the node: gradients are off, and
    no functorch transform, forward-mode level or tracer is active, which Function.apply would have to answer or refuse."""
    if (torch.is_grad_enabled() or not _can_tell or torch.autograd.forward_ad._current_level >= 0 or _functorch_level() is not None
            or _tracing_state() is not None):
        return function.apply(*args)
    return function.forward(_Untracked(), *args)


def stream_wait(waiter, signaller):
    """Work queued on raw stream `waiter` from here on starts after everything now queued on `signaller`."""
    check_rc(lib().tb_stream_wait(waiter, signaller), "stream wait")


def pad8(n):
    return (n + 7) // 8 * 8


def empty_padded(rows, cols, dtype, device):
    """A [rows, cols] view of [rows, pad8(cols)] storage: every row starts 16-byte aligned."""
    ld = pad8(cols)
    if ld == cols:
        return torch.empty(rows, cols, dtype=dtype, device=device)
    return torch.empty(rows, ld, dtype=dtype, device=device)[:, :cols]


# The kernels take addresses and sizes: what would read beyond an operand is refused here, before a launch.
def need(ok, what):
    if not ok:
        raise ValueError(what)


def need_bf16(*tensors):
    first = None
    for t in tensors:
        if t is None:
            continue
        if not t.is_cuda or t.dtype != torch.bfloat16:
            raise TypeError("the sm_100a operators take bf16 CUDA tensors (cast the model with .bfloat16())")
        first = t if first is None else first
        need(t.device == first.device, "the operands lie on different devices")


def need_ids(ids, beside):
    if not ids.is_cuda or ids.dtype != torch.int64:
        raise TypeError("token ids and targets are int64 CUDA tensors")
    need(ids.device == beside.device, "the operands lie on different devices")


def need_product(x, w, bias):
    """x . w^T + bias: of w's rows only their distance is free."""
    need(x.dim() > 0 and w.dim() == 2, "a product takes an input of rows and a 2-D weight")
    need(x.shape[-1] == w.shape[1], "the input's width is not the weight's")
    need(w.stride(1) == 1 or w.shape[1] == 1, "the weight's rows have to be contiguous")
    need(bias is None or bias.numel() == w.shape[0], "the bias has not one value per output")


def vectors_of(t):
    """t, or a copy of it, for kernels that read it as a run of 16-byte vectors."""
    t = t.contiguous()
    return t.clone() if t.data_ptr() % 16 else t
