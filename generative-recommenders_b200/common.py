"""Types shared by the ops: the backend selector the reference threads through every call."""

from enum import Enum, unique

import torch
from torch._C._profiler import _RecordFunctionFast
from torch.autograd import forward_ad
from torch.compiler import is_compiling

from . import _cabi


@unique
class HammerKernel(Enum):
    """Same members as generative_recommenders/common.py:112-119.

    This library implements exactly one backend, ``CUDA`` (hand-written sm_100a kernels).
    The reference leaves ``CUDA`` unhandled in ``hstu_mha`` (it falls through to the PyTorch
    branch, generative_recommenders/ops/hstu_attention.py:191-207); here it is the only value
    that runs, every other member raises so that nothing silently takes a slower path.
    """

    TRITON = "TRITON"
    TLX = "TLX"
    PYTORCH = "PYTORCH"
    CUDA = "CUDA"
    TRITON_CC = "TRITON_CC"
    CUTEDSL = "CUTEDSL"


def _require_cuda_backend(kernel) -> None:
    name = getattr(kernel, "name", kernel)
    if name != "CUDA":
        raise NotImplementedError(
            "generative-recommenders_b200 only implements HammerKernel.CUDA (got %r); "
            "other backends are not part of this library" % (kernel,)
        )


_DTYPES = {torch.float32: _cabi.F32, torch.bfloat16: _cabi.BF16, torch.float16: _cabi.F16}


def dtype_code(t: torch.Tensor) -> int:
    try:
        return _DTYPES[t.dtype]
    except KeyError:
        raise TypeError("unsupported dtype %s (float32, bfloat16 and float16 are)" % t.dtype)


def require_cuda(*tensors) -> None:
    for t in tensors:
        if t is not None and not t.is_cuda:
            raise RuntimeError("tensors must live on a CUDA device; this library has no CPU path")


# The calls of a layer on a small batch are bound by host time, so the helpers below do what the torch
# functions beside them do without building Python objects on the way (per call: a stream object 6 us,
# a device context 7 us, a profiler range 18 us, a no-op ``.to`` 1 us, an autograd node about 15 us).
def stream_ptr(device) -> int:
    index = getattr(device, "index", None)
    if type(index) is not int:
        return torch.cuda.current_stream(device).cuda_stream
    return torch._C._cuda_getCurrentRawStream(index)


class _Nothing:
    __slots__ = ()

    def __enter__(self):
        return None

    def __exit__(self, *exc):
        return False


_NOTHING = _Nothing()


def on_device(device):
    """``torch.cuda.device(device)`` around a launch; nothing where that is the thread's device already."""
    index = getattr(device, "index", None)   # (an int or None has none, a str a method)
    return _NOTHING if index == torch._C._cuda_getDevice() else torch.cuda.device(device)


def span(name: str):
    """``record_function(name)`` while a profiler runs, else its light form (other observers see it too).
    The compiler knows the former only."""
    if is_compiling() or torch.autograd._profiler_enabled():
        return torch.autograd.profiler.record_function(name)
    return _RecordFunctionFast(name)


def as_dtype(t: torch.Tensor, dtype) -> torch.Tensor:
    return t if t.dtype is dtype else t.to(dtype)


def outside_autograd(*tensors) -> bool:
    """True where an ``autograd.Function`` would do no more than run its forward: no input asks for a
    gradient, and there is no forward-mode level, functorch transform, tracer or compiler that has to see
    the node (or to refuse it)."""
    if is_compiling():   # (first: the compiler need not see the rest)
        return False
    if torch.is_grad_enabled():
        for t in tensors:
            if t is not None and t.requires_grad:
                return False
    return (forward_ad._current_level < 0 and not torch._C._are_functorch_transforms_active()
            and torch._C._get_tracing_state() is None)


def last_dim_contiguous(t: torch.Tensor) -> torch.Tensor:
    """Same rule as the reference's switch_to_contiguous_if_needed
    (generative_recommenders/common.py:262-269): only a non-unit last stride forces a copy."""
    if t.dim() > 0 and t.stride(-1) != 1 and t.shape[-1] > 1:
        return t.contiguous()
    return t
