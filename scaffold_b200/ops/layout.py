"""Activation layout helpers.

Modules exchange ordinary NCDHW-shaped tensors whose memory is channels-last
(``torch.channels_last_3d``); the kernels see the same memory as a contiguous
voxel-major ``[N, D, H, W, C]`` tensor. Both conversions are views when the
memory format already matches.
"""
from __future__ import annotations

import torch
import torch.nn.functional as F

AMP_DTYPE = torch.bfloat16


_aten_only = [False]


class aten_only:
    """Context manager: route every module through ATen (the oracle of the parity tests)."""

    def __enter__(self):
        self._old = _aten_only[0]
        _aten_only[0] = True
        return self

    def __exit__(self, *exc):
        _aten_only[0] = self._old


def use_cuda_kernels(x: torch.Tensor) -> bool:
    """True when the sm_100a kernel path applies: CUDA tensor, bf16 or autocast-to-bf16."""
    if not x.is_cuda or _aten_only[0]:
        return False
    if x.dtype == torch.bfloat16:
        return True
    return torch.is_autocast_enabled("cuda") and torch.get_autocast_dtype("cuda") == torch.bfloat16


def to_vm(x: torch.Tensor, pad16: bool = False, pad_to: int = 16) -> torch.Tensor:
    """NCDHW-shaped tensor -> contiguous voxel-major bf16 ``[N, D, H, W, C]``."""
    if (pad16 and x.is_cuda and x.dim() == 5 and x.shape[1] < 16 and x.is_contiguous()
            and x.dtype in (torch.float32, torch.bfloat16) and not x.requires_grad):
        # input staging kernel: layout change + down-cast + channel padding in one pass
        from . import _lib
        n, c, d, h, w = x.shape
        y = torch.empty((n, d, h, w, pad_to), dtype=torch.bfloat16, device=x.device)
        _lib.check(_lib.lib().sb_stage_input(x.data_ptr(), int(x.dtype == torch.bfloat16), n, c, d * h * w,
                                             y.data_ptr(), pad_to, _lib.stream_ptr()), "sb_stage_input")
        return y
    v = x.permute(0, 2, 3, 4, 1)
    if v.dtype != torch.bfloat16:
        v = v.to(torch.bfloat16)
    c = v.shape[4]
    if pad16 and c % pad_to != 0:
        v = F.pad(v, (0, pad_to - c % pad_to))
    return v.contiguous()


def from_vm(y: torch.Tensor) -> torch.Tensor:
    """Voxel-major ``[N, D, H, W, C]`` -> NCDHW-shaped view (channels-last memory)."""
    return y.permute(0, 4, 1, 2, 3)


# Parameters updated through raw pointers (the fused optimizer) do not bump the
# tensors' version counters; packed operand caches also key on weights_epoch().
_weights_epoch = [0]  # any weights may have changed (a checkpoint was restored)
_flat_steps = [0]     # steps of all flat optimizers together
EPOCH_CELL_ATTR = "_sb_epoch_cell"  # on a parameter of a flat optimizer: the one-element step counter of that optimizer


def bump_weights_epoch() -> None:
    _weights_epoch[0] += 1


def bump_flat_step(cell) -> None:
    """A flat optimizer updated its parameters, and only those, through raw pointers."""
    cell[0] += 1
    _flat_steps[0] += 1


def weights_epoch(w=None):
    """Changes when ``w`` may have been updated through raw pointers: with the steps of its own optimizer, or, for a
    tensor that no optimizer has marked (a view of a parameter), with every optimizer's steps."""
    cell = getattr(w, EPOCH_CELL_ATTR, None)
    return (_weights_epoch[0], _flat_steps[0] if cell is None else cell[0])


# Parameters whose ``.grad`` is a view into a flat gradient buffer (set up by the fused optimizer) are marked
# with this attribute; the convolution and GroupNorm backward passes then add their parameters' gradients straight into
# those views (no temporary tensor, no autograd accumulation kernel) and tell the listeners below that they are there.
FLAT_GRAD_ATTR = "_sb_flat_grad"
_grad_written_listeners = []


def _autograd_accumulates(ctx, param) -> bool:
    """Whether the running backward pass adds a gradient to ``param.grad`` that ``ctx``'s node returns for it: not when
    the caller asked for other tensors' gradients (``backward(inputs=...)``), nor when for this one's as a result
    (``autograd.grad``)."""
    for node, _ in ctx.next_functions:
        if getattr(node, "variable", None) is param:
            try:
                return torch._C._will_engine_execute_node(node)
            except RuntimeError:  # the parameter is one of autograd.grad()'s inputs
                return False
    return False


def direct_grad_target(param, ctx=None):
    """The flat-buffer gradient view of ``param`` when the kernels may accumulate into it directly, else None. ``ctx`` is
    the autograd node in whose backward pass this is asked; without one nothing is known of the pass."""
    if not getattr(param, FLAT_GRAD_ATTR, False) or param._backward_hooks:
        return None  # a hook on the parameter wants to see its gradient: autograd's own accumulation
    g = param.grad
    if g is None or g.dtype != torch.float32 or not g.is_contiguous() or g.shape != param.shape:
        return None
    return g if ctx is None or _autograd_accumulates(ctx, param) else None


def add_grad_written_listener(fn) -> None:
    """Register a bound method (held weakly: a reducer that is dropped stops listening by itself)."""
    import weakref
    _grad_written_listeners.append(weakref.WeakMethod(fn) if hasattr(fn, "__self__") else (lambda f=fn: f))


def remove_grad_written_listener(fn) -> None:
    _grad_written_listeners[:] = [r for r in _grad_written_listeners if r() is not None and r() != fn]


def notify_grad_written(param) -> None:
    """Called by a backward pass that wrote ``param.grad`` itself (autograd's accumulate hooks do not fire then)."""
    dead = False
    for ref in list(_grad_written_listeners):
        fn = ref()
        if fn is None:
            dead = True
        else:
            fn(param)
    if dead:
        _grad_written_listeners[:] = [r for r in _grad_written_listeners if r() is not None]
