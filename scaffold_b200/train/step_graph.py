"""CUDA graphs of the training and validation passes of a :class:`TrainEngine`.

A step of a small network is bound by its launches: at scale 5 (32 cubed, base width 64) an ordinary step takes 4.2 ms
and a replayed one 1.0, and even at scale 7 and base width 32 the gaps between launches are 3 % of the step. After a few ordinary passes over batches of one shape the engine therefore captures that pass and
replays it: one graph for forward and loss, one for backward (so that the loss can be copied to the host between the
two). The optimizer's update, whose learning rate and step count change from step to step, stays outside.

A graph replays kernels on fixed addresses, so it is used only while nothing that the ordinary pass would have looked
at has changed: the same parameters at the same addresses, the same modules with the same settings, no hook on any of
them (see :class:`_Fingerprint`). Otherwise the ordinary pass runs. The batch is copied into the graph's own buffers,
the results out of them, so inputs may live anywhere and results are the caller's to keep.

Limits: batches whose widest feature map is at most ``MAX_MAP_BYTES``, since the graph keeps the memory of one pass's
activations (2 x 128 cubed x 64 channels gains 1.0 to 1.7 % for 7.4 GB, 2 x 160 cubed 1.0 to 1.8 % for 14.4 GB, 256
cubed nothing for 29.5 GB; the limit stands above the first); at most ``MAX_SHAPES`` batch shapes
per engine, and ``1 / MEMORY_SHARE`` of the device's memory. The memory is given back with the engine, when a pass is
found out of date, and when an ordinary pass of the engine runs out of memory.
"""
from __future__ import annotations

import math
import threading
import weakref
from itertools import chain
from operator import eq, is_
from time import perf_counter
from types import FunctionType
from typing import Optional

import torch
import torch.nn as nn

from ..models import unet
from ..models.unet import UNet
from ..ops import _lib, conv_kernels as ck, layout, loss as losses, pool_kernels
from ..ops import conv3d as c3
from ..ops.group_norm import GroupNorm
from ..ops.optim import FusedClipAdam
from ..ops.pool import MaxPool3d
from ..utils import perf

WARM_PASSES = 2        # ordinary passes over a shape before its capture (kernels set up, operand layouts known)
MAX_SHAPES = 4         # graphs per engine and kind of pass
MAX_MAP_BYTES = 640 << 20
_CAPTURES = threading.Lock()  # torch captures on one stream of the process
MEMORY_SHARE = 8       # an engine's graphs together keep at most 1 / this of the device's memory


def _watched() -> bool:
    """True while something follows single operations or tensors (dispatch and function modes, saved-tensor hooks,
    forward-mode AD, functorch transforms, tracing): it would see nothing of a replayed pass."""
    return bool(torch._C._len_torch_dispatch_stack() or torch._C._len_torch_function_stack()
                or torch._C._autograd._top_saved_tensors_default_hooks(True) is not None
                or torch.autograd.forward_ad._current_level >= 0
                or torch._C._functorch.maybe_current_level() is not None or torch._C._get_tracing_state() is not None)


# The modules whose passes are known to be kernels and nothing else. Any other one (a dropout in an Identity's place, a
# subclass) may keep state of its own in Python.
_MODULES = (UNet, unet.DoubleConv, unet.Down, unet.Up, unet.OutConv, unet._FirstConvSequential, c3.Conv3d,
            c3.ConvTranspose3d, GroupNorm, MaxPool3d, nn.Sequential, nn.ModuleList, nn.Identity, nn.Upsample)
_ENGINE_STEPS = ("to_device", "_autocast", "forward_loss", "_eval_pass")


def _functions(engine_type) -> list:
    """The functions that a pass runs, wherever they could be replaced for all instances."""
    return [t.forward for t in _MODULES] + [getattr(engine_type, n) for n in _ENGINE_STEPS] + [
        UNet.forward_padded_logits, UNet.features, UNet._run, unet.Down.forward_with_skip, unet.Down._after_pool,
        c3.Conv3d.forward_padded, c3.Conv3d._cuda_forward, ck.conv_same, ck.conv_wgrad, ck.convT_fwd, ck.convT_dgrad,
        losses.segmentation_loss_fused, losses.hard_dice_fused]


def remember_functions(engine_type) -> None:
    """Called where the engine is defined: a pass with other functions than these is not captured. (One that, say, reads
    a value on the host ends a capture with an error, see ``_capture_failed``.)"""
    _OWN_FUNCTIONS[:] = _functions(engine_type)


_OWN_FUNCTIONS: list = []


def _capture_failed(device, rng_state) -> None:
    """An error of the runtime inside a capture leaves torch's generator of the device in its capture state, where every
    later use of it raises: it gets a state of its own again, the one from before the capture."""
    torch.cuda.synchronize(device)
    index = torch.cuda.current_device() if device.index is None else device.index
    fresh = torch.Generator(device=device)
    fresh.set_state(rng_state)
    torch.cuda.default_generators[index].graphsafe_set_state(fresh)


def _replaced_steps(engine) -> bool:
    """True for an engine whose steps are not TrainEngine's: a subclass, or functions of its own."""
    from .engine import TrainEngine
    t = type(engine)
    return any(n in engine.__dict__ or (t is not TrainEngine and getattr(t, n) is not getattr(TrainEngine, n))
               for n in _ENGINE_STEPS)


class _Fingerprint:
    """What a captured pass depends on besides the batch's values; ``holds()`` is some thousand identity checks."""

    def __init__(self, engine):
        modules = list(engine.model.modules())
        # every attribute of every module: settings, mode, a forward or a compiled call of its own, ... (dicts compare
        # their values by identity first; tensors are looked at by identity alone)
        self._dicts = [d for m in modules for d in (m.__dict__, m._modules) if d]
        self._were = [dict(d) for d in self._dicts]
        self._tensors = [d for m in modules for d in (m._parameters, m._buffers) if d]
        self._named = list(chain.from_iterable(map(dict.values, self._tensors)))
        self._hooks = [h for m in modules for h in (m._forward_hooks, m._forward_pre_hooks, m._backward_hooks,
                                                    m._backward_pre_hooks)]
        self._params = list(engine.model.parameters())
        self._ptrs = [p.data_ptr() for p in self._params]
        self._needs = [p.requires_grad for p in self._params]
        self._known = all(type(m) in _MODULES and m._compiled_call_impl is None
                          and not any(isinstance(getattr(type(m), n, None), FunctionType) for n in m.__dict__)
                          for m in modules)
        self._settings = self._read(engine)

    @staticmethod
    def _read(engine):
        cw = engine.class_weights
        return (engine.amp, engine.n_classes, id(cw), 0 if cw is None else cw.data_ptr(), engine.flat.data.data_ptr(),
                engine.flat.grad.data_ptr(), ck.PAIR_CONV, c3._GN_FROM_EPILOGUE, pool_kernels._USE_INDEX)

    def holds(self, engine) -> bool:
        if not self._known or any(self._hooks):
            return False
        try:
            if not all(map(eq, self._dicts, self._were)):
                return False
        except (RuntimeError, TypeError, ValueError):  # an attribute that has no truth value, so it is another one
            return False
        now = list(chain.from_iterable(map(dict.values, self._tensors)))
        if len(now) != len(self._named) or not all(map(is_, now, self._named)):
            return False
        ps = self._params
        if ([p.data_ptr() for p in ps] != self._ptrs or [p.requires_grad for p in ps] != self._needs
                or any([p._backward_hooks or p._post_accumulate_grad_hooks for p in ps])):
            return False
        return self._settings == self._read(engine) and _functions(type(engine)) == _OWN_FUNCTIONS


class _Pass:
    """One captured pass: forward + loss (+ backward), with its own input buffers."""

    def __init__(self, engine, images, masks, train: bool):
        dev = engine.device
        self._lock = threading.Lock()
        self.images = torch.empty(images.shape, dtype=images.dtype, device=dev)
        self.masks = torch.empty(masks.shape, dtype=masks.dtype, device=dev)
        self._load(images, masks)
        self.fingerprint = _Fingerprint(engine)
        self.class_weights = engine.class_weights  # the kernels read it at its address: keep it alive
        convs = [c for m in engine.model.modules() for c in (getattr(m, "_cache", None), getattr(m, "_cache_b", None))
                 if c is not None]
        # Operand copies that the forward pass makes itself (k = 1 and transposed convolutions, padded biases) must be
        # made inside the graph, where a replay renews them; the ones of the 3x3x3 layers are persistent buffers that
        # the optimizer step renews.
        for c in convs:
            c._vals = {}
        engine.flat.rebind_grads()
        c3.repack_all(engine.flat)
        # ... so every layout that a layer uses has to be one that the optimizer step (and refresh_packs) renews
        layouts = {}
        for m in engine.model.modules():
            if isinstance(m, c3.Conv3d):
                c = m._cache
                if c._asked and c3.packed_weight(engine.flat, c) is not m.weight:
                    raise RuntimeError("a layer's operand copies are not the optimizer's to renew")
                layouts[c] = set(c._asked), set(c._fresh), dict(c._bufs)
        self.packs = c3.pack_buffers(engine.flat)
        pool = torch.cuda.graph_pool_handle()
        self.forward_graph, self.backward_graph = torch.cuda.CUDAGraph(), None
        before = _lib.launch_count()
        try:
            with torch.cuda.graph(self.forward_graph, pool=pool, capture_error_mode="thread_local"):
                if train:
                    loss, ce, fg, _ = engine.forward_loss(self.images, self.masks)
                    out = (loss.detach(), ce.detach(), fg.detach())
                else:
                    with torch.no_grad():
                        out = engine._eval_pass(self.images, self.masks)
            self.launches = _lib.launch_count() - before
            if train:
                before = _lib.launch_count()
                self.backward_graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(self.backward_graph, pool=pool, capture_error_mode="thread_local"):
                    loss.backward()
                self.back_launches = _lib.launch_count() - before
            if any(c._asked != asked or c._bufs.keys() != bufs.keys() for c, (asked, _, bufs) in layouts.items()):
                raise RuntimeError("a layer asked for a layout that the passes before had not")
        finally:
            for c in convs:
                c._vals = {}  # these tensors live in the graph's memory
            for c, (asked, fresh, bufs) in layouts.items():
                c._asked, c._bufs = asked, bufs
                c._fresh &= fresh  # packing that was recorded has not run
        self.out = out
        self.stream = torch.cuda.current_stream()
        # what the graphs keep: their pool, the buffers of the batch
        self.bytes = sum(s["total_size"] for s in torch.cuda.memory_snapshot() if tuple(s["segment_pool_id"]) == tuple(pool))
        self.bytes += sum(t.numel() * t.element_size() for t in (self.images, self.masks))

    def _load(self, images, masks):  # (neither side needs a gradient)
        self.images.copy_(images, non_blocking=True)
        self.masks.copy_(masks, non_blocking=True)

    def forward(self, engine, images, masks):
        with self._lock:  # one set of buffers: threads take turns, each on its own stream behind the last one's
            return self._forward(engine, images, masks)

    def _forward(self, engine, images, masks):
        stream = torch.cuda.current_stream()
        if stream != self.stream:  # the buffers are the graph's: a pass on another stream comes after the last one
            stream.wait_stream(self.stream)
            self.stream = stream
            self.images.record_stream(stream)  # made on another one, and dropped whenever the pass is
            self.masks.record_stream(stream)
        c3.refresh_packs(engine.flat)
        # the regions of the ordinary pass, without their context managers (14 us of a 600 us step); the loss is part of
        # the graph, so its host time counts as the prediction's
        t0 = perf_counter()
        self._load(images, masks)
        t1 = perf_counter()
        self.forward_graph.replay()
        t2 = perf_counter()
        out = tuple([t.clone() for t in self.out])
        perf.count_region("image_to_device", t1 - t0)
        perf.count_region("predict", t2 - t1)
        perf.count_region("calculate_loss", perf_counter() - t2)
        _lib.lib().sb_count_launch(self.launches)
        return out

    def backward(self):
        self.backward_graph.replay()
        _lib.lib().sb_count_launch(self.back_launches)


class StepGraphs:
    """The captured passes of one engine."""

    def __init__(self):
        self._passes = {}   # key -> _Pass, or the number of ordinary passes seen, or None (cannot be captured)
        self._model = None  # weak reference to the model that these passes are of
        self._lock = threading.Lock()

    def __reduce__(self):  # a copy of the engine has captured nothing yet
        return StepGraphs, ()

    @staticmethod
    def _usable(engine, images, masks) -> bool:
        model = engine.model
        if not (engine.cuda and engine.fused_loss and engine.flat is not None and type(model) is UNet
                and isinstance(engine.optimizer, FusedClipAdam) and engine.reducer.world == 1
                and engine.spatial is None and model._spatial is None and not _replaced_steps(engine)):
            return False
        widest = images.shape[0] * math.prod(images.shape[2:]) * model.base_width * 2
        return (widest <= MAX_MAP_BYTES and not model.checkpointing and not layout._aten_only[0]
                and not torch.is_anomaly_enabled() and not perf._nvtx_enabled()
                and not torch.nn.modules.module._has_any_global_hook() and not _watched()
                and not torch.cuda.is_current_stream_capturing())

    def get(self, engine, images, masks, train: bool) -> Optional[_Pass]:
        """The captured pass for this batch's shape, or None: run the ordinary pass."""
        with self._lock:
            return self._get(engine, images, masks, train)

    def _get(self, engine, images, masks, train):
        if self._model is None or self._model() is not engine.model:  # the engine has another model now
            self._passes = {}
            self._model = weakref.ref(engine.model)
        if images.dim() != 5 or not self._usable(engine, images, masks) or torch.is_grad_enabled() is not train:
            return None
        if torch.is_inference_mode_enabled():  # buffers made in it could not be written outside of it
            return None
        if images.requires_grad:  # the caller wants the gradient of the batch itself (and its first layer takes another path)
            return None
        key = (train, tuple(images.shape), images.dtype, tuple(masks.shape), masks.dtype)
        seen = self._passes.get(key, 0)
        if isinstance(seen, _Pass):
            if seen.fingerprint.holds(engine):
                return seen
            # the model was changed: start over, and keep no memory for the other shapes' passes either
            self._passes = {k: 0 if k[0] == train and isinstance(p, _Pass) else p for k, p in self._passes.items()}
            seen = 0
        if seen is None:
            return None
        if seen < WARM_PASSES:
            if key in self._passes or len(self._passes) < 4 * MAX_SHAPES:
                self._passes[key] = seen + 1
            return None
        owned = all(getattr(p, layout.EPOCH_CELL_ATTR, None) is engine.flat.epoch_cell
                    for p in engine.model.parameters())
        if not owned:  # a parameter outside the optimizer: nothing would renew its operand copies
            self._passes[key] = None
            return None
        kept = {k: p for k, p in self._passes.items() if isinstance(p, _Pass)}
        room = torch.cuda.get_device_properties(engine.device).total_memory // MEMORY_SHARE
        room -= sum(p.bytes for p in kept.values())
        if sum(k[0] == train for k in kept) >= MAX_SHAPES or room <= 0:
            return None
        probe = _Fingerprint(engine)
        if not probe.holds(engine):  # hooks are set, or a module is not one of the model's own: look again later
            self._passes[key] = 0
            return None
        rng_state = torch.cuda.get_rng_state(engine.device)
        try:
            # (the caller's stream is current again whatever ends a capture)
            with _CAPTURES, torch.cuda.stream(torch.cuda.current_stream()):
                new = _Pass(engine, images, masks, train)
            if new.bytes > room:
                raise RuntimeError(f"its {new.bytes >> 20} MB are over the limit")
            self._passes[key] = new
        except RuntimeError as exc:  # no memory for the graph's buffers, or an operation that cannot be captured
            import logging
            logging.getLogger("scaffold").warning("the %s pass stays uncaptured: %s", "training" if train else
                                                  "validation", str(exc).splitlines()[0])
            self._passes[key] = new = None
            _capture_failed(engine.device, rng_state)
        return self._passes[key]

    def release(self) -> bool:
        """Give the memory of all captured passes back; False when there was none."""
        with self._lock:
            held = any(isinstance(p, _Pass) for p in self._passes.values())
            self._passes = {k: None if isinstance(p, _Pass) else p for k, p in self._passes.items()}
        if held:
            torch.cuda.synchronize()
            torch.cuda.empty_cache()
        return held
