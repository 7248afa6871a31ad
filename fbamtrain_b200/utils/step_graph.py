"""Forward and backward of a launch-bound training step as a CUDA graph.

A step of a small configuration is some two hundred launches of a few microseconds each, which take the host several
times as long to issue as the GPU to run (toy configuration, 4 x 64 frames of 24 x 80: 4.5 ms a step, GPU busy for 1.1).
:class:`StepGraph` watches the steps of a trainer; where the host is what a step waits for, forward and backward of the
next step of that shape are captured once and replayed from then on.  Gradients are added to the flat buffers and the
parameters read where they lie, so the optimizer, gradient accumulation and checkpoints see no difference; inputs are
copied into the graph's own buffers, the loss out of them.

What is captured is what the host would have done for the step at hand.  Before every replay the settings of the model, of
this package and of the libraries that this depends on are compared (:meth:`_setting`); with anything out of the ordinary —
hooks, saved-tensor hooks, dispatch modes, anomaly detection, debug switches, a recording of launches or shapes — the step
runs as usual.  ``FBAMTRAIN_STEP_GRAPH=0`` keeps every step that way.

The activations of the captured steps stay with the graphs, in one pool of memory that is as large as the largest step
needs and goes to nobody else.  It is at most ``MEMORY_SHARE`` of the memory that is free at a capture, and is given back
(:meth:`StepGraph.release`) where a large step of the trainer would otherwise have to recompute its activations.

The reference has no counterpart: its executor launches kernel by kernel (reference:
``tensorlib/src/execution_backend.cpp``).
"""
from __future__ import annotations

import gc
import os
import time
from collections import OrderedDict
from typing import Optional

import torch
from torch.nn.modules import module as _module

from ..ops import dispatch, embconv, native, native_ops, tuning
from . import debug, flops, plan
from .logging import LOG, enabled as log_enabled

# Cells of a step (frames x positions) up to which steps are watched: a step of the headline configuration has 63 million
# and keeps the GPU busy three times as long as the host; its graph would hold 28 GB of activations.
MAX_CELLS = 8 << 20
WATCHED_STEPS = 2        # steps of a shape that run as usual before one may be captured
HOST_SHARE = 0.7         # captured where the host takes at least this share of the step's time on the GPU's clock
MAX_GRAPHS = 2           # per trainer; the least recently used one is given back
MAX_WATCHES = 8
# Part of the device memory that is free at a capture which the graphs of a trainer may hold: what they hold is lost to
# everything else for as long as they live.
MEMORY_SHARE = 0.125


_PLAIN = frozenset((bool, int, float, str, torch.dtype))


def _module_setting(m: torch.nn.Module) -> tuple:
    """What a module's part of a step depends on besides parameters: its code, its plain attributes and its buffers."""
    kind = type(m)
    setting = [kind, kind.forward, kind.__call__]
    setting += [item for item in vars(m).items() if type(item[1]) in _PLAIN]
    if m._buffers:
        setting += [None if b is None else b.data_ptr() for b in m._buffers.values()]
    return tuple(setting)


def _library_setting() -> tuple:
    """Switches of the library paths, which fp32 models and the tables of the first layer take."""
    b = torch.backends
    return (torch.get_float32_matmul_precision(), b.fp32_precision, b.cuda.matmul.fp32_precision, b.cudnn.fp32_precision,
            b.cudnn.conv.fp32_precision, b.cudnn.rnn.fp32_precision, b.cuda.matmul.allow_fp16_reduced_precision_reduction,
            b.cuda.matmul.allow_bf16_reduced_precision_reduction, b.cudnn.enabled, b.cudnn.benchmark, b.cudnn.deterministic,
            b.cuda.flash_sdp_enabled(), b.cuda.mem_efficient_sdp_enabled(), b.cuda.math_sdp_enabled(),
            b.cuda.cudnn_sdp_enabled(), b.cuda.preferred_blas_library())


class _Watch:
    """Host and GPU time of the steps of one shape that ran as usual (the smallest of each).  ``wait``: how many there have
    to be before a capture; it doubles whenever a graph of the shape is given back, so that shapes that take turns and do
    not fit ``MAX_GRAPHS`` cost some ten captures in a thousand steps each and not one at every turn."""

    def __init__(self) -> None:
        self.wait: float = WATCHED_STEPS
        self.kept = 0              # bytes that the forward leaves for the backward
        self.restart(None)

    def restart(self, setting: Optional[tuple]) -> None:
        self.steps, self.host_ms, self.gpu_ms, self.pending = 0, float("inf"), float("inf"), []
        self.setting = setting     # what the steps run under; asked for from the last one before a capture on

    def given_back(self) -> None:
        self.steps, self.wait = 0, 2 * self.wait

    def launch_bound(self) -> bool:
        """Looks at finished events only, so it never waits for the device."""
        while self.pending and self.pending[0][1].query():
            start, end = self.pending.pop(0)
            self.gpu_ms = min(self.gpu_ms, start.elapsed_time(end))
        return self.steps >= self.wait and self.gpu_ms < float("inf") and self.host_ms >= HOST_SHARE * self.gpu_ms


class _Captured:
    def __init__(self, cells, targets):
        self.cells, self.targets = torch.empty_like(cells), torch.empty_like(targets)
        self.graph = torch.cuda.CUDAGraph()
        self.loss: Optional[torch.Tensor] = None
        self.flops = (0.0, 0.0)
        self.launches = 0


class StepGraph:
    def __init__(self, model: torch.nn.Module, device: torch.device):
        self.model = model
        self.device = torch.device("cuda", torch.cuda.current_device() if device.index is None else device.index)
        self._watches: "OrderedDict[tuple, _Watch]" = OrderedDict()
        self._graphs: "OrderedDict[tuple, _Captured]" = OrderedDict()
        self._stream: Optional[torch.cuda.Stream] = None
        self.pool_bytes = 0        # device memory that the allocator holds for the graphs and gives to nobody else

    # ------------------------------------------------------------------------------------------
    def _ordinary(self) -> bool:
        """Nothing is active that a replay would pass by."""
        if (os.environ.get("FBAMTRAIN_STEP_GRAPH", "1") == "0" or dispatch.get_backend() != "auto" or tuning.active()
                or plan.active() is not None or debug.SYNC_EVERY_OP or debug.POISON_ALLOC or debug.DEBUG_KERNEL_LAUNCH
                or debug.PROFILE_LABELS or debug.BREAK_ON_LAUNCH or log_enabled("INFO")):
            return False
        if (not torch.is_grad_enabled() or torch.is_inference_mode_enabled() or torch.is_anomaly_enabled()
                or torch.is_autocast_enabled("cuda") or torch._C._len_torch_dispatch_stack()
                or torch._C._len_torch_function_stack() or torch._C._autograd._top_saved_tensors_default_hooks(True)
                or torch.cuda.is_current_stream_capturing() or torch.cuda.current_device() != self.device.index):
            return False
        if (_module._global_forward_hooks or _module._global_forward_pre_hooks or _module._global_backward_hooks
                or _module._global_backward_pre_hooks):
            return False
        cfg, action = self.model.cfg, self.model.action_model
        # recomputed chunks and the streamed recurrence (which reads a value back) run as usual
        return not (cfg.frame_head_recompute or cfg.frame_replay or action.streaming or action.host_offload)

    def _setting(self) -> Optional[tuple]:
        """What the launches of a step depend on besides its shape and the values of inputs and parameters; ``None`` where
        the model has something that a replay would pass by."""
        no = native_ops
        setting = [self.model.frame_chunk, no.TWO_CTA, no.USE_MN_MAJOR, no.WEIGHT_GRAD_SPLIT_K, no.FUSE_DGRAD_CLASSES,
                   no.FUSED_LM_HEAD_CE, no.LM_HEAD_CHUNK_ROWS, no.RESIDUAL_NORM_MAX_DIM,
                   tuple(dispatch._prefer.values()), os.environ.get("FBAMTRAIN_EMBCONV"),
                   os.environ.get("FBAMTRAIN_ATTENTION_FWD2"), torch.are_deterministic_algorithms_enabled(),
                   native.lib(self.model.action_model.head_weight).fbam_reserved_sms(), *_library_setting(),
                   repr(self.model.cfg)]
        for m in self.model.modules():       # one walk: 0.2 ms for the headline model, in which nothing is launched
            if (m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or m._backward_pre_hooks
                    or "forward" in m.__dict__):
                return None
            setting.append(_module_setting(m))
            for p in m._parameters.values():
                if p is not None:
                    grad = p.grad
                    if grad is None or p._backward_hooks or p._post_accumulate_grad_hooks:
                        return None
                    setting += (p.data_ptr(), grad.data_ptr(), p.requires_grad)
        return tuple(setting)

    # ------------------------------------------------------------------------------------------
    def forward_backward(self, cells: torch.Tensor, targets: torch.Tensor, loss_scale: float, run) -> Optional[torch.Tensor]:
        """The loss of ``run(cells, targets, after_forward)`` (forward and backward on device tensors, with a call between the
        two where one is given), or ``None`` where the step is not one to watch."""
        chunk = self.model.frame_chunk
        frames = cells.shape[0] * cells.shape[1]
        if frames * cells.shape[2] > MAX_CELLS or (chunk and frames > chunk) or not self._ordinary():
            return None
        if not (cells.is_contiguous() and targets.is_contiguous()):
            return None
        shape = (tuple(cells.shape), cells.dtype, tuple(targets.shape), targets.dtype, loss_scale)
        watch = self._watch(shape)
        # The setting of the model is looked at where a graph may be replayed or captured now or in the next step: the first
        # step of a shape, which may be its only one, and steps that the GPU bounds go without.
        if (not any(of == shape for of, _ in self._graphs) and watch.steps + 1 != watch.wait
                and not watch.launch_bound()):
            return self._watched(watch, cells, targets, run)
        setting = self._setting()
        if setting is None:
            return None
        key = (shape, setting)
        captured = self._graphs.get(key)
        if captured is None:
            if watch.setting != setting:
                if watch.setting is None:
                    watch.setting = setting
                else:
                    watch.restart(setting)
                return self._watched(watch, cells, targets, run)
            if not watch.launch_bound():
                return self._watched(watch, cells, targets, run)
            if not self._room(watch):
                watch.given_back()
                return self._watched(watch, cells, targets, run)
            try:
                captured = self._capture(cells, targets, run)
            except RuntimeError as e:        # nothing of a capture has run: the step does now, as usual
                LOG("WARN", f"step graph: capture failed, steps of this shape run launch by launch ({e})")
                watch.wait = float("inf")
                return self._watched(watch, cells, targets, run)
            self._graphs[key] = captured
            while len(self._graphs) > MAX_GRAPHS:
                # its kernels may still be running: the memory goes back to the allocator only behind them
                torch.cuda.current_stream().synchronize()
                self._give_back()
        self._graphs.move_to_end(key)
        captured.cells.copy_(cells)
        captured.targets.copy_(targets)
        captured.graph.replay()
        flops.add_counted(*captured.flops)
        native.add_launches(captured.launches)
        return captured.loss.clone()

    def _room(self, watch: _Watch) -> bool:
        """Gradients of activations come to less than the activations, hence the two."""
        more = max(0, 2 * watch.kept + (64 << 20) - self.pool_bytes)
        return self.pool_bytes + more <= MEMORY_SHARE * (torch.cuda.mem_get_info(self.device)[0] + self.pool_bytes)

    def release(self) -> int:
        """Gives all graphs back, for a step that needs their memory; the bytes that are free for it now."""
        if self._graphs:
            torch.cuda.current_stream().synchronize()
        while self._graphs:
            self._give_back()
        freed, self.pool_bytes = self.pool_bytes, 0
        return freed

    def _give_back(self) -> None:
        (shape, _), _graph = self._graphs.popitem(last=False)
        self._watch(shape).given_back()

    def _watch(self, shape: tuple) -> _Watch:
        """The watch of a shape; those of the last ``MAX_WATCHES`` shapes are kept."""
        watch = self._watches.get(shape)
        if watch is None:
            watch = self._watches[shape] = _Watch()
        self._watches.move_to_end(shape)
        while len(self._watches) > MAX_WATCHES:
            self._watches.popitem(last=False)
        return watch

    def _watched(self, watch: _Watch, cells, targets, run) -> torch.Tensor:
        start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        after_forward = None
        if watch.steps > 0:              # not in the first step of a shape, which may be its only one
            before = torch.cuda.memory_allocated(self.device)

            def after_forward():
                watch.kept = max(watch.kept, torch.cuda.memory_allocated(self.device) - before)
        start.record()
        t0 = time.perf_counter()
        loss = run(cells, targets, after_forward)
        watch.host_ms = min(watch.host_ms, 1e3 * (time.perf_counter() - t0))
        end.record()
        watch.steps += 1
        watch.pending = (watch.pending + [(start, end)])[-4:]
        return loss

    def _capture(self, cells, targets, run) -> _Captured:
        captured = _Captured(cells, targets)
        if self._stream is None:
            self._stream = torch.cuda.Stream(self.device)
        token = embconv.cache_token()
        before, launches = flops.snapshot(), native.launches()
        # tables that depend on parameters are built inside the graph, in every replay, and none of its memory is
        # left to calls outside
        embconv.set_cache_token(("graph", id(captured)))
        compute = torch.cuda.current_stream()
        self._stream.wait_stream(compute)
        collecting = gc.isenabled()
        gc.disable()                     # what a collection frees may not be freed during a capture
        try:
            with torch.cuda.stream(self._stream):
                # other threads (logger, prefetch) may use CUDA meanwhile: only this thread's calls are looked at.  Not
                # torch.cuda.graph(), which waits for the device and gives the allocator's cache back first.
                # Graphs share a pool: what a step leaves behind in it is its loss, which is copied out at once, and replays
                # follow one another on the trainer's stream.
                pool = next((c.graph.pool() for c in self._graphs.values()), None) or torch.cuda.graph_pool_handle()
                captured.graph.capture_begin(pool=pool, capture_error_mode="thread_local")
                try:
                    captured.loss = run(captured.cells, captured.targets, None)
                finally:
                    captured.graph.capture_end()
            self.pool_bytes = sum(s["total_size"] for s in torch.cuda.memory_snapshot(pool, include_traces=False))
        finally:
            if collecting:
                gc.enable()
            embconv.set_cache_token(token)
            after = flops.snapshot()
            captured.flops = (after[0] - before[0], after[1] - before[1])
            captured.launches = native.launches() - launches
            flops.add_counted(-captured.flops[0], -captured.flops[1])     # counted with each replay
            native.add_launches(-captured.launches)
        compute.wait_stream(self._stream)
        return captured
