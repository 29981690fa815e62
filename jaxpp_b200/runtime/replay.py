"""Replays of launch-bound steps as CUDA graphs.

A step of a small model is a few hundred kernels of a few microseconds each, launched from generated Python at 10 to
17 microseconds apiece: the GPU idles most of the time.  From its third call on, a single-process program whose inputs
are small is replayed from a graph recorded over buffers of its own: the call's inputs are copied into them, the graph
is launched, and the results are copied into fresh tensors (or, where the step updates an input in place, back into the
caller's tensor).  Nothing refers to the caller's buffers between calls, so every call may bring others.

Only what a recording reproduces is replayed: programs made of capturable ops, on one device, called outside of
profiling, tracing and other recordings, with the flags of the time of the recording.  Everything else, and every
program whose recording fails, runs op by op as before.
"""
from __future__ import annotations

import gc
import os
import threading
from typing import Sequence

import torch

from ..compiler.program import Accum, Delete, Program, RunTask, SendDone, Slice
from ..utils import config, logger, optimes
from .. import fault

# The copies in and back cost 4 x bytes / HBM bandwidth per call (1 MB: 0.6 us) and the op-by-op launches that they replace
# at least 10 us per op: 64 MB (40 us) are always worth it, and 1 MB per op beyond.  With more than MAX_BYTES a step is
# bound by its kernels and the memory kept here would count.
FREE_BYTES, BYTES_PER_OP, MAX_BYTES = 64 << 20, 1 << 20, 256 << 20
MIN_OPS = 8
MAX_POOL_BYTES = 512 << 20       # memory that one recording may keep for its intermediate values
TOTAL_POOL_BYTES = 1 << 30       # what all recordings of the process keep together, their copies of the inputs included;
                                 # programs that come when it is used up run op by op
EAGER_CALLS = 2                  # calls that run op by op first: allocator, kernels and workspaces are warm, and a
                                 # program that is called once or twice is never recorded

_pool_lock = threading.Lock()
_pool_bytes = [0]
_FLAGS = [v for v in vars(config).values() if isinstance(v, config.OverwriteableVar)]
_MOE_OPS = {"router", "route_tokens", "route_tokens_bwd", "slots", "dispatch_rows", "combine_rows", "combine_rows_bwd"}
# ATen ops that synchronise or allocate by value for some arguments although their schemas do not say so
_ATEN_REFUSED = {"index", "index_put", "index_put_", "_index_put_impl_", "masked_select", "nonzero", "repeat_interleave", "item",
                 "_local_scalar_dense", "bincount", "lift_fresh", "lift_fresh_copy", "pin_memory", "is_pinned"}


def _settings() -> tuple:
    """What an op-by-op run would look up while it runs: a recording holds for the settings that it was made under."""
    return (tuple(f._override for f in _FLAGS), torch.are_deterministic_algorithms_enabled(), torch.get_float32_matmul_precision(),
            torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction, torch.get_default_dtype())


def _capturable(op) -> bool:
    if not isinstance(op, torch._ops.OpOverload):
        return False
    tags = op.tags
    if torch.Tag.dynamic_output_shape in tags or torch.Tag.data_dependent_output in tags or torch.Tag.nondeterministic_seeded in tags:
        return False
    name = op._schema.name.split("::")[1]
    if op.namespace == "b200":
        return True
    if op.namespace == "b200moe":
        return name in _MOE_OPS
    return op.namespace == "aten" and name not in _ATEN_REFUSED


def _program_ok(prog: Program) -> bool:
    if prog.n_ranks != 1:
        return False
    ops = 0
    for ins in prog.instrs:
        if isinstance(ins, RunTask):
            if ins.hooks or not all(_capturable(t) for t in ins.code.targets):
                return False
            if any(isinstance(c, torch.Tensor) for c in ins.code.consts):     # copied from the host on every run
                return False
            ops += ins.code.n_ops
        elif not isinstance(ins, (Slice, Accum, Delete, SendDone)):
            return False
    in_bytes = sum(prog.values[vid].nbytes for vid, ranks in prog.inputs if ranks)
    out_bytes = sum(prog.values[o[1]].nbytes for o in prog.outputs if o[0] != "c")
    return ops >= MIN_OPS and max(in_bytes, out_bytes) <= min(MAX_BYTES, FREE_BYTES + ops * BYTES_PER_OP)


def _plain(x, device: torch.device) -> bool:
    return (type(x) in (torch.Tensor, torch.nn.Parameter) and x.device == device and x.layout == torch.strided and x.is_contiguous()
            and not x.is_conj() and not x.is_neg() and not x.is_inference())


def _same_memory(a: torch.Tensor, b: torch.Tensor) -> bool:
    return a.data_ptr() == b.data_ptr() and a.shape == b.shape and a.stride() == b.stride() and a.dtype == b.dtype


def _by_dtype(tensors: Sequence, which: Sequence) -> list:
    """Positions and tensors of ``which``, grouped for one multi-tensor copy per dtype."""
    groups: dict = {}
    for k in which:
        if tensors[k].numel():
            g = groups.setdefault(tensors[k].dtype, ([], []))
            g[0].append(k)
            g[1].append(tensors[k])
    return list(groups.values())


def _copy(dst: list, src: list) -> None:
    torch._foreach_copy_(dst, src)


def _input_bytes(inputs: Sequence) -> int:
    return sum(x.nbytes for x in inputs if x is not None)


class _Recording:
    def __init__(self, prog: Program, inputs: Sequence, device: torch.device, execute):
        from ..ops import native

        self.device = device
        self.settings = _settings()
        self.static = [None if x is None else torch.empty_like(x, requires_grad=False).copy_(x) for x in inputs]
        self.stream = torch.cuda.Stream(device)
        self.graph = torch.cuda.CUDAGraph()
        self.done = torch.cuda.Event()
        launches = native.LAUNCHES[0]
        versions = [None if s is None else s._version for s in self.static]
        self.stream.wait_stream(torch.cuda.current_stream(device))
        native._recording.written = set()
        collecting = gc.isenabled()
        gc.disable()      # a collection in the middle could give back CUDA objects with calls that a recording forbids
        try:
            with torch.cuda.stream(self.stream):
                # other threads may allocate and launch meanwhile
                self.graph.capture_begin(capture_error_mode="thread_local")
                try:
                    outs = execute(list(self.static))
                finally:
                    self.graph.capture_end()
            written = native._recording.written
        finally:
            native._recording.written = None
            if collecting:
                gc.enable()
        self.launches = native.LAUNCHES[0] - launches
        native.LAUNCHES[0] = launches
        # the graph's own segments: other threads allocate meanwhile
        self.pool_bytes = sum(seg["total_size"] for seg in torch.cuda.memory_snapshot(mempool_id=self.graph.pool(), include_traces=False))
        self.kept_bytes = self.pool_bytes + _input_bytes(self.static)
        # (every static tensor has a storage of its own)
        self.written = [k for k, s in enumerate(self.static)
                        if s is not None and (s.untyped_storage().data_ptr() in written or s._version != versions[k])]
        # every output: a constant, an input (passed through or updated in place), or the n-th result of the graph
        self.results: list = []
        self.outputs: list = []
        starts = {s.untyped_storage().data_ptr(): k for k, s in enumerate(self.static) if s is not None and s.numel()}
        for o, val in zip(prog.outputs, outs):
            if o[0] == "c":
                self.outputs.append(("c", val))
                continue
            ((rank, t),) = val.items()
            if t.device != device:
                raise NotImplementedError("a result on another device")
            k = starts.get(t.untyped_storage().data_ptr()) if t.numel() else None
            if k is not None:
                if not _same_memory(t, self.static[k]):
                    raise NotImplementedError("a result that is a view of an input")
                self.outputs.append(("in", rank, k))
                continue
            n = next((i for i, r in enumerate(self.results) if _same_memory(r, t)), None)
            if n is None:
                if t.numel() and any(r.untyped_storage().data_ptr() == t.untyped_storage().data_ptr() for r in self.results):
                    raise NotImplementedError("results that share memory")
                n = len(self.results)
                self.results.append(t)
            self.outputs.append(("out", rank, n))
        self._plan()
        self.done.record(torch.cuda.current_stream(device))     # the first copies into the buffers

    def _plan(self) -> None:
        """What a call looks up: worked out here, since the calls are bound by the host."""
        self.forms = [None if s is None else (s.dtype, s.shape) for s in self.static]
        self.sizes = [0 if s is None else s.nbytes for s in self.static]
        self.into = _by_dtype(self.static, [k for k, s in enumerate(self.static) if s is not None])
        self.back = _by_dtype(self.static, self.written)
        self.out = _by_dtype(self.results, range(len(self.results)))

    def covers(self, inputs: Sequence) -> bool:
        """A compiled step runs on whatever tensors it is called with; the recording is one of these shapes and dtypes.  A
        step that updates an input in place is not replayed if another input sees the update: their order matters."""
        for x, form in zip(inputs, self.forms):
            if x is None or form is None:
                if x is not form:
                    return False
            elif x.dtype != form[0] or x.shape != form[1]:
                return False
        if self.written:
            end = 0
            for a, n in sorted([(x.data_ptr(), n) for x, n in zip(inputs, self.sizes) if n]):
                if a < end:
                    return False
                end = a + n
        return True

    def run(self, inputs: Sequence) -> list:
        from ..ops import native

        stream = torch.cuda.current_stream(self.device)
        stream.wait_event(self.done)       # the buffers may still be in use by a replay on another stream
        fresh = [torch.empty_like(t) for t in self.results]     # (if there is no memory for them, nothing has run yet)
        try:
            for which, buffers in self.into:
                _copy(buffers, [inputs[k] for k in which])      # (what requires grad is not replayed where grad is recorded)
            self.graph.replay()
            native.LAUNCHES[0] += self.launches
            for which, results in self.out:
                _copy([fresh[n] for n in which], results)
            for which, buffers in self.back:
                # (.data: like the kernels' own in-place updates, this does not touch autograd's version counters)
                _copy([inputs[k].data for k in which], buffers)
        finally:
            self.done.record(stream)       # whatever is in flight uses the buffers, also after an error
        return [o[1] if o[0] == "c" else {o[1]: inputs[o[2]] if o[0] == "in" else fresh[o[2]]} for o in self.outputs]

    def release(self) -> None:
        try:
            self.done.synchronize()        # nothing that uses the buffers is in flight when they are given back
        except Exception:  # pragma: no cover - the context is gone at interpreter exit
            pass
        self.graph = None
        self.static, self.results, self.into, self.back, self.out = [], [], [], [], []


class StepReplay:
    """The recording of one compiled program, made and used by :meth:`run`."""

    def __init__(self, prog: Program):
        self.prog = prog
        self.lock = threading.Lock()
        self.calls = 0
        self.recording: _Recording | None = None
        self.ok: bool | None = None       # may this program be recorded at all?

    def _applies(self, inputs: Sequence, device: torch.device) -> bool:
        from . import executor

        if self.ok is None:
            self.ok = device.type == "cuda" and _program_ok(self.prog)
        if not self.ok or not config.step_graphs.value or executor._TIMES or optimes.ACTIVE[0] or fault._PLAN[0] is not None or config.nvtx_ranges.value:
            return False
        if os.environ.get("JAXPP_B200_TRACK_LIVE_BYTES") == "1" or torch.cuda.current_device() != (device.index or 0):
            return False
        grad = torch.is_grad_enabled()
        for x in inputs:
            if x is not None and (not _plain(x, device) or (grad and x.requires_grad)):
                return False
        # dispatch and function modes (tracing, fake tensors, profilers of ops) see every op of an op-by-op run
        if torch.utils._python_dispatch._get_current_dispatch_mode() is not None or torch.overrides._get_current_function_mode() is not None:
            return False
        return not torch.is_autocast_enabled("cuda") and not torch.cuda.is_current_stream_capturing()

    def run(self, inputs: Sequence, device: torch.device, execute) -> list | None:
        """The outputs of one step (as ``run_single_controller`` returns them), or ``None``: run it op by op.
        ``execute(inputs)`` runs the program op by op and returns its outputs."""
        if self.ok is False or not self._applies(inputs, device):
            return None
        with self.lock:
            rec = self.recording
            if rec is None:
                self.calls += 1
                if self.calls <= EAGER_CALLS:
                    return None
                rec = self._record(inputs, device, execute)
            if rec is None or rec.settings != _settings() or rec.device != device or not rec.covers(inputs):
                return None
            return rec.run(inputs)

    def _record(self, inputs, device, execute) -> _Recording | None:
        most = MAX_POOL_BYTES + _input_bytes(inputs)
        with _pool_lock:
            if _pool_bytes[0] + most > TOTAL_POOL_BYTES:
                return None
            _pool_bytes[0] += most      # reserved until the size is known
        rec = None
        try:
            rec = _Recording(self.prog, inputs, device, execute)
        except Exception as e:
            # not capturable after all, or no memory for it: nothing has run, the caller runs the step op by op
            logger.info("step is not replayed as a CUDA graph: %s", e)
        keep = rec is not None and rec.pool_bytes <= MAX_POOL_BYTES
        with _pool_lock:
            _pool_bytes[0] += (rec.kept_bytes if keep else 0) - most
        if not keep:
            self.ok = False
            if rec is not None:
                rec.release()
        self.recording = rec if keep else None
        return self.recording

    def _drop(self) -> None:
        rec, self.recording = self.recording, None
        if rec is not None:
            with _pool_lock:
                _pool_bytes[0] -= rec.kept_bytes
            rec.release()

    def __del__(self):
        try:
            self._drop()
        except Exception:  # pragma: no cover - interpreter exit
            pass
