"""Run a packaged recipe on the current CUDA device with torch tensors as caller buffers.

This is the call a user makes: ``Runner(aim).run(inputs, outputs)`` wraps
``Runtime.create -> Model.load -> Session.create -> Session.enqueue`` of ``runtime.py`` and
submits on torch's current stream.  torch only owns device memory and streams here; every
kernel comes from the AIM's CUBIN through the native loader.
"""
from __future__ import annotations

from collections import OrderedDict
from pathlib import Path
from typing import Mapping

from . import runtime as rt

TORCH_DTYPES = {"F32": "float32", "F16": "float16", "BF16": "bfloat16", "F8_E4M3": "uint8", "I32": "int32"}


MAX_BINDINGS = 8       # sets of tensor addresses whose packed views are kept (the loader keeps as many graphs)


class Runner:
    def __init__(self, aim_path: str | Path, profile: str = "", flags: int = 0, probe_libraries: bool = False):
        import torch
        if not torch.cuda.is_available():
            raise RuntimeError("aginfer_b200.Runner needs a CUDA device; there is no CPU execution path")
        torch.cuda.current_stream().synchronize()  # make sure torch's context is the current one
        overrides = {} if probe_libraries else dict(cuda_runtime_version_override=12080, cublaslt_abi_override=12,
                                                    cudnn_abi_override=9)
        self.runtime = rt.Runtime.create(**overrides)
        self.model = rt.Model.load(aim_path)
        self.session = rt.Session.create(self.runtime, self.model, profile, flags)
        self.inputs = self.session.input_info()
        self.outputs = self.session.output_info()
        self._dtypes = {t.name: t.dtype for t in self.inputs + self.outputs}
        self._bindings: OrderedDict = OrderedDict()    # tensor names and addresses -> (packed views, layouts)
        self._side = None
        self._replays = not flags & rt.NO_GRAPH_REPLAY
        # the raw handle of torch's current stream, without building a Stream object on every call
        raw, device = getattr(torch._C, "_cuda_getCurrentRawStream", None), getattr(torch._C, "_cuda_getDevice", None)
        self._current_stream = ((lambda: raw(device())) if raw is not None and device is not None
                                else (lambda: torch.cuda.current_stream().cuda_stream))

    def empty_outputs(self, device="cuda") -> dict:
        import torch
        return {t.name: torch.empty(t.shape, dtype=getattr(torch, TORCH_DTYPES[t.dtype]), device=device)
                for t in self.outputs}

    def run(self, inputs: Mapping[str, "object"], outputs: Mapping[str, "object"] | None = None, stream=None,
            denoising_steps: int = 0, noise_override=None) -> dict:
        """``denoising_steps`` / ``noise_override`` (a tensor) travel as the reference's RunOptions: another
        number of Euler steps runs the package's sibling profile for it, and the override replaces the ``noise``
        input (which may then be left out of ``inputs``)."""
        outputs = dict(outputs) if outputs is not None else self.empty_outputs()
        options = None
        if denoising_steps or noise_override is not None:
            view = None
            if noise_override is not None:
                view = rt.TensorView.from_torch("noise_override", noise_override, self._dtypes.get("noise"))
                self._override_keep = noise_override
            options = rt.run_options(denoising_steps, view)
        key = (*inputs, *outputs, *[t.data_ptr() for t in inputs.values()], *[t.data_ptr() for t in outputs.values()])
        tensors = (*inputs.values(), *outputs.values())
        # What the packed views say about a tensor beside its address, looked at on every call: a tensor can be given
        # another shape or stride in place, and another one can stand at the same address.
        layout = [(t.shape, t.stride(), t.dtype, t.storage_offset(), t.untyped_storage().nbytes()) for t in tensors]
        bound = self._bindings.get(key)
        if bound is None or bound[1] != layout:
            packed = self.session.bind(
                [rt.TensorView.from_torch(n, t, self._dtypes.get(n)) for n, t in inputs.items()],
                [rt.TensorView.from_torch(n, t, self._dtypes.get(n)) for n, t in outputs.items()])
            if bound is None and len(self._bindings) >= MAX_BINDINGS:
                self._bindings.popitem(last=False)
            bound = self._bindings[key] = (packed, layout)
        self._bindings.move_to_end(key)
        self._keep = tensors       # in use until the next call at least
        raw = self._current_stream() if stream is None else stream.cuda_stream
        if raw == 0 and not self._replays:
            # Replay switched off: every launch goes to a stream of its own, ordered after and before the work on the
            # default stream.  With replay on, graphs and the first pass over a further set of addresses (launched one
            # by one) go into the default stream itself.
            import torch
            if self._side is None:
                self._side = torch.cuda.Stream()
            default = stream if stream is not None else torch.cuda.current_stream()
            self._side.wait_stream(default)
            self.session.enqueue_packed(bound[0], self._side.cuda_stream, options)
            default.wait_stream(self._side)
        else:
            self.session.enqueue_packed(bound[0], raw, options)
        return outputs

    def stats(self) -> dict:
        return self.session.stats()
