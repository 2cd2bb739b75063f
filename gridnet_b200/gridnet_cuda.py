"""Module-shaped stand-in for the reference's native extension ``gridnet_cuda``.

Same four functions, same positional arguments and the same contract as the
pybind11 module in src/gridnet_cuda.cpp:188-194: tensors must be CUDA and
contiguous (RuntimeError otherwise), outputs are caller-allocated, nothing is
returned. Work is queued on torch's current stream (the reference launches on
the legacy default stream, src/gridnet_cuda_kernels.cu:761).

The gradient outputs are overwritten; the reference accumulates into tensors its
caller zeroes first (gridnet/backend_cuda.py:78-81), which gives the same values.
"""
from __future__ import annotations

import functools

import torch

from ._lib import GN_ERR_UNSUPPORTED, GridnetB200Error, activation_id, check, lib


def _check_input(t: torch.Tensor, name: str) -> None:
    if not t.is_cuda:
        raise GridnetB200Error(f"{name} must be a CUDA tensor")
    if not t.is_contiguous():
        raise GridnetB200Error(f"{name} must be contiguous")


def _suffix(t: torch.Tensor) -> str:
    if t.dtype == torch.float32:
        return "f32"
    if t.dtype == torch.float64:
        return "f64"
    raise GridnetB200Error(f"unsupported dtype {t.dtype}: float32 and float64 only")


def _same(ts, names):
    dtype, device = ts[0].dtype, ts[0].device
    for t, n in zip(ts, names):
        if not (t.is_cuda and t.is_contiguous()):
            _check_input(t, n)
        if t.dtype != dtype or t.device != device:
            raise GridnetB200Error(f"{n}: dtype/device differs from {names[0]}")


def _stream(t: torch.Tensor) -> int:
    return torch._C._cuda_getCurrentRawStream(t.device.index)


def forward(weight, bias, scale, initActivations, outActivations, innerIterations, blockSize, eps,
            normalize, activation) -> None:
    _same((weight, bias, scale, initActivations, outActivations),
          ("weight", "bias", "scale", "initActivations", "outActivations"))
    B, M, N, K = initActivations.shape
    fn = getattr(lib, "gn_step_forward_" + _suffix(weight))
    with torch.cuda.device(weight.device):
        check(fn(weight.data_ptr(), bias.data_ptr(), scale.data_ptr(), initActivations.data_ptr(),
                 outActivations.data_ptr(), B, M, N, K, int(innerIterations), int(blockSize), float(eps),
                 int(bool(normalize)), activation_id(activation), _stream(weight)))


def backward(weight, bias, scale, initActivations, outGrads, weightGradOut, biasGradOut, scaleGradOut,
             activationsGradOut, innerIterations, blockSize, eps, normalize, activation) -> None:
    _same((weight, bias, scale, initActivations, outGrads, weightGradOut, biasGradOut, scaleGradOut,
           activationsGradOut),
          ("weight", "bias", "scale", "initActivations", "outGrads", "weightGradOut", "biasGradOut",
           "scaleGradOut", "activationsGradOut"))
    B, M, N, K = initActivations.shape
    sfx = _suffix(weight)
    with torch.cuda.device(weight.device):
        need = 0
        if sfx == "f32" and B > 0:
            need = int(lib.gn_step_backward_workspace_bytes(B, M, N, K, int(innerIterations), int(blockSize),
                                                            int(bool(normalize)), 4))
        if need:
            # scratch for the tuned four-kernel path (torch's caching allocator, stream ordered)
            ws = torch.empty(need, dtype=torch.uint8, device=weight.device)
            check(lib.gn_step_backward_ws_f32(
                weight.data_ptr(), bias.data_ptr(), scale.data_ptr(), initActivations.data_ptr(), outGrads.data_ptr(),
                weightGradOut.data_ptr(), biasGradOut.data_ptr(), scaleGradOut.data_ptr(),
                activationsGradOut.data_ptr(), B, M, N, K, int(innerIterations), int(blockSize), float(eps),
                int(bool(normalize)), activation_id(activation), ws.data_ptr(), ws.numel(), _stream(weight)))
            return
        fn = getattr(lib, "gn_step_backward_" + sfx)
        check(fn(weight.data_ptr(), bias.data_ptr(), scale.data_ptr(), initActivations.data_ptr(),
                 outGrads.data_ptr(), weightGradOut.data_ptr(), biasGradOut.data_ptr(),
                 scaleGradOut.data_ptr(), activationsGradOut.data_ptr(), B, M, N, K, int(innerIterations),
                 int(blockSize), float(eps), int(bool(normalize)), activation_id(activation),
                 _stream(weight)))


def forward_with_stash(weight, bias, scale, initActivations, outActivations, innerIterations, blockSize, activation,
                       stash=None):
    """:func:`forward` (normalize off, float32) that also keeps what the backward pass would otherwise
    recompute, in ``stash`` (``gn_step_stash_bytes`` of uint8) or a new tensor. Returns that tensor, or ``None`` (after running the ordinary forward) where the
    tuned path does not apply. Not part of the reference's module: it always recomputes."""
    _same((weight, bias, scale, initActivations, outActivations),
          ("weight", "bias", "scale", "initActivations", "outActivations"))
    B, M, N, K = initActivations.shape
    need = 0
    if weight.dtype == torch.float32 and B > 0:
        need = int(lib.gn_step_stash_bytes(B, M, N, K, int(innerIterations), int(blockSize)))
    with torch.cuda.device(weight.device):
        if need:
            if stash is None:
                stash = torch.empty(need, dtype=torch.uint8, device=weight.device)
            rc = lib.gn_step_forward_stash_f32(
                weight.data_ptr(), bias.data_ptr(), scale.data_ptr(), initActivations.data_ptr(),
                outActivations.data_ptr(), B, M, N, K, int(innerIterations), int(blockSize), activation_id(activation),
                stash.data_ptr(), stash.numel(), _stream(weight))
            if rc == 0:
                return stash
            if rc != GN_ERR_UNSUPPORTED:  # anything but "the tuned path does not apply here"
                check(rc)
    forward(weight, bias, scale, initActivations, outActivations, innerIterations, blockSize, 1e-5, False, activation)
    return None


def backward_with_stash(weight, bias, scale, initActivations, outGrads, weightGradOut, biasGradOut, scaleGradOut,
                        activationsGradOut, innerIterations, blockSize, activation, stash) -> None:
    """:func:`backward` for a step whose forward pass went through :func:`forward_with_stash`."""
    _same((weight, bias, scale, initActivations, outGrads, weightGradOut, biasGradOut, scaleGradOut,
           activationsGradOut),
          ("weight", "bias", "scale", "initActivations", "outGrads", "weightGradOut", "biasGradOut",
           "scaleGradOut", "activationsGradOut"))
    B, M, N, K = initActivations.shape
    with torch.cuda.device(weight.device):
        need = int(lib.gn_step_backward_stash_workspace_bytes(B, M, N, K, int(innerIterations), int(blockSize)))
        ws = torch.empty(need, dtype=torch.uint8, device=weight.device)
        check(lib.gn_step_backward_stash_f32(
            weight.data_ptr(), bias.data_ptr(), scale.data_ptr(), initActivations.data_ptr(), outGrads.data_ptr(),
            weightGradOut.data_ptr(), biasGradOut.data_ptr(), scaleGradOut.data_ptr(), activationsGradOut.data_ptr(),
            B, M, N, K, int(innerIterations), int(blockSize), activation_id(activation), stash.data_ptr(), stash.numel(),
            ws.data_ptr(), ws.numel(), _stream(weight)))


@functools.lru_cache(maxsize=512)
def _step_bytes(device: int, B: int, M: int, N: int, K: int, inner: int, block: int, normalize: bool):
    """(what a step keeps, scratch forward without and with keeping it, scratch backward without and with what was kept),
    in bytes; None where the kernels of :func:`forward_kept` do not apply. Asked once per shape: five calls into the
    library cost as much as two launches."""
    with torch.cuda.device(device):
        kept = int(lib.gn_step_kept_bytes(B, M, N, K, inner, block, normalize))
        if not kept:
            return None
        return (kept, *(int(lib.gn_step_kept_workspace_bytes(B, M, N, K, inner, block, normalize, b, k))
                        for b in (0, 1) for k in (0, 1)))


def step_bytes(weight, initActivations, innerIterations, blockSize, normalize):
    if weight.dtype != torch.float32 or not weight.is_cuda:
        return None
    return _step_bytes(weight.device.index, *initActivations.shape, int(innerIterations), int(blockSize), bool(normalize))


def forward_kept(weight, bias, scale, initActivations, outActivations, innerIterations, blockSize, eps, normalize, activation,
                 kept=None) -> None:
    """:func:`forward` on the kernels that hold the weights in tensor memory; ``kept`` (``gn_step_kept_bytes`` of uint8)
    receives what :func:`backward_kept` would otherwise compute again."""
    _same((weight, bias, scale, initActivations, outActivations),
          ("weight", "bias", "scale", "initActivations", "outActivations"))
    B, M, N, K = initActivations.shape
    with torch.cuda.device(weight.device):
        need = step_bytes(weight, initActivations, innerIterations, blockSize, normalize)[2 if kept is not None else 1]
        ws = torch.empty(need, dtype=torch.uint8, device=weight.device)
        check(lib.gn_step_forward_kept_f32(
            weight.data_ptr(), bias.data_ptr(), scale.data_ptr(), initActivations.data_ptr(), outActivations.data_ptr(), B, M, N, K,
            int(innerIterations), int(blockSize), float(eps), int(bool(normalize)), activation_id(activation),
            None if kept is None else kept.data_ptr(), 0 if kept is None else kept.numel(), ws.data_ptr(), need, _stream(weight)))


def backward_kept(weight, bias, scale, initActivations, outGrads, weightGradOut, biasGradOut, scaleGradOut, activationsGradOut,
                  innerIterations, blockSize, eps, normalize, activation, kept=None) -> None:
    """:func:`backward` for a step whose forward pass went through :func:`forward_kept`."""
    _same((weight, bias, scale, initActivations, outGrads, weightGradOut, biasGradOut, scaleGradOut,
           activationsGradOut),
          ("weight", "bias", "scale", "initActivations", "outGrads", "weightGradOut", "biasGradOut",
           "scaleGradOut", "activationsGradOut"))
    B, M, N, K = initActivations.shape
    with torch.cuda.device(weight.device):
        need = step_bytes(weight, initActivations, innerIterations, blockSize, normalize)[4 if kept is not None else 3]
        ws = torch.empty(need, dtype=torch.uint8, device=weight.device)
        check(lib.gn_step_backward_kept_f32(
            weight.data_ptr(), bias.data_ptr(), scale.data_ptr(), initActivations.data_ptr(), outGrads.data_ptr(),
            weightGradOut.data_ptr(), biasGradOut.data_ptr(), scaleGradOut.data_ptr(), activationsGradOut.data_ptr(), B, M, N, K,
            int(innerIterations), int(blockSize), float(eps), int(bool(normalize)), activation_id(activation),
            None if kept is None else kept.data_ptr(), 0 if kept is None else kept.numel(), ws.data_ptr(), ws.numel(), _stream(weight)))


def forward_gated(weight, bias, initActivations, outActivations, innerIterations, blockSize,
                  activation) -> None:
    _same((weight, bias, initActivations, outActivations),
          ("weight", "bias", "initActivations", "outActivations"))
    B, M, N, K = initActivations.shape
    fn = getattr(lib, "gn_gated_forward_" + _suffix(weight))
    with torch.cuda.device(weight.device):
        check(fn(weight.data_ptr(), bias.data_ptr(), initActivations.data_ptr(), outActivations.data_ptr(),
                 B, M, N, K, int(innerIterations), int(blockSize), activation_id(activation),
                 _stream(weight)))


def backward_gated(weight, bias, initActivations, outGrads, weightGradOut, biasGradOut, activationsGradOut,
                   innerIterations, blockSize, activation) -> None:
    _same((weight, bias, initActivations, outGrads, weightGradOut, biasGradOut, activationsGradOut),
          ("weight", "bias", "initActivations", "outGrads", "weightGradOut", "biasGradOut",
           "activationsGradOut"))
    B, M, N, K = initActivations.shape
    fn = getattr(lib, "gn_gated_backward_" + _suffix(weight))
    with torch.cuda.device(weight.device):
        need = 0
        if _suffix(weight) == "f32" and B > 0:
            need = int(lib.gn_gated_backward_workspace_bytes(B, M, N, K, int(innerIterations), int(blockSize), 4))
        if need:
            # scratch for the tuned four-kernel path (torch's caching allocator, stream ordered)
            ws = torch.empty(need, dtype=torch.uint8, device=weight.device)
            check(lib.gn_gated_backward_ws_f32(
                weight.data_ptr(), bias.data_ptr(), initActivations.data_ptr(), outGrads.data_ptr(),
                weightGradOut.data_ptr(), biasGradOut.data_ptr(), activationsGradOut.data_ptr(), B, M, N, K,
                int(innerIterations), int(blockSize), activation_id(activation), ws.data_ptr(), ws.numel(),
                _stream(weight)))
            return
        check(fn(weight.data_ptr(), bias.data_ptr(), initActivations.data_ptr(), outGrads.data_ptr(),
                 weightGradOut.data_ptr(), biasGradOut.data_ptr(), activationsGradOut.data_ptr(), B, M, N, K,
                 int(innerIterations), int(blockSize), activation_id(activation), _stream(weight)))
