"""Autograd ops with the reference's op surface (gridnet/backend_cuda.py:5-190).

``GridnetCudaOp.apply(weight, bias, residual_scale, init_activations, inner_iters,
block_size, eps, normalize, activation)`` and ``GatedGridnetCudaOp.apply(weight,
bias, init_activations, inner_iters, block_size, activation)`` take the same
arguments, make the same shape/dtype/device assertions (AssertionError), return a
clone for an empty batch and hand back the same gradient tuples as the reference
classes, so ``gridnet/__init__.py:14-18`` can import them in place of the originals.

Added on top of that surface, for the whole-grid normalisation the reference's
models run between steps (gridnet/scripts/train_mnist.py:54,62-64):
``GridNormOp`` (LayerNorm over [M,N,K] per sample, forward and backward) and
``outer_forward`` (the fused inference loop).
"""
from __future__ import annotations

import ctypes
import functools

import torch

from . import gridnet_cuda, patch_loop
from ._lib import activation_id, check, lib


def _assert_step_args(weight, bias, residual_scale, init_activations, block_size, gated):
    batch_size, m, n, k = init_activations.shape
    assert m % block_size == 0 and n % block_size == 0 and k % block_size == 0, (
        f"{block_size=} incompatible with {init_activations.shape=}")
    want = (27, 2, m, n, k) if gated else (27, m, n, k)
    assert tuple(weight.shape) == want, f"{weight.shape=} invalid for {init_activations.shape=}"
    assert bias.shape == weight.shape[1:], f"{bias.shape=} invalid for {weight.shape=}"
    others = [("bias", bias), ("init_activations", init_activations)]
    if not gated:
        assert bias.shape == residual_scale.shape, f"{bias.shape=} invalid for {residual_scale.shape=}"
        others.insert(1, ("residual_scale", residual_scale))
    for name, t in others:
        assert weight.dtype == t.dtype, f"mismatching dtypes: {weight.dtype=} {name}.dtype={t.dtype}"
    for name, t in others:
        assert weight.device == t.device, f"mismatching devices: {weight.device=} {name}.device={t.device}"
    return batch_size


_keep_forward_stash = None  # None: decide per call from the free device memory


def keep_forward_stash(enabled):
    """Trade memory for time in training: a forward pass of a step or a loop that will be differentiated (float32) can also keep
    what its inner iterations computed, so that its backward skips computing that again (about a quarter of the backward time;
    same gradient bits): of a step (:class:`GridnetCudaOp`) ``inner_iters`` to ``2 * inner_iters - 1`` extra activation tensors,
    two and the statistics of the blocks more with per-block normalisation; of a loop ``inner_iters`` per outer step (gated:
    three times that). The reference always recomputes. ``True`` / ``False`` force the choice; ``None`` (the default)
    decides by memory. Steps keep it while all steps alive keep less than 2 GiB on the device together, and beyond that while it
    is at most a tenth of the device memory that is free at that moment. The loops decide once per loop how many of their LAST
    outer steps keep theirs: all where the loop holds less than a GiB, else as many as fit into 70 % of the free memory.
    What cannot be allocated after all is recomputed. Returns the previous setting."""
    global _keep_forward_stash
    previous, _keep_forward_stash = _keep_forward_stash, (None if enabled is None else bool(enabled))
    return previous


def _free_bytes(device) -> int:
    """Free memory of the device as a caller of torch sees it: what the caching allocator holds but has not handed out
    counts. Asks the driver: 0.3 ms on a quiet host, now and then tens or hundreds where other programs use it."""
    free, _ = torch.cuda.mem_get_info(device)
    return free + torch.cuda.memory_reserved(device) - torch.cuda.memory_allocated(device)


class _Kept:
    """``nbytes`` of device memory that a step keeps for its backward pass. Knows how much all of them hold together on a
    device, which is what makes it unnecessary to ask the driver for the free memory before every small step."""

    # device index -> {id: bytes} of the objects alive. Single dict operations only, no lock: __del__ may run in the middle
    # of __init__ of another one, on the same thread, when the garbage collector decides so
    _alive = {}
    UNASKED = 2 << 30

    def __init__(self, nbytes: int, device):
        self.buffer = torch.empty(nbytes, dtype=torch.uint8, device=device)
        self.alive = _Kept._alive.setdefault(self.buffer.device.index, {})
        self.alive[id(self)] = nbytes

    def __del__(self):
        alive = getattr(self, "alive", None)
        if alive is not None:
            alive.pop(id(self), None)

    @staticmethod
    def room_for(need: int, device) -> bool:
        """As :func:`keep_forward_stash` says; otherwise while all steps together keep less than 2 GiB on the device, and
        beyond that while ``need`` is at most a tenth of its free memory."""
        if _keep_forward_stash is not None:
            return _keep_forward_stash
        if sum(list(_Kept._alive.get(device.index, {}).values())) + need <= _Kept.UNASKED:
            return True
        return need * 10 <= _free_bytes(device)


# Time of a step forward and backward in microseconds, measured over 16 x 32 x 24 .. 96^3 grids, batches of 2 to 128 and one to
# five inner iterations: max(host, fixed + per neuron * P + B * P * (a + b * inner)). The kernels of forward_kept re-order 27 weights per
# neuron three times but do a sample in a half to two thirds of the time (a seventh against the general kernels, which are the
# others' choice for normalised blocks of 4).
_STEP_COST_KEPT = {False: (195, 0, 4.2e-4, 14e-6, 6e-6), True: (195, 0, 4.2e-4, 18e-6, 8e-6)}  # by normalize
_STEP_COST_OTHER = {(8, False): (175, 85, 5e-5, 11e-6, 10.5e-6), (8, True): (170, 100, 7e-5, 20e-6, 19.7e-6),
                    (4, False): (175, 60, 6e-5, 12e-6, 15.5e-6), (4, True): (152, 45, 0, 0, 120e-6)}


def _step_cost(c, P: int, B: int, inner: int) -> float:
    host, fixed, per_neuron, a, b = c
    return max(host, fixed + per_neuron * P + B * P * (a + b * inner))


@functools.lru_cache(maxsize=512)
def _kept_is_faster(shape, inner: int, block: int, normalize: bool) -> bool:
    B, M, N, K = shape
    P = M * N * K
    return (block, normalize) in _STEP_COST_OTHER and _step_cost(_STEP_COST_KEPT[normalize], P, 4 * ((B + 3) // 4), inner) < _step_cost(
        _STEP_COST_OTHER[block, normalize], P, B, inner)


def _quad_step(weight, x, inner_iters: int, block_size: int, normalize: bool):
    """What :func:`gridnet_cuda.step_bytes` says if the step should run on the kernels of :func:`gridnet_cuda.forward_kept`."""
    if weight.dtype != torch.float32 or not _kept_is_faster(x.shape, int(inner_iters), int(block_size), bool(normalize)):
        return None
    return gridnet_cuda.step_bytes(weight, x, inner_iters, block_size, normalize)


class _Op(torch.autograd.Function):
    """An op that keeps things for its backward pass. Where gradients are off there is none, but a parameter still says that it
    requires one (``ctx.needs_input_grad``), so it comes detached."""

    @classmethod
    def apply(cls, *args):
        if not torch.is_grad_enabled():
            args = [a.detach() if isinstance(a, torch.Tensor) else a for a in args]
        return super().apply(*args)


class GridnetCudaOp(_Op):
    """One outer-loop step of the plain gridnet (gridnet/backend_cuda.py:5-108)."""

    @staticmethod
    def forward(ctx, weight, bias, residual_scale, init_activations, inner_iters: int, block_size: int,
                eps: float, normalize: bool, activation: str):
        batch_size = _assert_step_args(weight, bias, residual_scale, init_activations, block_size, False)
        if not batch_size:
            return init_activations.clone()
        ctx.save_for_backward(weight, bias, residual_scale, init_activations)
        ctx.cfg = (inner_iters, block_size, eps, normalize, activation)
        ctx.kept = None
        outputs = torch.empty_like(init_activations)
        args = (weight, bias, residual_scale, init_activations, outputs, inner_iters, block_size)
        quad = _quad_step(weight, init_activations, inner_iters, block_size, normalize)
        ctx.quad = quad is not None
        need = 0
        if weight.dtype == torch.float32 and any(ctx.needs_input_grad[:4]):
            if quad is not None:
                need = quad[0]
            elif not normalize:
                need = int(lib.gn_step_stash_bytes(*init_activations.shape, int(inner_iters), int(block_size)))
        if need and _Kept.room_for(need, weight.device):
            try:
                ctx.kept = _Kept(need, weight.device)
            except torch.cuda.OutOfMemoryError:
                pass  # the backward pass runs the step again
        if ctx.quad:
            gridnet_cuda.forward_kept(*args, eps, normalize, activation, None if ctx.kept is None else ctx.kept.buffer)
        elif ctx.kept is not None:
            if gridnet_cuda.forward_with_stash(*args, activation, ctx.kept.buffer) is None:
                ctx.kept = None
        else:
            gridnet_cuda.forward(*args, eps, normalize, activation)
        return outputs

    @staticmethod
    def backward(ctx, grad_output):
        weight, bias, residual_scale, init_activations = ctx.saved_tensors
        inner_iters, block_size, eps, normalize, activation = ctx.cfg
        # every gradient buffer is written in full by the library: no zero fill
        grads = [torch.empty_like(t) for t in ctx.saved_tensors]
        args = (weight, bias, residual_scale, init_activations, grad_output.contiguous(), *grads, inner_iters, block_size)
        kept, ctx.kept = ctx.kept, None
        if ctx.quad:
            gridnet_cuda.backward_kept(*args, eps, normalize, activation, None if kept is None else kept.buffer)
        elif kept is not None:
            gridnet_cuda.backward_with_stash(*args, activation, kept.buffer)
        else:
            gridnet_cuda.backward(*args, eps, normalize, activation)
        return (*grads, None, None, None, None, None)


class GatedGridnetCudaOp(torch.autograd.Function):
    """One outer-loop step of the gated gridnet (gridnet/backend_cuda.py:111-190)."""

    @staticmethod
    def forward(ctx, weight, bias, init_activations, inner_iters: int, block_size: int, activation: str):
        batch_size = _assert_step_args(weight, bias, None, init_activations, block_size, True)
        if not batch_size:
            return init_activations.clone()
        ctx.save_for_backward(weight, bias, init_activations)
        ctx.cfg = (inner_iters, block_size, activation)
        outputs = torch.empty_like(init_activations)
        gridnet_cuda.forward_gated(weight, bias, init_activations, outputs, inner_iters, block_size, activation)
        return outputs

    @staticmethod
    def backward(ctx, grad_output):
        weight, bias, init_activations = ctx.saved_tensors
        inner_iters, block_size, activation = ctx.cfg
        weight_grad = torch.empty_like(weight)
        bias_grad = torch.empty_like(bias)
        act_grad = torch.empty_like(init_activations)
        gridnet_cuda.backward_gated(weight, bias, init_activations, grad_output.contiguous(), weight_grad,
                                    bias_grad, act_grad, inner_iters, block_size, activation)
        return weight_grad, bias_grad, act_grad, None, None, None


def _workspace(nbytes: int, device) -> torch.Tensor:
    return torch.empty(max(int(nbytes), 256), dtype=torch.uint8, device=device)


def _require_f32_cuda(**tensors):
    for name, t in tensors.items():
        if not t.is_cuda:
            raise RuntimeError(f"{name} must be a CUDA tensor")
        if t.dtype != torch.float32:
            raise RuntimeError(f"{name} must be float32")
        if not t.is_contiguous():
            raise RuntimeError(f"{name} must be contiguous")


class GridNormOp(torch.autograd.Function):
    """``torch.nn.LayerNorm`` over the whole grid of each sample, float32.

    ``GridNormOp.apply(x, gamma, beta, eps)`` with x [B, M, N, K] and gamma, beta
    [M, N, K] equals ``F.layer_norm(x, x.shape[1:], gamma, beta, eps)``.
    """

    @staticmethod
    def forward(ctx, x, gamma, beta, eps: float = 1e-5):
        assert x.shape[1:] == gamma.shape == beta.shape, f"{gamma.shape=} {beta.shape=} invalid for {x.shape=}"
        if not x.shape[0]:
            return x.clone()
        _require_f32_cuda(x=x, gamma=gamma, beta=beta)
        B, P = x.shape[0], x[0].numel()
        y = torch.empty_like(x)
        ws = _workspace(lib.gn_norm_workspace_bytes(B, P), x.device)
        with torch.cuda.device(x.device):
            check(lib.gn_norm_forward_f32(x.data_ptr(), gamma.data_ptr(), beta.data_ptr(), y.data_ptr(), None, B,
                                          P, float(eps), ws.data_ptr(), ws.numel(),
                                          torch.cuda.current_stream().cuda_stream))
        ctx.save_for_backward(x, gamma)
        ctx.eps = float(eps)
        return y

    @staticmethod
    def backward(ctx, grad_y):
        x, gamma = ctx.saved_tensors
        grad_y = grad_y.contiguous()
        B, P = x.shape[0], x[0].numel()
        gx, gg, gb = torch.empty_like(x), torch.empty_like(gamma), torch.empty_like(gamma)
        ws = _workspace(lib.gn_norm_workspace_bytes(B, P), x.device)
        with torch.cuda.device(x.device):
            check(lib.gn_norm_backward_f32(x.data_ptr(), gamma.data_ptr(), grad_y.data_ptr(), gx.data_ptr(),
                                           gg.data_ptr(), gb.data_ptr(), B, P, ctx.eps, ws.data_ptr(), ws.numel(),
                                           torch.cuda.current_stream().cuda_stream))
        return gx, gg, gb, None


_STAGGER = 4352  # bytes: 17 x 256, keeps 256-byte alignment
_BIG = 1 << 30


def _staggered(nbytes: int, device, k: int) -> torch.Tensor:
    """``nbytes`` of device memory; from a GiB up starting ``(k % 7 + 1) * 4352`` bytes into its allocation. The tensors a
    training step streams side by side (input, output, kept iterations) are each an exact power of two in size at the
    benchmark's shapes, so fresh allocations start at the same offset inside every 2 MB page. Different offsets were meant to keep the
    streams off the same memory channels; with the kernels of today they make no difference (C3's forward pass 51.8 ms with
    them, 51.4 without, six processes each), and what made single passes longer was :func:`_free_bytes`."""
    if nbytes < _BIG:
        return torch.empty(nbytes, dtype=torch.uint8, device=device)
    off = (k % 7 + 1) * _STAGGER
    return torch.empty(nbytes + 8 * _STAGGER, dtype=torch.uint8, device=device)[off:off + nbytes]


def _pointers(tensors):
    return (ctypes.c_void_p * len(tensors))(*[None if t is None else t.data_ptr() for t in tensors])


class _Piece:
    """A piece of an allocation, where a tensor of its own would only be asked for its address."""
    __slots__ = ("of", "address")
    dtype = torch.uint8

    def __init__(self, of: torch.Tensor, offset: int):
        self.of, self.address = of, of.data_ptr() + offset

    def data_ptr(self) -> int:
        return self.address


class _Pool:
    """What a small loop keeps for its backward pass, in one allocation: a tensor to save and to unpack instead of one per step
    and kind (32^3, 8 steps: 17 of them, 60 us of the host's time)."""

    def __init__(self, memory: torch.Tensor, layout):
        self.memory, self.layout = memory, layout

    def _cut(self, piece):
        outer, stat, one, keep, stash = self.layout
        kept = stat + (outer + 1) * one
        return (piece(stat, one), piece(0, stat), [piece(stat + (k + 1) * one, one) for k in range(outer)],
                [None] * (outer - keep) + [piece(kept + k * stash, stash) for k in range(keep)])

    def pieces(self):
        """(x_il4, stats, outs, stashes) of :func:`_loop_forward`, as addresses."""
        return self._cut(lambda off, nbytes: _Piece(self.memory, off))

    def __iter__(self):
        """The same as tensors."""
        return iter(self._cut(lambda off, nbytes: self.memory[off:off + nbytes]))


def _kept_steps(nbytes_out: int, nbytes_stash: int, outer: int, device) -> int:
    """How many of the ``outer`` steps of a differentiated loop keep their inner iterations (the LAST ones: their
    backward comes first): all or none when :func:`keep_forward_stash` forces it; otherwise as many as fit into 70 % of the
    device memory that is free when the loop starts. A loop that needs less than a GiB in all does not ask (the driver's
    answer takes longer than a small model's forward pass)."""
    if _keep_forward_stash is not None:
        return outer if _keep_forward_stash else 0
    per_step = nbytes_out + nbytes_stash
    if per_step * outer < _BIG:
        return outer
    return max(0, min(outer, int(0.7 * _free_bytes(device)) // per_step))


def _allocate_stashes(outer: int, keep: int, nbytes: int, device):
    """Room for the iterations of the last ``keep`` of ``outer`` steps, None for the others."""
    stashes = [None] * outer
    try:
        for k in reversed(range(outer - keep, outer)):  # the last ones first: where memory ends, the others go without
            stashes[k] = _staggered(nbytes, device, k + 3)
    except torch.cuda.OutOfMemoryError:
        # what is left free is the backward pass's: give back what it takes to run iterations again
        for k in range(outer):
            if stashes[k] is not None:
                stashes[k] = None
                break
    return stashes


def on_patches(B: int, M: int, N: int, K: int) -> bool:
    """Whether a loop with gradients runs on the register-patch kernels (gated, one sample: as its steps and norms one by one).
    The quad kernels compute, keep and walk back four samples whatever the batch. On small grids they are faster all the same
    (one sample, 2 x 8 iterations: 64^3 0.71 ms against 2.9, 128^3 4.5 against 4.5); beyond 128^3 one sample, beyond twice that two
    are better off with the other kernels, which also hold no more activations than there are. ms and GB, quad / patches: 160^3,
    2 x 8, one sample 8.5, 4.1 / 7.8, 2.6, two 8.4 / 8.9; 256^3, 2 x 4, one 17.8, 13.5 / 14.7, 9.5, two 18.1, 13.8 / 17.0, 11.0,
    three 17.9 / 19.8; blocks of 4, 4 x 4, one 24.5, 16.4 / 18.9, 10.6, two 24.4, 16.6 / 24.2, 13.2; gated 160^3, 2 x 4, one 8.1,
    6.4 / 7.5, 3.1, two 8.1 / 8.9."""
    return B <= 2 and M * N * K > B << 21


def _patch_forward(plist, norm_weight, norm_bias, x, inner: int, outer: int, block: int, activation: str, ln_eps: float,
                   residual: bool, need_grad: bool):
    """:func:`_loop_forward` where :func:`on_patches`: x, outs and stashes are in the grid's own layout, x in float32."""
    one, dev = x.numel() * 4, x.device
    with torch.cuda.device(dev):
        stash = patch_loop.stash_bytes(x, inner, block)
        keep = _kept_steps(one, stash, outer, dev) if need_grad and stash else 0
        stats = torch.empty(outer, x.shape[0], 2, dtype=torch.float32, device=dev)
        outs = [_staggered(one, dev, k).view(torch.float32).view(x.shape) for k in range(outer if need_grad else min(2, outer))]
        stashes = _allocate_stashes(outer, keep, stash, dev)
        y = patch_loop.forward(plist, norm_weight, norm_bias, x, inner, outer, block, activation, ln_eps, residual,
                               [outs[k % len(outs)] for k in range(outer)], stats, stashes)
    return y, (x, stats, outs, stashes)


def _loop_forward(plist, norm_weight, norm_bias, x, inner: int, outer: int, block: int, activation: str, ln_eps: float,
                  residual: bool, need_grad: bool, gated: bool = False):
    """The loop forward through ``gn_loop_forward_f32``; ``plist``: one (weight, bias, residual_scale) for all steps, or one
    per step; gated: one (weight, bias), through ``gn_gated_loop_forward_f32``. Returns the output and what the backward pass needs: (x_il4,
    stats, outs, stashes), or a :class:`_Pool` of them."""
    B, M, N, K = x.shape
    for params in plist:
        _assert_step_args(*params, *([None] if gated else []), x, block, gated)
        assert norm_weight.shape == params[1].shape[-3:] == norm_bias.shape, f"{norm_weight.shape=} invalid for {params[1].shape=}"
        _require_f32_cuda(**dict(zip(("weight", "bias", "residual_scale"), params)))
    _require_f32_cuda(norm_weight=norm_weight, norm_bias=norm_bias, x=x)
    # the register-patch kernels read by bulk tensor copies and in pairs
    if not gated and on_patches(B, M, N, K) and all(t.data_ptr() % 16 == 0 for t in (x, norm_weight, norm_bias, *(t for p in plist for t in p))):
        return _patch_forward(plist, norm_weight, norm_bias, x, inner, outer, block, activation, ln_eps, residual, need_grad)
    dev = x.device
    one = int(lib.gn_loop_tensor_bytes(B, M, N, K))
    stat = outer * 4 * ((B + 3) // 4) * 8
    stat = (stat + 255) // 256 * 256
    y = torch.empty_like(x)
    with torch.cuda.device(dev):
        if gated:
            wbytes = int(lib.gn_gated_loop_workspace_bytes(B, M, N, K, inner, outer, 0, 0))
        else:
            wbytes = int(lib.gn_loop_forward_workspace_bytes(B, M, N, K, inner, outer, block, int(residual)))
        if wbytes == 0:
            raise RuntimeError(f"the fused loop does not cover {tuple(x.shape)}, block {block}, {inner} inner iterations")
        ws = torch.empty(wbytes, dtype=torch.uint8, device=dev)
        stashes, pool = [None] * outer, None
        if need_grad:
            stash_bytes = (3 if gated else 1) * inner * one
            keep = _kept_steps(one, stash_bytes, outer, dev)
            total = (outer + 1) * one + stat + keep * stash_bytes
            if total < _BIG:  # one allocation, cut up
                try:
                    pool = torch.empty(total, dtype=torch.uint8, device=dev)
                except torch.cuda.OutOfMemoryError:
                    keep = 0
                    pool = torch.empty((outer + 1) * one + stat, dtype=torch.uint8, device=dev)
                pool = _Pool(pool, (outer, stat, one, keep, stash_bytes))
                x_il4, stats, outs, stashes = pool.pieces()
            else:
                stats = torch.empty(stat, dtype=torch.uint8, device=dev)
                x_il4 = _staggered(one, dev, 6)
                outs = [_staggered(one, dev, k) for k in range(outer)]
                stashes = _allocate_stashes(outer, keep, stash_bytes, dev)
        else:
            stats = torch.empty(stat, dtype=torch.uint8, device=dev)
            x_il4 = torch.empty(one, dtype=torch.uint8, device=dev)
            pair = [torch.empty(one, dtype=torch.uint8, device=dev) for _ in range(min(2, outer))]
            outs = [pair[k & 1] for k in range(outer)]
        if gated:
            weight, bias = plist[0]
            check(lib.gn_gated_loop_forward_f32(weight.data_ptr(), bias.data_ptr(), norm_weight.data_ptr(), norm_bias.data_ptr(), x.data_ptr(),
                                                y.data_ptr(), x_il4.data_ptr(), _pointers(outs), stats.data_ptr(), _pointers(stashes), B, M,
                                                N, K, inner, outer, ln_eps, activation_id(activation), ws.data_ptr(), ws.numel(),
                                                torch.cuda.current_stream().cuda_stream))
            return y, pool or (x_il4, stats, outs, stashes)
        weights, biases, scales = ([p[i] for p in plist] for i in range(3))
        check(lib.gn_loop_forward_f32(_pointers(weights), _pointers(biases), _pointers(scales), len(plist),
                                      norm_weight.data_ptr(), norm_bias.data_ptr(), x.data_ptr(), y.data_ptr(),
                                      x_il4.data_ptr(), _pointers(outs), stats.data_ptr(), _pointers(stashes), B, M, N, K,
                                      inner, outer, block, ln_eps, activation_id(activation), int(residual), ws.data_ptr(),
                                      ws.numel(), torch.cuda.current_stream().cuda_stream))
    return y, pool or (x_il4, stats, outs, stashes)


def _loop_backward(plist, norm_weight, norm_bias, saved, grad_y, inner: int, outer: int, block: int, activation: str,
                   residual: bool, gated: bool = False):
    """The gradients of :func:`_loop_forward` through ``gn_loop_backward_f32``: one (weight, bias, residual_scale) triple per
    entry of ``plist``, then those of the norm's weight and bias and of x."""
    x_il4, stats, outs, stashes = saved
    g = grad_y.contiguous()
    B, M, N, K = g.shape
    dev = g.device
    if x_il4.dtype == torch.float32:  # _patch_forward
        with torch.cuda.device(dev):
            return patch_loop.backward(plist, norm_weight, norm_bias, x_il4, outs, stats, stashes, g, inner, outer, block, activation, residual)
    grads = [tuple(torch.empty_like(t) for t in params) for params in plist]
    gg, gb, gx = torch.empty_like(norm_weight), torch.empty_like(norm_bias), torch.empty_like(g)
    with torch.cuda.device(dev):
        replay = int(any(t is None for t in stashes))
        if gated:
            (weight, bias), (gw, gb_) = plist[0], grads[0]
            ws = torch.empty(int(lib.gn_gated_loop_workspace_bytes(B, M, N, K, inner, outer, 1, replay)), dtype=torch.uint8, device=dev)
            check(lib.gn_gated_loop_backward_f32(weight.data_ptr(), bias.data_ptr(), norm_weight.data_ptr(), norm_bias.data_ptr(),
                                                 x_il4.data_ptr(), _pointers(outs), stats.data_ptr(), _pointers(stashes), g.data_ptr(),
                                                 gw.data_ptr(), gb_.data_ptr(), gg.data_ptr(), gb.data_ptr(), gx.data_ptr(), B, M, N, K,
                                                 inner, outer, activation_id(activation), ws.data_ptr(), ws.numel(),
                                                 torch.cuda.current_stream().cuda_stream))
            return grads, gg, gb, gx
        ws = torch.empty(int(lib.gn_loop_backward_workspace_bytes(B, M, N, K, inner, outer, block, int(residual), replay)),
                         dtype=torch.uint8, device=dev)
        columns = [_pointers([p[i] for p in plist]) for i in range(3)] + [_pointers([p[i] for p in grads]) for i in range(3)]
        check(lib.gn_loop_backward_f32(*columns[:3], len(plist), norm_weight.data_ptr(), norm_bias.data_ptr(), x_il4.data_ptr(),
                                       _pointers(outs), stats.data_ptr(), _pointers(stashes), g.data_ptr(), *columns[3:],
                                       gg.data_ptr(), gb.data_ptr(), gx.data_ptr(), B, M, N, K, inner, outer, block,
                                       activation_id(activation), int(residual), ws.data_ptr(), ws.numel(),
                                       torch.cuda.current_stream().cuda_stream))
    return grads, gg, gb, gx


def _save_loop(ctx, params, saved):
    ctx.layout = None
    if isinstance(saved, _Pool):
        ctx.layout = saved.layout
        ctx.save_for_backward(*params, saved.memory)
        return
    x_il4, stats, outs, stashes = saved
    ctx.kept = [t is not None for t in stashes]
    ctx.save_for_backward(*params, x_il4, stats, *outs, *[t for t in stashes if t is not None])


def _restore_loop(ctx, nparams: int, outer: int):
    t = ctx.saved_tensors
    params, rest = t[:nparams], t[nparams:]
    if ctx.layout:
        return params, _Pool(rest[0], ctx.layout).pieces()
    outs, kept = rest[2:2 + outer], iter(rest[2 + outer:])
    return params, (rest[0], rest[1], outs, [next(kept) if k else None for k in ctx.kept])


class FusedLoopTrainOp(_Op):
    """The model loop of the reference's scripts with gradients:

        h = x
        for _ in range(outer_iters):
            h = layer_norm(gridnet_step(weight, bias, residual_scale, h, ..., normalize=False), norm_weight, norm_bias)

    (gridnet/scripts/train_mnist.py:62-64) as ONE autograd node, float32, shared parameters, on the quad kernels
    (``gn_loop_forward_f32`` / ``gn_loop_backward_f32``) or, for one or two samples of a large grid, on the register-patch
    kernels (:func:`on_patches`): every step kernel reduces the statistics of what it writes and
    normalises its input while loading it, so between steps only the RAW step outputs (and their statistics) exist and are
    saved - half the activations that the step-by-step composition saves. The last steps also keep their inner iterations
    for the backward pass, as many as the memory allows (:func:`keep_forward_stash`).

    ``FusedLoopTrainOp.apply(weight, bias, residual_scale, norm_weight, norm_bias, x, inner_iters, outer_iters,
    block_size, activation, ln_eps)``."""

    @staticmethod
    def supported(weight, x, inner_iters: int, block_size: int) -> bool:
        if weight.dtype != torch.float32 or not weight.is_cuda or inner_iters < 1 or x.shape[0] == 0:
            return False
        return bool(lib.gn_loop_train_supported(*x.shape, int(inner_iters), int(block_size)))

    @staticmethod
    def forward(ctx, weight, bias, residual_scale, norm_weight, norm_bias, x, inner_iters: int, outer_iters: int,
                block_size: int, activation: str, ln_eps: float):
        ctx.cfg = (int(inner_iters), int(outer_iters), int(block_size), activation)
        if not ctx.cfg[1]:
            ctx.save_for_backward(weight, bias, residual_scale, norm_weight, norm_bias)
            return x.clone()
        y, saved = _loop_forward([(weight, bias, residual_scale)], norm_weight, norm_bias, x.contiguous(), *ctx.cfg,
                                 float(ln_eps), False, any(ctx.needs_input_grad[:6]))
        _save_loop(ctx, (weight, bias, residual_scale, norm_weight, norm_bias), saved)
        return y

    @staticmethod
    def backward(ctx, grad_y):
        outer = ctx.cfg[1]
        if not outer:
            return (*(torch.zeros_like(t) for t in ctx.saved_tensors), grad_y, None, None, None, None, None)
        params, saved = _restore_loop(ctx, 5, outer)
        grads, gg, gb, gx = _loop_backward([params[:3]], *params[3:], saved, grad_y, *ctx.cfg, False)
        return (*grads[0], gg, gb, gx, None, None, None, None, None)


class FusedGatedLoopTrainOp(_Op):
    """:class:`FusedLoopTrainOp` for the gated step (gridnet/scripts/train_mnist.py:36-44, 62-64), block 8:

        for _ in range(outer_iters):
            h = layer_norm(gated_gridnet_step(weight, bias, h, ...), norm_weight, norm_bias)

    ``FusedGatedLoopTrainOp.apply(weight, bias, norm_weight, norm_bias, x, inner_iters, outer_iters, block_size, activation,
    ln_eps)``."""

    @staticmethod
    def supported(weight, x, inner_iters: int, block_size: int) -> bool:
        return block_size == 8 and not (x.shape[0] == 1 and on_patches(*x.shape)) and FusedLoopTrainOp.supported(weight, x, inner_iters,
                                                                                                                  block_size)

    @staticmethod
    def forward(ctx, weight, bias, norm_weight, norm_bias, x, inner_iters: int, outer_iters: int, block_size: int,
                activation: str, ln_eps: float):
        ctx.cfg = (int(inner_iters), int(outer_iters), int(block_size), activation)
        if not ctx.cfg[1]:
            ctx.save_for_backward(weight, bias, norm_weight, norm_bias)
            return x.clone()
        y, saved = _loop_forward([(weight, bias)], norm_weight, norm_bias, x.contiguous(), *ctx.cfg, float(ln_eps), False,
                                 any(ctx.needs_input_grad[:5]), gated=True)
        _save_loop(ctx, (weight, bias, norm_weight, norm_bias), saved)
        return y

    @staticmethod
    def backward(ctx, grad_y):
        outer = ctx.cfg[1]
        if not outer:
            return (*(torch.zeros_like(t) for t in ctx.saved_tensors), grad_y, None, None, None, None, None)
        params, saved = _restore_loop(ctx, 4, outer)
        grads, gg, gb, gx = _loop_backward([params[:2]], *params[2:], saved, grad_y, *ctx.cfg, False, gated=True)
        return (*grads[0], gg, gb, gx, None, None, None, None, None)


class FusedLoopSeparateTrainOp(_Op):
    """:class:`FusedLoopTrainOp` for a loop in which every outer step has its own network
    (``separate_params`` of gridnet/scripts/train_imagenet.py:54-58,76-79): the same fused forward and the same
    reverse walk, each step's parameter gradients going to that step's parameters.

    ``FusedLoopSeparateTrainOp.apply(norm_weight, norm_bias, x, inner_iters, block_size, activation, ln_eps,
    weight_0, bias_0, residual_scale_0, weight_1, ...)``: three tensors per outer step."""

    @staticmethod
    def forward(ctx, norm_weight, norm_bias, x, inner_iters: int, block_size: int, activation: str, ln_eps: float,
                *step_params):
        assert len(step_params) % 3 == 0, "three tensors (weight, bias, residual_scale) per outer step"
        plist = [tuple(step_params[i:i + 3]) for i in range(0, len(step_params), 3)]
        ctx.cfg = (int(inner_iters), len(plist), int(block_size), activation)
        if not plist:
            ctx.save_for_backward(norm_weight, norm_bias)
            return x.clone()
        y, saved = _loop_forward(plist, norm_weight, norm_bias, x.contiguous(), *ctx.cfg, float(ln_eps), False,
                                 any(ctx.needs_input_grad))
        _save_loop(ctx, (norm_weight, norm_bias, *step_params), saved)
        return y

    @staticmethod
    def backward(ctx, grad_y):
        outer = ctx.cfg[1]
        if not outer:
            return (*(torch.zeros_like(t) for t in ctx.saved_tensors), grad_y, None, None, None, None)
        params, saved = _restore_loop(ctx, 2 + 3 * outer, outer)
        plist = [params[i:i + 3] for i in range(2, 2 + 3 * outer, 3)]
        grads, gg, gb, gx = _loop_backward(plist, *params[:2], saved, grad_y, *ctx.cfg, False)
        return (gg, gb, gx, None, None, None, None) + tuple(t for triple in grads for t in triple)


class FusedLoopResidualTrainOp(_Op):
    """The residual form of the model loop with gradients (gridnet/scripts/train_imagenet.py:81-83):

        for net in nets:  n = layer_norm(h);  h = h + (net(n) - n)

    as one autograd node. Forward: the step kernel normalises h while loading it, one pass writes
    ``h + (y - layer_norm(h))`` and reduces the statistics of the result; saved are the step inputs h_k and their
    statistics (and the inner iterations of the last steps, memory permitting). Backward, per step in reverse: the step
    backward on the rebuilt ``n``, then one pass for the sums of the LayerNorm gradient of ``grad_step - grad`` and one
    that adds it to ``grad``.

    ``FusedLoopResidualTrainOp.apply(norm_weight, norm_bias, x, inner_iters, block_size, activation, ln_eps,
    outer_iters, *params)`` with ``params`` either one (weight, bias, residual_scale) shared by all outer steps or
    ``outer_iters`` of them, one after the other."""

    @staticmethod
    def forward(ctx, norm_weight, norm_bias, x, inner_iters: int, block_size: int, activation: str, ln_eps: float,
                outer_iters: int, *params):
        outer = int(outer_iters)
        assert len(params) in (3, 3 * outer), "one (weight, bias, residual_scale), or one per outer step"
        ctx.cfg = (int(inner_iters), outer, int(block_size), activation)
        if not outer:
            ctx.save_for_backward(norm_weight, norm_bias, *params)
            return x.clone()
        plist = [tuple(params[i:i + 3]) for i in range(0, len(params), 3)]
        y, saved = _loop_forward(plist, norm_weight, norm_bias, x.contiguous(), *ctx.cfg, float(ln_eps), True,
                                 any(ctx.needs_input_grad))
        ctx.nparams = 2 + len(params)
        _save_loop(ctx, (norm_weight, norm_bias, *params), saved)
        return y

    @staticmethod
    def backward(ctx, grad_out):
        outer = ctx.cfg[1]
        if not outer:
            z = [torch.zeros_like(t) for t in ctx.saved_tensors]
            return (z[0], z[1], grad_out, None, None, None, None, None, *z[2:])
        params, saved = _restore_loop(ctx, ctx.nparams, outer)
        plist = [params[i:i + 3] for i in range(2, ctx.nparams, 3)]
        grads, gg, gb, gx = _loop_backward(plist, *params[:2], saved, grad_out, *ctx.cfg, True)
        return (gg, gb, gx, None, None, None, None, None) + tuple(t for triple in grads for t in triple)


def fused_loop_forward(step_params, norm_weight, norm_bias, x, inner_iters: int, block_size: int,
                       activation: str = "silu", ln_eps: float = 1e-5, outer_residual: bool = False) -> torch.Tensor:
    """The model loop of gridnet/scripts/train_imagenet.py:76-86 without gradients, for the variants that
    :func:`outer_forward` does not take: ``step_params`` is one ``(weight, bias, residual_scale)`` per outer step
    (``separate_params``; repeat one tuple for shared parameters), and with ``outer_residual`` a step is
    ``n = norm(h); h = h + (net(n) - n)`` instead of ``h = norm(net(h))``. Float32, whole 8^3 regions, block 4 or 8. The
    normalised tensor is never stored: the step kernel normalises while it loads, and either it (plain form) or the
    combining pass (residual form) reduces the next statistics."""
    plist = [tuple(p) for p in step_params]
    outer = len(plist)
    if not outer or not x.shape[0]:
        return x.clone()
    if all(t is u for p in plist[1:] for t, u in zip(p, plist[0])):
        plist = plist[:1]  # shared parameters: re-ordered once
    with torch.no_grad():
        return _loop_forward(plist, norm_weight, norm_bias, x.contiguous(), int(inner_iters), outer, int(block_size),
                             activation, float(ln_eps), bool(outer_residual), False)[0]


def device_status(clear: bool = True, device=None) -> bool:
    """True if, since the last clear, a kernel on ``device`` gave up a bounded wait on a bulk tile copy and had
    no workspace flag to report it in, or a persistent kernel of :func:`outer_forward` one on its other blocks (the results of that
    call are invalid). Synchronises the device."""
    dev = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    with torch.cuda.device(dev):
        torch.cuda.synchronize(dev)
        rc = int(lib.gn_device_status(1 if clear else 0))
    if rc < 0:
        check(rc)
    return rc == 1


def outer_forward_failed(workspace: torch.Tensor, batch: int, shape, block_size: int) -> bool:
    """True if the last :func:`outer_forward` that used ``workspace`` recorded a device-side failure
    (a bounded wait that gave up). Synchronises the device."""
    m, n, k = shape
    off = int(lib.gn_outer_forward_error_flag_offset(batch, m, n, k, block_size))
    torch.cuda.synchronize(workspace.device)
    return bool(workspace[off:off + 4].view(torch.int32).item())


def outer_forward_workspace(batch: int, shape, block_size: int, device) -> torch.Tensor:
    """Scratch buffer for :func:`outer_forward`; reusable across calls of the same size."""
    m, n, k = shape
    return _workspace(lib.gn_outer_forward_workspace_bytes(batch, m, n, k, block_size), device)


@functools.lru_cache(maxsize=512)
def _outer_workspace_bytes(device: int, batch: int, m: int, n: int, k: int, block_size: int) -> int:
    with torch.cuda.device(device):
        return max(256, int(lib.gn_outer_forward_workspace_bytes(batch, m, n, k, block_size)))


@torch.no_grad()
def outer_forward(weight, bias, residual_scale, norm_weight, norm_bias, init_activations, inner_iters: int,
                  outer_iters: int, block_size: int, activation: str = "silu", ln_eps: float = 1e-5,
                  out: torch.Tensor | None = None, workspace: torch.Tensor | None = None) -> torch.Tensor:
    """Inference loop of the reference's models, fused:

        h = init_activations
        for _ in range(outer_iters):
            h = gridnet_step(weight, bias, residual_scale, h, inner_iters, block_size, normalize=False, ...)
            h = layer_norm(h, (M, N, K), norm_weight, norm_bias, ln_eps)

    (gridnet/scripts/train_mnist.py:62-64). float32, no autograd.
    """
    batch_size = _assert_step_args(weight, bias, residual_scale, init_activations, block_size, False)
    assert norm_weight.shape == bias.shape == norm_bias.shape, f"{norm_weight.shape=} invalid for {bias.shape=}"
    if not batch_size:
        return init_activations.clone()
    _require_f32_cuda(weight=weight, bias=bias, residual_scale=residual_scale, norm_weight=norm_weight,
                      norm_bias=norm_bias, init_activations=init_activations)
    B, M, N, K = init_activations.shape
    y = torch.empty_like(init_activations) if out is None else out
    flags, key = 0, None
    if workspace is None:
        ws = torch.empty(_outer_workspace_bytes(weight.device.index, B, M, N, K, block_size), dtype=torch.uint8, device=weight.device)
    else:
        # A caller-owned workspace keeps the parameters re-ordered for the quad or the large-batch kernel between calls. They
        # are rebuilt unless this very workspace tensor was used by the previous call with the same parameter tensors, by the
        # same of these two kernels, and neither they nor the workspace have been written to through torch since (torch
        # counts in-place writes).
        ws = workspace
        with torch.cuda.device(weight.device):
            plan = int(lib.gn_outer_forward_plan(B, M, N, K, int(inner_iters), int(outer_iters), int(block_size)))
        if plan in (2, 5):
            params = (weight, bias, residual_scale, norm_weight, norm_bias)
            key = (plan, tuple((t.data_ptr(), t._version) for t in params), (B, M, N, K, int(block_size)))
            if getattr(ws, "_gn_packed_for", None) == (key, ws._version):
                flags = 1  # GN_OUTER_PARAMS_UNCHANGED
    with torch.cuda.device(weight.device):
        check(lib.gn_outer_forward_flags_f32(weight.data_ptr(), bias.data_ptr(), residual_scale.data_ptr(),
                                             norm_weight.data_ptr(), norm_bias.data_ptr(),
                                             init_activations.data_ptr(), y.data_ptr(), B, M, N, K, int(inner_iters),
                                             int(outer_iters), int(block_size), float(ln_eps),
                                             activation_id(activation), ws.data_ptr(), ws.numel(), flags,
                                             gridnet_cuda._stream(weight)))
    if workspace is not None:
        ws._gn_packed_for = None if key is None else (key, ws._version)
    return y


def step_stats_partials(shape, block_size: int) -> int:
    """Number of (sum, sum of squares) pairs per sample that :func:`fused_step` writes."""
    m, n, k = shape
    return int(lib.gn_step_stats_partials(m, n, k, block_size))


@torch.no_grad()
def fused_step(weight, bias, residual_scale, x, out, inner_iters: int, block_size: int, activation: str = "silu",
               norm_weight=None, norm_bias=None, in_mean_rstd=None, out_partials=None) -> torch.Tensor:
    """One step of the fused loop (``gn_step_forward_fused_f32``): ``x`` may be the raw
    output of the previous step, normalised on load with ``in_mean_rstd`` [B, 2] and
    ``norm_weight`` / ``norm_bias``; ``out_partials`` [B, nparts, 2] float64 receives the
    statistics partials of ``out``. Block size 8, float32."""
    _require_f32_cuda(weight=weight, bias=bias, residual_scale=residual_scale, x=x, out=out)
    B, M, N, K = x.shape
    ptr = lambda t: None if t is None else t.data_ptr()
    with torch.cuda.device(weight.device):
        check(lib.gn_step_forward_fused_f32(weight.data_ptr(), bias.data_ptr(), residual_scale.data_ptr(),
                                            x.data_ptr(), out.data_ptr(), ptr(norm_weight), ptr(norm_bias),
                                            ptr(in_mean_rstd), ptr(out_partials), B, M, N, K, int(inner_iters),
                                            int(block_size), activation_id(activation),
                                            torch.cuda.current_stream().cuda_stream))
    return out


@torch.no_grad()
def norm_finalize(partials, mean_rstd, P: int, eps: float = 1e-5) -> torch.Tensor:
    """[B, nparts, 2] float64 partial sums -> [B, 2] float32 (mean, 1/sqrt(var + eps))."""
    B, nparts = partials.shape[0], partials.shape[1]
    with torch.cuda.device(partials.device):
        check(lib.gn_norm_finalize_f32(partials.data_ptr(), nparts, mean_rstd.data_ptr(), B, int(P), float(eps),
                                       torch.cuda.current_stream().cuda_stream))
    return mean_rstd


@torch.no_grad()
def norm_apply(x, norm_weight, norm_bias, mean_rstd, out) -> torch.Tensor:
    """out = (x - mean) * rstd * norm_weight + norm_bias per sample."""
    _require_f32_cuda(x=x, norm_weight=norm_weight, norm_bias=norm_bias, out=out)
    B, P = x.shape[0], x[0].numel()
    with torch.cuda.device(x.device):
        check(lib.gn_norm_apply_f32(x.data_ptr(), norm_weight.data_ptr(), norm_bias.data_ptr(),
                                    mean_rstd.data_ptr(), out.data_ptr(), B, P,
                                    torch.cuda.current_stream().cuda_stream))
    return out


# ---- building blocks of the large-batch step kernel (gn_pair64_* in include/gridnet_b200.h) ----------------
def _il64_groups(batch: int) -> int:
    return (int(batch) + 63) // 64


@torch.no_grad()
def pair64_pack_weights(weight, bias, residual_scale, norm_weight=None, norm_bias=None) -> torch.Tensor:
    """weight [27,M,N,K], bias, residual_scale [M,N,K] (float32, M, N, K multiples of 8) and, if steps are to
    normalise their input on load, the whole-grid norm's weight and bias [M,N,K] -> the parameters in the order
    the large-batch step kernel reads them (one flat float32 tensor)."""
    _require_f32_cuda(weight=weight, bias=bias, residual_scale=residual_scale)
    ptr = lambda t: None if t is None else t.data_ptr()
    M, N, K = bias.shape
    nbytes = int(lib.gn_pair64_packed_weight_bytes(M, N, K))
    if nbytes == 0:
        raise RuntimeError(f"grid {tuple(bias.shape)} is not a multiple of 8 in every dimension")
    packed = torch.empty(nbytes // 4, dtype=torch.float32, device=weight.device)
    with torch.cuda.device(weight.device):
        check(lib.gn_pair64_pack_weights_f32(weight.data_ptr(), bias.data_ptr(), residual_scale.data_ptr(),
                                             ptr(norm_weight), ptr(norm_bias), packed.data_ptr(), M, N, K,
                                             torch.cuda.current_stream().cuda_stream))
    return packed


@torch.no_grad()
def pair64_interleave(x, out: torch.Tensor | None = None) -> torch.Tensor:
    """x [B,M,N,K] -> the same activations interleaved by groups of 64 samples, [ceil(B/64), M, N, K, 64]
    (samples beyond B are zero)."""
    _require_f32_cuda(x=x)
    B, M, N, K = x.shape
    if out is None:
        out = torch.empty(_il64_groups(B), M, N, K, 64, dtype=torch.float32, device=x.device)
    with torch.cuda.device(x.device):
        check(lib.gn_pair64_interleave_f32(x.data_ptr(), out.data_ptr(), B, M, N, K,
                                           torch.cuda.current_stream().cuda_stream))
    return out


@torch.no_grad()
def pair64_deinterleave(x_il64, batch: int, shape, mean_rstd=None, norm_weight=None, norm_bias=None,
                        out: torch.Tensor | None = None) -> torch.Tensor:
    """Inverse of :func:`pair64_interleave`; with ``mean_rstd`` the whole-grid normalisation is applied on the
    way: ``(v - mean) * rstd * norm_weight + norm_bias``."""
    _require_f32_cuda(x_il64=x_il64)
    M, N, K = shape
    if out is None:
        out = torch.empty(batch, M, N, K, dtype=torch.float32, device=x_il64.device)
    ptr = lambda t: None if t is None else t.data_ptr()
    with torch.cuda.device(x_il64.device):
        check(lib.gn_pair64_deinterleave_f32(x_il64.data_ptr(), ptr(mean_rstd), ptr(norm_weight), ptr(norm_bias),
                                             out.data_ptr(), int(batch), M, N, K,
                                             torch.cuda.current_stream().cuda_stream))
    return out


@torch.no_grad()
def pair64_step(packed, x_il64, y_il64, batch: int, shape, inner_iters: int, activation: str = "silu",
                in_mean_rstd=None, out_partials=None, error_flag=None) -> torch.Tensor:
    """One step of the large-batch kernel on interleaved activations (``gn_step_forward_pair64_f32``); the
    optional arguments have the meaning they have in :func:`fused_step`, with ``64 * ceil(B/64)`` rows (the
    norm's weight and bias that ``in_mean_rstd`` goes with are the ones given to :func:`pair64_pack_weights`)."""
    M, N, K = shape
    ptr = lambda t: None if t is None else t.data_ptr()
    nparts = 0 if out_partials is None else int(out_partials.shape[1])
    with torch.cuda.device(x_il64.device):
        check(lib.gn_step_forward_pair64_f32(packed.data_ptr(), x_il64.data_ptr(), y_il64.data_ptr(),
                                             ptr(in_mean_rstd), ptr(out_partials), nparts, int(batch),
                                             M, N, K, int(inner_iters), activation_id(activation), ptr(error_flag),
                                             torch.cuda.current_stream().cuda_stream))
    return y_il64


class HostPipelinedForward:
    """The fused inference loop for batches that live in (pinned) HOST memory.

    ``submit(host_x, host_y)`` queues host->device copy, :func:`outer_forward` and device->host
    copy of one batch on three streams with ``depth`` device buffer sets, so the copies of one
    batch overlap the compute of its neighbours; ``synchronize()`` waits for everything queued.
    A buffer set is busy for copy-in + compute + copy-out, so three sets (the default) are what
    keeps all three stages running at once; with two, a step takes half of that sum.
    ``host_x`` / ``host_y`` are ``[B, M, N, K]`` float32 CPU tensors (pinned for real overlap).
    """

    def __init__(self, weight, bias, residual_scale, norm_weight, norm_bias, batch: int, inner_iters: int,
                 outer_iters: int, block_size: int, activation: str = "silu", ln_eps: float = 1e-5, depth: int = 3):
        self.params = (weight, bias, residual_scale, norm_weight, norm_bias)
        self.cfg = (int(inner_iters), int(outer_iters), int(block_size), activation, float(ln_eps))
        dev = weight.device
        shape = tuple(bias.shape)
        self.device = dev
        self.depth = depth
        self.dx = [torch.empty(batch, *shape, device=dev) for _ in range(depth)]
        self.dy = [torch.empty(batch, *shape, device=dev) for _ in range(depth)]
        self.ws = outer_forward_workspace(batch, shape, block_size, dev)
        self.s_in, self.s_compute, self.s_out = (torch.cuda.Stream(dev) for _ in range(3))
        self.ev_in = [torch.cuda.Event() for _ in range(depth)]
        self.ev_compute = [torch.cuda.Event() for _ in range(depth)]
        self.ev_out = [torch.cuda.Event() for _ in range(depth)]
        self.count = 0
        torch.cuda.synchronize(dev)

    def submit(self, host_x: torch.Tensor, host_y: torch.Tensor) -> None:
        j = self.count % self.depth
        reuse = self.count >= self.depth
        self.count += 1
        inner, outer, block, act, eps = self.cfg
        if reuse:  # buffer set j is free once its previous result has left the device
            self.s_in.wait_event(self.ev_out[j])
            self.s_compute.wait_event(self.ev_out[j])
        with torch.cuda.stream(self.s_in):
            self.dx[j].copy_(host_x, non_blocking=True)
            self.ev_in[j].record(self.s_in)
        self.s_compute.wait_event(self.ev_in[j])
        with torch.cuda.stream(self.s_compute):
            outer_forward(*self.params, self.dx[j], inner, outer, block, act, eps, out=self.dy[j], workspace=self.ws)
            self.ev_compute[j].record(self.s_compute)
        self.s_out.wait_event(self.ev_compute[j])
        with torch.cuda.stream(self.s_out):
            host_y.copy_(self.dy[j], non_blocking=True)
            self.ev_out[j].record(self.s_out)

    def join(self, stream=None) -> None:
        """Make ``stream`` (default: the current stream) wait for everything queued so far."""
        stream = stream or torch.cuda.current_stream(self.device)
        for ev in self.ev_out[: min(self.count, self.depth)]:
            stream.wait_event(ev)

    def synchronize(self) -> None:
        for s in (self.s_in, self.s_compute, self.s_out):
            s.synchronize()
