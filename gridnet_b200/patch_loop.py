"""The model loop with gradients step by step on the register-patch kernels (``gn_step_forward_train_f32`` and the tuned step
backward), activations in the grid's own layout: for batches of one or two on large grids, where the quad kernels' four
samples per lane are mostly copies (``on_patches`` in backend_cuda.py). Same tensors in, kept and out as ``_loop_forward`` and
``_loop_backward`` there, the same bits forward.

    plain     h = layer_norm(step(h))                  gridnet/scripts/train_mnist.py:62-64
    residual  n = layer_norm(h);  h = h + step(n) - n  gridnet/scripts/train_imagenet.py:81-83
"""
from __future__ import annotations

import torch

from . import gridnet_cuda
from ._lib import GN_ERR_UNSUPPORTED, activation_id, check, lib


def _workspace(nbytes: int, device) -> torch.Tensor:
    return torch.empty(max(256, int(nbytes)), dtype=torch.uint8, device=device)


def stash_bytes(x, inner: int, block: int) -> int:
    """What a step keeps of its inner iterations; 0: such a step always runs them again."""
    return int(lib.gn_step_stash_bytes(*x.shape, inner, block))


def forward(plist, norm_weight, norm_bias, x, inner: int, outer: int, block: int, activation: str, ln_eps: float, residual: bool,
            outs, stats, stashes):
    """Runs the loop; ``outs``: a tensor like x per step for its raw output (residual: the next h), ``stats`` [outer, B, 2] for
    the (mean, rstd) of outs[k] (residual: of the input of step k), ``stashes``: per step ``stash_bytes`` bytes or None."""
    B, M, N, K = x.shape
    P, act, st = M * N * K, activation_id(activation), torch.cuda.current_stream().cuda_stream
    y = torch.empty_like(x)
    nws = _workspace(lib.gn_norm_workspace_bytes(B, P), x.device)
    nparts = int(lib.gn_step_stats_partials(M, N, K, block))
    partials = torch.empty(B, nparts, 2, dtype=torch.float64, device=x.device)
    if residual:
        check(lib.gn_norm_local_sums_f32(x.data_ptr(), partials.data_ptr(), B, P, nws.data_ptr(), nws.numel(), st))
        check(lib.gn_norm_finalize_f32(partials.data_ptr(), 1, stats[0].data_ptr(), B, P, ln_eps, st))
    last = torch.empty(B, 2, dtype=torch.float32, device=x.device)  # residual: statistics that nobody needs
    h = x
    for k in range(outer):
        weight, bias, scale = plist[k % len(plist)]
        mr = stats[k] if residual else (stats[k - 1] if k else None)
        stash = stashes[k]
        check(lib.gn_step_forward_train_f32(weight.data_ptr(), bias.data_ptr(), scale.data_ptr(), h.data_ptr(),
                                            (y if residual else outs[k]).data_ptr(), norm_weight.data_ptr(), norm_bias.data_ptr(),
                                            None if mr is None else mr.data_ptr(), None if residual else partials.data_ptr(), B, M, N, K, inner,
                                            block, act, None if stash is None else stash.data_ptr(), 0 if stash is None else stash.numel(), st))
        if residual:
            following = stats[k + 1] if k + 1 < outer else last
            check(lib.gn_norm_residual_combine_f32(h.data_ptr(), y.data_ptr(), norm_weight.data_ptr(), norm_bias.data_ptr(), mr.data_ptr(),
                                                   outs[k].data_ptr(), following.data_ptr(), B, P, ln_eps, nws.data_ptr(), nws.numel(), st))
        else:
            check(lib.gn_norm_finalize_f32(partials.data_ptr(), nparts, stats[k].data_ptr(), B, P, ln_eps, st))
        h = outs[k]
    if residual:
        return y.copy_(h)
    check(lib.gn_norm_apply_f32(h.data_ptr(), norm_weight.data_ptr(), norm_bias.data_ptr(), stats[outer - 1].data_ptr(), y.data_ptr(), B, P, st))
    return y


def _step_backward(params, grads, h, mr, norm_weight, norm_bias, gy, gx, inner: int, block: int, activation: str, stash) -> None:
    """The step's gradients for the input layer_norm(h) with the statistics ``mr`` (None: h itself), which the backward kernels
    rebuild while they load h where they can (block 8), a pass here otherwise."""
    B, M, N, K = h.shape
    st = torch.cuda.current_stream().cuda_stream
    if mr is not None and block == 8:
        if stash is not None:
            need = int(lib.gn_step_backward_stash_workspace_bytes(B, M, N, K, inner, block))
        else:
            need = int(lib.gn_step_backward_workspace_bytes(B, M, N, K, inner, block, 0, 4))
        if need > 0:
            ws = _workspace(need, h.device)
            rc = lib.gn_step_backward_fused_in_f32(*(t.data_ptr() for t in (*params, h, mr, norm_weight, norm_bias, gy, *grads, gx)), B, M, N, K,
                                                   inner, block, activation_id(activation), None if stash is None else stash.data_ptr(),
                                                   0 if stash is None else stash.numel(), ws.data_ptr(), ws.numel(), st)
            if rc != GN_ERR_UNSUPPORTED:
                check(rc)
                return
    if mr is not None:
        n = torch.empty_like(h)
        check(lib.gn_norm_apply_f32(h.data_ptr(), norm_weight.data_ptr(), norm_bias.data_ptr(), mr.data_ptr(), n.data_ptr(), B, M * N * K, st))
        h = n
    if stash is not None:
        gridnet_cuda.backward_with_stash(*params, h, gy, *grads, gx, inner, block, activation, stash)
    else:
        gridnet_cuda.backward(*params, h, gy, *grads, gx, inner, block, 1e-5, False, activation)


def backward(plist, norm_weight, norm_bias, x, outs, stats, stashes, grad_y, inner: int, outer: int, block: int, activation: str, residual: bool):
    """One (weight, bias, scale) gradient per entry of ``plist``, those of the norm's weight and bias, and that of x."""
    B, M, N, K = x.shape
    P, st = M * N * K, torch.cuda.current_stream().cuda_stream
    nws = _workspace(lib.gn_norm_workspace_bytes(B, P), x.device)
    sums = torch.empty(B, 2, dtype=torch.float64, device=x.device)
    grads, gg, gb = [None] * len(plist), None, None

    def norm_backward(h, mr, g):
        gh, dg, db = torch.empty_like(h), torch.empty_like(norm_weight), torch.empty_like(norm_weight)
        check(lib.gn_norm_backward_local_sums_f32(h.data_ptr(), norm_weight.data_ptr(), g.data_ptr(), mr.data_ptr(), sums.data_ptr(), B, P,
                                                  nws.data_ptr(), nws.numel(), st))
        check(lib.gn_norm_backward_apply_f32(h.data_ptr(), norm_weight.data_ptr(), g.data_ptr(), mr.data_ptr(), sums.data_ptr(), P, gh.data_ptr(),
                                             dg.data_ptr(), db.data_ptr(), B, P, nws.data_ptr(), nws.numel(), st))
        return gh, (dg if gg is None else gg.add_(dg)), (db if gb is None else gb.add_(db))

    g = grad_y
    for k in reversed(range(outer)):
        kp = k % len(plist)
        h = outs[k - 1] if k else x
        mr = stats[k] if residual else (stats[k - 1] if k else None)
        if not residual:
            g, gg, gb = norm_backward(outs[k], stats[k], g)
        here, gx = [torch.empty_like(t) for t in plist[kp]], torch.empty_like(x)
        _step_backward(plist[kp], here, h, mr, norm_weight, norm_bias, g, gx, inner, block, activation, stashes[k])
        if residual:
            gx -= g  # h' = h + net(n) - n: n also enters with a minus sign
            gh, gg, gb = norm_backward(h, mr, gx)
            g = g + gh
        else:
            g = gx
        if grads[kp] is None:
            grads[kp] = here
        else:  # steps that share parameters
            for total, part in zip(grads[kp], here):
                total += part
    return [tuple(t) for t in grads], gg, gb, g
