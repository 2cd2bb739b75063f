"""Module wrappers and the host-buffer pipeline on the GPU: the fused model loop equals the
step-by-step composition with autograd, reference-style state dicts load, training gradients
flow through both ops, and HostPipelinedForward returns what outer_forward returns."""
import numpy as np
import pytest
import torch

from oracle import gridnet_oracle as orc

from util import assert_close

pytestmark = pytest.mark.gpu


def test_model_fused_inference_equals_training_path_and_oracle():
    import gridnet_b200 as gb

    torch.manual_seed(0)
    shape = (16, 16, 16)
    dev = torch.device("cuda")
    model = gb.GridnetModel(shape, inner_iters=2, outer_iters=3, block_size=8, device=dev)
    with torch.no_grad():
        model.network.bias.normal_(0, 0.1)
        model.norm.weight.normal_(1, 0.1)
        model.norm.bias.normal_(0, 0.1)
    assert set(model.state_dict()) == {"network.weight", "network.bias", "network.residual_scale", "norm.weight", "norm.bias"}
    x = torch.zeros(3, *shape, device=dev)
    x[..., 0] = torch.randn(3, 16, 16, device=dev)
    with torch.no_grad():
        fused = model(x)
    stepwise = model(x)  # grad enabled: GridnetCudaOp + GridNormOp per outer step
    assert stepwise.requires_grad
    assert torch.allclose(fused, stepwise, rtol=1e-4, atol=1e-5)
    sd = {k: v.detach().cpu().numpy().astype(np.float64) for k, v in model.state_dict().items()}
    want = orc.outer_forward(sd["network.weight"], sd["network.bias"], sd["network.residual_scale"], sd["norm.weight"],
                             sd["norm.bias"], x.cpu().numpy().astype(np.float64), 2, 3, 8)
    err = np.abs(fused.cpu().numpy() - want)
    assert (err <= 1e-5 + 1e-4 * np.abs(want)).all()
    # a training step: the gradients of all five parameters and of the input against the oracle's chain
    # step_backward o layernorm_backward over the three outer steps (float64 oracle, float32 oracle for the noise)
    from util import assert_close

    gy = torch.linspace(-1, 1, stepwise.numel(), device=dev).view_as(stepwise).contiguous()
    xg = x.clone().requires_grad_(True)
    out = model(xg)
    names = ["network.weight", "network.bias", "network.residual_scale", "norm.weight", "norm.bias"]
    params = dict(model.named_parameters())
    grads = torch.autograd.grad(out, [params[n] for n in names] + [xg], gy)
    args64 = [sd[n] for n in names] + [x.cpu().numpy().astype(np.float64), gy.cpu().numpy().astype(np.float64)]
    want64 = orc.outer_backward(*args64, 2, 3, 8)
    want32 = orc.outer_backward(*(a.astype(np.float32) for a in args64), 2, 3, 8)
    for name, g, r64, r32 in zip(names + ["input"], grads, want64, want32):
        assert_close(g.cpu().numpy(), r64, r32, f"model gradient of {name}")
    # the fused training node against the step-by-step composition of the two autograd ops (same library kernels
    # underneath, different order of a few float32 operations), with the forward stash on and off
    for keep in (False, True):
        previous = gb.keep_forward_stash(keep)
        try:
            xs = x.clone().requires_grad_(True)
            h = xs
            for _ in range(3):
                h = model.norm(model.network(h))
            want = torch.autograd.grad(h, [params[n] for n in names] + [xs], gy)
            xf = x.clone().requires_grad_(True)
            outf = model(xf)
            got = torch.autograd.grad(outf, [params[n] for n in names] + [xf], gy)
        finally:
            gb.keep_forward_stash(previous)
        assert torch.allclose(outf, h, rtol=1e-5, atol=1e-6)
        for name, a, c in zip(names + ["input"], got, want):
            assert torch.allclose(a, c, rtol=1e-3, atol=1e-4 * (1 + c.abs().max().item())), (name, keep, (a - c).abs().max().item())


@pytest.mark.parametrize("block,shape,B", [(8, (16, 8, 24), 5), (4, (8, 16, 8), 3)])
def test_fused_training_loop_op(block, shape, B):
    """FusedLoopTrainOp directly: both block sizes, odd batch, a non-cubic grid, zero outer iterations, and
    gradients against the float64 oracle chain."""
    import gridnet_b200 as gb
    from util import assert_close

    r = np.random.default_rng(61)
    f = np.float32
    w = (r.standard_normal((27, *shape)) / np.sqrt(27)).astype(f)
    b = (0.1 * r.standard_normal(shape)).astype(f)
    s = (1 + 0.1 * r.standard_normal(shape)).astype(f)
    ga = (1 + 0.1 * r.standard_normal(shape)).astype(f)
    be = (0.1 * r.standard_normal(shape)).astype(f)
    x = r.standard_normal((B, *shape)).astype(f)
    gy = r.standard_normal((B, *shape)).astype(f)
    inner, outer = 2, 3
    leaves = [torch.from_numpy(a).cuda().requires_grad_(True) for a in (w, b, s, ga, be, x)]
    assert gb.FusedLoopTrainOp.supported(leaves[0], leaves[5], inner, block)
    y = gb.FusedLoopTrainOp.apply(*leaves, inner, outer, block, "silu", 1e-5)
    grads = torch.autograd.grad(y, leaves, torch.from_numpy(gy).cuda())
    a64 = [a.astype(np.float64) for a in (w, b, s, ga, be, x)]
    assert_close(y.detach().cpu().numpy(), orc.outer_forward(*a64, inner, outer, block), None, "fused training forward")
    want64 = orc.outer_backward(*a64, gy.astype(np.float64), inner, outer, block)
    want32 = orc.outer_backward(w, b, s, ga, be, x, gy, inner, outer, block)
    for name, g, r64, r32 in zip(("weight", "bias", "scale", "gamma", "beta", "input"), grads, want64, want32):
        assert_close(g.cpu().numpy(), r64, r32, f"fused training gradient of {name} (block {block})")
    y0 = gb.FusedLoopTrainOp.apply(*leaves, inner, 0, block, "silu", 1e-5)
    assert torch.equal(y0, leaves[5])


def test_gated_model_and_readout_run():
    import gridnet_b200 as gb

    dev = torch.device("cuda")
    shape = (8, 8, 8)
    model = gb.GridnetModel(shape, 2, 2, 4, dev, activation="tanh", gated=True)
    ro = gb.Readout(shape, 10, dev)
    x = torch.randn(2, *shape, device=dev)
    out = ro(model(x))
    assert out.shape == (2, 10)
    out.sum().backward()
    assert model.network.weight.grad.abs().sum() > 0
    with pytest.raises(RuntimeError):
        gb.gridnet_step(torch.zeros(27, *shape), torch.zeros(shape), torch.zeros(shape), torch.zeros(1, *shape), 1, 8)


def test_host_pipelined_forward_matches_outer_forward():
    import gridnet_b200 as gb

    g = torch.Generator().manual_seed(3)
    shape, B = (16, 16, 16), 4
    w = (torch.randn(27, *shape, generator=g) / 27 ** 0.5).cuda()
    b = (0.1 * torch.randn(shape, generator=g)).cuda()
    s = torch.ones(shape).cuda()
    gamma = (1 + 0.1 * torch.randn(shape, generator=g)).cuda()
    beta = (0.1 * torch.randn(shape, generator=g)).cuda()
    hx = [torch.randn(B, *shape, generator=g).pin_memory() for _ in range(5)]
    hy = [torch.empty(B, *shape).pin_memory() for _ in range(5)]
    pipe = gb.HostPipelinedForward(w, b, s, gamma, beta, B, 2, 3, 8)
    for xi, yi in zip(hx, hy):  # more batches than buffer sets: buffers are reused
        pipe.submit(xi, yi)
    pipe.synchronize()
    for xi, yi in zip(hx, hy):
        want = gb.outer_forward(w, b, s, gamma, beta, xi.cuda(), 2, 3, 8).cpu()
        assert torch.equal(yi, want)


@pytest.mark.parametrize("block", [8, 4])
def test_fused_loop_variants_equal_the_step_by_step_composition(block):
    """Per-step parameters (with gradients, through FusedLoopSeparateTrainOp) and the residual form (without,
    through fused_loop_forward) against the composition of the step op and the norm op, which the other tests pin
    to the oracle (gridnet/scripts/train_imagenet.py:76-86)."""
    import gridnet_b200 as gb

    g = torch.Generator().manual_seed(17)
    shape, B, inner, outer = (16, 8, 16), 3, 2, 3
    dev = "cuda"
    mk = lambda *sz, scale=1.0, shift=0.0: (shift + scale * torch.randn(*sz, generator=g)).to(dev)
    plist = [(mk(27, *shape, scale=27 ** -0.5), mk(*shape, scale=0.1), mk(*shape, scale=0.1, shift=1.0))
             for _ in range(outer)]
    gamma, beta = mk(*shape, scale=0.1, shift=1.0), mk(*shape, scale=0.1)
    x, gy = mk(B, *shape), mk(B, *shape)

    def composition(leaves_p, ga, be, xin, residual):
        h = xin
        for w, b, s in leaves_p:
            if residual:
                n = gb.GridNormOp.apply(h, ga, be, 1e-5)
                h = h + (gb.GridnetCudaOp.apply(w, b, s, n, inner, block, 1e-5, False, "silu") - n)
            else:
                h = gb.GridNormOp.apply(gb.GridnetCudaOp.apply(w, b, s, h, inner, block, 1e-5, False, "silu"), ga, be, 1e-5)
        return h

    # inference, both forms
    with torch.no_grad():
        for residual in (False, True):
            want = composition(plist, gamma, beta, x, residual)
            got = gb.fused_loop_forward(plist, gamma, beta, x, inner, block, "silu", 1e-5, outer_residual=residual)
            assert torch.allclose(got, want, rtol=1e-4, atol=1e-5), (residual, (got - want).abs().max().item())
        assert torch.equal(gb.fused_loop_forward([], gamma, beta, x, inner, block, "silu", 1e-5, outer_residual=True), x)

    # training with per-step parameters
    def leaves():
        ps = [tuple(t.clone().requires_grad_(True) for t in p) for p in plist]
        return ps, gamma.clone().requires_grad_(True), beta.clone().requires_grad_(True), x.clone().requires_grad_(True)

    ps, ga, be, xl = leaves()
    flat = [t for p in ps for t in p]
    want_y = composition(ps, ga, be, xl, False)
    want = torch.autograd.grad(want_y, [ga, be, xl] + flat, gy)
    ps, ga, be, xl = leaves()
    flat = [t for p in ps for t in p]
    got_y = gb.FusedLoopSeparateTrainOp.apply(ga, be, xl, inner, block, "silu", 1e-5, *flat)
    got = torch.autograd.grad(got_y, [ga, be, xl] + flat, gy)
    assert torch.allclose(got_y, want_y, rtol=1e-4, atol=1e-5)
    for i, (a, c) in enumerate(zip(got, want)):
        assert torch.allclose(a, c, rtol=1e-3, atol=1e-4 * (1 + c.abs().max().item())), (i, (a - c).abs().max().item())

    # training in the residual form: per-step parameters, then one shared set, with the stash forced on and off
    for shared in (False, True):
        for keep in (True, False):
            previous = gb.keep_forward_stash(keep)
            try:
                ps, ga, be, xl = leaves()
                if shared:
                    ps = [ps[0]] * outer
                uniq = list(ps[0]) if shared else [t for p in ps for t in p]
                want_y = composition(ps, ga, be, xl, True)
                want = torch.autograd.grad(want_y, [ga, be, xl] + uniq, gy)
                ps, ga, be, xl = leaves()
                if shared:
                    ps = [ps[0]] * outer
                uniq = list(ps[0]) if shared else [t for p in ps for t in p]
                got_y = gb.FusedLoopResidualTrainOp.apply(ga, be, xl, inner, block, "silu", 1e-5, outer, *uniq)
                got = torch.autograd.grad(got_y, [ga, be, xl] + uniq, gy)
            finally:
                gb.keep_forward_stash(previous)
            assert torch.allclose(got_y, want_y, rtol=1e-4, atol=1e-5), (shared, keep)
            for i, (a, c) in enumerate(zip(got, want)):
                assert torch.allclose(a, c, rtol=1e-3, atol=1e-4 * (1 + c.abs().max().item())), \
                    (shared, keep, i, (a - c).abs().max().item())
    y0 = gb.FusedLoopResidualTrainOp.apply(gamma, beta, x, inner, block, "silu", 1e-5, 0, *plist[0])
    assert torch.equal(y0, x)


@pytest.mark.parametrize("name,grid,block,inner,outer,B", [("C3", 128, 8, 2, 16, 1), ("C4", 64, 4, 8, 16, 2)])
def test_training_configurations_at_their_own_grid_and_depth(name, grid, block, inner, outer, B):
    """The two forward + backward configurations of the benchmark at their own grid size, block size and
    iteration counts (128^3 / 8 / 2 x 16 and 64^3 / 4 / 8 x 16), one or two samples of the batch (samples only meet
    in the parameter gradients, which are sums over them): the fused training node's output and all six gradients
    against the float64 oracle's chain rule over the whole loop, the float32 oracle giving the noise floor."""
    import gridnet_b200 as gb
    from util import assert_close

    r = np.random.default_rng(73)
    f = np.float32
    shape = (grid, grid, grid)
    w = (r.standard_normal((27, *shape)) / np.sqrt(27)).astype(f)
    b = np.zeros(shape, f)
    s = np.ones(shape, f)
    ga = (1 + 0.05 * r.standard_normal(shape)).astype(f)
    be = (0.05 * r.standard_normal(shape)).astype(f)
    x = np.zeros((B, *shape), f)
    x[..., 0] = r.standard_normal((B, grid, grid))  # the input face, as in the benchmark
    gy = r.standard_normal((B, *shape)).astype(f)
    leaves = [torch.from_numpy(a).cuda().requires_grad_(True) for a in (w, b, s, ga, be, x)]
    assert gb.FusedLoopTrainOp.supported(leaves[0], leaves[5], inner, block)
    y = gb.FusedLoopTrainOp.apply(*leaves, inner, outer, block, "silu", 1e-5)
    grads = torch.autograd.grad(y, leaves, torch.from_numpy(gy).cuda())
    assert not gb.device_status(clear=True)
    a64 = [a.astype(np.float64) for a in (w, b, s, ga, be, x)]
    y64 = orc.outer_forward(*a64, inner, outer, block)
    y32 = orc.outer_forward(w, b, s, ga, be, x, inner, outer, block)
    assert_close(y.detach().cpu().numpy(), y64, y32, f"{name} forward")
    want64 = orc.outer_backward(*a64, gy.astype(np.float64), inner, outer, block)
    want32 = orc.outer_backward(w, b, s, ga, be, x, gy, inner, outer, block)
    # noise factor 3 instead of 2: the comparison is between the MAXIMA of two realisations of float32 rounding
    # noise over up to 5.7e7 elements after 32 chained stencil passes (gradients up to 4e3 in magnitude; measured:
    # the float32 oracle's worst error 1.3e-3, ours 3.0e-3, i.e. 7e-7 of max|ref|; 25 against 29 elements outside)
    for label, g, r64, r32 in zip(("weight", "bias", "scale", "gamma", "beta", "input"), grads, want64, want32):
        assert_close(g.cpu().numpy(), r64, r32, f"{name} gradient of {label}", noise_factor=3.0)


@pytest.mark.parametrize("keep", [True, False])
@pytest.mark.parametrize("shape,batch,inner,outer,act", [((8, 16, 24), 5, 1, 2, "tanh"), ((24, 8, 8), 2, 3, 3, "silu"), ((16, 16, 8), 9, 2, 1, "leaky_relu")])
def test_gated_loop_matches_oracle(shape, batch, inner, outer, act, keep):
    """The gated loop as one autograd node, ragged quads, kept iterations and replay, against the float64 oracle."""
    import gridnet_b200 as gb

    r = np.random.default_rng(11)
    w = (r.standard_normal((27, 2, *shape)) / np.sqrt(27)).astype(np.float32)
    b, x, gy = ((0.3 * r.standard_normal(n)).astype(np.float32) for n in ((2, *shape), (batch, *shape), (batch, *shape)))
    ga, be = (1 + 0.1 * r.standard_normal(shape)).astype(np.float32), (0.1 * r.standard_normal(shape)).astype(np.float32)
    t = [torch.from_numpy(a).cuda().requires_grad_(True) for a in (w, b, ga, be, x)]
    previous = gb.keep_forward_stash(keep)
    try:
        y = gb.FusedGatedLoopTrainOp.apply(*t, inner, outer, 8, act, 1e-5)
        y.backward(torch.from_numpy(gy).cuda())
    finally:
        gb.keep_forward_stash(previous)
    w, b, ga, be, h, g = (a.astype(np.float64) for a in (w, b, ga, be, x, gy))
    ins, mids = [], []
    for _ in range(outer):
        ins.append(h)
        mids.append(orc.gated_forward(w, b, h, inner, 8, act))
        h = orc.layernorm_forward(mids[-1], ga, be)
    assert_close(y.detach().cpu().numpy(), h, None, "y")
    sums = [0.0] * 4
    for k in reversed(range(outer)):
        g, dga, dbe = orc.layernorm_backward(mids[k], ga, g)
        dw, db, g = orc.gated_backward(w, b, ins[k], g, inner, 8, act)
        sums = [s + d for s, d in zip(sums, (dw, db, dga, dbe))]
    for got, ref, name in zip(t, (*sums, g), ("weight", "bias", "norm.weight", "norm.bias", "x")):
        assert_close(got.grad.cpu().numpy(), ref, None, f"grad {name}")


@pytest.mark.parametrize("block,shape,batch,inner,outer,act", [(8, (8, 16, 24), 5, 1, 3, "leaky_relu"), (8, (40, 24, 16), 9, 4, 4, "silu"),
                                                               (4, (16, 8, 24), 7, 3, 4, "relu"), (4, (24, 24, 24), 4, 8, 6, "silu")])
def test_loops_with_gradients_give_the_bits_of_the_register_patch_kernels(block, shape, batch, inner, outer, act):
    """What rounding differs by in a forward pass is amplified in the gradients, without bound where a pre-activation crosses
    the kink of an activation function. So the loops with gradients, whichever kernels they run on, have the forward pass
    of the register-patch kernels bit for bit: plain and residual, with the iterations kept and run again, and a single step."""
    import gridnet_b200 as gb
    from gridnet_b200 import gridnet_cuda
    from gridnet_b200._lib import activation_id, check, lib

    g = torch.Generator().manual_seed(23)
    mk = lambda *sz, scale=1.0, shift=0.0: (shift + scale * torch.randn(*sz, generator=g)).cuda()
    params = mk(27, *shape, scale=27 ** -0.5), mk(*shape, scale=0.1), mk(*shape, scale=0.1, shift=1.0)
    gamma, beta, x, gy = mk(*shape, scale=0.1, shift=1.0), mk(*shape, scale=0.1), mk(batch, *shape, shift=2.0), mk(batch, *shape)
    P, st = x[0].numel(), torch.cuda.current_stream().cuda_stream
    ptr = lambda t: None if t is None else t.data_ptr()
    nws = torch.empty(lib.gn_norm_workspace_bytes(batch, P), dtype=torch.uint8, device="cuda")

    def step(h, mr, partials):
        y = torch.empty_like(h)
        check(lib.gn_step_forward_train_f32(*map(ptr, params), ptr(h), ptr(y), ptr(gamma), ptr(beta), ptr(mr), ptr(partials), batch, *shape, inner,
                                            block, activation_id(act), None, 0, st))
        return y

    def plain(h):
        n = lib.gn_step_stats_partials(*shape, block)
        partials, mr = torch.empty(batch, n, 2, dtype=torch.float64, device="cuda"), None
        for _ in range(outer):
            h, mr = step(h, mr, partials), torch.empty(batch, 2, device="cuda")
            check(lib.gn_norm_finalize_f32(ptr(partials), n, ptr(mr), batch, P, 1e-5, st))
        y = torch.empty_like(h)
        check(lib.gn_norm_apply_f32(ptr(h), ptr(gamma), ptr(beta), ptr(mr), ptr(y), batch, P, st))
        return y

    def residual(h):
        sums, mr = torch.empty(batch, 2, dtype=torch.float64, device="cuda"), torch.empty(batch, 2, device="cuda")
        check(lib.gn_norm_local_sums_f32(ptr(h), ptr(sums), batch, P, ptr(nws), nws.numel(), st))
        check(lib.gn_norm_finalize_f32(ptr(sums), 1, ptr(mr), batch, P, 1e-5, st))
        for _ in range(outer):
            out, nxt = torch.empty_like(h), torch.empty(batch, 2, device="cuda")
            check(lib.gn_norm_residual_combine_f32(ptr(h), ptr(step(h, mr, None)), ptr(gamma), ptr(beta), ptr(mr), ptr(out), ptr(nxt), batch, P,
                                                   1e-5, ptr(nws), nws.numel(), st))
            h, mr = out, nxt
        return h

    grads = []
    for keep in (True, False):
        previous = gb.keep_forward_stash(keep)
        try:
            for form, want in (("plain", plain(x)), ("residual", residual(x))):
                leaves = [t.clone().requires_grad_(True) for t in (*params, gamma, beta, x)]
                if form == "plain":
                    y = gb.FusedLoopTrainOp.apply(*leaves, inner, outer, block, act, 1e-5)
                else:
                    y = gb.FusedLoopResidualTrainOp.apply(*leaves[3:], inner, block, act, 1e-5, outer, *leaves[:3])
                assert torch.equal(y, want), (form, keep, (y - want).abs().max().item())
                grads.append(torch.autograd.grad(y, leaves, gy))
        finally:
            gb.keep_forward_stash(previous)
    for a, c in zip(grads[0] + grads[1], grads[2] + grads[3]):
        assert torch.equal(a, c)  # iterations that are run again are the ones that were kept
    one, two = torch.empty_like(x), torch.empty_like(x)
    gridnet_cuda.forward(*params, x, one, inner, block, 1e-5, False, act)
    gridnet_cuda.forward_kept(*params, x, two, inner, block, 1e-5, False, act)
    assert torch.equal(one, two)


def test_gated_loop_takes_its_statistics_as_the_norm_op_does():
    """Step outputs whose mean is 300 deviations from zero: the statistics that the gated loop's kernel takes from them are those
    that the norm op's kernels take (floats of four values, doubles above), to a rounding of the result."""
    import gridnet_b200 as gb
    from gridnet_b200 import backend_cuda
    from gridnet_b200._lib import check, lib

    shape, batch = (16, 8, 24), 6
    P = shape[0] * shape[1] * shape[2]
    g = torch.Generator().manual_seed(3)
    w = torch.zeros(27, 2, *shape, device="cuda")
    b = torch.stack([300 + torch.randn(shape, generator=g), torch.randn(shape, generator=g)]).cuda()
    x = (300 + torch.randn(batch, *shape, generator=g)).cuda()
    gamma, beta = torch.ones(shape, device="cuda"), torch.zeros(shape, device="cuda")
    _, (_, stats, outs, _) = backend_cuda._loop_forward([(w, b)], gamma, beta, x, 2, 1, 8, "silu", 1e-5, False, True, gated=True)
    raw = outs[0].view(torch.float32).view(-1, P, 4).permute(0, 2, 1).reshape(-1, P)[:batch].contiguous()
    got = stats.view(torch.float32).view(-1, 2)[:batch]
    sums, want = torch.empty(batch, 2, dtype=torch.float64, device="cuda"), torch.empty(batch, 2, device="cuda")
    ws = torch.empty(lib.gn_norm_workspace_bytes(batch, P), dtype=torch.uint8, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    check(lib.gn_norm_local_sums_f32(raw.data_ptr(), sums.data_ptr(), batch, P, ws.data_ptr(), ws.numel(), st))
    check(lib.gn_norm_finalize_f32(sums.data_ptr(), 1, want.data_ptr(), batch, P, 1e-5, st))
    assert raw.mean() / raw.std() > 200
    assert torch.allclose(got, want, rtol=2.0 ** -22, atol=0), (got, want)


@pytest.mark.parametrize("batch", [1, 3, 4, 6])
def test_samples_that_fill_up_a_quad_leave_no_trace(batch):
    """The quad kernels work on four samples at a time. With an eps of zero a constant grid or block divides by zero; where no
    sample of the batch is constant, what fills up the last quad must not be either."""
    import gridnet_b200 as gb
    from gridnet_b200 import gridnet_cuda as gc

    g = torch.Generator().manual_seed(9)
    shape, inner, outer = (8, 16, 8), 2, 2
    mk = lambda *sz, scale=1.0, shift=0.0: (shift + scale * torch.randn(*sz, generator=g)).cuda()
    w, b, s = mk(27, *shape, scale=27 ** -0.5), torch.zeros(shape, device="cuda"), torch.ones(shape, device="cuda")
    gamma, beta, x, gy = mk(*shape, scale=0.1, shift=1.0), mk(*shape, scale=0.1), mk(batch, *shape), mk(batch, *shape)
    w2, b2 = mk(27, 2, *shape, scale=27 ** -0.5), torch.zeros(2, *shape, device="cuda")

    def plain(step):
        def f(w, b, *rest):
            *s, ga, be, h = rest
            for _ in range(outer):
                h = torch.nn.functional.layer_norm(step(w, b, *s, h), shape, ga, be, 0.0)
            return h
        return f

    def check(f, ref, leaves):
        a, c = ([t.clone().requires_grad_(True) for t in leaves] for _ in range(2))
        got, want = torch.autograd.grad(f(*a), a, gy), torch.autograd.grad(ref(*c), c, gy)
        for i, (p, q) in enumerate(zip(got, want)):
            assert torch.isfinite(q).all() and torch.allclose(p, q, rtol=1e-3, atol=1e-4 * (1 + q.abs().max().item())), i

    check(lambda *t: gb.FusedLoopTrainOp.apply(*t, inner, outer, 8, "silu", 0.0),
          plain(lambda w, b, s, h: gb.GridnetCudaOp.apply(w, b, s, h, inner, 8, 1e-5, False, "silu")), (w, b, s, gamma, beta, x))
    check(lambda *t: gb.FusedGatedLoopTrainOp.apply(*t, inner, outer, 8, "tanh", 0.0),
          plain(lambda w, b, h: gb.GatedGridnetCudaOp.apply(w, b, h, inner, 8, "tanh")), (w2, b2, gamma, beta, x))
    got, want = ([torch.empty_like(t) for t in (w, b, s, x)] for _ in range(2))
    gc.backward_kept(w, b, s, x, gy, *got, inner, 8, 0.0, True, "silu")
    gc.backward(w, b, s, x, gy, *want, inner, 8, 0.0, True, "silu")
    for i, (p, q) in enumerate(zip(got, want)):
        assert torch.isfinite(q).all() and torch.allclose(p, q, rtol=1e-3, atol=1e-4 * (1 + q.abs().max().item())), i


@pytest.mark.parametrize("shape,batch", [((8, 8, 8), 129), ((32, 32, 32), 37), ((16, 24, 8), 3), ((32, 40, 64), 5)])
@pytest.mark.parametrize("gated", [False, True])
def test_layer_norm_sums_taken_with_the_border_or_apart(shape, batch, gated):
    """The backward pass of small grids takes the sums of the norm's gradient in the border pass, quads split over a cluster of CTAs
    (7 of them, 4, 1); 160 regions have them apart. Against the composition of the step op and torch's layer norm. The sums run
    over at most 2 x 129 x 512 values of order one in another order: 1e-4 of the largest gradient is twenty times their rounding."""
    import gridnet_b200 as gb

    g = torch.Generator().manual_seed(17)
    inner, outer = 2, 3
    mk = lambda *sz, scale=1.0, shift=0.0: (shift + scale * torch.randn(*sz, generator=g)).cuda()
    params = [mk(27, *([2] if gated else []), *shape, scale=27 ** -0.5), mk(*([2] if gated else []), *shape, scale=0.1)]
    if not gated:
        params.append(mk(*shape, scale=0.1, shift=1.0))
    leaves = params + [mk(*shape, scale=0.1, shift=1.0), mk(*shape, scale=0.1), mk(batch, *shape)]
    gy = mk(batch, *shape)

    def loop(*t):
        if gated:
            return gb.FusedGatedLoopTrainOp.apply(*t, inner, outer, 8, "tanh", 1e-5)
        return gb.FusedLoopTrainOp.apply(*t, inner, outer, 8, "silu", 1e-5)

    def composed(*t):
        *p, gamma, beta, h = t
        for _ in range(outer):
            h = gb.GatedGridnetCudaOp.apply(*p, h, inner, 8, "tanh") if gated else gb.GridnetCudaOp.apply(*p, h, inner, 8, 1e-5, False, "silu")
            h = torch.nn.functional.layer_norm(h, shape, gamma, beta, 1e-5)
        return h

    grads = []
    for f in (loop, loop, composed):
        t = [a.clone().requires_grad_(True) for a in leaves]
        grads.append(torch.autograd.grad(f(*t), t, gy))
    for i, (a, again, want) in enumerate(zip(*grads)):
        assert torch.equal(a, again), i
        assert torch.allclose(a, want, rtol=0, atol=1e-4 * want.abs().max().item()), (i, (a - want).abs().max().item(), want.abs().max().item())


@pytest.mark.parametrize("gated", [False, True])
def test_what_a_loop_keeps_survives_being_packed_and_unpacked(gated):
    """A small loop saves what it keeps as one tensor and finds its pieces by their addresses. Hooks that move saved tensors away and
    bring back others, and a second walk over the same graph, give the same gradients."""
    import gridnet_b200 as gb

    g = torch.Generator().manual_seed(23)
    shape, batch, inner, outer = (16, 8, 24), 5, 2, 3
    mk = lambda *sz, scale=1.0, shift=0.0: (shift + scale * torch.randn(*sz, generator=g)).cuda()
    leaves = [mk(27, *([2] if gated else []), *shape, scale=27 ** -0.5), mk(*([2] if gated else []), *shape, scale=0.1)]
    leaves += ([] if gated else [mk(*shape, scale=0.1, shift=1.0)]) + [mk(*shape, scale=0.1, shift=1.0), mk(*shape, scale=0.1), mk(batch, *shape)]
    leaves = [t.requires_grad_(True) for t in leaves]
    op, gy = gb.FusedGatedLoopTrainOp if gated else gb.FusedLoopTrainOp, mk(batch, *shape)
    y = op.apply(*leaves, inner, outer, 8, "tanh", 1e-5)
    want = torch.autograd.grad(y, leaves, gy, retain_graph=True)
    again = torch.autograd.grad(y, leaves, gy)
    with torch.autograd.graph.save_on_cpu():
        y = op.apply(*leaves, inner, outer, 8, "tanh", 1e-5)
    moved = torch.autograd.grad(y, leaves, gy)
    for a, b, c in zip(want, again, moved):
        assert torch.equal(a, b) and torch.equal(a, c)


def test_separate_networks_of_a_small_grid_kept_and_recomputed():
    """A network per step on a grid of 64 regions, whose reverse sweeps follow the re-ordering of their parameters directly where the
    iterations are kept, and a forward pass where they are not: the same gradients, bit for bit, over many repeats."""
    import gridnet_b200 as gb

    g = torch.Generator().manual_seed(31)
    shape, batch, inner, outer = (32, 32, 32), 40, 2, 6
    mk = lambda *sz, scale=1.0, shift=0.0: (shift + scale * torch.randn(*sz, generator=g)).cuda()
    leaves = [mk(*shape, scale=0.1, shift=1.0), mk(*shape, scale=0.1), mk(batch, *shape)]
    sets = [t for _ in range(outer) for t in (mk(27, *shape, scale=27 ** -0.5), mk(*shape, scale=0.1), mk(*shape, scale=0.1, shift=1.0))]
    leaves, sets, gy = [t.requires_grad_(True) for t in leaves], [t.requires_grad_(True) for t in sets], mk(batch, *shape)

    def grads(keep):
        previous = gb.keep_forward_stash(keep)
        try:
            y = gb.FusedLoopSeparateTrainOp.apply(*leaves, inner, 8, "silu", 1e-5, *sets)
        finally:
            gb.keep_forward_stash(previous)
        return torch.autograd.grad(y, leaves + sets, gy)

    want = grads(False)
    for _ in range(10):
        for i, (a, b) in enumerate(zip(grads(True), want)):
            assert torch.equal(a, b), i


@pytest.mark.parametrize("shape,block,gated", [((16, 8, 24), 8, False), ((16, 8, 24), 8, True), ((16, 8, 24), 4, False), ((32, 40, 64), 8, False)])
def test_statistics_need_no_more_than_their_own_alignment(shape, block, gated):
    """A caller of the C interface may keep the loop's statistics at any address that pairs of floats may have: 8 bytes off a multiple of
    16 they give the same bits (with sums in the border pass, of both branches, apart from it, and with blocks of 4)."""
    from gridnet_b200 import backend_cuda as bc

    g = torch.Generator().manual_seed(37)
    batch, inner, outer, act = 6, 2, 3, "tanh"
    mk = lambda *sz, scale=1.0, shift=0.0: (shift + scale * torch.randn(*sz, generator=g)).cuda()
    two = [2] if gated else []
    params = [mk(27, *two, *shape, scale=27 ** -0.5), mk(*two, *shape, scale=0.1)] + ([] if gated else [mk(*shape, scale=0.1, shift=1.0)])
    gamma, beta, x, gy = mk(*shape, scale=0.1, shift=1.0), mk(*shape, scale=0.1), mk(batch, *shape), mk(batch, *shape)
    _, saved = bc._loop_forward([params], gamma, beta, x, inner, outer, block, act, 1e-5, False, True, gated=gated)
    x_il4, stats, outs, stashes = saved
    assert stats.data_ptr() % 16 == 0
    moved = torch.empty(stats.numel() + 16, dtype=torch.uint8, device="cuda")[8:8 + stats.numel()].copy_(stats)
    assert moved.data_ptr() % 16 == 8
    (want, *more), (got, *moved_more) = (bc._loop_backward([params], gamma, beta, (x_il4, s, outs, stashes), gy, inner, outer, block, act, False, gated=gated)
                                         for s in (stats, moved))
    for i, (a, b) in enumerate(zip([*want[0], *more], [*got[0], *moved_more])):
        assert torch.equal(a, b), i


def test_what_does_not_fit_is_recomputed(monkeypatch):
    """The bookkeeping of kept iterations: per device, without a lock that a finaliser could meet held, and a loop that runs out of
    memory while it allocates them goes on with those it has (allocation made to fail here; the gradients are the same bits)."""
    import gc

    import gridnet_b200 as gb
    from gridnet_b200 import backend_cuda

    kept = backend_cuda._Kept
    device = torch.device("cuda", torch.cuda.current_device())
    held = lambda: sum(kept._alive.get(device.index, {}).values())
    base = held()
    a, b = kept(1 << 20, device), kept(2 << 20, device)
    assert held() == base + (3 << 20)
    b.itself = b  # a cycle: its finaliser runs inside a collection, whenever that is
    del b
    gc.collect()
    assert held() == base + (1 << 20)
    monkeypatch.setattr(kept, "UNASKED", held() + 100)
    assert kept.room_for(100, device)
    monkeypatch.setattr(backend_cuda, "_free_bytes", lambda d: 5000)
    assert kept.room_for(500, device) and not kept.room_for(501, device)
    monkeypatch.setitem(kept._alive, device.index + 1, {1: 1 << 40})  # another device's does not count
    assert kept.room_for(100, device)
    del a

    monkeypatch.undo()
    g = torch.Generator().manual_seed(2)
    shape, batch, inner, outer = (16, 8, 8), 5, 2, 4
    mk = lambda *sz, scale=1.0: (scale * torch.randn(*sz, generator=g)).cuda()
    leaves = [mk(27, *shape, scale=27 ** -0.5), mk(*shape, scale=0.1), mk(*shape), mk(*shape), mk(*shape), mk(batch, *shape)]
    gy = mk(batch, *shape)

    def grads():
        t = [u.clone().requires_grad_(True) for u in leaves]
        return torch.autograd.grad(gb.FusedLoopTrainOp.apply(*t, inner, outer, 8, "silu", 1e-5), t, gy)

    want = grads()
    monkeypatch.setattr(backend_cuda, "_BIG", 0)  # the path of loops that hold more than a GiB
    real, calls = backend_cuda._staggered, []

    def scarce(nbytes, dev, k):
        calls.append(nbytes)
        if len(calls) > 1 + outer + 2:  # the input, the outputs and two steps' iterations
            raise torch.cuda.OutOfMemoryError("out of memory")
        return real(nbytes, dev, k)

    for f in (real, scarce):
        monkeypatch.setattr(backend_cuda, "_staggered", f)
        for u, v in zip(grads(), want):
            assert torch.equal(u, v)
    assert len(calls) == 1 + outer + 3


@pytest.mark.parametrize("kind", ["gated", "step", "loop"])
def test_nothing_is_kept_where_gradients_are_off(kind):
    """Under no_grad a model's parameters still require gradients; its forward pass must not keep anything for them all the
    same: a gated loop of eight steps would hold 50 activation tensors, a normalised step the pre-activations."""
    import gridnet_b200 as gb

    shape, batch, inner, outer = (32, 32, 32), 64, 2, 8
    device = torch.device("cuda")
    x = torch.randn(batch, *shape, device=device)
    one = x.numel() * 4
    if kind == "gated":
        model = gb.GridnetModel(shape, inner, outer, 8, device, activation="tanh", gated=True)
    elif kind == "step":
        model = gb.Gridnet(shape, inner, 8, device)
    else:
        net, norm = gb.Gridnet(shape, inner, 8, device, normalize=False), gb.GridNorm(shape, device)
        model = lambda h: gb.FusedLoopTrainOp.apply(net.weight, net.bias, net.residual_scale, norm.weight, norm.bias, h, inner, outer, 8, "silu", 1e-5)
    want = model(x).detach()
    torch.cuda.synchronize()
    base = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    with torch.no_grad():
        y = model(x)
    assert not y.requires_grad and torch.equal(y, want)
    # the output, input and outputs of a step in the kernels' layout, and at most 8.2 MB of parameters in another order
    assert torch.cuda.max_memory_allocated() - base < 4 * one + 10e6, kind


def test_gated_loop_calls_modules_that_are_listened_to():
    """Forward hooks on the gated network or its norm, and a network with a forward of its own, see every outer step."""
    import gridnet_b200 as gb

    shape, outer = (8, 8, 16), 3
    device = torch.device("cuda")
    torch.manual_seed(4)
    model = gb.GridnetModel(shape, 2, outer, 8, device, activation="tanh", gated=True)
    x = torch.randn(5, *shape, device=device)
    want = model(x)
    for module in (model.network, model.norm):
        seen = []
        handle = module.register_forward_hook(lambda m, args, out: seen.append(out))
        y = model(x)
        handle.remove()
        assert len(seen) == outer
        assert torch.allclose(y, want, rtol=1e-4, atol=1e-5)

    class Doubled(gb.GatedGridnet):
        def forward(self, h):
            return 2 * super().forward(h)

    model.network.__class__ = Doubled
    h = x
    for _ in range(outer):
        h = model.norm(model.network(h))
    assert torch.equal(model(x), h)


@pytest.mark.parametrize("block,batch", [(8, 1), (8, 2), (4, 1)])
def test_loops_on_patches_match_the_quad_kernels(block, batch, monkeypatch):
    """Loops with gradients of one or two samples of a large grid run on the register-patch kernels: the same output bits, and
    gradients, as on the quad kernels; plain, per-step parameters and residual; iterations kept and run again. On a small grid
    that the rule is made to cover; an input that these kernels cannot read stays on the quad kernels."""
    import gridnet_b200 as gb
    from gridnet_b200 import backend_cuda

    for n, first in ((1, (128, 128, 136)), (2, (128, 136, 256))):
        assert backend_cuda.on_patches(n, *first) and not backend_cuda.on_patches(n, 128, 128, n * 128)
    assert not backend_cuda.on_patches(3, 256, 256, 256)
    g = torch.Generator().manual_seed(31)
    shape, inner, outer = (16, 24, 8), 3, 3
    mk = lambda *sz, scale=1.0, shift=0.0: (shift + scale * torch.randn(*sz, generator=g)).cuda()
    plist = [(mk(27, *shape, scale=27 ** -0.5), mk(*shape, scale=0.1), mk(*shape, scale=0.1, shift=1.0)) for _ in range(outer)]
    gamma, beta, x, gy = mk(*shape, scale=0.1, shift=1.0), mk(*shape, scale=0.1), mk(batch, *shape), mk(batch, *shape)

    def run(form, keep, x=x):
        ps = [tuple(t.clone().requires_grad_(True) for t in p) for p in (plist if form == "separate" else plist[:1])]
        ga, be, xl = gamma.clone().requires_grad_(True), beta.clone().requires_grad_(True), x.detach().requires_grad_(True)
        flat = [t for p in ps for t in p]
        previous = gb.keep_forward_stash(keep)
        try:
            if form == "plain":
                y = gb.FusedLoopTrainOp.apply(*flat, ga, be, xl, inner, outer, block, "silu", 1e-5)
            elif form == "separate":
                y = gb.FusedLoopSeparateTrainOp.apply(ga, be, xl, inner, block, "silu", 1e-5, *flat)
            else:
                y = gb.FusedLoopResidualTrainOp.apply(ga, be, xl, inner, block, "silu", 1e-5, outer, *flat)
            return [y] + list(torch.autograd.grad(y, [ga, be, xl] + flat, gy))
        finally:
            gb.keep_forward_stash(previous)

    def inference(form):
        with torch.no_grad():
            return gb.fused_loop_forward(plist if form == "separate" else plist[:1] * outer, gamma, beta, x, inner, block, "silu", 1e-5, form == "residual")

    for form in ("plain", "separate", "residual"):
        want = run(form, True)
        assert torch.equal(inference(form), want[0])
        with monkeypatch.context() as m:
            m.setattr(backend_cuda, "on_patches", lambda *a: True)
            for keep in (True, False):
                got = run(form, keep)
                assert torch.equal(got[0], want[0]), (form, keep)
                for i, (a, c) in enumerate(zip(got[1:], want[1:])):
                    assert torch.allclose(a, c, rtol=1e-3, atol=1e-5 * (1 + c.abs().max().item())), (form, keep, i)
            assert torch.equal(inference(form), want[0])
            shifted = torch.empty(x.numel() + 1, device="cuda")[1:].view(x.shape).copy_(x)
            for a, c in zip(run(form, True, shifted), want):
                assert torch.equal(a, c), form
