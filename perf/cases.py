"""The work that users of this framework have it do, as cases that can be timed: inference of the model loop, training
steps of the models, and single steps of the update through the module and autograd surface.

A case is a dict of plain values; ``listed()`` names the fixed ones, ``draw(rng)`` gives more of the same ranges,
``prepare(case, seed)`` builds the model and its inputs on the GPU, ``run(state)`` is one pass, ``work(case)`` the
bytes and operations that a pass cannot do without, ``tolerance(case)`` how far two correct implementations may differ.
"""
import torch
import torch.nn.functional as F

import gridnet_b200 as gb
from gridnet_b200.script_models import ImageNetModel, MnistModel


def _case(name, kind, grid, block, inner, outer, batch, activation="silu", **more):
    m, n, k = grid
    case = dict(kind=kind, m=m, n=n, k=k, block=block, inner=inner, outer=outer, batch=batch, activation=activation)
    case.update(more)
    if name:
        case["name"] = name
    return case


def listed():
    return [
        # -- inference: GridnetModel without gradients
        # the MNIST-shaped network on a handful of images: launches and latency are what it costs
        _case("infer mnist", "infer", (32, 32, 32), 8, 2, 8, 8),
        # one sample through the 64^3 network: an interactive request
        _case("infer one sample", "infer", (64, 64, 64), 8, 4, 12, 1),
        # the headline throughput configuration: 64^3, 4 x 12 iterations, a batch of 64
        _case("infer 64^3", "infer", (64, 64, 64), 8, 4, 12, 64),
        # a grid that is not a cube, the odd last batch of a data set, and the activation of the ImageNet script
        _case("infer ragged", "infer", (40, 56, 72), 8, 3, 6, 37, "leaky_relu"),
        # the largest grid: 16.8 M neurons, 1.8 GB of weights
        _case("infer 256^3", "infer", (256, 256, 256), 8, 2, 32, 32),
        # -- training: forward and backward of the whole model
        # the MNIST script's model and loss on a mini-batch
        _case("train mnist", "mnist", (32, 32, 32), 8, 2, 8, 64, gated=False),
        # the same with the gated network and its default activation
        _case("train mnist gated", "mnist", (32, 32, 32), 8, 2, 8, 64, "tanh", gated=True),
        # the ImageNet-shaped loop (128^3, 2 x 16) on the share of the batch that one of eight GPUs gets
        _case("train 128^3", "train", (128, 128, 128), 8, 2, 16, 32),
        # the ImageNet script's model at its default grid of 64^3 in its residual form
        _case("train imagenet residual", "imagenet", (64, 64, 64), 8, 2, 8, 16, "leaky_relu", separate=False),
        # block size 4 with eight inner iterations: the halo-heavy configuration
        _case("train block 4", "train", (64, 64, 64), 4, 8, 16, 128),
        # -- one step through the module, forward and backward
        # the Gridnet class as it is by default: normalisation per block
        _case("step normalised", "step", (64, 64, 64), 8, 2, 1, 64, normalize=True, double=False),
        # double precision, block 4, odd sizes: what a gradient check or a reference run does
        _case("step double", "step", (20, 12, 28), 4, 3, 1, 5, normalize=True, double=True),
    ]


def _log_int(rng, lo, hi):
    """A whole number from lo to hi, spread over its logarithm."""
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def _grid(rng, block, lo, hi):
    """Three sides, multiples of the block, each between lo and hi."""
    return tuple(block * _log_int(rng, max(1, lo // block), hi // block) for _ in range(3))


def draw(rng):
    kind = rng.choice(["infer", "infer", "infer", "infer", "train", "train", "mnist", "imagenet", "step", "step"])
    act = rng.choice(["silu", "silu", "leaky_relu", "tanh", "relu"])
    if kind == "mnist":
        gated = rng.random() < 0.4
        return _case(None, kind, (32, 32, 32), 8, rng.randint(1, 4), rng.randint(2, 12), _log_int(rng, 4, 256),
                     "tanh" if gated else act, gated=gated)
    if kind == "imagenet":
        g = rng.choice([32, 64])
        return _case(None, kind, (g, g, g), 8, rng.randint(1, 4), rng.randint(2, 10), _log_int(rng, 4, 64), act,
                     separate=rng.random() < 0.5)
    if kind == "step":
        double = rng.random() < 0.3
        block = rng.choice([8, 8, 4])
        grid = _grid(rng, block, 8, 32 if double else 96)
        voxels = grid[0] * grid[1] * grid[2]
        batch = _log_int(rng, 1, max(2, min(128, (1 << (19 if double else 24)) // voxels)))
        return _case(None, kind, grid, block, rng.randint(1, 6), 1, batch, act, normalize=rng.random() < 0.6, double=double)
    # the whole loop: up to the work of the largest listed case of its kind, in neuron updates and in memory
    block = rng.choice([8, 8, 8, 4])
    inner, outer = (rng.randint(2, 8) if block == 4 else rng.randint(1, 5)), rng.randint(4, 16)
    grid = _grid(rng, block, 16, 128)
    voxels = grid[0] * grid[1] * grid[2]
    updates = (1 << 34) if kind == "infer" else (1 << 31)
    batch = _log_int(rng, 1, max(2, min(256, (1 << 27) // voxels, updates // (voxels * inner * outer))))
    return _case(None, kind, grid, block, inner, outer, batch, act)


def prepare(case, seed):
    device = torch.device("cuda", torch.cuda.current_device())
    torch.manual_seed(seed)
    grid = (case["m"], case["n"], case["k"])
    B, block, inner, outer, act = case["batch"], case["block"], case["inner"], case["outer"], case["activation"]
    kind = case["kind"]
    state = {"kind": kind}
    if kind in ("infer", "train"):
        model = gb.GridnetModel(grid, inner, outer, block, device, activation=act)
        # activations as a model starts with them: the input on the first plane along K, zero elsewhere
        x = torch.zeros(B, *grid, device=device)
        x[..., 0] = torch.randn(B, *grid[:2], device=device)
        if kind == "train":
            state["grad"] = torch.randn(B, *grid, device=device)  # what the readout and the loss send back
            x.requires_grad_(True)
    elif kind == "mnist":
        model = MnistModel(inner, outer, init_scale=1.0, residual_scale=1.0, gated=case["gated"], remember_bias=1.0,
                           activation=act, device=device)
        x = torch.rand(B, 28, 28, device=device)
        state["labels"] = torch.randint(10, (B,), device=device)
    elif kind == "imagenet":
        model = ImageNetModel(inner_iters=inner, outer_iters=outer, outer_residual=True, init_scale=1.0, residual_scale=1.0,
                              emb_channels=4, grid_size=grid[0], activation=act, separate_params=case["separate"],
                              device=device)
        x = torch.randn(B, 3, 256, 256, device=device)
        state["labels"] = torch.randint(1000, (B,), device=device)
    else:
        dtype = torch.float64 if case["double"] else torch.float32
        model = gb.Gridnet(grid, inner, block, device, dtype=dtype, normalize=case["normalize"], activation=act)
        x = torch.randn(B, *grid, device=device, dtype=dtype).requires_grad_(True)
        state["grad"] = torch.randn(B, *grid, device=device, dtype=dtype)
    with torch.no_grad():  # biases, scales and norm parameters as training leaves them, not as it finds them
        for name, p in model.named_parameters():
            if name.endswith(("bias", "residual_scale", "norm.weight")):
                p += 0.1 * torch.randn_like(p)
    state["model"], state["x"] = model, x
    return state


def run(state):
    model, x = state["model"], state["x"]
    if state["kind"] == "infer":
        with torch.no_grad():
            return model(x)
    model.zero_grad(set_to_none=True)
    x.grad = None
    out = model(x)
    if "labels" in state:
        F.cross_entropy(out, state["labels"]).backward()
    else:
        out.backward(state["grad"])
    grads = {name: p.grad for name, p in model.named_parameters()}
    if x.requires_grad:
        grads["x"] = x.grad
    return {"out": out.detach(), "grads": grads}


def work(case):
    voxels = case["m"] * case["n"] * case["k"]
    acts = case["batch"] * voxels
    size = 8 if case.get("double") else 4
    gated = bool(case.get("gated"))
    nets = case["outer"] if case.get("separate") else 1
    params = voxels * ((54 + 2 if gated else 27 + 2) * nets + (2 if case["kind"] != "step" else 0))
    madds = (54 if gated else 27) * acts * case["inner"] * case["outer"]
    if case["kind"] == "infer":
        return {"bytes": size * (params + 2 * acts), "flops": 2 * madds}
    # training: parameters and inputs read, their gradients written; the forward sum and its two transposes
    ends = {"train": 4, "step": 4}.get(case["kind"], 0) * acts
    return {"bytes": size * (2 * params + ends), "flops": 6 * madds}


def tolerance(case):
    if case.get("double"):
        return {"rel": 1e-12}
    # float32 throughout: against a float64 composition of the same steps the listed loops and their gradients are off by
    # 1e-7 to 6e-7 (2-norm) and single values by up to 4e-5; another order of the sums may double that and more
    return {"rel": 1e-5, "max": 1e-3}
