"""The work that programs have this package do, as measurable cases.

A case is a dict of plain values.  ``kind`` says what a pass is:

* ``train``      one Euler step of a model in the middle of a training rollout, forward and backward to
                 the incoming positions and states and to the MLP weights (``stepping.step_euler``);
* ``step``       the same step under ``torch.no_grad``, as an evaluation loop makes it;
* ``graphed``    the step recorded in a CUDA graph (``graphs.GraphedEulerStep``), as an interactive or
                 long rollout makes it;
* ``perceive``   binning, reorder, the fused perception operators and their backward with respect to
                 positions and features (``sphops.perceive``);
* ``operators``  the same through the per-operator API that a model written for ``sphops`` calls
                 (density, blur, gradient_hybrid, density_gradient), with or without ``enable_fusion``;
* ``rollout``    several perception steps with re-binning and the backward of the last one
                 (``rollout.PerceptionRollout``);
* ``splat``      a batch of particle images and their backward (``splatting.splat_particles_batch``).

Particles are drawn with the spatial distributions of the benchmark configurations (uniform, blobs,
strokes, ball with a dense shell), features and upstream gradients are N(0, 1).
"""
from __future__ import annotations

import math

import torch

from npa_b200 import sphops as sph
from npa_b200 import splatting
from npa_b200.graphs import GraphedEulerStep
from npa_b200.rollout import PerceptionRollout, VelocityField
from npa_b200.stepping import step_euler

HIDDEN = 128  # width of the per-particle MLP


def _case(kind, dim, B, N, C, eps, grid, boundary="clamped", mode="grid", sampler="uniform", mpb=32, **more):
    """``grid`` is the number of cells per axis; ``mass`` and ``fuse`` are off unless given."""
    return dict(kind=kind, dim=dim, B=B, N=N, C=C, eps=eps, grid=grid, boundary=boundary, mode=mode,
                sampler=sampler, mpb=mpb, **more)


def listed():
    return [
        # A growing shape: 8 systems of 4,096 particles with 16 channels, the everyday training step in 2D.
        dict(name="train_2d_growing", **_case("train", 2, 8, 4096, 16, 0.1, 16)),
        # Point-cloud digits: many small systems of 512 particles drawn as strokes, 64 of them in a training batch.
        dict(name="train_2d_strokes", **_case("train", 2, 64, 512, 16, 0.1, 16, sampler="strokes", mpb=64)),
        # A growing 3D shape on Morton-ordered cells: 4 systems of 16,384 particles.
        dict(name="train_3d_growing", **_case("train", 3, 4, 16384, 16, 0.1, 32, mode="particle", sampler="ball_shell", mpb=64)),
        # The largest 3D training step: 4 systems of 65,536 particles with 32 channels, ~41 neighbours each.
        dict(name="train_3d_splat", **_case("train", 3, 4, 65536, 32, 0.0879, 24, sampler="ball_shell")),
        # Evaluation of a texture: one periodic system with long-range neighbourhoods (~128 neighbours).
        dict(name="step_2d_texture", **_case("step", 2, 1, 4096, 16, 0.2, 10, boundary="periodic")),
        # An interactive rollout of one small system, where launches and latency are all there is.
        dict(name="graphed_2d_growing", **_case("graphed", 2, 1, 2500, 16, 0.1, 16)),
        # A model written for sphops, unchanged, in training: one launch per operator and direction.
        dict(name="operators_2d_growing", **_case("operators", 2, 8, 4096, 16, 0.1, 16, fuse=False)),
        # The same with operator fusion switched on, odd sizes, per-particle masses, periodic box.
        dict(name="operators_2d_fused_odd", **_case("operators", 2, 3, 5001, 13, 0.05, 20, boundary="periodic", fuse=True, mass=True)),
        # Strongly clustered 2D particles: cells from empty to hundreds of particles.
        dict(name="perceive_2d_blobs", **_case("perceive", 2, 8, 16384, 32, 0.025, 40, sampler="blobs")),
        # The largest single perception step with position gradients (the benchmark's headline workload).
        dict(name="perceive_3d_splat", **_case("perceive", 3, 4, 65536, 32, 0.0879, 24, sampler="ball_shell")),
        # Periodic 3D systems of 262,144 particles, re-binned every step, backward through the last one.
        dict(name="rollout_3d_periodic", **_case("rollout", 3, 2, 262144, 16, 0.03125, 32, boundary="periodic", steps=4, slots=128)),
        # Rendering for an image loss: 8 systems of 4,096 particles into 256 x 256 images, forward and backward.
        dict(name="splat_images", **_case("splat", 2, 8, 4096, 3, 0.0, 0, img=256)),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "step", "graphed", "operators", "operators", "perceive", "perceive",
                       "perceive", "rollout", "splat"])
    if kind == "splat":
        B = _log_uniform(rng, 1, 16)
        return _case(kind, 2, B, _log_uniform(rng, 256, min(8192, 32768 // B)), 3, 0.0, 0, img=rng.randint(64, 256))
    dim = 3 if kind == "rollout" else rng.choice([2, 3])
    most = {"step": 65536, "graphed": 32768, "rollout": 262144}.get(kind, 131072)  # particles in all
    B = _log_uniform(rng, 1, 4 if kind == "rollout" else 64)
    N = _log_uniform(rng, 256 if B > 1 else 1024, min(65536, most // B))
    C = rng.choice([8, 12, 13, 16, 16, 20, 24, 32])
    boundary = "periodic" if kind == "rollout" else rng.choice(["clamped", "clamped", "periodic"])
    mode = "particle" if dim == 3 and rng.random() < 0.25 else "grid"
    sampler = "uniform"
    if boundary == "clamped":
        sampler = rng.choice(["uniform", "blobs", "strokes"]) if dim == 2 else rng.choice(["uniform", "ball_shell"])
    # smoothing radius for 12 to 64 neighbours at the mean density, never more than a quarter of the box
    want = math.exp(rng.uniform(math.log(12.0), math.log(64.0)))
    if dim == 2:
        eps, side = math.sqrt(want / (math.pi * N)), 1.0
    elif sampler == "ball_shell":
        eps, side = (want / (0.9 * N)) ** (1.0 / 3.0), 2.0
    else:
        eps, side = (3.0 * want / (4.0 * math.pi * N)) ** (1.0 / 3.0), 1.0
    eps = min(eps, side / 4.0)
    if sampler in ("blobs", "strokes"):
        eps *= 0.6  # clustered particles: shorter radius for the same neighbourhoods
    cells = max(4, int(side / eps)) if boundary == "periodic" else max(4, math.ceil(side / eps))
    if mode == "particle":
        cells = 1 << (cells - 1).bit_length()
        if boundary == "periodic" and cells > side / eps:
            cells = max(4, cells // 2)
    cells = min(cells, 64)
    eps = round(side / cells, 6) if boundary == "periodic" else round(max(eps, side / cells), 6)
    c = _case(kind, dim, B, N, C, eps, cells, boundary=boundary, mode=mode, sampler=sampler, mpb=rng.choice([32, 64]))
    if kind == "operators":
        c["fuse"] = rng.random() < 0.5
    if kind in ("operators", "perceive"):
        c["mass"] = rng.random() < 0.25
    if kind == "rollout":
        c.update(steps=rng.randint(2, 4), slots=rng.choice([64, 128]))
    return c


# ---- inputs ----------------------------------------------------------------------------------------------------------
def _uniform(c, g):
    """Uniform in the periodic box, or in a square / cube one unit wide (or as wide as the grid, when that is larger)."""
    wide = c["grid"] * c["eps"]
    side = wide if c["boundary"] == "periodic" or wide > 1.5 else 1.0
    return (torch.rand(c["B"], c["N"], c["dim"], generator=g, device="cuda") - 0.5) * side


def _blobs(c, g):
    B, N, dev = c["B"], c["N"], "cuda"
    centres = torch.rand(B, 64, 2, generator=g, device=dev)
    pick = torch.randint(0, 64, (B, N, 1), generator=g, device=dev).expand(-1, -1, 2)
    x = torch.gather(centres, 1, pick) + 0.04 * torch.randn(B, N, 2, generator=g, device=dev)
    return x.clamp_(0.0, 1.0) - 0.5


def _strokes(c, g):
    """12 random segments per system in 4 polylines, particles spread evenly over their length with a little jitter."""
    B, N, dev = c["B"], c["N"], "cuda"
    points = torch.rand(B, 4, 4, 2, generator=g, device=dev)
    a, b = points[:, :, :-1].reshape(B, 12, 2), points[:, :, 1:].reshape(B, 12, 2)
    length = (b - a).norm(dim=-1)
    end = torch.cumsum(length, dim=1)
    t = torch.rand(B, N, generator=g, device=dev) * end[:, -1:]
    k = torch.searchsorted(end, t).clamp_(max=11)
    u = ((t - torch.gather(end - length, 1, k)) / torch.gather(length, 1, k).clamp_min(1e-9)).unsqueeze(-1)
    k = k.unsqueeze(-1).expand(-1, -1, 2)
    x = torch.lerp(torch.gather(a, 1, k), torch.gather(b, 1, k), u)
    return (x + 0.01 * torch.randn(B, N, 2, generator=g, device=dev)).clamp_(0.0, 1.0) - 0.5


def _ball_shell(c, g):
    """Nine particles in ten uniform in the unit ball, one in ten in a thin shell at its surface."""
    B, N, dev = c["B"], c["N"], "cuda"
    direction = torch.nn.functional.normalize(torch.randn(B, N, 3, generator=g, device=dev), dim=-1)
    u = torch.rand(B, N, generator=g, device=dev)
    shell = torch.rand(B, N, generator=g, device=dev) < 0.1
    return direction * torch.where(shell, 0.98 + 0.02 * u, u ** (1.0 / 3.0)).unsqueeze(-1)


_SAMPLERS = {"uniform": _uniform, "blobs": _blobs, "strokes": _strokes, "ball_shell": _ball_shell}


class _Model(torch.nn.Module):
    """What a step reads of an NPA model: the MLP, its scalars and the perception flags (with their defaults)."""

    def __init__(self, dim, C, eps, g):
        super().__init__()
        self.spatial_dims = dim
        self.eps0, self.alpha = eps, 1.0
        self.state_grad = self.density_grad = self.log_norm_grad = self.log_norm_density_grad = True
        self.stopgrad_pos, self.stopgrad_state = True, False
        width = 2 * C + C * dim + dim
        self.model = torch.nn.Sequential(torch.nn.Linear(width, HIDDEN), torch.nn.ReLU(),
                                         torch.nn.Linear(HIDDEN, dim + C, bias=False)).cuda()
        with torch.no_grad():
            for p in self.model.parameters():
                fan_in = p.shape[-1] if p.dim() == 2 else width
                p.copy_((2.0 * torch.rand(p.shape, generator=g, device="cuda") - 1.0) / math.sqrt(fan_in))


def prepare(case, seed):
    c = case
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    B, N, C, D = c["B"], c["N"], c["C"], c["dim"]

    def randn(*shape):
        return torch.randn(*shape, generator=g, device="cuda")

    if c["kind"] == "splat":
        x = (torch.rand(B, N, 2, generator=g, device="cuda") - 0.5) * 1.6
        return dict(kind="splat", x=x, color=torch.rand(B, N, 3, generator=g, device="cuda"), img=c["img"],
                    up=randn(B, c["img"], c["img"], 4))

    grid = sph.HashGrid(dim=D, boundary=c["boundary"], mode=c["mode"], grid_size=(c["grid"],) * D, eps=c["eps"],
                        num_particles=N, batch_size=B, max_particles_per_block=c["mpb"])
    x = _SAMPLERS[c["sampler"]](c, g)
    if D == 3:  # 3D positions are stored four wide
        x = torch.cat([x, torch.zeros_like(x[..., :1])], dim=-1)
    st = dict(kind=c["kind"], grid=grid, x=x.contiguous(), s=randn(B, N, C), dim=D, seed=int(seed))
    if c["kind"] in ("train", "step", "graphed"):
        st["model"] = _Model(D, C, c["eps"], g)
    if c["kind"] == "train":
        # in the middle of a rollout both come from the step before and take gradients
        st["x"].requires_grad_(True)
        st["s"].requires_grad_(True)
        st["leaves"] = [st["x"], st["s"], *st["model"].model.parameters()]
        st["ups"] = [randn(*x.shape), randn(B, N, C)]
    elif c["kind"] == "graphed":
        st["graph"] = GraphedEulerStep(st["model"], grid, C, update_prob=1.0)
    elif c["kind"] in ("perceive", "operators"):
        st["x"].requires_grad_(True)
        st["s"].requires_grad_(True)
        st["fuse"] = bool(c.get("fuse"))
        st["mass"] = 0.5 + torch.rand(B, N, generator=g, device="cuda") if c.get("mass") else None
        st["ups"] = [randn(B, N), randn(B, N, C), randn(B, N, C, D), randn(B, N, D)]
    elif c["kind"] == "rollout":
        dt = 0.05 * c["eps"]  # a particle crosses a cell in about twenty steps
        st["rollout"] = PerceptionRollout(grid, C, c["steps"], dt, VelocityField(D, x.device, seed=int(seed)), list_slots=c["slots"])
        st["work_x"], st["work_s"] = torch.empty_like(st["x"]), torch.empty_like(st["s"])
        st["ups"] = dict(g_rho=randn(B, N), g_blur=randn(B, N, C), g_grad=randn(B, N, C, D))
    return st


# ---- passes ----------------------------------------------------------------------------------------------------------
def _train(st):
    # the update mask is drawn from torch's CUDA generator: seeded, as a reproducible training run seeds it
    torch.cuda.default_generators[st["x"].device.index].manual_seed(st["seed"])
    x_new, s_new, _ = step_euler(st["model"], st["x"], st["s"], st["grid"], update_prob=0.5)
    grads = torch.autograd.grad([x_new, s_new], st["leaves"], st["ups"])
    return [x_new.detach(), s_new.detach(), *grads]


def _step(st):
    with torch.no_grad():
        x_new, s_new, _ = step_euler(st["model"], st["x"], st["s"], st["grid"], update_prob=1.0)
    return [x_new, s_new]


def _graphed(st):
    return list(st["graph"](st["x"], st["s"]))


def _binned(st):
    snap = st["grid"].instantiate(st["x"])
    if st["mass"] is None:
        return (snap, *sph.bin_particles(st["x"], st["s"], snap), None)
    return (snap, *sph.bin_particles(st["x"], st["s"], snap, st["mass"]))


def _perceive(st):
    snap, x, s, mass = _binned(st)
    out = sph.perceive(x, s, snap, mass)
    grads = torch.autograd.grad(out, [st["x"], st["s"]], st["ups"])
    return [snap.permutation, snap.bin_offsets, *(t.detach() for t in out), *grads]


def _operators(st):
    sph.enable_fusion(st["fuse"])
    snap, x, s, mass = _binned(st)
    rho = sph.density(x, snap, mass)
    out = [rho, sph.blur(x, rho, s, snap, mass), sph.gradient_hybrid(x, rho, s, snap, mass), sph.density_gradient(x, snap, mass)]
    grads = torch.autograd.grad(out, [st["x"], st["s"]], st["ups"])
    return [snap.permutation, *(t.detach() for t in out), *grads]


def _rollout(st):
    st["work_x"].copy_(st["x"])
    st["work_s"].copy_(st["s"])
    r = st["rollout"]
    grads = r.run(st["work_x"], st["work_s"], st["ups"])
    return [r.x_bin, r.s_bin, r.rho, r.blur, r.grad, *grads]


def _splat(st):
    x, color = st["x"].detach().requires_grad_(True), st["color"].detach().requires_grad_(True)
    image = splatting.splat_particles_batch(x, color, img_size=st["img"])
    return [image.detach(), *torch.autograd.grad(image, [x, color], st["up"])]


_PASSES = {"train": _train, "step": _step, "graphed": _graphed, "perceive": _perceive, "operators": _operators,
           "rollout": _rollout, "splat": _splat}


def run(state):
    return _PASSES[state["kind"]](state)


# ---- what a pass cannot do without -----------------------------------------------------------------------------------
def _neighbours(c):
    """Mean number of neighbours of a particle, from the density of its distribution (an estimate)."""
    N, h = c["N"], c["eps"]
    ball = math.pi * h * h if c["dim"] == 2 else 4.0 / 3.0 * math.pi * h ** 3
    if c["sampler"] == "ball_shell":
        return 1.0 + 0.9 * N * h ** 3
    if c["sampler"] == "strokes":  # ~6 units of line per system
        return 1.0 + min(N * 2.0 * h / 6.0 * 1.5, float(N))
    if c["sampler"] == "blobs":    # its own blob plus the others, which cover the square about evenly
        return 1.0 + N / 64.0 * (1.0 - math.exp(-h * h / (4.0 * 0.04 ** 2))) + N * ball
    wide = c["grid"] * h
    side = wide if c["boundary"] == "periodic" or wide > 1.5 else 1.0
    return 1.0 + N * ball / side ** c["dim"]


def work(case):
    c = case
    B, N, C, D = c["B"], c["N"], c["C"], c["dim"]
    if c["kind"] == "splat":
        img, n = c["img"], B * N
        sigma = 2.0 * img * (2.0 / 128.0) / 2.0
        patch = (2 * max(1, math.ceil(5 * sigma)) + 1) ** 2
        return {"bytes": 4.0 * (2 * B * img * img * 4 + 2 * n * 5), "flops": float(n) * patch * (10 + 16)}
    P, n = (2 if D == 2 else 4), float(B * N)
    pairs = n * _neighbours(c)
    F, Y = 2 * C + C * D + D, D + C
    binning = n * 4 * (2 * P + 2 * C + 1)                      # positions and features in, in cell order out, permutation
    forward = n * 4 * (P + C + 1 + C + C * D + D)              # rho, blur, gradient, density gradient
    full = n * 4 * (1 + C + C * D + D + P + C)                 # upstream gradients in, both gradients out
    pair_forward = pairs * (2.0 * C * (1 + D) + 20)
    pair_sums = pairs * (2.0 * C * (1 + D) + 20)               # feature gradients of the backward
    pair_full = pairs * (2.0 * C * (1 + D) * 3 + 40)           # and the dot products of the position gradients
    if c["kind"] in ("train", "step", "graphed"):
        nbytes = binning + n * 4 * (P + C + P + C)
        flops = pair_forward + 2.0 * n * HIDDEN * (F + Y)
        if c["kind"] == "train":
            nbytes += n * 4 * (2 * (P + C) + C + Y)            # upstream gradients in, gradients out, what the step saves
            flops += pair_sums + 4.0 * n * HIDDEN * (F + Y)
        return {"bytes": nbytes, "flops": flops}
    if c["kind"] == "rollout":
        return {"bytes": c["steps"] * (binning + forward) + full, "flops": c["steps"] * pair_forward + pair_full}
    return {"bytes": binning + forward + full, "flops": pair_forward + pair_full}


def tolerance(case):
    """32-bit sums of tens of terms, in any order.  A step's MLP adds the kinks of its ReLU: a hidden unit that is zero
    to rounding error may be switched on in one implementation and off in another, which moves single gradient values."""
    if case["kind"] == "train":
        return {"rel": 2e-5, "max": 0.5}
    return {"rel": 1e-5, "max": 2e-3}
