"""One Euler step of an NPA model on the fused kernels.

``step_euler`` has the contract of the reference's ``step_euler`` (models/npa.py:168-204) and
works on the reference's ``NPA`` module unchanged (it reads ``model.model``, ``alpha``, ``eps0``,
``spatial_dims`` and the perception flags), but runs

    grid build -> reorder -> packed perception (two neighbour sweeps) -> model.model (torch GEMMs,
    weight gradients by one fused kernel)
    -> fused limiter + update (+ wrap)

instead of five neighbour sweeps and ~25 elementwise torch kernels.  Values and gradients are
those of ``NPA.forward`` followed by the reference's update (tests/test_gpu_step_update.py).
"""
from __future__ import annotations

import math

import torch

from . import sphops as sph
from .sphops import sph as sph_ops
from .mlp import apply_mlp, on_tensor_memory


def _scalar(v) -> float:
    return float(v.item()) if isinstance(v, torch.Tensor) else float(v)


def _buffer_scalar(model, name) -> float:
    """``model.<name>`` (a one-element buffer such as ``eps0`` or ``alpha``) as a Python float, read from
    the device once and cached on the module until the buffer is modified in place or replaced: a step
    then makes no device-to-host copy (the reference keeps these as device tensors and never syncs)."""
    v = getattr(model, name)
    if not isinstance(v, torch.Tensor):
        return float(v)
    cache = model.__dict__.setdefault("_npa_b200_scalars", {})
    hit = cache.get(name)
    if hit is not None and hit[0] is v and hit[1] == v._version:
        return hit[2]
    value = float(v.item())
    cache[name] = (v, v._version, value)
    return value


class _FrozenView:
    """The attributes of an NPA module that a step reads, with ``eps0`` and ``alpha`` as Python floats."""

    def __init__(self, model):
        self.model = model.model
        self.eps0, self.alpha = _scalar(model.eps0), _scalar(model.alpha)
        self.spatial_dims = model.spatial_dims
        for flag, default in (("state_grad", True), ("density_grad", True), ("log_norm_grad", True),
                              ("log_norm_density_grad", True), ("stopgrad_pos", True), ("stopgrad_state", False)):
            setattr(self, flag, getattr(model, flag, default))
        self.last_snapshot = None


def frozen_view(model):
    """A stand-in for ``model`` whose scalar buffers were read once: ``step_euler`` on it makes no
    device-to-host copy, which a step recorded in a CUDA graph must not."""
    return model if isinstance(model, _FrozenView) else _FrozenView(model)


def perceive(model, x, s, grid):
    """``NPA.perceive`` (models/npa.py:87-137) on the packed perception call; returns
    ``(z, x_bin, s_bin, snapshot)`` like the reference."""
    if not (getattr(model, "state_grad", True) and getattr(model, "density_grad", True)):
        raise NotImplementedError("the packed perception covers state_grad=True, density_grad=True "
                                  "(every shipped configuration); use the per-operator API otherwise")
    with torch.no_grad():
        snapshot = grid.instantiate(x)
    x_bin, s_bin = sph.bin_particles(x, s, snapshot)
    x_perceive = x_bin.detach() if getattr(model, "stopgrad_pos", True) else x_bin
    s_perceive = s_bin.detach() if getattr(model, "stopgrad_state", False) else s_bin
    z = sph.perceive_features(x_perceive, s_perceive, snapshot, _buffer_scalar(model, "eps0"),
                              log_norm_grad=getattr(model, "log_norm_grad", True),
                              log_norm_density_grad=getattr(model, "log_norm_density_grad", True))
    return z, x_bin, s_bin, snapshot


def _one_node(model, x, s, grid) -> bool:
    """Whether a step of this model is covered by the single autograd node: the adaptation MLP on the default
    engine, gradient features on, rows one warp pass covers, neighbour lists on, single precision by default."""
    C, module = s.shape[-1], model.model
    if not (getattr(model, "state_grad", True) and getattr(model, "density_grad", True) and sph_ops.packable(C)
            and sph_ops._columns(grid.hashgrid) > 0 and on_tensor_memory(module)):
        return False
    if torch.get_default_dtype() != torch.float32:  # the update mask is drawn in the default type
        return False
    first, _, last = module
    return (first.weight.device == x.device and first.in_features == 2 * C + C * grid.dim + grid.dim
            and last.out_features == grid.dim + C)


def step_euler(model, x, s, grid, dt=1.0, update_prob=0.5, intermediate=False, noise_std=0.0, wrap=False):
    """``x, s, stats`` after one step; the particles come back in cell order, as in the reference.

    ``wrap=True`` additionally applies ``grid.wrap_positions`` (the reference's trainers call it
    after the rollout, train.py:238); the 3D padding column is kept either way.
    """
    B, N, C = s.shape
    alpha = _buffer_scalar(model, "alpha")
    stats = None
    if not intermediate and _one_node(model, x, s, grid):
        first, _, last = model.model
        x_new, s_new, model.last_snapshot, uniforms = sph_ops.euler_step(
            grid, x, s, (first.weight, first.bias, last.weight), _buffer_scalar(model, "eps0"), alpha, dt, update_prob, wrap,
            getattr(model, "log_norm_grad", True), getattr(model, "log_norm_density_grad", True),
            getattr(model, "stopgrad_pos", True), getattr(model, "stopgrad_state", False))
    else:
        z, x_bin, s_bin, snapshot = perceive(model, x, s, grid)
        model.last_snapshot = snapshot
        y = apply_mlp(model.model, z)  # (B, N, dim + C)
        if intermediate:
            d = y[..., : model.spatial_dims]
            dx = alpha * d * grid.eps / (1.0 + d.norm(dim=-1, keepdim=True))
            stats = {"dx_norm": dx.norm(dim=-1).mean()}
        uniforms = torch.rand(B, N, 1, device=x.device) if update_prob < 1.0 else None
        if uniforms is None:
            x_new, s_new = sph.step_update(y, x_bin, s_bin, snapshot, alpha, dt, None, wrap)
        else:
            x_new, s_new = sph_ops.step_update_where(y, x_bin, s_bin, snapshot, alpha, dt, uniforms, update_prob, wrap)
    if noise_std > 0:
        noise = torch.randn_like(x_new) * noise_std * math.sqrt(dt)
        x_new = x_new + (noise if uniforms is None else noise * (uniforms < update_prob).float())
    return x_new, s_new, stats
