"""The ``sphops`` operator API on top of the B200 kernels.

Same public names, signatures, defaults and autograd behaviour as the
reference's ``sphops/sph.py`` (HashGrid :42-123, Permute :127-184,
unbin_particles :187-198, Count :201-229, Density :232-267, Blur :270-321,
Gradient :324-376, DensityGradient :379-413, MomentMatrix :416-464,
safe_inv_sym_mat :467-471, gradient_hybrid :474-484), so ``models/npa.py`` and
the trainers of the reference run unchanged on it.  Two additions that the
reference does not have: :func:`perceive`, the fused forward/backward of the
whole perception step, and the ``device`` argument of :class:`HashGrid`.

Semantics kept from the reference: default mass is 1.0 per particle; ``rho`` is
a density and the operators form ``mass / rho`` themselves; 3D positions are
``[B, N, 4]`` with an ignored fourth column whose gradient is 0; gradients of
inputs that do not require grad are returned as ``None``.
"""
from __future__ import annotations

import math
import weakref
from dataclasses import dataclass, field

import torch

from . import sph_cuda
from .._native import ops as _ops


def _mass(mass):
    """``[B, N]`` masses (a trailing axis of one is dropped), or None = 1.0 per particle."""
    return mass.squeeze(-1) if mass is not None and mass.dim() == 3 and mass.shape[-1] == 1 else mass


_GRID_CLASSES = {
    (2, "periodic", "grid"): "HashGrid2DPeriodic",
    (3, "periodic", "grid"): "HashGrid3DPeriodic",
    (2, "clamped", "grid"): "HashGrid2DBox",
    (3, "clamped", "grid"): "HashGrid3DBox",
    (2, "periodic", "particle"): "VHashGrid2DPeriodic",
    (3, "periodic", "particle"): "VHashGrid3DPeriodic",
    (2, "clamped", "particle"): "VHashGrid2DBox",
    (3, "clamped", "particle"): "VHashGrid3DBox",
}


def get_hashgrid_cls(dim, boundary, mode):
    return getattr(sph_cuda, _GRID_CLASSES[(dim, boundary, mode)])


@dataclass
class HashGridSnapshot:
    """Result of one binning pass; every tensor a later operator needs lives here."""

    grid: object
    bin_offsets: torch.Tensor
    permutation: torch.Tensor
    block_info: torch.Tensor
    dim: int
    # outputs computed ahead of their call by a fused sweep (see enable_fusion); not part of the
    # reference's dataclass, defaulted so positional construction still works
    parked: dict = field(default_factory=dict, repr=False, compare=False)
    # neighbour lists of the positions the last density sweep saw: (key, tensor), see _lists_of
    lists: tuple = field(default=None, repr=False, compare=False)

    def __getstate__(self):
        # what is kept for tensor objects of this process (by weak reference) is of no use to a copy
        return {**self.__dict__, "parked": {}, "lists": None}


class HashGrid:
    """Uniform grid over ``[-G*eps/2, G*eps/2)`` per axis, cell size = cut-off ``eps``.

    ``mode="grid"`` orders cells linearly, ``mode="particle"`` along a Morton
    curve (power-of-two sizes only); both run the same kernels here.
    ``max_particles_per_block`` bounds the particles of one work item.
    """

    def __init__(self, dim=2, boundary="periodic", mode="grid", grid_size=(16, 16), eps=0.1,
                 num_particles=4096, batch_size=8, max_particles_per_block=64, device=None):
        self.dim = dim
        self.boundary = boundary
        self.mode = mode
        self.grid_size = grid_size
        self.eps = eps
        self.num_particles = num_particles
        self.batch_size = batch_size
        self.max_particles_per_block = max_particles_per_block
        if mode == "particle":
            for size in grid_size:
                assert (size & (size - 1)) == 0, "grid_size must be a power of 2"
        self.num_cells = math.prod(grid_size)
        self.hashgrid_cls = get_hashgrid_cls(dim, boundary, mode)
        self.hashgrid = self.hashgrid_cls(*grid_size, eps, num_particles, batch_size, max_particles_per_block)
        self.device = torch.device("cuda") if device is None else torch.device(device)
        self._last_snapshot = None

    def instantiate(self, x):
        """Bin positions ``x [B, N, P]`` and return the snapshot the operators take."""
        return self.adopt(*_ops.instantiate(self.hashgrid.native, x))

    def adopt(self, bin_offsets, permutation, block_info):
        """The snapshot of a binning pass whose arrays are there already."""
        # outputs a fused sweep parked on the previous snapshot and nobody claimed, and its neighbour lists, are
        # dropped now: they would otherwise live (with the autograd graph they hang on) as long as that snapshot does
        previous = self._last_snapshot() if self._last_snapshot is not None else None
        if previous is not None:
            previous.parked.clear()
            previous.lists = None
        snapshot = HashGridSnapshot(grid=self.hashgrid, bin_offsets=bin_offsets, permutation=permutation,
                                    block_info=block_info, dim=self.dim)
        self._last_snapshot = weakref.ref(snapshot)
        return snapshot

    def wrap_positions(self, x):
        """Periodic: map each of the ``dim`` coordinates into ``[-L/2, L/2)``; clamped: identity."""
        if self.boundary != "periodic":
            return x
        cols = []
        for d in range(self.dim):
            L = torch.tensor(self.grid_size[d] * self.eps, device=x.device)
            cols.append(torch.remainder(x[..., d] + 0.5 * L, L) - 0.5 * L)
        return torch.stack(cols, dim=-1)


# ---------------------------------------------------------------------------------------------
# Operator fusion behind the per-operator API.
#
# NPA.perceive (models/npa.py:105-126) calls density, blur, moment_matrix, gradient and
# density_gradient one after the other with the SAME tensor objects; each is a full sweep over the
# neighbour cells in the reference.  With fusion enabled, density() also computes the density
# gradient and blur() also computes the feature gradient and the moment matrix, in the same sweep,
# and parks the extra outputs on the snapshot; the later call returns the parked tensor when it
# is made with the very same input objects (identity and version), otherwise it runs its own
# kernel as usual.  Five sweeps become two, and autograd sees one node per sweep, so the backward
# is fused too.  Off by default: a caller that only wants blur would pay for the gradient.
# ---------------------------------------------------------------------------------------------
_FUSION = {"enabled": False}
# Columns of the neighbour lists the density sweep records for the other sweeps of its snapshot
# (row = count, j_0, j_1, ...; particles with more neighbours are searched again); 0 = off, None = by the grid.
_PAIR_CACHE = {"columns": None}


def set_pair_cache(columns=128):
    """Length of the per-particle neighbour lists that the sweeps of a snapshot share (4 * columns bytes
    per particle while the snapshot or the autograd graph is alive); 0 disables them, None is the default: by the
    number of neighbours that the grid's mean density gives, and for the density, ``perceive`` and the single operators up to 512
    as long as the lists of a call take at most 128 MiB.  A backward through many recorded steps of those keeps the lists of all of
    them: ``set_pair_cache(128)`` bounds them at 512 bytes per particle and step, for more time where particles have more neighbours."""
    columns = None if columns is None else int(columns)
    if columns is not None and columns != 0 and not 2 <= columns <= 513:
        raise ValueError("columns must be 0 or between 2 and 513")
    _PAIR_CACHE["columns"] = columns


def _columns(grid):
    set_by_user = _PAIR_CACHE["columns"]
    return grid.list_columns if set_by_user is None else set_by_user


def _roomy_columns(grid):
    set_by_user = _PAIR_CACHE["columns"]
    return grid.roomy_list_columns if set_by_user is None else set_by_user


def _lists_of(snapshot, x_bin):
    """Neighbour lists recorded on this snapshot for the very same positions object, or None."""
    return snapshot.lists[1] if snapshot.lists is not None and _same(snapshot.lists[0], x_bin) else None


def _density(x_bin, mass, snapshot, want_density_gradient):
    """``(rho, density gradient or None)``, with neighbour lists for the backward and for the later operators on the same
    positions.  Every call records its own lists: positions can change without a new version (a replayed CUDA graph, a
    kernel that writes through the pointer, ``.data``), and then the density is computed anew as well.  The snapshot
    gets the lists when the sweep that fills them has been issued, never before."""
    key = _key(x_bin)
    columns = _roomy_columns(snapshot.grid) if key is not None else 0
    pairs = torch.empty(*x_bin.shape[:2], columns, dtype=torch.int32, device=x_bin.device) if columns else None
    out = _ops.density(*_sweep_args(snapshot), x_bin, mass, pairs, True, want_density_gradient, columns > 0)
    snapshot.lists = (key, pairs) if columns else None
    return out


def _sweep_args(snapshot):
    return snapshot.grid.native, snapshot.bin_offsets, snapshot.block_info


def enable_fusion(flag=True):
    """Turn speculative sibling-output fusion of the per-operator API on or off (process wide)."""
    _FUSION["enabled"] = bool(flag)


def fusion_enabled():
    return _FUSION["enabled"]


def _key(*tensors):
    """Identity + version of the input tensor objects (None allowed), held weakly: a parked output never
    keeps its inputs alive, and an input that has died can never match again.  None when one of them is an
    inference tensor: those have no version, a change in place would go unnoticed."""
    try:
        return tuple((None if t is None else weakref.ref(t), None if t is None else t._version) for t in tensors)
    except RuntimeError:  # "Inference tensors do not track version counter"
        return None


def _same(key, *tensors):
    return len(key) == len(tensors) and all(
        (t is None and kt is None) or (t is not None and kt is not None and kt() is t and kv == t._version)
        for (kt, kv), t in zip(key, tensors))


def _park(snapshot, name, key, value):
    if key is not None:
        snapshot.parked[name] = (key, value)


def _claim(snapshot, name, *tensors):
    entry = snapshot.parked.get(name)
    if entry is None or not _same(entry[0], *tensors):
        return None
    del snapshot.parked[name]
    return entry[1]


class DensityPair:
    """density and density_gradient of the same positions in one sweep."""

    @staticmethod
    def apply(x_bin, mass, snapshot):
        return _density(x_bin, mass, snapshot, True)


class BlurGradient:
    """blur, feature gradient and (not differentiated) moment matrix in one sweep."""

    @staticmethod
    def apply(x_bin, s_bin, rho, mass, snapshot):
        pairs = _lists_of(snapshot, x_bin)
        return _ops.blur_gradient(*_sweep_args(snapshot), x_bin, rho, s_bin, mass, pairs, pairs is not None, True, True, True)


class Permute:
    """Reorder into cell order (gradients: the inverse reorder)."""

    @staticmethod
    def apply(x, s, mass, snapshot):
        return _ops.reorder(snapshot.grid.native, snapshot.permutation, x, s, mass)


def bin_particles(x, s, snapshot, mass=None):
    return Permute.apply(x, s, _mass(mass), snapshot)


def unbin_particles(x_bin, s_bin, snapshot, mass_bin=None):
    return _ops.unreorder(snapshot.grid.native, snapshot.permutation, x_bin, s_bin, _mass(mass_bin))


class Count:
    @staticmethod
    def apply(x_bin, snapshot):
        # a neighbour count is piecewise constant in the positions: its node gives no gradient
        return _ops.count(*_sweep_args(snapshot), x_bin)


def count(x_bin, snapshot):
    return Count.apply(x_bin, snapshot)


class Density:
    @staticmethod
    def apply(x_bin, mass, snapshot):
        return _density(x_bin, mass, snapshot, False)[0]


def density(x_bin, snapshot, mass=None):
    if _FUSION["enabled"]:
        rho, rho_grad = DensityPair.apply(x_bin, _mass(mass), snapshot)
        _park(snapshot, "density_gradient", _key(x_bin, mass), rho_grad)
        return rho
    return Density.apply(x_bin, _mass(mass), snapshot)


class Blur:
    @staticmethod
    def apply(x_bin, s_bin, rho, mass, snapshot):
        pairs = _lists_of(snapshot, x_bin)
        return _ops.blur_gradient(*_sweep_args(snapshot), x_bin, rho, s_bin, mass, pairs, pairs is not None, True, False, False)[0]


def blur(x_bin, rho, s_bin, snapshot, mass=None):
    if _FUSION["enabled"]:
        s_blur, s_grad, moment = BlurGradient.apply(x_bin, s_bin, rho, _mass(mass), snapshot)
        _park(snapshot, "gradient", _key(x_bin, rho, s_bin, mass), s_grad)
        _park(snapshot, "moment_matrix", _key(x_bin, rho, mass), moment)
        return s_blur
    return Blur.apply(x_bin, s_bin, rho, _mass(mass), snapshot)


class Gradient:
    @staticmethod
    def apply(x_bin, s_bin, rho, mass, snapshot):
        pairs = _lists_of(snapshot, x_bin)
        return _ops.blur_gradient(*_sweep_args(snapshot), x_bin, rho, s_bin, mass, pairs, pairs is not None, False, True, False)[1]


def gradient(x_bin, rho, s_bin, snapshot, mass=None):
    parked = _claim(snapshot, "gradient", x_bin, rho, s_bin, mass)
    if parked is not None:
        return parked
    return Gradient.apply(x_bin, s_bin, rho, _mass(mass), snapshot)


class DensityGradient:
    @staticmethod
    def apply(x_bin, mass, snapshot):
        return _ops.density(*_sweep_args(snapshot), x_bin, mass, _lists_of(snapshot, x_bin), False, True, False)[1]


def density_gradient(x_bin, snapshot, mass=None):
    parked = _claim(snapshot, "density_gradient", x_bin, mass)
    if parked is not None:
        return parked
    return DensityGradient.apply(x_bin, _mass(mass), snapshot)


class MomentMatrix:
    @staticmethod
    def apply(x_bin, rho, mass, snapshot):
        return _ops.moment_matrix(*_sweep_args(snapshot), x_bin, rho, mass)


def moment_matrix(x_bin, rho, snapshot, mass=None):
    # the parked matrix carries no autograd history: usable when none is wanted (gradient_hybrid)
    if not (torch.is_grad_enabled() and (x_bin.requires_grad or rho.requires_grad)):
        parked = _claim(snapshot, "moment_matrix", x_bin, rho, mass)
        if parked is not None:
            return parked
    return MomentMatrix.apply(x_bin, rho, _mass(mass), snapshot)


@torch.no_grad()
def safe_inv_sym_mat(M, rtol=1e-6):
    M_inv = torch.empty_like(M)
    sph_cuda.safe_inv_sym_mat(M, M_inv, rtol)
    return M_inv


def gradient_hybrid(x_bin, rho, s_bin, snapshot, mass=None):
    """Moment-corrected gradient: value ``raw @ inv(M)``, gradient of the raw SPH gradient."""
    pairs = _lists_of(snapshot, x_bin)
    if pairs is not None and "gradient" not in snapshot.parked:
        return _ops.gradient_hybrid(*_sweep_args(snapshot), x_bin, rho, s_bin, _mass(mass), pairs, 1e-3)
    with torch.no_grad():
        M = moment_matrix(x_bin, rho, snapshot, mass=mass)
    raw = gradient(x_bin, rho, s_bin, snapshot, mass=mass)
    return _ops.corrected_gradient(raw, M, 1e-3)


# ---------------------------------------------------------------------------------------------
# Fused perception step (extension; the reference issues one launch per operator).
# ---------------------------------------------------------------------------------------------
class Perception:
    """rho = density(x); blur(x, rho, s); gradient(x, rho, s); density_gradient(x) as one node.

    Forward runs two sweeps over the neighbour cells instead of four launches; backward runs the
    chained two-sweep backward, or the features-only variant when ``x_bin`` needs no gradient.
    """

    @staticmethod
    def apply(x_bin, s_bin, mass, snapshot, want_density_gradient):
        return _ops.perception(*_sweep_args(snapshot), x_bin, s_bin, mass, want_density_gradient, _roomy_columns(snapshot.grid))


def perceive(x_bin, s_bin, snapshot, mass=None, with_density_gradient=True):
    """Fused ``(rho, blur, gradient[, density_gradient])`` of binned particles.

    Equivalent to ``rho = density(x_bin, snapshot, mass)``, ``blur(x_bin, rho, s_bin, ...)``,
    ``gradient(x_bin, rho, s_bin, ...)`` and ``density_gradient(x_bin, ...)`` with gradients
    flowing through ``rho`` into ``x_bin``.
    """
    return Perception.apply(x_bin, s_bin, _mass(mass), snapshot, with_density_gradient)


class PerceiveFeatures:
    """The packed perception row of NPA.perceive (models/npa.py:87-137) as one autograd node."""

    @staticmethod
    def apply(x_bin, s_bin, mass, snapshot, coef, dg_scale, inv_tol, log_norm_grad, log_norm_dg):
        return _ops.packed_perception(*_sweep_args(snapshot), x_bin, s_bin, mass, coef, dg_scale, inv_tol, log_norm_grad, log_norm_dg,
                                      _columns(snapshot.grid))


def packable(C):
    """Whether one warp pass of the packed sweep covers rows of ``C`` features."""
    return (C % 4 == 0 and C <= 128) or C <= 32


def perceive_features(x_bin, s_bin, snapshot, eps0, mass=None, log_norm_grad=True, log_norm_density_grad=True,
                      inv_rtol=1e-3):
    """The perception vector ``z [B, N, 2C + C*dim + dim]`` an NPA model feeds its MLP, in two sweeps.

    Same value and gradients as the body of ``NPA.perceive`` with its defaults (state and density
    gradients on): ``[s | blur(s) | LN(coef * gradient_hybrid(s)) | LN(coef^(1+dim)/N * density_gradient)]``
    with ``coef = eps / eps0`` and ``LN(w) = log(1+|w|) w/|w|`` (skipped when the flag is False).
    Pass ``x_bin.detach()`` to stop gradients into the positions, as NPA does by default.
    """
    mass = _mass(mass)
    B, N, C = s_bin.shape
    coef = float(snapshot.grid.eps) / float(eps0)
    dg_scale = coef ** (1 + snapshot.dim) / N
    if not packable(C):
        # wider feature rows than one warp pass covers: same result from the separate operators
        def _ln(v):
            return torch.log(1.0 + v.norm(dim=-1, keepdim=True)) * torch.nn.functional.normalize(v, dim=-1)
        rho = density(x_bin, snapshot, mass)
        s_blur = blur(x_bin, rho, s_bin, snapshot, mass)
        with torch.no_grad():
            L = safe_inv_sym_mat(moment_matrix(x_bin, rho, snapshot, mass), rtol=inv_rtol)
        raw = gradient(x_bin, rho, s_bin, snapshot, mass)
        g = (raw + (raw @ L - raw).detach()) * coef
        dg = density_gradient(x_bin, snapshot, mass) * dg_scale
        if log_norm_grad:
            g = _ln(g)
        if log_norm_density_grad:
            dg = _ln(dg)
        return torch.cat([s_bin, s_blur, g.reshape(B, N, -1), dg], dim=-1)
    return PerceiveFeatures.apply(x_bin, s_bin, mass, snapshot, coef, dg_scale, float(inv_rtol),
                                  bool(log_norm_grad), bool(log_norm_density_grad))


class StepUpdate:
    """The Euler update of step_euler (models/npa.py:183-203) with the displacement limiter of
    NPA.forward (models/npa.py:145-153) as one elementwise kernel and one autograd node."""

    @staticmethod
    def apply(y, x_bin, s_bin, mask, snapshot, alpha, dt, wrap):
        return _ops.step_update(snapshot.grid.native, y, x_bin, s_bin, mask, alpha, dt, wrap, -1.0)


def step_update(y, x_bin, s_bin, snapshot, alpha, dt=1.0, update_mask=None, wrap=False):
    """``(x, s)`` after one Euler step, from the MLP output ``y [B, N, dim + C]`` in cell order.

    ``dx = alpha * y[..., :dim] * eps / (1 + |y[..., :dim]|)``, ``x = x_bin + dt * dx * mask`` (the 3D
    padding column is carried over), ``s = s_bin + dt * y[..., dim:] * mask``; ``update_mask`` is the
    reference's ``(rand(B, N, 1) < update_prob).float()`` (or None); ``wrap=True`` also applies
    ``HashGrid.wrap_positions`` on a periodic grid (keeping the padding column).
    """
    if update_mask is not None:
        update_mask = update_mask.reshape(y.shape[0], y.shape[1]).to(torch.float32).contiguous()
    return StepUpdate.apply(y.contiguous(), x_bin.contiguous(), s_bin.contiguous(), update_mask, snapshot,
                            float(alpha), float(dt), bool(wrap))


def step_update_where(y, x_bin, s_bin, snapshot, alpha, dt, uniforms, update_prob, wrap=False):
    """``step_update`` with ``update_mask = (uniforms < update_prob).float()``, the comparison made in the kernel."""
    if uniforms.dtype != torch.float32 or not update_prob >= 0.0:  # (the kernel's threshold; negative: the mask itself)
        return step_update(y, x_bin, s_bin, snapshot, alpha, dt, (uniforms < update_prob).float(), wrap)
    return _ops.step_update(snapshot.grid.native, y.contiguous(), x_bin.contiguous(), s_bin.contiguous(),
                            uniforms.reshape(y.shape[0], y.shape[1]), float(alpha), float(dt), bool(wrap), float(update_prob))


def euler_step(grid, x, s, weights, eps0, alpha, dt, update_prob, wrap, log_norm_grad, log_norm_density_grad, stopgrad_pos,
               stopgrad_state, inv_rtol=1e-3):
    """``instantiate``, ``bin_particles``, ``perceive_features``, the MLP ``weights`` = (W1, b1, W2) and ``step_update`` as
    one call and one autograd node: ``(x_new, s_new, snapshot, uniforms of the update mask or None)``."""
    coef = float(grid.eps) / float(eps0)
    x_new, s_new, bin_offsets, permutation, block_info, uniforms = _ops.euler_step(
        grid.hashgrid.native, x, s, *weights, coef, coef ** (1 + grid.dim) / x.shape[1], float(inv_rtol), bool(log_norm_grad),
        bool(log_norm_density_grad), bool(stopgrad_pos), bool(stopgrad_state), float(alpha), float(dt), float(update_prob), bool(wrap),
        _columns(grid.hashgrid))
    return x_new, s_new, grid.adopt(bin_offsets, permutation, block_info), uniforms
