"""What the operators keep between calls, on the host: no kernel is launched."""
import copy
import pickle

import pytest
import torch

from npa_b200 import sphops as sph


def _grid(dim=2, B=2, N=16, **kw):
    return sph.HashGrid(dim=dim, boundary="clamped", mode="grid", grid_size=(8,) * dim, eps=0.1, num_particles=N,
                        batch_size=B, **kw)


def _snapshot(grid):
    B = grid.batch_size
    return sph.HashGridSnapshot(grid=grid.hashgrid, bin_offsets=torch.zeros(B * grid.num_cells + 1, dtype=torch.int32),
                                permutation=None, block_info=torch.zeros(grid.hashgrid.max_blocks, 4, dtype=torch.int32), dim=grid.dim)


@pytest.mark.parametrize("fused", [False, True])
def test_a_refused_density_leaves_no_lists_behind(fused):
    """Lists that no sweep has filled must not be found by the next operator: their entries are indices."""
    grid = _grid()
    snap = _snapshot(grid)
    sph.enable_fusion(fused)
    try:
        with pytest.raises((TypeError, RuntimeError)):
            sph.density(torch.zeros(2, 16, 2), snap)       # CPU tensors are refused before any launch
    finally:
        sph.enable_fusion(False)
    assert snap.lists is None


class _Ops:
    """Stands in for the native operators: records the lists a density is given."""

    def __init__(self):
        self.recorded = []

    def density(self, grid, offs, info, x, mass, pairs, want_rho, want_dg, record):
        self.recorded.append((pairs, record))
        return torch.zeros(x.shape[:2]), torch.zeros(*x.shape[:2], 2) if want_dg else None


@pytest.mark.parametrize("fused", [False, True])
def test_density_of_inference_tensors(monkeypatch, fused):
    """Inference tensors have no version to compare: they are computed with, but nothing is kept for them."""
    from npa_b200.sphops import sph as impl

    ops = _Ops()
    monkeypatch.setattr(impl, "_ops", ops)
    snap = _snapshot(_grid())
    sph.enable_fusion(fused)
    try:
        with torch.inference_mode():
            assert impl.density(torch.zeros(2, 16, 2), snap).shape == (2, 16)
    finally:
        sph.enable_fusion(False)
    assert ops.recorded == [(None, False)] and snap.lists is None and not snap.parked


def test_every_density_records_its_own_lists(monkeypatch):
    """Positions may change without a new tensor version (a replayed graph, a raw pointer): a second density on the same
    tensor object must not take the lists of the first."""
    from npa_b200.sphops import sph as impl

    ops = _Ops()
    recorded = ops.recorded
    monkeypatch.setattr(impl, "_ops", ops)
    snap, x = _snapshot(_grid()), torch.zeros(2, 16, 2)
    for _ in range(2):
        impl.density(x, snap)
        assert recorded[-1][1] and snap.lists[1] is recorded[-1][0]
    assert recorded[0][0] is not recorded[1][0]
    sph.set_pair_cache(0)
    try:
        impl.density(x, snap)          # lists switched off in between: the old ones are not left behind either
        assert recorded[-1] == (None, False) and snap.lists is None
    finally:
        impl._PAIR_CACHE["columns"] = None


@pytest.mark.parametrize("duplicate", [copy.deepcopy, lambda o: pickle.loads(pickle.dumps(o))], ids=["deepcopy", "pickle"])
def test_grids_and_snapshots_are_copied_and_pickled(duplicate):
    """A model that holds a grid or its last snapshot is copied (for a moving average) and saved whole."""
    from npa_b200.sphops import sph as impl

    grid = _grid(dim=3, N=600)
    twin = duplicate(grid)
    assert twin.hashgrid is not grid.hashgrid and twin.hashgrid.max_blocks == grid.hashgrid.max_blocks
    assert twin.hashgrid.native is not grid.hashgrid.native and twin.hashgrid.list_columns == grid.hashgrid.list_columns
    snap, x = _snapshot(grid), torch.zeros(2, 600, 4)
    snap.lists = (impl._key(x), torch.zeros(2, 600, 128, dtype=torch.int32))
    snap.parked["gradient"] = (impl._key(x), torch.zeros(1))
    other = duplicate(snap)
    assert other.lists is None and other.parked == {} and torch.equal(other.bin_offsets, snap.bin_offsets)
    assert snap.lists is not None and other.grid.cell_count == 512


def test_forward_mode_derivatives_are_refused():
    """An operator without a forward-mode derivative must not drop the tangent of a dual number."""
    from torch.autograd import forward_ad
    from npa_b200 import _native

    grid, f = _grid(), torch.zeros
    snap = _snapshot(grid)
    sweep = (grid.hashgrid.native, snap.bin_offsets, snap.block_info)
    with forward_ad.dual_level():
        def dual(*shape):
            return forward_ad.make_dual(f(*shape), torch.ones(*shape))

        x, s, rho = dual(2, 16, 2), f(2, 16, 4), f(2, 16)
        calls = {
            "reorder": (grid.hashgrid.native, f(2, 16, dtype=torch.int32), x, s, None),
            "count": (*sweep, x),
            "density": (*sweep, x, None, None, True, False, False),
            "blur_gradient": (*sweep, f(2, 16, 2), dual(2, 16), s, None, None, False, True, False, False),
            "gradient_hybrid": (*sweep, x, rho, s, None, f(2, 16, 128, dtype=torch.int32), 1e-3),
            "moment_matrix": (*sweep, x, rho, None),
            "corrected_gradient": (dual(2, 16, 4, 2), f(2, 16, 2, 2), 1e-3),
            "perception": (*sweep, f(2, 16, 2), dual(2, 16, 4), None, True, 128),
            "packed_perception": (*sweep, x, s, None, 1.0, 1.0, 1e-3, True, True, 128),
            "step_update": (grid.hashgrid.native, dual(2, 16, 6), f(2, 16, 2), s, None, 1.0, 1.0, False, -1.0),
            "mlp": (f(32, 8), dual(128, 8), f(128), f(4, 128)),
            "euler_step": (grid.hashgrid.native, x, s, f(128, 18), f(128), f(6, 128), 1.0, 1.0, 1e-3, True, True, True, False, 1.0, 1.0,
                           0.5, False, 128),
            "splat": (dual(2, 16, 2), f(2, 16, 3), 32, 1.0, 5, -1.0, 1.0, False, False, 1.0)}
        for name, args in calls.items():
            with pytest.raises(NotImplementedError, match="forward-mode"):
                getattr(_native.ops, name)(*args)


def test_the_move_kernel_takes_only_fields_of_the_shapes_it_reads():
    """The kernel reads dim x modes products and phases by pointer: parameters that torch would broadcast, refuse or record stay
    with the tensor operations."""
    from npa_b200.rollout import PerceptionRollout, VelocityField, _writable

    class Another(VelocityField):
        pass

    def native(change=lambda field: None, kind=VelocityField, modes=8):
        field = kind(2, torch.device("cpu"), modes=modes)
        roll = PerceptionRollout(_grid(), 4, 2, 0.1, field)
        change(field)
        return roll._native_move()

    assert native() and native(modes=64)
    assert not native(modes=65) and not native(kind=Another)
    assert not native(lambda f: setattr(f, "phase", f.phase[:1]))            # broadcast over the modes
    assert not native(lambda f: setattr(f, "phase", torch.zeros(9)))
    assert not native(lambda f: setattr(f, "phase", f.phase.view(2, 4)))
    assert not native(lambda f: setattr(f, "k_t", f.k_t[:, :7].contiguous()))
    assert not native(lambda f: setattr(f, "k_t", torch.zeros(3, 8)))
    assert not native(lambda f: setattr(f, "amp", torch.zeros(7, 2)))
    assert not native(lambda f: setattr(f, "amp", f.amp.t().contiguous()))
    assert not native(lambda f: setattr(f, "amp", f.amp.double()))
    assert not native(lambda f: f.amp.requires_grad_(True))
    assert not native(lambda f: setattr(f, "amp", torch._neg_view(f.amp)))
    # positions and states
    x = torch.zeros(2, 3)
    with torch.inference_mode():
        inference = torch.zeros(2, 3)
        assert _writable(inference)
    leaf = torch.zeros(2, 3, requires_grad=True)
    with torch.no_grad():
        view = leaf[:1]
    assert _writable(x) and _writable(x[:1]) and not _writable(inference) and not _writable(leaf) and not _writable(view)


@pytest.mark.parametrize("dim", [2, 3])
def test_memory_of_the_default_lists(dim):
    """Longer lists than 128 columns stay below 128 MiB for a call, so that a recorded step never keeps over 96 MiB more than with 128;
    a setting of the user's is taken as it is."""
    from npa_b200.sphops import sph as impl
    for B, N in ((1, 16), (64, 512), (8, 4096), (3, 5001), (1, 65536), (8, 16384), (1, 131073), (4, 65536), (16, 65536), (2, 1 << 20)):
        cells = max(3, round((N / (16 if dim == 2 else 8)) ** (1.0 / dim)))
        grid = sph.HashGrid(dim=dim, boundary="clamped", mode="grid", grid_size=(cells,) * dim, eps=1.0 / cells, num_particles=N, batch_size=B).hashgrid
        if grid.list_columns > 128:
            assert grid.roomy_list_columns == grid.list_columns
            continue
        columns, narrow = grid.roomy_list_columns, 4 * 128 * B * N
        assert 128 <= columns <= 512 and (columns == 128 or 4 * columns * B * N <= 128 << 20)
        assert 4 * columns * B * N - narrow <= 96 << 20
        try:
            sph.set_pair_cache(128)
            assert impl._roomy_columns(grid) == impl._columns(grid) == 128
        finally:
            sph.set_pair_cache(None)
        assert impl._roomy_columns(grid) == columns and impl._columns(grid) == 128
