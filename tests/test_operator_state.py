"""What the operators keep between calls, on the host: no kernel is launched."""
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
