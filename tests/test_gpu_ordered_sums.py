"""The packed perception's sums in one fixed order (density_ordered.cu, packed_ordered.cuh): every branch of the density
search (tiles of one and of merged work items, a lane per candidate with 1, 2 and 4 classes), every row layout, lists that
overflow, runs of more than 96 neighbours, masses; against the operators one by one, whose kernels sum in another order."""
import pytest
import torch

from helpers import make_grid
from npa_b200.workloads import Workload, make_inputs

pytestmark = pytest.mark.gpu


def _log_normalize(v):
    return torch.log(1.0 + v.norm(dim=-1, keepdim=True)) * torch.nn.functional.normalize(v, dim=-1)


@pytest.mark.parametrize("dim,boundary,mode,B,N,cells,C,columns", [
    (2, "clamped", "grid", 3, 4097, 16, 16, 128),      # tiles
    (3, "clamped", "grid", 1, 20011, 28, 8, 128),      # tiles of merged work items
    (2, "clamped", "grid", 1, 1001, 10, 13, 128),      # a lane per candidate: 2 classes
    (3, "clamped", "grid", 2, 1501, 6, 30, 128),
    (2, "periodic", "grid", 1, 4099, 8, 20, 512),      # 1 class, ~200 neighbours
    (2, "periodic", "grid", 1, 200, 3, 5, 128),        # an axis of three cells
    (2, "periodic", "grid", 9, 1203, 16, 32, 24),      # tiles; most lists overflow
    (3, "periodic", "grid", 2, 2047, 5, 16, 128),      # 4 classes
    (3, "clamped", "particle", 2, 3001, 8, 32, 24),    # 4 classes; most lists overflow
    (2, "periodic", "particle", 2, 33, 4, 4, 128)])
def test_packed_perception_in_every_branch(dim, boundary, mode, B, N, cells, C, columns):
    from npa_b200 import sphops as sph
    from npa_b200.sphops import sph as ops
    w = Workload("ordered", dim=dim, B=B, N=N, C=C, eps=1.0 / cells, grid_size=(cells,) * dim, boundary=boundary, mode=mode)
    x, s, _ = make_inputs(w, seed=N)
    x[..., :dim] *= 0.99 / x[..., :dim].abs().max() * 0.5
    x[:, 1] = x[:, 0]                   # a coincident pair
    grid, eps0 = make_grid(sph, w), 0.07
    mass = (0.5 + torch.rand(B, N, generator=torch.Generator().manual_seed(3))).cuda()
    snap = grid.instantiate(x.cuda())
    xb, sb, mb = sph.bin_particles(x.cuda(), s.cuda(), snap, mass)
    before = ops._PAIR_CACHE["columns"]
    try:
        sph.set_pair_cache(columns)
        for m in (None, mb):
            rho = sph.density(xb, snap, m)
            grad = sph.gradient_hybrid(xb, rho, sb, snap, m) * (grid.eps / eps0)
            dg = sph.density_gradient(xb, snap, m) * ((grid.eps / eps0) ** (1 + dim)) / N
            want = torch.cat([sb, sph.blur(xb, rho, sb, snap, m), _log_normalize(grad).view(B, N, -1), _log_normalize(dg)], dim=-1)
            z = sph.perceive_features(xb, sb, snap, eps0, m)
            # fp32 sums of up to ~200 terms of both signs, and an inverse moment matrix: as for the fused sweeps
            assert torch.allclose(z, want, rtol=1e-4, atol=1e-5 * float(want.abs().max())), float((z - want).abs().max())
            again = sph.perceive_features(xb, sb.clone().requires_grad_(True), snap, eps0, m).detach()
            if columns <= 128:          # the same order whether a backward will follow or not
                assert torch.equal(again, z)
            else:                       # a recorded step searches for more than 127 neighbours anew
                assert torch.allclose(again, z, rtol=1e-4, atol=1e-5 * float(z.abs().max()))
    finally:
        ops._PAIR_CACHE["columns"] = before
