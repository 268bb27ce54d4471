"""Operators given other positions than the ones that were binned (a perturbed copy on the same snapshot), and positions where
the cell's image is not what the coordinate says: on the edge of a periodic box, and outside it."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _make(dim, boundary, mode, B, N, cells, seed=0):
    from npa_b200 import sphops as sph
    h = 1.0 / cells
    grid = sph.HashGrid(dim=dim, boundary=boundary, mode=mode, grid_size=(cells,) * dim, eps=h, num_particles=N, batch_size=B)
    g = torch.Generator().manual_seed(seed)
    x = torch.rand(B, N, dim, generator=g) - 0.5
    return sph, grid, h, x, g


def _padded(x):
    return torch.cat([x, torch.zeros_like(x[..., :1])], dim=-1).cuda().contiguous() if x.shape[-1] == 3 else x.cuda().contiguous()


def _pairs(x, h, periodic):
    """(r^2 < h^2 with a little less, with a little more) of all pairs of a system, minimum image of the unit box, fp64."""
    d = x[:, None, :] - x[None, :, :]
    if periodic:
        d = d - torch.round(d)
    q = (d * d).sum(-1)
    return q, q < h * h * (1 - 1e-5), q < h * h * (1 + 1e-5)


def _density(q, inside, h, dim):
    c = 4 / (np.pi * h ** 8) if dim == 2 else 315 / (64 * np.pi * h ** 9)
    return c * (torch.clamp(h * h - q, min=0) ** 3 * inside).sum(1)


@pytest.mark.parametrize("dim,boundary,mode", [(2, "clamped", "grid"), (2, "periodic", "grid"), (3, "clamped", "grid"), (3, "periodic", "grid"),
                                               (2, "clamped", "particle"), (3, "periodic", "particle")])
@pytest.mark.parametrize("B", [3, 20])         # below and above the switch between the two searches
def test_candidates_are_those_around_the_binned_cell(dim, boundary, mode, B):
    from npa_b200.sphops import sph as impl
    N, cells = 1001, 8
    sph, grid, h, x, g = _make(dim, boundary, mode, B, N, cells)
    periodic = boundary == "periodic"
    snap = grid.instantiate(_padded(x))
    xb, sb = sph.bin_particles(_padded(x), torch.zeros(B, N, 1, device="cuda"), snap)
    moved = xb.clone()
    moved[..., :dim] += (torch.rand(B, N, dim, generator=g).cuda() - 0.5) * 0.8 * h
    count, rho = sph.count(moved, snap).cpu().double(), sph.density(moved, snap).cpu().double()
    z = sph.perceive_features(moved, sb, snap, h)         # the search of the packed perception
    rho2 = sph.perceive(moved, sb, snap)[0].cpu().double()
    sph.set_pair_cache(4)                                  # lists that overflow: every sweep searches
    try:
        z2 = sph.perceive_features(moved, sb, snap, h)
        rho3, blur3, grad3, dg3 = sph.perceive(moved, sb + 1.0, snap)
    finally:
        impl._PAIR_CACHE["columns"] = None
    assert torch.allclose(z2, z, rtol=1e-4, atol=1e-4 * float(z.abs().max()))
    for b in range(B):
        cell = torch.floor(xb[b, :, :dim].cpu().double() * cells).long()
        gap = (cell[:, None, :] - cell[None, :, :]).abs()
        if periodic:
            gap = torch.minimum(gap, cells - gap)
        near = gap.max(-1).values <= 1                     # cells that every search has to look into
        q, less, more = _pairs(moved[b, :, :dim].cpu().double(), h, periodic)
        assert (count[b] >= (less & near).sum(1)).all() and (count[b] <= more.sum(1)).all()
        low, high = _density(q, near, h, dim), _density(q, torch.ones_like(near), h, dim)
        for r in (rho[b], rho2[b], rho3[b].cpu().double()):
            assert (r >= low * (1 - 1e-4)).all() and (r <= high * (1 + 1e-4)).all()


@pytest.mark.parametrize("dim,mode", [(2, "grid"), (3, "grid"), (2, "particle"), (3, "particle")])
@pytest.mark.parametrize("B", [2, 20])
@pytest.mark.parametrize("where", ["edge", "outside"])
def test_periodic_images_of_positions_on_the_edge_and_outside(dim, mode, B, where):
    """A coordinate of exactly half the box is binned into the first cell; one beyond it into the cell of its image."""
    N, cells = 997, 8
    sph, grid, h, x, g = _make(dim, "periodic", mode, B, N, cells, seed=4)
    some = torch.rand(B, N, dim, generator=g)
    if where == "edge":
        x = torch.where(some < 0.1, torch.full_like(x, 0.5), torch.where(some > 0.9, torch.full_like(x, -0.5), x))
    else:
        x = torch.where(some < 0.1, x + 1.0, torch.where(some > 0.9, x - 2.0, x))
    snap = grid.instantiate(_padded(x))
    xb, sb = sph.bin_particles(_padded(x), torch.randn(B, N, 4, generator=g).cuda(), snap)
    count, rho = sph.count(xb, snap).cpu().double(), sph.density(xb, snap).cpu().double()
    out = sph.perceive(xb, sb, snap)
    hat = sph.gradient_hybrid(xb, out[0], sb, snap)
    z = sph.perceive_features(xb, sb, snap, h, log_norm_grad=False)
    C = 4
    assert torch.allclose(z[..., C: 2 * C], out[1], rtol=1e-4, atol=1e-4 * float(out[1].abs().max()))
    assert torch.allclose(z[..., 2 * C: 2 * C + C * dim].reshape(hat.shape), hat, rtol=1e-3, atol=1e-4 * float(hat.abs().max()))
    for b in range(B):
        q, less, more = _pairs(xb[b, :, :dim].cpu().double(), h, True)
        assert (count[b] >= less.sum(1)).all() and (count[b] <= more.sum(1)).all()
        want = _density(q, torch.ones_like(less), h, dim)
        for r in (rho[b], out[0][b].cpu().double()):
            assert ((r - want).abs() <= 1e-4 * want).all()


@pytest.mark.parametrize("dim,B,N", [(3, 1, 65535), (3, 4, 16384), (2, 1, 3001)])   # either side of the count's dispatch
def test_counts_on_periodic_grids_against_brute_force(dim, B, N):
    cells = 16
    sph, grid, h, x, g = _make(dim, "periodic", "grid", B, N, cells, seed=9)
    snap = grid.instantiate(_padded(x))
    xb, _ = sph.bin_particles(_padded(x), torch.zeros(B, N, 1, device="cuda"), snap)
    count = sph.count(xb, snap)
    for b in range(B):
        p = xb[b, :, :dim].double()
        rows = torch.randint(0, N, (500,), generator=g).cuda()
        d = p[rows][:, None, :] - p[None, :, :]
        q = ((d - torch.round(d)) ** 2).sum(-1)
        assert (count[b][rows] >= (q < h * h * (1 - 1e-5)).sum(1)).all() and (count[b][rows] <= (q < h * h * (1 + 1e-5)).sum(1)).all()
