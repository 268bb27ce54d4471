"""Feature gradients of a step as dense products on the tensor cores (positions as binned), against float64 and the sums over lists."""
import ctypes
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


class Call:
    """The backward of the packed perception for given rows of dL/dz, by lists or as a step calls it."""

    def __init__(self, x, cells, eps, boundary, C, mass=None):
        from npa_b200 import _native as n, sphops as sph
        from npa_b200.sphops import sph as impl
        self.n, self.C, self.eps, self.boundary = n, C, eps, boundary
        self.B, self.N = x.shape[:2]
        self.dim = 2 if x.shape[2] == 2 else 3
        grid = sph.HashGrid(dim=self.dim, boundary=boundary, mode="grid", grid_size=(cells,) * self.dim, eps=eps, num_particles=self.N,
                            batch_size=self.B, max_particles_per_block=32)
        self.gd = n.make_grid(self.dim, boundary, "grid", (cells,) * self.dim, eps, self.B, self.N, 32)
        self.box = cells * eps
        s = torch.randn(self.B, self.N, C, device="cuda")
        self.snap = grid.instantiate(x)
        self.x, self.s, *m = sph.bin_particles(x, s, self.snap, *(() if mass is None else (mass,)))
        self.mass = m[0] if m else None
        Z, self.K = 2 * C + C * self.dim + self.dim, impl._columns(grid.hashgrid)
        e = lambda *shape, **kw: torch.empty(self.B, self.N, *shape, device="cuda", **kw)
        self.rho, self.dg, self.z, self.v, self.packed, self.pairs = e(), e(self.dim), e(Z), e(C, self.dim), e(4), e(self.K, dtype=torch.int32)
        self.st, p = n.current_stream(), n.ptr
        n.check(n.lib.npa_perceive_features_forward_lists(ctypes.byref(self.gd), C, p(self.x), p(self.mass), p(self.s), 1.0, 1.0, 1e-3, 0, 0, p(self.rho), p(self.dg),
                                                          p(self.z), p(self.v), p(self.packed), p(self.snap.bin_offsets), p(self.snap.block_info),
                                                          p(self.pairs), self.K, self.st))
        self.dz = torch.randn(self.B, self.N, Z, device="cuda")
        self.add = torch.randn(self.B, self.N, C, device="cuda")

    def __call__(self, binned, add=None):
        n, p = self.n, self.n.ptr
        f = n.lib.npa_perceive_features_backward_binned if binned else n.lib.npa_perceive_features_backward_lists
        nbytes = n.lib.npa_lists_backward_scratch_bytes(ctypes.byref(self.gd), self.C)
        work, out = torch.empty(nbytes // 4, device="cuda"), torch.full((self.B, self.N, self.C), float("nan"), device="cuda")
        n.check(f(ctypes.byref(self.gd), self.C, p(self.x), p(self.mass), p(self.s), p(self.rho), p(self.dg), p(self.v), p(self.packed), p(self.dz), 1.0, 1.0, 0, 0,
                  p(add), None, p(out), p(work), nbytes, p(self.snap.bin_offsets), p(self.pairs), self.K, self.st))
        return out

    def exact(self, b, idx):
        """Float64 value for particles ``idx`` of system ``b``, and the sum of the magnitudes of its terms with weights that bound how
        the rounding of a distance moves them: (h^2 - q)^3 by 3 (h^2 - q)^2 h^2, (h - d)^2 by 2 (h - d) h."""
        C, D = self.C, self.dim
        X, V, dz = self.x[b, :, :D].double(), 1.0 / self.rho[b].double(), self.dz[b].double()
        gB, gG = dz[:, C:2 * C], dz[:, 2 * C:2 * C + C * D].reshape(-1, C, D)
        f32 = lambda v: float(torch.tensor(v, dtype=torch.float32))
        h, h2 = f32(self.eps), f32(self.eps ** 2)
        cs = f32(4 / (math.pi * self.eps ** 8) if D == 2 else 315 / (64 * math.pi * self.eps ** 9))
        cg = f32(10 / (math.pi * self.eps ** 5) if D == 2 else 15 / (math.pi * self.eps ** 6))
        r = X[None] - X[idx][:, None]
        if self.boundary == "periodic":
            r = r - self.box * torch.round(r / self.box)
        q = (r * r).sum(-1)
        t, d = (h2 - q).clamp_min(0), (q + 1e-12).sqrt()
        near = (q > 0) & (q < h2)
        phi = torch.where(near, cg * 3 * (h - d).clamp_min(0) ** 2 / d, 0.0)
        wide = torch.where(near, cg * 6 * (h - d).clamp_min(0) * h / d, 0.0)
        K, Kw = phi[..., None] * r, wide[..., None] * r.abs()
        value = cs * t ** 3 @ gB - torch.einsum("ijd,jfd->if", K, gG)
        size = cs * 3 * h2 * t ** 2 @ gB.abs() + torch.einsum("ijd,jfd->if", Kw, gG.abs())
        T, Tw = torch.einsum("j,ijd->id", V, K), torch.einsum("j,ijd->id", V, Kw)
        own = lambda T, g: torch.einsum("id,ifd->if", T, g)
        return (value * V[idx, None] - own(T, gG[idx]) + dz[idx, :C], size * V[idx, None] + own(Tw, gG[idx].abs()) + dz[idx, :C].abs())


def _positions(dim, B, N, side, spread="uniform"):
    x = (torch.rand(B, N, dim, device="cuda") - 0.5) * side
    if spread == "lines":                                   # crowded cells beside empty ones
        x[..., 1:] = torch.round(x[..., 1:] * 4 / side) * side / 4 + 0.002 * torch.randn_like(x[..., 1:])
    if dim == 3:
        x = torch.cat([x, torch.zeros_like(x[..., :1])], -1)
    return x.contiguous()


# tiles of eight particles, blocks of sixteen features; a tile over the end of a row of cells and of a system; one particle, one tile and one more
@pytest.mark.parametrize("dim,B,N,cells,boundary,spread", [
    (2, 1, 9, 1, "clamped", "uniform"), (2, 3, 701, 6, "clamped", "uniform"), (2, 2, 4096, 16, "clamped", "lines"), (2, 3, 1003, 7, "periodic", "uniform"),
    (2, 1, 200, 4, "periodic", "uniform"), (3, 3, 6700, 9, "clamped", "uniform"), (3, 1, 20001, 11, "clamped", "lines")])
@pytest.mark.parametrize("C", [1, 4, 13, 16, 17, 32])
def test_against_float64(dim, B, N, cells, boundary, spread, C):
    torch.manual_seed(C)
    side = 1.0 if boundary == "periodic" else 0.97
    call = Call(_positions(dim, B, N, side, spread), cells, 1.0 / cells, boundary, C)
    got, lists = call(True), call(False)
    assert not torch.equal(got, lists)                      # two kernels
    assert torch.equal(call(True), got)                     # the same bits every time
    assert torch.allclose(call(True, call.add), got + call.add, rtol=1e-6, atol=0)
    for b in range(B):
        for idx in torch.arange(0, N, max(1, N // 300), device="cuda").split(64):
            want, size = call.exact(b, idx)
            # four roundings of a weight's distance, 2^-22 of the split operands, and of the sums
            assert ((got[b, idx].double() - want).abs() <= 16 * 2.0 ** -24 * size).all()


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan"), 3.0e38])
def test_rows_that_are_not_finite_reach_their_neighbours_only(value):
    torch.manual_seed(3)
    call = Call(_positions(2, 2, 700, 0.97), 6, 1 / 6, "clamped", 16)
    clean = call(True)
    call.dz[0, 100, 20] = call.dz[1, 350, 40] = value       # of the blur and of the gradient
    got, want = call(True), call(False)
    fine = torch.isfinite(want)
    assert torch.equal(torch.isfinite(got), fine)
    assert torch.allclose(got[fine], want[fine], rtol=2e-5, atol=1e-4) and (~fine).any() and fine.float().mean() > 0.9
    touched = (got != clean).any(-1)
    assert touched.float().mean() < 0.5


@pytest.mark.parametrize("dim,B,N,cells", [(2, 2, 700, 6), (3, 1, 20003, 12)])
@pytest.mark.parametrize("volume", [None, float("inf"), float("nan")])
def test_volumes_that_are_not_finite_reach_their_neighbours_only(dim, B, N, cells, volume):
    """A particle of no mass and no neighbour has the volume 0 / 0: particles beside it in memory that have no pair with it keep their sums,
    as over the lists."""
    torch.manual_seed(7)
    x = _positions(dim, B, N, 0.97)
    eps = 1 / cells
    alone = torch.tensor([0.49] * dim, device="cuda")
    x[(x[..., :dim] - alone).norm(dim=-1) < 1.01 * eps] *= 0.5                  # nobody in reach of the corner
    x[:, 5, :dim] = alone
    mass = 0.5 + torch.rand(B, N, device="cuda")
    mass[:, 5] = 0.0
    call = Call(x, cells, eps, "clamped", 16, mass)
    lone = (call.x[..., :dim] == alone).all(-1)
    assert int(lone.sum()) == B and bool(torch.isnan(call.packed[lone][:, 3]).all())
    if volume is not None:
        call.packed[..., 3][lone] = volume
    got, want = call(True), call(False)
    assert not torch.isfinite(got[lone]).any() and torch.isfinite(want[~lone]).all()
    assert torch.allclose(got[~lone], want[~lone], rtol=2e-5, atol=1e-4)


@pytest.mark.parametrize("dim,N,cells,boundary,C,most", [
    (2, 6144, 39, "clamped", 16, 1.0), (2, 6144, 39, "clamped", 32, 1.0), (2, 6144, 24, "periodic", 8, 1.0), (2, 6144, 16, "clamped", 13, 1.0),
    (3, 20480, 17, "clamped", 16, 1.0), (3, 20480, 13, "clamped", 32, 1.0),                          # 13 to 35 neighbours
    (2, 6144, 55, "clamped", 16, 1.05)])                                                             # 7
def test_error_is_not_larger_than_that_of_the_lists(dim, N, cells, boundary, C, most):
    """2-norm against float64: operands in two pieces and sums that the tensor cores truncate have to be as good as single precision."""
    torch.manual_seed(N + C)
    call = Call(_positions(dim, 1, N, 1.0), cells, 1.0 / cells, boundary, C)
    dense, lists = call(True), call(False)
    error = [0.0, 0.0]
    for idx in torch.arange(0, N, N // 6144, device="cuda").split(64):
        want, _ = call.exact(0, idx)
        for k, out in enumerate((dense, lists)):
            error[k] += float((out[0, idx].double() - want).square().sum())
    assert 0 < error[0] ** 0.5 <= most * error[1] ** 0.5


# per cell, particles and features on either side of the lines
@pytest.mark.parametrize("dim,boundary,cells,N,C,dense", [
    (2, "clamped", 40, 3200, 16, True), (2, "clamped", 40, 3199, 16, False), (2, "clamped", 80, 13999, 17, False), (2, "clamped", 80, 14000, 17, True),
    (2, "clamped", 20, 3200, 32, True), (2, "periodic", 79, 44000, 16, True), (2, "periodic", 79, 43999, 16, False),
    (2, "periodic", 80, 44000, 16, False),
    (2, "periodic", 74, 44000, 12, True), (2, "periodic", 75, 44000, 12, False),
    (2, "periodic", 104, 44000, 32, True), (2, "periodic", 20, 4799, 8, False), (3, "clamped", 14, 21952, 16, True),
    (3, "clamped", 14, 21951, 16, False),
    (3, "clamped", 21, 40000, 13, True),
    (3, "clamped", 21, 40000, 12, False),
    (3, "clamped", 18, 40000, 12, True), (3, "clamped", 14, 23680, 32, True),
    (3, "clamped", 14, 23681, 32, False), (3, "clamped", 14, 27440, 32, True),
    (3, "clamped", 14, 27439, 32, False),
    (3, "clamped", 22, 60000, 29, True), (3, "clamped", 22, 59999, 29, False),
    (3, "clamped", 24, 69119, 32, False),
    (3, "clamped", 24, 69120, 28, False), (3, "clamped", 21, 60000, 28, True),
    (3, "clamped", 35, 200000, 32, True), (3, "clamped", 35, 199999, 32, False),
    (3, "clamped", 34, 200000, 20, True),
    (3, "clamped", 34, 199999, 20, False), (3, "periodic", 12, 40000, 16, False)])
def test_lines_between_the_two_sweeps(dim, boundary, cells, N, C, dense):
    torch.manual_seed(C)
    call = Call(_positions(dim, 1, N, 1.0), cells, 1.0 / cells, boundary, C)
    got, lists = call(True), call(False)
    assert torch.equal(got, lists) != dense
    assert torch.allclose(got, lists, rtol=2e-5, atol=2e-5 * float(lists.abs().max()))


# boxes of one, two and three cells, whose rows of cells are each other's neighbours on both sides; positions boxes away; positions beyond the cells,
# which are binned into those at the edge
@pytest.mark.parametrize("dim,B,N,cells,boundary,away", [
    (2, 2, 61, 1, "periodic", 0), (2, 3, 133, 2, "periodic", 0), (2, 1, 403, 3, "periodic", 0), (2, 2, 133, 2, "periodic", 3), (2, 2, 1003, 7, "periodic", 3),
    (2, 1, 48000, 61, "periodic", 100), (2, 2, 4097, 16, "clamped", 0.5), (3, 1, 20011, 11, "clamped", 0.3)])
@pytest.mark.parametrize("C", [8, 16, 32])
def test_small_boxes_and_positions_beyond_them(dim, B, N, cells, boundary, away, C):
    torch.manual_seed(cells + C)
    x = _positions(dim, B, N, 1.0)
    if boundary == "periodic":
        x += torch.randint(-away, away + 1, x.shape, device="cuda")
    else:
        x *= 1 + away
    call = Call(x, cells, 1.0 / cells, boundary, C)
    got, lists = call(True), call(False)
    assert not torch.equal(got, lists)
    for b in range(B):
        for idx in torch.arange(0, N, max(1, N // 300), device="cuda").split(64):
            want, size = call.exact(b, idx)
            for out in (got, lists):
                assert ((out[b, idx].double() - want).abs() <= 16 * 2.0 ** -24 * size).all()


@pytest.mark.parametrize("dim,B,N,cells,C", [(2, 5, 701, 6, 16), (2, 5, 1003, 8, 32), (3, 3, 6701, 9, 13)])
def test_a_system_alone_and_in_a_batch(dim, B, N, cells, C):
    """Tiles of eight particles begin elsewhere, and the batch decides between the sweeps: the sums agree within their rounding, not to the bit."""
    torch.manual_seed(N)
    batch = Call(_positions(dim, B, N, 0.97), cells, 1.0 / cells, "clamped", C)
    together = batch(True, batch.add)
    for b in (1, B - 1):
        alone = Call(batch.x[b:b + 1].clone(), cells, 1.0 / cells, "clamped", C)
        assert torch.equal(alone.x[0], batch.x[b]) and torch.equal(alone.rho[0], batch.rho[b])
        alone.dz, add = batch.dz[b:b + 1].clone(), batch.add[b:b + 1].clone()
        got = alone(True, add)[0]
        idx = torch.arange(0, N, max(1, N // 256), device="cuda")
        for part in idx.split(64):
            _, size = batch.exact(b, part)
            assert ((got[part] - together[b, part]).abs() <= 2 * 16 * 2.0 ** -24 * (size + add[0, part].abs())).all()
