"""The sweeps over neighbour lists (a sub-group of lanes per particle): channel counts at the edges of the
lane layouts, odd channel counts, particle counts that do not fill a warp, lists that overflow for some
particles of a warp, masses; and the spiky kernel values of single pairs."""
import numpy as np
import pytest
import torch

from conftest import assert_close
from helpers import make_grid
from npa_b200.workloads import Workload, make_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,boundary", [(2, "periodic"), (3, "clamped")])
@pytest.mark.parametrize("C", [1, 3, 4, 16, 17, 32, 33, 64, 65, 128, 132])
def test_channel_counts_against_oracle(dim, boundary, C):
    import oracle
    from npa_b200 import sphops as sph
    w = Workload("lists", dim=dim, B=2, N=331, C=C, eps=0.2 if dim == 2 else 0.3, grid_size=(5,) * dim if dim == 2 else (4,) * 3,
                 boundary=boundary)
    x, s, _ = make_inputs(w, seed=C)
    x[..., :dim] *= 0.98 * w.grid_size[0] * w.eps
    grid = make_grid(sph, w)
    g = torch.Generator().manual_seed(3)
    mass = (0.5 + torch.rand(w.B, w.N, generator=g)).cuda()
    snap = grid.instantiate(x.cuda())
    xb, sb, mb = sph.bin_particles(x.cuda(), s.cuda(), snap, mass)
    kw = dict(mass=mb.cpu().numpy())
    if boundary == "periodic":
        kw.update(periodic=True, box_size=[n * w.eps for n in w.grid_size])
    ups = [torch.randn(*shape, generator=g) for shape in ((w.B, w.N), (w.B, w.N, C), (w.B, w.N, C, dim), (w.B, w.N, dim))]
    try:
        for columns in (128, 24):       # 24: lists overflow for many particles, next to some that fit
            sph.set_pair_cache(columns)
            xr, sr = xb.clone().requires_grad_(True), sb.clone().requires_grad_(True)
            out = sph.perceive(xr, sr, snap, mb)
            torch.autograd.backward(out, [u.cuda() for u in ups])
            got = [t.detach().cpu().numpy() for t in (*out, sr.grad, xr.grad)]
            if columns == 128:
                want = _oracle_chain(oracle, w, xb, sb, out[0], ups, kw)
            for name, a, b in zip(("rho", "blur", "grad", "rho_grad", "grad_s", "grad_x"), got, want):
                # fp32 sums of up to ~100 terms of both signs: a few 1e-6 of the largest value
                assert_close(a[..., :dim] if name == "grad_x" else a, b, 1e-5, 5e-6, f"{name}, C={C}, columns={columns}")
    finally:
        sph.set_pair_cache(None)


def test_default_length_of_the_lists_follows_the_grid():
    """4,096 particles in 10 x 10 cells have 128 neighbours each: the default lists hold them, and every sweep agrees with shorter
    lists that overflow."""
    from npa_b200 import sphops as sph
    grid = sph.HashGrid(dim=2, boundary="periodic", mode="grid", grid_size=(10, 10), eps=0.1, num_particles=4096, batch_size=1)
    g = torch.Generator().manual_seed(1)
    x = (torch.rand(1, 4096, 2, generator=g) - 0.5).cuda()
    snap = grid.instantiate(x)
    xb, sb = sph.bin_particles(x, torch.randn(1, 4096, 8, generator=g).cuda(), snap)
    rho = sph.density(xb, snap)
    lists = snap.lists[1]
    assert lists.shape[2] == grid.hashgrid.list_columns == 256 and int(lists[..., 0].min()) > 0 and int(lists[..., 0].max()) > 127
    assert float((lists[..., 0].float() - sph.count(xb, snap)).abs().max()) <= 1.0     # (a pair on the cut-off itself)
    want = sph.blur(xb, rho, sb, snap)
    sph.set_pair_cache(64)
    try:
        sph.density(xb, snap)
        assert int(snap.lists[1][..., 0].max()) == -1
        got = sph.blur(xb, rho, sb, snap)
    finally:
        sph.set_pair_cache(None)
    assert torch.allclose(got, want, rtol=1e-4, atol=1e-5 * float(want.abs().max()))


def _oracle_chain(oracle, w, xb, sb, rho, ups, kw):
    xn, sn, rn = xb.cpu().numpy(), sb.cpu().numpy(), rho.detach().cpu().numpy()
    g_rho, g_blur, g_grad, g_dg = (u.numpy() for u in ups)
    fw = oracle.forward(xn, w.eps, w.dim, s=sn, rho_in=rn, want=("rho", "rho_grad", "blur", "grad"), **kw)
    dx1, ds, drho = oracle.backward(xn, w.eps, w.dim, s=sn, rho_in=rn, g_blur=g_blur, g_grad=g_grad, **kw)
    dx2, _, _ = oracle.backward(xn, w.eps, w.dim, g_rho=(g_rho + drho).astype(np.float32), g_rho_grad=g_dg, **kw)
    return fw["rho"], fw["blur"], fw["grad"], fw["rho_grad"], ds, dx1 + dx2


def test_spiky_kernel_of_single_pairs():
    """Two particles per system at a known distance: the density gradient is c_g m 3 (h - d)^2 / d r."""
    from npa_b200 import sphops as sph
    h, B = 0.25, 4096
    grid = sph.HashGrid(dim=2, boundary="clamped", grid_size=(4, 4), eps=h, num_particles=2, batch_size=B)
    rng = np.random.default_rng(5)
    r = (10.0 ** rng.uniform(-5, np.log10(0.98 * h), (B, 1)) * np.array([[np.cos(0.7), np.sin(0.7)]])).astype(np.float32)
    x = np.zeros((B, 2, 2), dtype=np.float32)
    x[:, 1] = r
    xt = torch.from_numpy(x).cuda()
    snap = grid.instantiate(xt)
    xb, _ = sph.bin_particles(xt, torch.zeros(B, 2, 1, device="cuda"), snap)
    sph.density(xb, snap)              # records the lists
    got = sph.unbin_particles(torch.zeros_like(xb), sph.density_gradient(xb, snap), snap)[1][:, 0].cpu().numpy().astype(np.float64)
    rd = r.astype(np.float64)
    d = np.sqrt((rd ** 2).sum(1) + 1e-12)
    hf = float(np.float32(h))
    want = 10.0 / (np.pi * h ** 5) * (3.0 * (hf - d) ** 2 / d)[:, None] * rd
    # relative: rounding of q and d (2^-24 each, doubled by the square and amplified by d / (h - d)) and of six operations
    bound = 2.0 ** -24 * (8.0 + 4.0 * d / (hf - d))
    assert (np.abs(got - want) <= bound[:, None] * np.abs(want).max(axis=1, keepdims=True)).all()


@pytest.mark.parametrize("dim,C", [(3, 32), (3, 16), (2, 13), (3, 20)])
def test_full_backward_with_particles_of_no_mass_and_crowded_lists(dim, C):
    """Lists of the default length (longer than 128 where memory allows) against sweeps that search: gradients of particles without
    mass, whose volume is zero, and of clusters with more than 127 neighbours.  The searching backward divides by the mass: there the
    particles weigh 1e-20, which changes no sum."""
    from npa_b200 import sphops as sph
    N = 3000
    grid = sph.HashGrid(dim=dim, boundary="clamped", mode="grid", grid_size=(8,) * dim, eps=0.125, num_particles=N, batch_size=1)
    assert grid.hashgrid.roomy_list_columns == (512 if grid.hashgrid.list_columns == 128 else grid.hashgrid.list_columns)
    g = torch.Generator().manual_seed(C)
    x = torch.rand(1, N, 2 if dim == 2 else 4, generator=g) - 0.5
    x[:, : N // 4, :dim] *= 0.3
    mass = 0.5 + torch.rand(1, N, generator=g)
    mass[:, ::7] = 0.0
    s = torch.randn(1, N, C, generator=g)
    ups = [torch.randn(1, N, *t, generator=g).cuda() for t in ((), (C,), (C, dim), (dim,))]
    got = []
    for columns in (None, 0):
        sph.set_pair_cache(columns)
        try:
            xr, sr = x.cuda().requires_grad_(True), s.cuda().requires_grad_(True)
            snap = grid.instantiate(xr)
            xb, sb, mb = sph.bin_particles(xr, sr, snap, mass.clamp(min=0.0 if columns is None else 1e-20).cuda())
            out = sph.perceive(xb, sb, snap, mb)
            got.append([*(t.detach() for t in out), *torch.autograd.grad(out, [xr, sr], ups)])
        finally:
            sph.set_pair_cache(None)
    # two fp32 sums of up to a few hundred terms in different orders: 2e-5 of the largest value
    for a, b in zip(*got):
        assert torch.isfinite(a).all() and float((a - b).abs().max()) <= 2e-5 * float(b.abs().max())


def test_memory_that_recorded_steps_keep():
    """A chain of steps through ``perceive``: what every further step keeps until the backward is its tensors and its lists, at the
    default length and at 128 columns."""
    from npa_b200 import sphops as sph
    B, N, C = 8, 4096, 16
    grid = sph.HashGrid(dim=2, boundary="clamped", mode="grid", grid_size=(16, 16), eps=0.0625, num_particles=N, batch_size=B)
    g = torch.Generator(device="cuda").manual_seed(2)
    x0, s0 = torch.rand(B, N, 2, generator=g, device="cuda") - 0.5, torch.randn(B, N, C, generator=g, device="cuda")

    def kept(steps):
        """Bytes that are alive after ``steps`` recorded steps."""
        torch.cuda.synchronize()
        before = torch.cuda.memory_allocated()
        x, s = x0.clone().requires_grad_(True), s0.clone().requires_grad_(True)
        for _ in range(steps):
            snap = grid.instantiate(x)
            xb, sb = sph.bin_particles(x, s, snap)
            rho, blur, grad, dg = sph.perceive(xb, sb, snap)
            x, s = xb + 1e-4 * dg, blur
        return torch.cuda.memory_allocated() - before

    per_step = {}
    for columns in (None, 128):
        sph.set_pair_cache(columns)
        try:
            kept(2)
            per_step[columns] = (kept(5) - kept(2)) / 3
        finally:
            sph.set_pair_cache(None)
    lists = {None: 4 * grid.hashgrid.roomy_list_columns * B * N, 128: 4 * 128 * B * N}
    assert abs((per_step[None] - per_step[128]) - (lists[None] - lists[128])) <= 2 << 20
    assert per_step[128] <= lists[128] + (32 << 20)  # tensors of a step: positions, features, blur, gradient, density: 12 MiB
