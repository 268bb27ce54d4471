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
        sph.set_pair_cache(128)


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
