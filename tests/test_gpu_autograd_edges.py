"""Operators in the ways torch lets a caller run them: inference tensors, saved-tensor hooks, checkpointing, odd gradients."""
import pytest
import torch

from helpers import make_grid
from npa_b200.workloads import Workload, make_inputs

pytestmark = pytest.mark.gpu


def _inputs(dim=2, N=601, C=8, B=2):
    from npa_b200 import sphops as sph
    w = Workload("edges", dim=dim, B=B, N=N, C=C, eps=0.125, grid_size=(8,) * dim)
    x, s, _ = make_inputs(w, seed=N)
    x[..., :dim] *= 0.49 / x[..., :dim].abs().max()
    return sph, make_grid(sph, w), x.cuda(), s.cuda()


def test_operators_in_inference_mode():
    sph, grid, x, s = _inputs()

    def run():
        snap = grid.instantiate(x)
        xb, sb = sph.bin_particles(x, s, snap)
        rho = sph.density(xb, snap)
        return [rho, sph.blur(xb, rho, sb, snap), sph.gradient(xb, rho, sb, snap), sph.gradient_hybrid(xb, rho, sb, snap),
                sph.density_gradient(xb, snap), sph.moment_matrix(xb, rho, snap), sph.count(xb, snap)]

    with torch.no_grad():
        want = run()
    with torch.inference_mode():
        got = run()
    for a, b in zip(got, want):
        # without lists the sweeps search, and sum in another order
        assert torch.allclose(a, b, rtol=1e-4, atol=1e-5 * float(b.abs().max()))
