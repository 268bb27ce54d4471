"""The multi-step perception rollout (npa_b200.rollout) against the same loop written with the public
sphops API and autograd."""
import pytest
import torch

from npa_b200.workloads import Workload, make_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w", [
    Workload("r3", dim=3, B=2, N=3000, C=16, eps=0.125, grid_size=(8, 8, 8), boundary="periodic"),
    Workload("r2", dim=2, B=3, N=1500, C=8, eps=0.08, grid_size=(14, 14)),
], ids=lambda w: w.name)
def test_rollout_matches_the_public_api_loop(w):
    from npa_b200 import sphops as sph
    from npa_b200.rollout import PerceptionRollout, VelocityField
    steps, dt = 4, 0.004
    x0, s0, ups = make_inputs(w, seed=2)
    box = torch.tensor([g * w.eps for g in w.grid_size[: w.dim]])
    x0[..., : w.dim] *= box * (1.0 if w.boundary == "periodic" else 0.8)
    x0, s0 = x0.cuda(), s0.cuda()
    ups = {k: v.cuda() for k, v in ups.items()}
    grid = sph.HashGrid(dim=w.dim, boundary=w.boundary, mode="grid", grid_size=w.grid_size, eps=w.eps,
                        num_particles=w.N, batch_size=w.B, max_particles_per_block=32)
    vel = VelocityField(w.dim, x0.device, seed=4)
    roll = PerceptionRollout(grid, w.C, steps, dt, vel)
    x, s = x0.clone(), s0.clone()
    gx, gs = roll.run(x, s, ups)
    rho, blur, grad = roll.rho.clone(), roll.blur.clone(), roll.grad.clone()

    # the same loop with the public API: instantiate, bin, perceive, move, wrap; backward through the last step
    xr, sr = x0.clone(), s0.clone()
    for k in range(steps):
        last = k == steps - 1
        if last:
            xr.requires_grad_(True)
            sr.requires_grad_(True)
        snap = grid.instantiate(xr.detach())
        xb, sb = sph.bin_particles(xr, sr, snap)
        r, bl, gr = sph.perceive(xb, sb, snap, with_density_gradient=False)
        if not last:
            xn = xb[..., : w.dim] + dt * vel(xb)
            if w.boundary == "periodic":
                xn = grid.wrap_positions(xn)
            xr = xb.clone()
            xr[..., : w.dim] = xn
            sr = sb
    assert torch.equal(x, xr.detach()), "positions entering the last step differ"
    assert torch.equal(s, sr.detach())
    assert torch.equal(rho, r) and torch.equal(blur, bl) and torch.equal(grad, gr)
    torch.autograd.backward([r, bl, gr], [ups["g_rho"], ups["g_blur"], ups["g_grad"]])
    assert torch.equal(gx, xr.grad), "gradient with respect to the positions of the last step differs"
    assert torch.equal(gs, sr.grad)


@pytest.mark.parametrize("steps", [1, 2, 3])
@pytest.mark.parametrize("dim,N,boundary,modes,cells,eps,dt", [
    (3, 20011, "periodic", 8, 8, 0.125, 0.3), (2, 1001, "periodic", 64, 8, 0.125, 0.3), (3, 515, "clamped", 8, 8, 0.125, 0.3),
    (2, 1501, "periodic", 8, 9, 0.1, 5.0), (3, 3001, "periodic", 8, 24, 0.0879, 20.0)])
def test_the_native_move_gives_the_bits_of_the_tensor_operations(dim, N, boundary, modes, cells, eps, dt, steps):
    """A rollout whose velocity field is not the built-in type moves by tensor operations and copies the states: the same positions
    (bit for bit, or particles would change cells), states, outputs and gradients, with an odd and an even number of steps.  The last
    two boxes have lengths that are rounded, and moves of several lengths."""
    from npa_b200 import sphops as sph
    from npa_b200.rollout import PerceptionRollout, VelocityField

    class Another(VelocityField):
        pass

    grid = sph.HashGrid(dim=dim, boundary=boundary, mode="grid", grid_size=(cells,) * dim, eps=eps, num_particles=N, batch_size=2)
    g = torch.Generator(device="cuda").manual_seed(N)
    x0 = (torch.rand(2, N, 2 if dim == 2 else 4, generator=g, device="cuda") - 0.5) * (cells * eps)
    s0 = torch.randn(2, N, 8, generator=g, device="cuda")
    ups = {"g_rho": torch.randn(2, N, generator=g, device="cuda"), "g_blur": torch.randn(2, N, 8, generator=g, device="cuda"),
           "g_grad": torch.randn(2, N, 8, dim, generator=g, device="cuda")}
    got = []
    for field in (VelocityField, Another):
        roll = PerceptionRollout(grid, 8, steps, dt, field(dim, x0.device, seed=1, modes=modes))
        x, s = x0.clone(), s0.clone()
        versions = x._version, s._version
        grads = roll.run(x, s, ups)
        assert steps == 1 or (x._version > versions[0] and s._version > versions[1])
        got.append([t.clone() for t in (x, s, roll.x_bin, roll.s_bin, roll.rho, roll.blur, roll.grad, *grads)])
    for a, b in zip(*got):
        assert torch.equal(a, b)


def test_fields_and_tensors_that_the_move_kernel_does_not_take():
    """A phase that torch broadcasts over the modes moves as torch moves it, parameters of other shapes raise as in torch, and
    positions that may not be written in place are refused."""
    from npa_b200 import sphops as sph
    from npa_b200.rollout import PerceptionRollout, VelocityField

    class Another(VelocityField):
        pass

    grid = sph.HashGrid(dim=2, boundary="periodic", mode="grid", grid_size=(8, 8), eps=0.125, num_particles=300, batch_size=1)
    g = torch.Generator(device="cuda").manual_seed(1)
    x0, s0 = torch.rand(1, 300, 2, generator=g, device="cuda") - 0.5, torch.randn(1, 300, 4, generator=g, device="cuda")
    ups = {"g_rho": torch.randn(1, 300, generator=g, device="cuda"), "g_blur": torch.randn(1, 300, 4, generator=g, device="cuda"),
           "g_grad": torch.randn(1, 300, 4, 2, generator=g, device="cuda")}
    moved = []
    for kind in (VelocityField, Another):
        field = kind(2, x0.device, seed=1)
        field.phase = field.phase[:1].clone()
        x = x0.clone()
        PerceptionRollout(grid, 4, 2, 0.3, field).run(x, s0.clone(), ups)
        moved.append(x)
    assert torch.equal(*moved)
    for name, shape in (("phase", (9,)), ("k_t", (2, 7)), ("amp", (7, 2))):
        field = VelocityField(2, x0.device, seed=1)
        setattr(field, name, torch.zeros(shape, device="cuda"))
        with pytest.raises(RuntimeError):
            PerceptionRollout(grid, 4, 2, 0.3, field).run(x0.clone(), s0.clone(), ups)
    with torch.inference_mode():
        frozen = x0.clone()
    with pytest.raises(RuntimeError, match="[Ii]nference"):
        PerceptionRollout(grid, 4, 2, 0.3, VelocityField(2, x0.device, seed=1)).run(frozen, s0.clone(), ups)
