"""Contiguous tensors at addresses that vector loads cannot use (a view into a flat buffer): the same bits as at aligned ones."""
import pytest
import torch

from helpers import make_grid
from npa_b200.workloads import Workload, make_inputs

pytestmark = pytest.mark.gpu


def _at(t, floats):
    """A contiguous copy of ``t``, `floats` floats into a buffer."""
    flat = torch.empty(t.numel() + 8, dtype=t.dtype, device=t.device)
    view = flat[floats: floats + t.numel()].view(t.shape)
    view.copy_(t)
    assert view.data_ptr() % 16 == 4 * floats % 16 and view.is_contiguous()
    return view


def _setup(dim, C, boundary="clamped"):
    from npa_b200 import sphops as sph
    w = Workload("align", dim=dim, B=2, N=333, C=C, eps=0.2, grid_size=(5,) * dim, boundary=boundary)
    x, s, _ = make_inputs(w, seed=C)
    x[..., :dim] *= 0.49 / x[..., :dim].abs().max()
    grid = make_grid(sph, w)
    snap = grid.instantiate(x.cuda())
    return sph, grid, snap, *sph.bin_particles(x.cuda(), s.cuda(), snap)


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("C", [2, 6, 8, 16, 18, 32, 64])
@pytest.mark.parametrize("offset", [1, 2])
def test_packed_perception_of_features_at_any_address(dim, C, offset):
    from npa_b200.sphops import sph as impl
    sph, grid, snap, xb, sb = _setup(dim, C)
    before = impl._PAIR_CACHE["columns"]
    try:
        for columns in (128, 16):                       # 16: particles with more neighbours are searched for
            impl._PAIR_CACHE["columns"] = columns
            for rec in (False, True):
                want_s, got_s = (t.detach().requires_grad_(rec) for t in (sb, _at(sb, offset)))
                want = sph.perceive_features(xb, want_s, snap, 0.2)
                got = sph.perceive_features(xb, got_s, snap, 0.2)
                assert torch.equal(got, want)
                if rec:
                    up = torch.randn_like(want)
                    g = [torch.autograd.grad(z, s, u)[0] for z, s, u in ((want, want_s, up), (got, got_s, _at(up, offset)))]
                    assert torch.allclose(g[1], g[0], rtol=1e-5, atol=1e-6 * float(g[0].abs().max()))
    finally:
        impl._PAIR_CACHE["columns"] = before


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("C", [16, 32, 64, 128])        # rows that fill the lanes of their particle
def test_perception_of_features_at_any_address(dim, C):
    """The kernels that know the feature count and those that read float by float add the same products in the same order."""
    from npa_b200.sphops import sph as impl
    sph, grid, snap, xb, sb = _setup(dim, C, "periodic")
    before = impl._PAIR_CACHE["columns"]
    try:
        for columns in (128, 16):                       # 16: particles with more neighbours are searched for
            impl._PAIR_CACHE["columns"] = columns
            res, ups = [], None
            for offset in (0, 1):
                x, s = xb.detach().requires_grad_(True), _at(sb, offset).requires_grad_(True)
                out = sph.perceive(x, s, snap)
                ups = ups or [torch.randn_like(o) for o in out]
                res.append([*out, *torch.autograd.grad(out, [x, s], ups, retain_graph=True), torch.autograd.grad(out[1:3], s, ups[1:3])[0]])
            for a, b in zip(*res):
                assert torch.allclose(a, b, rtol=1e-5, atol=1e-6 * float(a.abs().max()))
            assert all(torch.equal(a, b) for a, b in zip(res[0][:4], res[1][:4]))
    finally:
        impl._PAIR_CACHE["columns"] = before


@pytest.mark.parametrize("C", [8, 16, 64])
def test_packed_perception_into_outputs_at_any_address(C):
    sph, grid, snap, xb, sb = _setup(2, C)
    z, v = torch.empty(2, 333, 4 * C + 2, device="cuda"), torch.empty(2, 333, C, 2, device="cuda")
    outs = []
    for offset in (0, 1):
        zo, vo = (_at(torch.zeros_like(t), offset) for t in (z, v))
        rho, dg = torch.empty(2, 333, device="cuda"), torch.empty(2, 333, 2, device="cuda")
        pairs = torch.empty(2, 333, 128, dtype=torch.int32, device="cuda")
        grid.hashgrid.perceive_features_forward(xb, None, sb, 1.0, 1.0, 1e-3, True, True, rho, dg, zo, vo, snap.bin_offsets,
                                                snap.block_info, pair_cache=pairs)
        outs.append((zo, vo, rho, dg))
    for a, b in zip(*outs):
        assert torch.allclose(a, b, rtol=1e-5, atol=1e-6 * float(b.abs().max()))


@pytest.mark.parametrize("dim", [2, 3])
def test_upstream_gradients_at_any_address(dim):
    from npa_b200 import splatting, stepping
    sph, grid, snap, xb, sb = _setup(dim, 8)
    rho = sph.density(xb, snap).detach()
    y = torch.randn(2, 333, dim + 8, device="cuda")
    calls = [
        lambda x, s: sph.bin_particles(x, s, snap), lambda x, s: sph.perceive(x, s, snap),
        lambda x, s: (sph.density(x, snap), sph.density_gradient(x, snap)), lambda x, s: (sph.blur(x, rho, s, snap),),
        lambda x, s: (sph.gradient_hybrid(x, rho, s, snap),), lambda x, s: (sph.moment_matrix(x, rho, snap),),
        lambda x, s: (sph.perceive_features(x, s, snap, 0.2),), lambda x, s: sph.step_update(y, x, s, snap, 1.0)]
    if dim == 2:
        calls.append(lambda x, s: (splatting.splat_particles_batch(x, s[..., :3], img_size=32),))
    for call in calls:
        g = torch.Generator(device="cuda").manual_seed(2)
        grads = []
        ups = None
        for offset in (0, 1):
            x, s = xb.detach().requires_grad_(True), sb.detach().requires_grad_(True)
            out = call(x, s)
            ups = ups or [torch.randn(o.shape, generator=g, device="cuda") for o in out]
            grads.append(torch.autograd.grad(out, [x, s], [_at(u, offset) for u in ups], allow_unused=True))
        for a, b in zip(*grads):
            assert a is b is None or torch.equal(a, b)


def test_euler_step_with_gradients_at_any_address():
    from test_gpu_autograd_edges import _steps
    x, s, steps, _ = _steps()
    grads = []
    for offset in (0, 1):
        a, b = x.clone().requires_grad_(True), s.clone().requires_grad_(True)
        out = steps["step"](a, b)
        grads.append(torch.autograd.grad(out, [a, b], [_at(torch.ones_like(o), offset) for o in out]))
    assert all(torch.equal(p, q) for p, q in zip(*grads))
