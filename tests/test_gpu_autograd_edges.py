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


def _operators():
    """Every differentiable operator as a function of positions and features in cell order (odd counts, both directions)."""
    from npa_b200 import splatting
    sph, grid, x, s = _inputs()
    snap = grid.instantiate(x)
    xb, sb = sph.bin_particles(x, s, snap)
    rho = sph.density(xb, snap).detach()
    first = lambda out: out if isinstance(out, tuple) else (out,)
    ops = {
        "bin_particles": lambda x, s: sph.bin_particles(x, s, snap),
        "count": lambda x, s: sph.count(x, snap),
        "density": lambda x, s: sph.density(x, snap),
        "density_gradient": lambda x, s: sph.density_gradient(x, snap),
        "blur": lambda x, s: sph.blur(x, rho, s, snap),
        "gradient": lambda x, s: sph.gradient(x, rho, s, snap),
        "gradient_hybrid": lambda x, s: sph.gradient_hybrid(x, rho, s, snap),
        "moment_matrix": lambda x, s: sph.moment_matrix(x, rho, snap),
        "perceive": lambda x, s: sph.perceive(x, s, snap),
        "perceive_features": lambda x, s: sph.perceive_features(x, s, snap, 0.125),
        "step_update": lambda x, s: sph.step_update(torch.cat([x, s], -1), x, s, snap, 1.0),
        "splat": lambda x, s: splatting.splat_particles_batch(x, s[..., :3], img_size=32),
        "chain": lambda x, s: sph.blur(x, sph.density(x, snap), s, snap)}
    return xb.detach(), sb.detach(), {k: (lambda f: lambda x, s: first(f(x, s)))(f) for k, f in ops.items()}


def _value_and_grads(f, x, s):
    x, s = x.clone().requires_grad_(True), s.clone().requires_grad_(True)
    out = f(x, s)
    g = torch.Generator(device="cuda").manual_seed(1)
    ups = [torch.randn(o.shape, generator=g, device="cuda") for o in out]
    return [o.detach() for o in out], torch.autograd.grad(out, [x, s], ups, allow_unused=True)


def _assert_same(got, want):
    for a, b in zip([*got[0], *got[1]], [*want[0], *want[1]]):
        assert (a is None) == (b is None)
        if a is not None:  # the same kernels, with or without lists: sums in another order
            assert torch.allclose(a, b, rtol=1e-4, atol=1e-5 * float(b.abs().max())), float((a - b).abs().max())


@pytest.mark.filterwarnings("ignore")
def test_traces_follow_their_inputs():
    """torch.jit.trace records an operator as a node that runs, not as the outputs it had while it was traced."""
    x, s, ops = _operators()
    moved, other = x + 0.002, s.flip(-1).contiguous()
    for name, f in ops.items():
        traced = torch.jit.trace(f, (x, s), check_trace=False)
        _assert_same(_value_and_grads(lambda x, s: tuple(traced(x, s)), moved, other), _value_and_grads(f, moved, other))


def test_outputs_require_a_gradient_wherever_an_input_does():
    """Also where that input gets none: a count of positions, masses outside the reorder."""
    sph, grid, x, s = _inputs()
    snap = grid.instantiate(x)
    mass = (0.5 + torch.rand(2, 601, device="cuda")).requires_grad_(True)
    xb, sb, mb = sph.bin_particles(x, s, snap, mass)
    xb, sb = xb.detach(), sb.detach()
    rho = sph.density(xb, snap, mb)
    outs = [rho, sph.density_gradient(xb, snap, mb), sph.blur(xb, rho.detach(), sb, snap, mb), sph.gradient(xb, rho.detach(), sb, snap, mb),
            sph.gradient_hybrid(xb, rho.detach(), sb, snap, mb), sph.moment_matrix(xb, rho.detach(), snap, mb),
            *sph.perceive(xb, sb, snap, mb), sph.perceive_features(xb, sb, snap, 0.125, mb),
            sph.count(xb.clone().requires_grad_(True), snap)]
    for out in outs:
        assert out.requires_grad
        out.sum().backward(retain_graph=True)
    assert mass.grad is None or not mass.grad.any()


class _Model(torch.nn.Module):
    """What step_euler reads of a model, in 2D with 8 channels."""

    def __init__(self, eps, seed=0):
        super().__init__()
        torch.manual_seed(seed)
        self.spatial_dims, self.eps0, self.alpha = 2, eps, 1.0
        self.state_grad = self.density_grad = self.log_norm_grad = self.log_norm_density_grad = True
        self.stopgrad_pos, self.stopgrad_state = False, False
        self.model = torch.nn.Sequential(torch.nn.Linear(34, 128), torch.nn.ReLU(), torch.nn.Linear(128, 10, bias=False)).cuda()


def _steps():
    """The step as one node and as four, as functions of positions and features."""
    from npa_b200 import stepping
    _, grid, x, s = _inputs()
    model = _Model(grid.eps)

    def step(x, s, intermediate):
        torch.manual_seed(3)
        return stepping.step_euler(model, x, s, grid, update_prob=0.5, intermediate=intermediate)[:2]

    return x, s, {"step": lambda x, s: step(x, s, False), "four_nodes": lambda x, s: step(x, s, True)}, grid


def test_saved_tensor_hooks_see_what_the_backward_reads():
    """Everything large moves to the host and comes back at another address; the gradients are the same bits."""
    x, s, ops = _operators()
    x2, s2, steps, _ = _steps()
    for name, f in {**ops, **steps}.items():
        a, b = (x2, s2) if name in steps else (x, s)
        want = _value_and_grads(f, a, b)
        packed = []

        def pack(t):
            packed.append(t.numel() * t.element_size())
            return t.cpu()

        with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t.cuda()):
            got = _value_and_grads(f, a, b)
        for p, q in zip([*got[0], *got[1]], [*want[0], *want[1]]):
            assert p is q is None or torch.equal(p, q), name
        if name in steps:  # the hidden layer alone is 128 floats per particle
            assert sum(packed) > a.shape[0] * a.shape[1] * 128 * 4


@pytest.mark.parametrize("name", ["step", "four_nodes"])
def test_checkpointed_steps_do_not_keep_what_they_recompute(name):
    from torch.utils.checkpoint import checkpoint
    x, s, steps, grid = _steps()
    f = steps[name]

    def rollout(call):
        a, b = x.clone().requires_grad_(True), s.clone().requires_grad_(True)
        p, q = a, b
        base = torch.cuda.memory_allocated()
        for _ in range(4):
            p, q = call(p, q)
        kept = torch.cuda.memory_allocated() - base
        return [p.detach(), q.detach()], torch.autograd.grad([p, q], [a, b], [torch.ones_like(p), torch.ones_like(q)]), kept

    plain = rollout(f)
    again = rollout(lambda p, q: checkpoint(f, p, q, use_reentrant=False))
    for p, q in zip([*again[0], *again[1]], [*plain[0], *plain[1]]):
        assert torch.equal(p, q)
    assert again[2] < plain[2] // 3, (again[2], plain[2])


def test_a_mask_changed_in_place_is_noticed():
    sph, grid, x, s = _inputs()
    snap = grid.instantiate(x)
    xb, sb = sph.bin_particles(x, s, snap)
    y = torch.randn(2, 601, 10, device="cuda", requires_grad=True)
    mask = torch.ones(2, 601, 1, device="cuda")
    out = sph.step_update(y, xb, sb, snap, 1.0, 1.0, mask)
    mask.zero_()
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        out[1].sum().backward()


@pytest.mark.parametrize("prob", [-1.0, 0.0, 0.3, 1.0])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_update_masks_below_any_threshold(prob, dtype):
    """Nothing moves below a probability of zero, and the mask follows the default type."""
    from npa_b200 import stepping
    x, s, _, grid = _steps()
    model = _Model(grid.eps)
    before = torch.get_default_dtype()
    torch.set_default_dtype(dtype)
    try:
        for intermediate in (False, True):          # one node, and the operators
            torch.manual_seed(5)
            x_new, s_new, _ = stepping.step_euler(model, x, s, grid, update_prob=prob, intermediate=intermediate)
            xb, sb = sph_bin(grid, x, s)
            moved = (s_new != sb).any(-1)
            torch.manual_seed(5)
            want = torch.rand(2, 601, 1, device="cuda").squeeze(-1) < prob if prob < 1.0 else torch.ones(2, 601, dtype=torch.bool, device="cuda")
            assert torch.equal(moved, want)
    finally:
        torch.set_default_dtype(before)


def sph_bin(grid, x, s):
    from npa_b200 import sphops as sph
    return sph.bin_particles(x, s, grid.instantiate(x))


def test_operators_without_features():
    sph, grid, x, s = _inputs()
    snap = grid.instantiate(x)
    empty = torch.empty(2, 601, 0, device="cuda")
    xb, sb = sph.bin_particles(x, empty, snap)
    xr, sr = xb.clone().requires_grad_(True), sb.clone().requires_grad_(True)
    rho, blur, grad, dg = sph.perceive(xr, sr, snap)
    assert blur.shape == (2, 601, 0) and grad.shape == (2, 601, 0, 2)
    want = sph.density(xb, snap)
    assert torch.allclose(rho, want, rtol=1e-6)
    up = torch.randn_like(rho)
    got, = torch.autograd.grad(rho, xr, up, retain_graph=True)
    ref = xb.clone().requires_grad_(True)
    want, = torch.autograd.grad(sph.density(ref, snap), ref, up)
    assert torch.allclose(got, want, rtol=1e-4, atol=1e-5 * float(want.abs().max()))
    out = sph.blur(xr, rho.detach(), sr, snap)
    gx, = torch.autograd.grad(out, xr, torch.empty_like(out))
    assert not gx.any()


def test_lists_read_on_another_stream_are_not_handed_out_again():
    """The next binning drops a snapshot's lists; memory that a side stream still reads must stay where it is."""
    sph, grid, x, s = _inputs(N=4001)
    snap = grid.instantiate(x)
    xb, sb = sph.bin_particles(x, s, snap)
    rho = sph.density(xb, snap)
    want = sph.gradient_hybrid(xb, rho, sb, snap)
    shape, where = snap.lists[1].shape, snap.lists[1].data_ptr()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        torch.cuda._sleep(100_000_000)                  # some 50 ms
        got = sph.gradient_hybrid(xb, rho, sb, snap)
    grid.instantiate(x)
    assert snap.lists is None
    fresh = [torch.full(shape, -7, dtype=torch.int32, device="cuda") for _ in range(3)]
    assert all(f.data_ptr() != where for f in fresh)
    torch.cuda.synchronize()
    assert torch.equal(got, want)


@pytest.mark.parametrize("change", ["short", "half", "offset"])
def test_what_a_hook_returns_for_a_step_is_checked(change):
    """The node of a step reads its saved block by offsets: another size or type is refused, another address is not."""
    x, s, steps, _ = _steps()
    want = _value_and_grads(steps["step"], x, s)

    def unpack(t):
        if t.numel() < 100_000:              # weights and mask
            return t
        if change == "short":
            return t[:-64]
        if change == "half":
            return t.half()
        flat = torch.empty(t.numel() + 1, device="cuda")
        flat[1:].copy_(t)
        return flat[1:]

    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
        if change == "offset":
            got = _value_and_grads(steps["step"], x, s)
            assert all(torch.equal(p, q) for p, q in zip([*got[0], *got[1]], [*want[0], *want[1]]))
        else:
            with pytest.raises(RuntimeError, match="saved-tensor hook"):
                _value_and_grads(steps["step"], x, s)
