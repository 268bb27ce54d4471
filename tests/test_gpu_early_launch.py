"""Kernels that may take their places before the one before them has completed (launch_early in csrc/common.cuh): every result is
that of the same calls with the GPU waited for in between, also behind copies, events of other streams and other kernels."""
import os
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu


def _grid(dim, N, B=2):
    from npa_b200 import sphops as sph
    return sph.HashGrid(dim=dim, boundary="periodic" if dim == 3 else "clamped", mode="grid", grid_size=(8,) * dim, eps=0.125, num_particles=N,
                        batch_size=B, max_particles_per_block=32)


def _positions(dim, N, g, B=2):
    x = torch.rand(B, N, 2 if dim == 2 else 4, generator=g, device="cuda") - 0.5
    return x


@pytest.mark.parametrize("dim,N,C", [(2, 700, 16), (3, 3000, 13), (3, 40000, 32)])
def test_chains_give_the_results_of_single_calls(dim, N, C):
    from npa_b200 import sphops as sph
    grid = _grid(dim, N)
    g = torch.Generator(device="cuda").manual_seed(N)

    def chain(x, s, ups, pause):
        xr, sr = x.clone().requires_grad_(True), s.clone().requires_grad_(True)
        pause()
        snap = grid.instantiate(xr)
        pause()
        xb, sb = sph.bin_particles(xr, sr, snap)
        pause()
        out = sph.perceive(xb, sb, snap)
        pause()
        grads = torch.autograd.grad(out, [xr, sr], ups)
        z = sph.perceive_features(xb.detach(), sb.detach(), snap, 0.125)
        return [snap.permutation, snap.bin_offsets, *out, *grads, z]

    for _ in range(8):
        x, s = _positions(dim, N, g), torch.randn(2, N, C, generator=g, device="cuda")
        ups = [torch.randn(2, N, *t, generator=g, device="cuda") for t in ((), (C,), (C, dim), (dim,))]
        want = chain(x, s, ups, torch.cuda.synchronize)
        got = chain(x, s, ups, lambda: None)
        for a, b in zip(got, want):
            assert torch.equal(a, b)


def test_inputs_written_by_copies_other_kernels_and_other_streams():
    from npa_b200 import sphops as sph
    grid, g = _grid(2, 5000), torch.Generator(device="cuda").manual_seed(3)
    old, new = _positions(2, 5000, g), _positions(2, 5000, g)
    s = torch.randn(2, 5000, 16, generator=g, device="cuda")
    host = new.cpu().pin_memory()
    want = grid.instantiate(new)
    permutation, x_bin = want.permutation.clone(), sph.bin_particles(new, s, want)[0].clone()
    by = new - old
    moved = old + by  # (the sum is rounded)
    want = grid.instantiate(moved)
    permutation_moved, x_bin_moved = want.permutation.clone(), sph.bin_particles(moved, s, want)[0].clone()
    torch.cuda.synchronize()

    def check(x, permutation=permutation, x_bin=x_bin):
        snap = grid.instantiate(x)
        xb, _ = sph.bin_particles(x, s, snap)
        torch.cuda.synchronize()
        assert torch.equal(snap.permutation, permutation) and torch.equal(xb, x_bin)

    # the host is ahead of the GPU from the pause on: the grid build is launched long before the positions are there
    for write, result in ((lambda x: x.copy_(host, non_blocking=True), (permutation, x_bin)), (lambda x: x.copy_(new), (permutation, x_bin)),
                          (lambda x: x.add_(by), (permutation_moved, x_bin_moved)), (lambda x: x.zero_().add_(new), (permutation, x_bin))):
        x = old.clone()
        grid.instantiate(x)
        torch.cuda._sleep(4_000_000)
        write(x)
        check(x, *result)
    # written on another stream behind an event, read here after a kernel of this stream
    side, x, done = torch.cuda.Stream(), old.clone(), torch.cuda.Event()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        torch.cuda._sleep(2_000_000)
        x.copy_(new)
        done.record()
    grid.instantiate(old)
    torch.cuda.current_stream().wait_event(done)
    check(x)
    # written here, read on another stream
    x = old.clone()
    torch.cuda._sleep(1_000_000)
    x.copy_(new)
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        check(x)


def test_a_recorded_step_after_joined_streams():
    """Launches inside a graph are plain ones: a fork and a join inside the recording, replayed with new inputs."""
    from npa_b200 import sphops as sph
    grid, g = _grid(3, 2000), torch.Generator(device="cuda").manual_seed(5)
    x, s = _positions(3, 2000, g), torch.randn(2, 2000, 8, generator=g, device="cuda")
    side = torch.cuda.Stream()
    other = _grid(3, 2000)

    def step():
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            a = other.instantiate(x)
        b = grid.instantiate(x)
        torch.cuda.current_stream().wait_stream(side)
        xb, sb = sph.bin_particles(x, s, a)
        return a.permutation, b.permutation, sph.perceive_features(xb, sb, a, 0.125)

    with torch.no_grad():
        warm = torch.cuda.Stream()
        warm.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(warm):
            step()
        torch.cuda.current_stream().wait_stream(warm)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = step()
        for _ in range(3):
            x.copy_(_positions(3, 2000, g))
            graph.replay()
            want = step()
            torch.cuda.synchronize()
            for a, b in zip(out, want):
                assert torch.equal(a, b)


# ---- whole steps, the single operators, images and rollouts, against a process that waits after every launch -----------------
class _Model:
    """What ``step_euler`` reads of a model."""

    def __init__(self, dim, C, g):
        out, width = dim + C, 2 * C + C * dim + dim
        self.model = torch.nn.Sequential(torch.nn.Linear(width, 128), torch.nn.ReLU(), torch.nn.Linear(128, out, bias=False)).cuda()
        with torch.no_grad():
            for p in self.model.parameters():
                p.copy_(torch.randn(p.shape, generator=g, device="cuda") / width ** 0.5)
        self.eps0, self.alpha, self.spatial_dims = 0.125, 0.5, dim


def _step_pass(dim, N, C, B):
    from npa_b200.stepping import step_euler
    grid = _grid(dim, N, B)
    model = _Model(dim, C, torch.Generator(device="cuda").manual_seed(1))

    def run(g):
        x, s = _positions(dim, N, g, B).requires_grad_(True), torch.randn(B, N, C, generator=g, device="cuda", requires_grad=True)
        ups = [torch.randn(x.shape, generator=g, device="cuda"), torch.randn(s.shape, generator=g, device="cuda")]
        torch.cuda.manual_seed(5)
        torch.cuda._sleep(1_000_000)
        x_new, s_new, _ = step_euler(model, x, s, grid, update_prob=0.5)
        grads = torch.autograd.grad([x_new, s_new], [x, s, *model.model.parameters()], ups)
        with torch.no_grad():
            further = step_euler(model, x_new, s_new, grid, update_prob=1.0)[:2]
        return [x_new, s_new, *grads, *further]
    return run


def _operators_pass(dim, N, C, B, fuse):
    from npa_b200 import sphops as sph
    grid = _grid(dim, N, B)

    def run(g):
        x, s = _positions(dim, N, g, B).requires_grad_(True), torch.randn(B, N, C, generator=g, device="cuda", requires_grad=True)
        mass = 0.5 + torch.rand(B, N, generator=g, device="cuda")
        ups = [torch.randn(B, N, *t, generator=g, device="cuda") for t in ((), (C,), (C, dim), (dim,))]
        torch.cuda._sleep(1_000_000)
        sph.enable_fusion(fuse)
        try:
            snap = grid.instantiate(x)
            xb, sb, mb = sph.bin_particles(x, s, snap, mass)
            rho = sph.density(xb, snap, mb)
            out = [rho, sph.blur(xb, rho, sb, snap, mb), sph.gradient_hybrid(xb, rho, sb, snap, mb), sph.density_gradient(xb, snap, mb)]
        finally:
            sph.enable_fusion(False)
        grads = torch.autograd.grad(out, [x, s], ups, retain_graph=True)
        z = sph.perceive_features(xb, sb, snap, 0.125)
        z_grads = torch.autograd.grad(z, [x, s], torch.ones_like(z))
        return [*out, sph.count(xb, snap), *grads, z, *z_grads]
    return run


def _splat_pass(B, N, img):
    from npa_b200 import splatting

    def run(g):
        x = ((torch.rand(B, N, 2, generator=g, device="cuda") - 0.5) * 2).requires_grad_(True)
        c = torch.rand(B, N, 3, generator=g, device="cuda", requires_grad=True)
        up = torch.randn(B, img, img, 4, generator=g, device="cuda")
        torch.cuda._sleep(1_000_000)
        image = splatting.splat_particles_batch(x, c, img_size=img)
        return [image, *torch.autograd.grad(image, [x, c], up)]
    return run


def _rollout_pass(dim, N, C, steps):
    from npa_b200.rollout import PerceptionRollout, VelocityField
    roll = PerceptionRollout(_grid(dim, N), C, steps, 0.1, VelocityField(dim, torch.device("cuda"), seed=1))

    def run(g):
        x, s = _positions(dim, N, g), torch.randn(2, N, C, generator=g, device="cuda")
        ups = {k: torch.randn(2, N, *t, generator=g, device="cuda") for k, t in (("g_rho", ()), ("g_blur", (C,)), ("g_grad", (C, dim)))}
        torch.cuda._sleep(1_000_000)
        grads = roll.run(x, s, ups)
        return [t.clone() for t in (x, s, roll.x_bin, roll.s_bin, roll.rho, roll.blur, roll.grad, *grads)]
    return run


PASSES = {
    "step, one CTA per system bins": lambda: _step_pass(2, 700, 16, 3),
    "step, a cluster per system bins": lambda: _step_pass(2, 4096, 16, 2),
    "step in 3D, six launches bin": lambda: _step_pass(3, 70001, 32, 1),
    "step with odd rows": lambda: _step_pass(3, 3001, 13, 2),
    "operators": lambda: _operators_pass(2, 4096, 16, 2, False),
    "operators fused, odd rows in 3D": lambda: _operators_pass(3, 5001, 13, 2, True),
    "image, few particles per tile": lambda: _splat_pass(2, 200, 200),
    "image, many particles per tile": lambda: _splat_pass(2, 3000, 210),
    "image, tiles shared by a cluster": lambda: _splat_pass(2, 4100, 64),
    "rollout": lambda: _rollout_pass(3, 3000, 16, 3),
}
SEEDS = (11, 12)


def _outputs(run, seed):
    return [t.detach().cpu() for t in run(torch.Generator(device="cuda").manual_seed(seed))]


@pytest.fixture(scope="module")
def waited(tmp_path_factory):
    """The outputs of all passes from a process in which every launch is waited for."""
    path = tmp_path_factory.mktemp("waited") / "outputs.pt"
    res = subprocess.run([sys.executable, __file__, str(path)], env={**os.environ, "CUDA_LAUNCH_BLOCKING": "1"}, capture_output=True, text=True,
                         timeout=300)
    assert res.returncode == 0, res.stderr[-2000:]
    return torch.load(path)


@pytest.mark.parametrize("name", PASSES)
def test_whole_passes_give_the_results_of_launches_that_are_waited_for(waited, name):
    """Two inputs in turn, so that memory that a pass uses again holds the answers of the other input; the host is ahead of the GPU."""
    run = PASSES[name]()
    for _ in range(4):
        for seed in SEEDS:
            got = _outputs(run, seed)
            assert len(got) == len(waited[name][seed])
            for k, (a, b) in enumerate(zip(got, waited[name][seed])):
                assert torch.equal(a, b), f"output {k}"


if __name__ == "__main__":
    sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    torch.save({name: {seed: _outputs(run, seed) for seed in SEEDS} for name, make in PASSES.items() for run in [make()]}, sys.argv[1])
