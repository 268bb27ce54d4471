"""Kernels that may take their places before the one before them has completed (launch_early in csrc/common.cuh): every result is
that of the same calls with the GPU waited for in between, also behind copies, events of other streams and other kernels."""
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
    torch.cuda.synchronize()

    def check(x):
        snap = grid.instantiate(x)
        xb, _ = sph.bin_particles(x, s, snap)
        torch.cuda.synchronize()
        assert torch.equal(snap.permutation, permutation) and torch.equal(xb, x_bin)

    for write in (lambda x: x.copy_(host, non_blocking=True), lambda x: x.copy_(new), lambda x: x.add_(new - old), lambda x: x.zero_().add_(new)):
        x = old.clone()
        grid.instantiate(x)
        torch.cuda._sleep(1_000_000)
        write(x)
        if not torch.equal(x, new):  # (the sum may be rounded)
            x.copy_(new)
        check(x)
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
