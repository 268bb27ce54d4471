"""A forward perception step recorded in a CUDA graph replays to the same result as the eager calls."""
import pytest
import torch

from helpers import make_grid
from npa_b200.workloads import CONFIGS, make_inputs, scaled

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,B", [("cfg1_2d_growing", 1), ("cfg3_2d_pointmnist_strokes", 32)])
def test_graphed_step_equals_eager(name, B):
    from npa_b200 import sphops as sph
    from npa_b200.graphs import GraphedPerception
    w = scaled(CONFIGS[name], B=B)
    grid = make_grid(sph, w)
    graphed = GraphedPerception(grid, w.C, eps0=0.1)
    for seed in (1, 2):                      # replay twice with different inputs
        x, s, _ = make_inputs(w, seed=seed)
        x, s = x.cuda(), s.cuda()
        z, xb, sb = graphed(x, s)
        with torch.no_grad():
            snap = grid.instantiate(x)
            xb_e, sb_e = sph.bin_particles(x, s, snap)
            z_e = sph.perceive_features(xb_e, sb_e, snap, 0.1)
        assert torch.equal(graphed.snapshot.permutation, snap.permutation)
        assert torch.equal(xb, xb_e) and torch.equal(sb, sb_e)
        assert torch.equal(z, z_e)


def test_graphed_euler_rollout_equals_eager():
    """Eight graphed steps of a small periodic system give the positions and states of eight eager
    steps (update_prob = 1: no random mask, so the two runs are comparable)."""
    from npa_b200 import sphops as sph
    from npa_b200.graphs import GraphedEulerStep
    from npa_b200.stepping import step_euler
    from npa_b200.workloads import Workload
    from test_gpu_step_update import _TinyNPA
    w = Workload("roll", dim=2, B=16, N=512, C=16, eps=0.06, grid_size=(16, 16), boundary="periodic")
    grid = make_grid(sph, w)
    torch.manual_seed(5)
    model = _TinyNPA(2, w.C).cuda()
    x, s, _ = make_inputs(w, seed=3)
    x, s = x.cuda(), s.cuda()
    graphed = GraphedEulerStep(model, grid, w.C, dt=1.0, update_prob=1.0, wrap=True)
    xg, sg = graphed.rollout(x, s, 8)
    with torch.no_grad():
        xe, se = x, s
        for _ in range(8):
            xe, se, _ = step_euler(model, xe, se, grid, dt=1.0, update_prob=1.0, wrap=True)
    assert torch.allclose(xg, xe, rtol=0, atol=1e-6) and torch.allclose(sg, se, rtol=1e-5, atol=1e-5)
    assert float(xg.abs().max()) <= 0.5 * 16 * 0.06 + 1e-6  # wrapped into the box


@pytest.mark.parametrize("N,C", [(501, 3), (2500, 16), (1027, 8)])
def test_inputs_of_a_recorded_step_by_one_launch_or_by_copies(N, C):
    """Contiguous, unaligned, strided, double and host inputs end in the same buffers."""
    from npa_b200.graphs import _load
    g = torch.Generator(device="cuda").manual_seed(N)
    x, s = torch.randn(1, N, 2, generator=g, device="cuda"), torch.randn(1, N, C, generator=g, device="cuda")
    wide, shifted = torch.zeros(1, N, C + 1, device="cuda"), torch.zeros(N * C + 1, device="cuda")
    wide[..., :C] = s
    shifted[1:] = s.flatten()
    for other in (s, wide[..., :C], shifted[1:].view(1, N, C), s.double(), s.cpu()):
        x_in, s_in = torch.full_like(x, 7.0), torch.full_like(s, 7.0)
        _load(x_in, x, s_in, other)
        assert torch.equal(x_in, x) and torch.equal(s_in, s)
        _load(x_in, x_in, s_in, s_in)
        assert torch.equal(x_in, x) and torch.equal(s_in, s)


def test_inputs_of_a_recorded_step_that_are_not_plain_memory():
    """Negated views and inputs that lie in the buffers are copied as torch copies them, one after the other."""
    from npa_b200.graphs import _load
    g = torch.Generator(device="cuda").manual_seed(9)
    x, s = torch.randn(1, 4096, 2, generator=g, device="cuda"), torch.randn(1, 4096, 2, generator=g, device="cuda")
    x_in, s_in = torch.zeros_like(x), torch.zeros_like(s)
    _load(x_in, torch._neg_view(x), s_in, torch._neg_view(s))
    assert torch.equal(x_in, -x) and torch.equal(s_in, -s)
    _load(x_in, x, s_in, s)
    for _ in range(20):  # the buffers in each other's place: the first is written before the second is read
        x_in.copy_(x)
        s_in.copy_(s)
        _load(x_in, s_in, s_in, x_in)
        assert torch.equal(x_in, s) and torch.equal(s_in, s)
