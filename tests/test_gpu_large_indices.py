"""Particle counts whose lanes no longer fit 32 bits: pairs (2 k, 2 k + 1) through hand-made lists, in 2D, and the last particles
of the output are looked at; and a renderer whose last window of particles ends beyond 2^31.  Needs 30 to 45 GB of device memory."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _pairs(n):
    x = torch.zeros(n, 2, device="cuda")
    x[1::2, 0] = 0.05
    lists = torch.empty(n, 2, dtype=torch.int32, device="cuda")
    lists[:, 0] = 1
    lists[:, 1] = torch.arange(n, dtype=torch.int32, device="cuda") ^ 1
    return x, lists


@pytest.mark.parametrize("which,n", [("density_gradient", 2 ** 29 + 1000), ("density_backward", 2 ** 30 + 1000)])
def test_the_last_particles_are_written(which, n):
    from npa_b200 import _native
    if torch.cuda.get_device_properties(0).total_memory < 60e9:
        pytest.skip("needs 30 GB of device memory")
    grid = _native.make_grid(2, "clamped", "grid", (4, 4), 0.25, 1, n, 64)
    offs = torch.zeros(17, dtype=torch.int32, device="cuda")          # not read: no list overflows
    info = torch.zeros(4, 4, dtype=torch.int32, device="cuda")
    x, lists = _pairs(n)
    out = torch.full((n, 2), float("nan"), device="cuda")
    st = _native.current_stream()
    if which == "density_gradient":
        _native.check(_native.lib.npa_density_gradient_forward_lists(ctypes.byref(grid), _native.ptr(x), None, _native.ptr(out), _native.ptr(offs),
                                                                     _native.ptr(lists), 2, st))
    else:
        up = torch.ones(n, device="cuda")
        _native.check(_native.lib.npa_density_chain_backward(ctypes.byref(grid), _native.ptr(x), None, _native.ptr(up), None, None, _native.ptr(out),
                                                             0, _native.ptr(offs), _native.ptr(info), _native.ptr(lists), 2, st))
    torch.cuda.synchronize()
    head = out[:2].clone()
    assert head[0, 0] > 0 and head[1, 0] < 0 and (head[:, 1] == 0).all()
    even, odd = out[0::2], out[1::2]
    assert bool((even == head[0]).all()) and bool((odd == head[1]).all())   # every particle, the last ones among them


def test_the_last_window_of_an_image_ends_beyond_32_bits():
    """2^31 - 1,000 particles far outside a 16 x 16 image but for the last one: eight slices, windows of 4,096 particles."""
    from npa_b200 import _native
    if torch.cuda.get_device_properties(0).total_memory < 90e9:
        pytest.skip("needs 45 GB of device memory")
    n, img = 2 ** 31 - 1000, 16
    x, color = torch.full((n, 2), 100.0, device="cuda"), torch.zeros(n, 3, device="cuda")
    x[n - 1] = 0.0
    color[n - 1] = torch.tensor([1.0, 2.0, 3.0])
    outs = []
    for first in (0, n - 1):  # all of them, and the last one alone
        out = torch.full((img, img, 4), float("nan"), device="cuda")
        at, ac = x[first:], color[first:].clone() if first else color
        _native.check(_native.lib.npa_splat_forward(_native.ptr(at), _native.ptr(ac), 1, n - first, img, 1.0, 5, -1.0, 1.0, 0, 0, 1.0, None,
                                                    _native.ptr(out), _native.current_stream()))
        outs.append(out)
    torch.cuda.synchronize()
    assert float(outs[1][7, 7, 3]) > 0.5 and torch.isfinite(outs[0]).all()
    assert float((outs[0] - outs[1]).abs().max()) <= 1e-6  # weights of one particle, by the product and by the pixel kernel
