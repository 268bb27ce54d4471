"""The adaptation MLP on the tensor-core linear kernels (three TF32 MMAs per product:
npa_linear_tcgen05 with the accumulators in tensor memory, and npa_linear_tf32x3 on mma.sync) and the
fused weight-gradient kernel (npa_mlp_weight_grad) against torch: values and gradients held to
float64 truth about as tightly as torch's own float32 run.  Every test runs once per engine."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True, params=["tcgen05", "mma.sync"])
def engine(request, monkeypatch):
    import npa_b200.mlp as mlp
    monkeypatch.setattr(mlp, "TENSOR_ENGINE", request.param)
    yield request.param
    if request.param == "tcgen05":   # no bounded wait of the kernel ever gave up
        from npa_b200 import _native as n
        status = ctypes.c_uint32(0)
        n.check(n.lib.npa_linear_tcgen05_status(ctypes.byref(status), 1))
        assert status.value == 0, f"linear_umma_kernel reported status {status.value}"


def _mlp(k, o, hidden=128, seed=0):
    torch.manual_seed(seed)
    return torch.nn.Sequential(torch.nn.Linear(k, hidden), torch.nn.ReLU(), torch.nn.Linear(hidden, o, bias=False)).cuda()


@pytest.mark.parametrize("rows,k,o", [(1000, 66, 18), (4096 + 7, 163, 35), (31, 176, 48), (2048, 5, 1), (65536 * 4, 163, 35)])
def test_gradients_match_float64_truth(rows, k, o):
    from npa_b200.mlp import apply_mlp, supported
    mlp = _mlp(k, o)
    assert supported(mlp)
    g = torch.Generator(device="cuda").manual_seed(1)
    shape = (2, rows // 2, k) if rows % 2 == 0 else (rows, k)
    z = torch.randn(*shape, generator=g, device="cuda")
    up = torch.randn(*shape[:-1], o, generator=g, device="cuda")

    def run(fn, module, dtype):
        module.zero_grad(set_to_none=True)
        zr = z.detach().clone().to(dtype).requires_grad_(True)
        y = fn(module, zr)
        y.backward(up.to(dtype))
        return [y.detach(), zr.grad] + [p.grad.clone() for p in module.parameters()]

    ours = run(apply_mlp, mlp, torch.float32)
    theirs = run(lambda m, t: m(t), mlp, torch.float32)
    truth = run(lambda m, t: m(t), _mlp(k, o).double(), torch.float64)
    names = ["y", "g_z", "g_W1", "g_b1", "g_W2"]
    for name, a, b, t in zip(names, ours, theirs, truth):
        scale = float(t.abs().max())
        err_ours = float((a.double() - t).abs().max())
        err_torch = float((b.double() - t).abs().max())
        # the split-precision products drop a term of 2^-22 per product: allow a few fp32 roundings more
        assert err_ours <= 4 * err_torch + 4e-6 * scale, (name, err_ours, err_torch, scale)
        print(f"{name}: error {err_ours:.3e} (torch fp32 {err_torch:.3e}) at scale {scale:.3e}")


def test_two_runs_are_bit_identical_and_unsupported_shapes_fall_back():
    from npa_b200.mlp import apply_mlp, supported
    mlp = _mlp(66, 18)
    z = torch.randn(3, 5000, 66, device="cuda")
    up = torch.randn(3, 5000, 18, device="cuda")
    grads = []
    for _ in range(2):
        mlp.zero_grad(set_to_none=True)
        apply_mlp(mlp, z.clone().requires_grad_(True)).backward(up)
        grads.append([p.grad.clone() for p in mlp.parameters()])
    for a, b in zip(*grads):
        assert torch.equal(a, b)
    wide = _mlp(66, 18, hidden=64)
    assert not supported(wide)
    zr = z.clone().requires_grad_(True)
    apply_mlp(wide, zr).backward(up)      # plain module call
    assert zr.grad is not None and wide[0].weight.grad is not None
    big = _mlp(200, 18)
    assert not supported(big)


@pytest.mark.parametrize("rows,k,n,out_by_in,relu,bias", [(1000, 163, 128, True, True, True), (777, 128, 35, True, False, False),
                                                          (4096, 35, 128, False, False, False), (130, 128, 163, False, False, False),
                                                          (64, 176, 128, True, True, True), (5, 3, 1, True, False, True),
                                                          (128 * 148 * 2 + 77, 163, 128, True, True, True),
                                                          (40000, 128, 163, False, False, False), (300, 200, 256, True, False, True)])
def test_linear_kernel_against_float64(rows, k, n, out_by_in, relu, bias, engine):
    """The linear kernel alone, both weight layouts, odd sizes, partial tiles, more tiles than CTAs."""
    from npa_b200.mlp import _linear
    if engine == "mma.sync" and max(k, n) > 176:
        pytest.skip("the mma.sync kernel holds the whole weight matrix in shared memory: up to 176 x 176")
    g = torch.Generator(device="cuda").manual_seed(2)
    a = torch.randn(rows, k, generator=g, device="cuda")
    w = torch.randn((n, k) if out_by_in else (k, n), generator=g, device="cuda")
    b = torch.randn(n, generator=g, device="cuda") if bias else None
    got = _linear(a, w, b, relu, out_by_in)
    want = a.double() @ (w.double().t() if out_by_in else w.double())
    if bias:
        want = want + b.double()
    if relu:
        want = want.relu()
    plain = (a @ (w.t() if out_by_in else w)) + (b if bias else 0)
    plain = plain.relu() if relu else plain
    scale = float(want.abs().max())
    err, err_torch = float((got.double() - want).abs().max()), float((plain.double() - want).abs().max())
    assert err <= 4 * err_torch + 4e-6 * scale, (err, err_torch, scale)


def test_gated_linear_is_the_relu_backward():
    from npa_b200.mlp import _linear
    g = torch.Generator(device="cuda").manual_seed(3)
    dy = torch.randn(3000, 35, generator=g, device="cuda")
    w2 = torch.randn(35, 128, generator=g, device="cuda")
    h = torch.randn(3000, 128, generator=g, device="cuda").relu()
    want = torch.where(h > 0, dy.double() @ w2.double(), torch.zeros((), dtype=torch.float64, device="cuda"))
    for force in (True, False):
        got = _linear(dy, w2, None, False, False, gate=h, force_tensor=force)
        assert float((got.double() - want).abs().max()) <= 4e-6 * float(want.abs().max())
        assert torch.equal(got == 0, want == 0) or float(((got == 0) != (want == 0)).float().mean()) < 1e-6


def test_a_wait_that_runs_out_ends_the_tcgen05_kernel_roles_cleanly(engine):
    """The bounded waits of linear_umma_kernel: a wait on an mbarrier that nothing completes gives up after
    its limit and raises the leave flag; a second role waiting elsewhere leaves through the flag; the
    context stays usable (no trap, no fault, no endless loop)."""
    if engine != "tcgen05":
        pytest.skip("the mma.sync kernel has no mbarrier waits")
    from npa_b200 import _native as n
    res = torch.full((2,), -1, dtype=torch.int32, device="cuda")
    n.check(n.lib.npa_linear_tcgen05_wait_selftest(2000, n.ptr(res), n.current_stream()))
    torch.cuda.synchronize()
    assert res.tolist() == [1, 1]
    assert float(torch.ones(4, device="cuda").sum().item()) == 4.0


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("C,N", [(4, 1), (13, 15), (16, 16), (16, 4097), (32, 17), (32, 40000), (45, 333)])   # eight rows per warp, up to 48 columns
@pytest.mark.parametrize("mask", [None, "weights", "uniforms"])
def test_hidden_gradient_of_a_step(dim, C, N, mask):
    """The update's backward and the hidden gradient in one pass: g_y to the bit as by the update's own kernel, dh to the bit as from that
    g_y, and dh against float64."""
    import ctypes
    from npa_b200 import _native as n
    gen = torch.Generator(device="cuda").manual_seed(C + N)
    randn = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    P, O = (2 if dim == 2 else 4), dim + C
    grid = n.make_grid(dim, "clamped", "grid", (8,) * dim, 0.1, 1, N, 32)
    y, gx, gs, W2, h = randn(N, O), randn(N, P), randn(N, C), randn(O, 128), randn(N, 128).relu()
    y[0, :dim] = 0                                          # the limiter's corner
    m = None if mask is None else torch.rand(N, generator=gen, device="cuda") if mask == "uniforms" else (randn(N) > 0).float()
    st, ref = n.current_stream(), ctypes.byref(grid)
    for up_x, up_s in ((gx, gs), (None, gs), (gx, None)):
        gy, gy_one, dh, dh_one = (torch.full(s, float("nan"), device="cuda") for s in ((N, O), (N, O), (N, 128), (N, 128)))
        if mask == "uniforms":
            n.check(n.lib.npa_step_update_backward_masked(ref, n.ptr(y), n.ptr(m), 0.5, C, 0.7, 0.9, n.ptr(up_x), n.ptr(up_s), n.ptr(gy), st))
        else:
            n.check(n.lib.npa_step_update_backward(ref, n.ptr(y), n.ptr(m), C, 0.7, 0.9, n.ptr(up_x), n.ptr(up_s), n.ptr(gy), st))
        n.check(n.lib.npa_mlp_hidden_grad(n.ptr(gy), n.ptr(W2), n.ptr(h), n.ptr(dh), N, 128, O, 128, 1, st))
        n.check(n.lib.npa_step_hidden_grad(ref, n.ptr(y), O, n.ptr(m), mask == "uniforms", 0.5, C, 0.7, 0.9, n.ptr(up_x), n.ptr(up_s), n.ptr(W2),
                                           n.ptr(h), n.ptr(gy_one), n.ptr(dh_one), 128, 128, 1, st))
        assert torch.equal(gy_one, gy) and torch.equal(dh_one, dh)
        want = (gy.double() @ W2.double()) * (h > 0)
        bound = 2.0 ** -24 * O * (gy.double().abs() @ W2.double().abs())    # a rounding per product of the chain
        assert ((dh.double() - want).abs() <= bound).all()


@pytest.mark.parametrize("dim,C,N", [(2, 4, 1), (2, 16, 127), (3, 12, 129), (3, 32, 128), (3, 32, 20001), (2, 28, 40000)])  # tiles of 128 rows, 148 at a time
@pytest.mark.parametrize("mask", [None, "weights", "uniforms"])
def test_forward_with_the_update(dim, C, N, mask):
    """The update in the MLP's epilogue: positions, states, hidden layer and raw displacements to the bit as by the two kernels."""
    import ctypes
    from npa_b200 import _native as n
    gen = torch.Generator(device="cuda").manual_seed(C + N)
    randn = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    P, O, K = (2 if dim == 2 else 4), dim + C, 2 * C + C * dim + dim
    z, W1, b1, W2, x, s = randn(N, K), randn(128, K) / K ** 0.5, randn(128), randn(O, 128) / 11, randn(N, P) * 0.3, randn(N, C)
    m = None if mask is None else torch.rand(N, generator=gen, device="cuda") if mask == "uniforms" else (randn(N) > 0).float()
    nan = lambda *s: torch.full(s, float("nan"), device="cuda")
    h, y, xo, so, h1, u1, x1, s1 = nan(N, 128), nan(N, O), nan(N, P), nan(N, C), nan(N, 128), nan(N, P), nan(N, P), nan(N, C)
    st, nbytes = n.current_stream(), n.lib.npa_mlp_forward_tcgen05_scratch_bytes(K, O)
    image = torch.empty(nbytes // 4, device="cuda")
    n.check(n.lib.npa_mlp_forward_tcgen05(n.ptr(z), n.ptr(W1), n.ptr(b1), n.ptr(W2), n.ptr(h), n.ptr(y), N, K, O, K, 1, 128, 1, n.ptr(image), nbytes, st))
    for boundary, wrap in (("clamped", 0), ("periodic", 1)):
        grid = ctypes.byref(n.make_grid(dim, boundary, "grid", (8,) * dim, 0.1, 1, N, 32))
        if mask == "uniforms":
            n.check(n.lib.npa_step_update_forward_masked(grid, n.ptr(y), n.ptr(x), n.ptr(s), n.ptr(m), 0.5, C, 0.7, 0.9, wrap, n.ptr(xo), n.ptr(so), st))
        else:
            n.check(n.lib.npa_step_update_forward(grid, n.ptr(y), n.ptr(x), n.ptr(s), n.ptr(m), C, 0.7, 0.9, wrap, n.ptr(xo), n.ptr(so), st))
        for hidden, u in ((h1, u1), (None, None)):
            x1.fill_(float("nan"))
            n.check(n.lib.npa_mlp_step_forward(grid, n.ptr(z), n.ptr(b1), n.ptr(hidden), K, n.ptr(image), nbytes, n.ptr(x), n.ptr(s), n.ptr(m),
                                               mask == "uniforms", 0.5, C, 0.7, 0.9, wrap, n.ptr(u), n.ptr(x1), n.ptr(s1), st))
            assert torch.equal(x1, xo) and torch.equal(s1, so)
        assert torch.equal(h1, h) and torch.equal(u1[:, :dim], y[:, :dim])


@pytest.mark.parametrize("k,o", [(95, 32), (96, 32), (95, 33), (94, 31), (175, 48)])   # both shapes of the kernel, on the lines between them
@pytest.mark.parametrize("rows", [1, 16, 17, 129, 40001])                               # a stage of rows, a segment, more than a segment per CTA
def test_weight_gradients_of_either_shape(engine, k, o, rows):
    from npa_b200 import _native as n
    if engine != "tcgen05":
        pytest.skip("the kernel of the tensor-memory engine")
    gen = torch.Generator(device="cuda").manual_seed(rows + k)
    randn = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    z, dh, h, dy = randn(rows, k), randn(rows, 128), randn(rows, 128), randn(rows, o)
    floats = n.lib.npa_mlp_weight_grad_tcgen05_scratch_floats(rows, k, o)
    scratch, gw1, gw2, gb1 = (torch.full(s, float("nan"), device="cuda") for s in ((floats,), (128, k), (o, 128), (128,)))
    n.check(n.lib.npa_mlp_weight_grad_tcgen05(n.ptr(z), n.ptr(dh), n.ptr(h), n.ptr(dy), rows, k, 128, o, n.ptr(scratch), floats, n.ptr(gw1), n.ptr(gw2),
                                              n.ptr(gb1), n.current_stream()))
    for got, a, b in ((gw1, dh, z), (gw2, dy, h), (gb1[:, None], dh, torch.ones_like(z[:, :1]))):
        a, b = a.double(), b.double()
        # heads and tails drop 2^-22 per product, a chain of 48 accumulations truncates by 2^-23 of its sum each
        assert ((got.double() - a.T @ b).abs() <= (2.0 ** -21 + 48 * 2.0 ** -23) * (a.abs().T @ b.abs())).all()
