"""dL/dz of a step taken apart as it leaves the tensor cores, against the product and the rows made one after the other."""
import ctypes

import pytest
import torch

from test_gpu_dense_backward import Call, _positions

pytestmark = pytest.mark.gpu


def _images(call, W1, W2, rows):
    """The image of W1 for the backward, in the order of the rows or in W1's own, made by the reorder's launch."""
    n, p, C, D = call.n, call.n.ptr, call.C, call.dim
    K, O = 2 * C + C * D + D, D + C
    nbytes = n.lib.npa_mlp_forward_tcgen05_scratch_bytes(K, O)
    size = n.lib.npa_step_rows_image_bytes(ctypes.byref(call.gd), C) if rows else n.lib.npa_linear_tcgen05_scratch_bytes(128, K)
    work, image = torch.empty(nbytes // 4, device="cuda"), torch.full((size // 4,), float("nan"), device="cuda")
    xo, so = torch.empty_like(call.x), torch.empty_like(call.s)
    head = (ctypes.byref(call.gd), C, p(call.x), p(call.s), p(call.snap.permutation), p(xo), p(so), p(W1), p(W2))
    tail = (W1.stride(0), W1.stride(1), W2.stride(0), W2.stride(1), p(work), nbytes, p(image), size, call.st)
    n.check(n.lib.npa_bin_particles_step_images(*head, *tail) if rows else n.lib.npa_bin_particles_mlp_images(*head, K, O, *tail))
    return image, size


# tiles of 128 rows: one row, one short of a tile, one more, a full round of 148 tiles and beyond; sections of 16 columns filled or not
@pytest.mark.parametrize("dim,boundary,B,N,C", [(2, "clamped", 1, 1, 16), (2, "periodic", 1, 127, 12), (2, "clamped", 3, 43, 20), (2, "clamped", 2, 9600, 32),
                                                (3, "clamped", 1, 129, 28), (3, "periodic", 2, 64, 24), (3, "clamped", 1, 19073, 16), (3, "clamped", 1, 2000, 12),
                                                (2, "clamped", 1, 300, 4), (3, "periodic", 1, 130, 8),
                                                (3, "clamped", 2, 10001, 32)])
@pytest.mark.parametrize("log_norm", [0, 1])
def test_rows_as_the_separate_kernels_make_them(dim, boundary, B, N, C, log_norm):
    """The same products and the same expression for each element: equal bits, also of rows that begin in another system."""
    torch.manual_seed(N + C)
    eps = 0.05 if dim == 2 else 0.1
    cells = max(4, round((N / 8) ** (1 / dim)))
    call = Call(_positions(dim, B, N, cells * eps), cells, eps, boundary, C)
    n, p, D = call.n, call.n.ptr, dim
    K = 2 * C + C * D + D
    W1, W2 = torch.randn(128, K, device="cuda"), torch.randn(D + C, 128, device="cuda")
    if log_norm:
        W1 = W1.t().contiguous().t()                        # strides of a transposed weight
    dh = torch.randn(B, N, 128, device="cuda") * (torch.rand(B, N, 128, device="cuda") < 0.5)
    call.v[0, 0] = 0.0                                      # a gradient of zero: the normalisation's own case
    plain, plain_bytes = _images(call, W1, W2, False)
    dz = torch.empty(B, N, K, device="cuda")
    n.check(n.lib.npa_linear_tcgen05_prepared(p(dh), p(plain), plain_bytes, p(dz), B * N, 128, K, call.st))
    ref = ctypes.byref(call.gd)
    nbytes = n.lib.npa_lists_backward_scratch_bytes(ref, C)
    work, want = torch.empty(nbytes // 4, device="cuda"), torch.empty(B, N, C, device="cuda")
    n.check(n.lib.npa_perceive_features_backward_binned(ref, C, p(call.x), None, p(call.s), p(call.rho), p(call.dg), p(call.v), p(call.packed), p(dz), 0.8, 0.3,
                                                        log_norm, 1, p(call.add), None, p(want), p(work), nbytes, p(call.snap.bin_offsets), p(call.pairs), call.K,
                                                        call.st))
    image, image_bytes = _images(call, W1, W2, True)
    nbytes = n.lib.npa_step_perceive_backward_scratch_bytes(ref, C)
    work, got = torch.full((nbytes // 4 + 64,), float("nan"), device="cuda"), torch.full((B, N, C), float("nan"), device="cuda")
    n.check(n.lib.npa_step_perceive_backward(ref, C, p(dh), p(image), image_bytes, p(call.x), p(call.s), p(call.rho), p(call.v), p(call.packed), 0.8, log_norm,
                                             p(call.add), p(got), p(work), nbytes, p(call.snap.bin_offsets), p(call.pairs), call.K, call.st))
    assert torch.equal(got, want)
    assert bool(torch.isnan(work[nbytes // 4:]).all())      # nothing beyond the scratch that was asked for
    status = ctypes.c_uint32(1)
    n.check(n.lib.npa_linear_tcgen05_status(ctypes.byref(status), 0))
    assert status.value == 0


# one system and several, binned by a CTA, a cluster or the general way; cells up to the line beyond which the work list has its own launch
@pytest.mark.parametrize("dim,B,N,cells,C", [(2, 1, 300, 16, 16), (2, 5, 1, 4, 12), (2, 64, 512, 9, 16), (2, 300, 33, 5, 8), (2, 3, 4096, 45, 16), (2, 3, 4096, 46, 16),
                                             (2, 7, 20000, 20, 13), (3, 4, 9000, 12, 32), (3, 2, 70000, 20, 16), (3, 3, 2000, 13, 16)])
def test_beginning_of_a_step_in_one_call(dim, B, N, cells, C):
    """Grid build, work list, reorder and images: the bytes of the separate calls."""
    from npa_b200 import _native as n, sphops as sph
    torch.manual_seed(N)
    p, st, eps = n.ptr, n.current_stream(), 0.05
    x, s = _positions(dim, B, N, cells * eps), torch.randn(B, N, C, device="cuda")
    grid = sph.HashGrid(dim=dim, boundary="clamped", mode="grid", grid_size=(cells,) * dim, eps=eps, num_particles=N, batch_size=B, max_particles_per_block=16)
    gd = n.make_grid(dim, "clamped", "grid", (cells,) * dim, eps, B, N, 16)
    ref, snap = ctypes.byref(gd), grid.instantiate(x)
    K, O = 2 * C + C * dim + dim, dim + C
    W1, W2 = torch.randn(128, K, device="cuda"), torch.randn(O, 128, device="cuda")
    strides = (K, 1, 128, 1)
    nbytes, build_bytes = n.lib.npa_mlp_forward_tcgen05_scratch_bytes(K, O), n.lib.npa_grid_scratch_bytes(ref)
    for rows in (0, 1) if C % 4 == 0 else (0,):
        size = n.lib.npa_step_rows_image_bytes(ref, C) if rows else n.lib.npa_linear_tcgen05_scratch_bytes(128, K)
        new = lambda: [torch.full((nbytes // 4,), -1.0, device="cuda"), torch.full((size // 4,), -1.0, device="cuda"), torch.empty_like(x), torch.empty_like(s)]
        want, got = new(), new()
        head, tail = (ref, C, p(x), p(s)), (*strides, p(want[0]), nbytes, p(want[1]), size)
        out = (p(want[2]), p(want[3]), p(W1), p(W2))
        n.check(n.lib.npa_bin_particles_step_images(*head, p(snap.permutation), *out, *tail, st) if rows
                else n.lib.npa_bin_particles_mlp_images(*head, p(snap.permutation), *out, K, O, *tail, st))
        lists = [torch.full_like(t, -7) for t in (snap.permutation, snap.bin_offsets, snap.block_info)]
        scratch = torch.empty(build_bytes, dtype=torch.uint8, device="cuda")
        n.check(n.lib.npa_step_bin(*head, *map(p, lists), p(scratch), build_bytes, p(got[2]), p(got[3]), p(W1), p(W2), *strides, p(got[0]), nbytes, p(got[1]), size,
                                   rows, st))
        for a, b in zip(got + lists, want + [snap.permutation, snap.bin_offsets, snap.block_info]):
            assert torch.equal(a, b)


@pytest.mark.parametrize("dim,B,N,C", [(2, 1, 5, 1), (2, 3, 43, 16), (2, 8, 4096, 16), (3, 1, 9001, 13), (3, 2, 700, 32)])
@pytest.mark.parametrize("which", ["both", "features", "positions"])
def test_weight_gradients_added_beside_the_inverse_reorder(dim, B, N, C, which):
    """The bits of the two separate calls: the runs and the order of the sums are the same."""
    from npa_b200 import _native as n
    torch.manual_seed(N)
    p, st, K, O, M = n.ptr, n.current_stream(), 2 * C + C * dim + dim, dim + C, B * N
    gd = n.make_grid(dim, "clamped", "grid", (4,) * dim, 0.1, B, N, 16)
    e = lambda *shape: torch.randn(*shape, device="cuda")
    z, dh, h, dy, x, s = e(M, K), e(M, 128), e(M, 128), e(M, O), e(B, N, 2 if dim == 2 else 4), e(B, N, C)
    perm = torch.stack([torch.randperm(N, device="cuda") for _ in range(B)]).to(torch.int32)
    size = n.lib.npa_mlp_weight_grad_tcgen05_scratch_floats(M, K, O)
    x_in, s_in = (x if which != "features" else None), (s if which != "positions" else None)

    def outputs():
        return [torch.full_like(t, float("nan")) for t in (x, s)] + [torch.full(q, float("nan"), device="cuda") for q in ((128, K), (O, 128), (128,))]

    want, got, work = outputs(), outputs(), torch.empty(size, device="cuda")
    of = lambda t, given: p(t) if given is not None else None
    rows = (p(z), p(dh), p(h), p(dy), M, K, 128, O, p(work), size)
    n.check(n.lib.npa_mlp_weight_grad_tcgen05(*rows, *map(p, want[2:]), st))
    n.check(n.lib.npa_unbin_particles(ctypes.byref(gd), C, p(x_in), p(s_in), None, p(perm), of(want[0], x_in), of(want[1], s_in), None, st))
    n.check(n.lib.npa_mlp_weight_grad_tcgen05_partial(*rows, st))
    n.check(n.lib.npa_step_unbin(ctypes.byref(gd), C, p(x_in), p(s_in), p(perm), of(got[0], x_in), of(got[1], s_in), K, O, p(work), size, *map(p, got[2:]), st))
    for a, b in zip(got, want):
        assert torch.equal(a.nan_to_num(7.0), b.nan_to_num(7.0))
    assert not bool(torch.isnan(got[2]).any() | torch.isnan(got[3]).any() | torch.isnan(got[4]).any())
