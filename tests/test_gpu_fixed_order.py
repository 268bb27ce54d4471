"""The packed perception's sums bit for bit against their stated order, evaluated on the CPU: pairs in list order, a feature's sum
split by (position mod classes) and added pairwise, the density gradient's by (position mod 32), distance 16 first; every
operation rounded to single precision, square root and quotient as IEEE rounds them."""
import numpy as np
import pytest
import torch

from helpers import make_grid
from npa_b200.workloads import Workload, make_inputs

pytestmark = pytest.mark.gpu
F, LONG = np.float32, np.longdouble


def _fma(a, b, c):
    """fl(a b + c) of single-precision values: the product is exact in extended precision, the sum nearly so."""
    return (LONG(1) * a * b + c).astype(F)


def _tree(parts):
    """Neighbours first."""
    while len(parts) > 1:
        parts = [(a + b).astype(F) for a, b in zip(parts[::2], parts[1::2])]
    return parts[0]


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("C,classes", [(4, 8), (16, 8), (20, 4), (32, 4), (6, 4), (18, 1)])
@pytest.mark.parametrize("N", [700, 9000])     # few particles and many: two density searches
def test_sums_in_their_stated_order(dim, C, classes, N):
    from npa_b200 import sphops as sph
    cells = {700: 6, 9000: 20}[N] if dim == 2 else {700: 4, 9000: 9}[N]
    w = Workload("order", dim=dim, B=1, N=N, C=C, eps=1.0 / cells, grid_size=(cells,) * dim)
    x, s, _ = make_inputs(w, seed=C)
    x[..., :dim] *= 0.49 / x[..., :dim].abs().max()
    grid = make_grid(sph, w)
    snap = grid.instantiate(x.cuda())
    xb, sb = sph.bin_particles(x.cuda(), s.cuda(), snap)
    rho, dg = torch.empty(1, N, device="cuda"), torch.empty(1, N, dim, device="cuda")
    z = torch.empty(1, N, 2 * C + C * dim + dim, device="cuda")
    pairs = torch.empty(1, N, 128, dtype=torch.int32, device="cuda")
    grid.hashgrid.perceive_features_forward(xb, None, sb, 1.0, 1.0, 1e-3, True, True, rho, dg, z, None, snap.bin_offsets, snap.block_info,
                                            pair_cache=pairs)
    X, S, R, L, Z, DG = (t[0].cpu().numpy() for t in (xb, sb, rho, pairs, z, dg))
    X = X[:, :dim]
    eps = grid.eps
    h, h2 = F(eps), F(eps * eps)
    c_s = F(4.0 / (np.pi * eps ** 8)) if dim == 2 else F(315.0 / (64.0 * np.pi * eps ** 9))
    c_g = F(10.0 / (np.pi * eps ** 5)) if dim == 2 else F(15.0 / (np.pi * eps ** 6))
    seen = 0
    for i in range(0, N, max(1, N // 150)):
        n = int(L[i, 0])
        if n < 0:
            continue
        seen += 1
        j = L[i, 1: 1 + n]
        r = (X[j] - X[i]).astype(F)
        q = _fma(r[:, 1], r[:, 1], (r[:, 0] * r[:, 0]).astype(F))
        if dim == 3:
            q = _fma(r[:, 2], r[:, 2], q)
        v = (F(1.0) / R[j]).astype(F)
        t = np.maximum((h2 - q).astype(F), F(0))
        weight = (v * ((t * t).astype(F) * t).astype(F)).astype(F)
        parts = [np.zeros(C, F) for _ in range(classes)]
        for e in range(n):
            parts[e % classes] = _fma(weight[e], S[j[e]], parts[e % classes])
        np.testing.assert_array_equal(Z[i, C: 2 * C], (c_s * _tree(parts)).astype(F), err_msg=f"blur of particle {i}")
        d = np.sqrt((q + F(1e-12)).astype(F)).astype(F)
        u = np.maximum((h - d).astype(F), F(0))
        phi = (((F(3.0) * u).astype(F) * u).astype(F) / d).astype(F)
        sums = [np.zeros(dim, F) for _ in range(32)]
        for e in range(n):
            if q[e] > 0:
                sums[e % 32] = _fma(phi[e], r[e], sums[e % 32])
        for half in (16, 8, 4, 2, 1):
            sums = [(sums[k] + sums[k + half]).astype(F) for k in range(half)]
        np.testing.assert_array_equal(DG[i], (c_g * sums[0]).astype(F), err_msg=f"density gradient of particle {i}")
    assert seen > 100
