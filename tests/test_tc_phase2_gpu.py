"""Phase 2 of the 128-column passes at the edges of its blocks of 4 row tiles:
blocks without sources (a single leaf whose diagonal block comes from the
coordinates), a last block of fewer row tiles, leaves of odd size (masked row
tiles, odd column-tile counts), dense leaf blocks, and block-row shards.

A 128-column pass and the same columns 16 at a time agree up to FP32
summation order and T's BF16 hi + lo rounding (2^-17 relative): 2e-6 in norm,
as for the whole pass."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def hm():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import hmatrix

    return hmatrix


def _compare(hm, H, n, nrhs, rows=slice(None)):
    import torch

    g = torch.Generator(device="cuda").manual_seed(4)
    X = torch.randn((nrhs, n), device="cuda", generator=g).t()
    Y = H.matvec(X)
    H.check()
    parts = torch.cat([H.matvec(X[:, c:min(c + 16, nrhs)].t().contiguous().t()) for c in range(0, nrhs, 16)], dim=1)
    Yo = H.matvec(X, original_order=True)  # gathered X, scattered Y
    assert torch.isfinite(Y[rows]).all()
    err = (torch.linalg.norm(Y[rows] - parts[rows]) / torch.linalg.norm(parts[rows])).item()
    assert err <= 2e-6, err
    return X, Y, Yo


@pytest.mark.parametrize("n,b,tol,diag,nrhs", [
    (20, 32, 1e-4, 1, 128),      # one leaf, no sources: Y is the fly diagonal alone
    (20, 32, 1e-4, 0, 70),       # one leaf, one dense block, one row tile
    (777, 32, 1e-4, 0, 128),     # 25 row tiles or so: a last block of fewer than four
    (3001, 64, 1e-5, 0, 65),     # odd leaves, dense leaf-level blocks
    (16411, 64, 1e-4, 0, 128),
])
def test_wide_pass_equals_narrow_passes(hm, n, b, tol, diag, nrhs):
    import torch

    pts = hm.generate_dataset(n, 3, seed=n)
    tree = hm.construct_kdtree(pts, n, 3, b)
    st = hm.construct_hmatrix_structure(tree, hm.BOX_CENTER, 1.0)
    H = hm.build_hmatrix(tree, st, pts, kernel=hm.K_MATERN32, ell=0.2, nugget=1e-3, tol=tol, max_rank=128,
                         precision=hm.PREC_MIXED, diag_from_coords=diag)
    X, Y, Yo = _compare(hm, H, n, nrhs)
    p = torch.from_numpy(tree.copy_out()["perm"]).cuda().long()
    Xt = X.t()[:, p].contiguous().t()
    assert torch.equal(Yo.t()[:, p], H.matvec(Xt).t())  # the same arithmetic in either order


def test_wide_pass_on_shards(hm):
    n = 9001
    pts = hm.generate_dataset(n, 3, seed=2)
    tree = hm.construct_kdtree(pts, n, 3, 64)
    st = hm.construct_hmatrix_structure(tree, hm.BOX_CENTER, 1.0)
    offs = tree.copy_out()["offsets"]
    for lo, hi in ((0, 37), (37, 128), (128, 129), (129, len(offs) - 1)):
        H = hm.build_hmatrix(tree, st, pts, kernel=hm.K_MATERN32, ell=0.2, tol=1e-4, max_rank=128,
                             precision=hm.PREC_MIXED, leaves=(lo, hi))
        _compare(hm, H, n, 128, slice(int(offs[lo]), int(offs[hi])))
