"""The product where the number of row tiles changes its shape: phase 2 shares
a row tile among 8, 4 or 1 warps (512, 3000 and 6000 row tiles), phase 1 cuts
its panels into shorter units on small matrices, a pass of up to 8 right-hand
sides multiplies one half of the FP32 tiles, and calls in the points' original
order read X and write Y through the permutation.

A call in original order does the same arithmetic as one in tree order, so the
two agree bit for bit; columns do not mix, so a column of a wide pass differs
from the same column alone by the order of FP32 sums only (2^-24 per addition,
at most some thousand additions that grow as a random walk: below 1e-5 of the
largest entry); both against dense FP64 rows at the build's tolerance."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def hm():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import hmatrix

    return hmatrix


# row tiles: 1 (one leaf), 16 (odd leaves), 512, 1024, 2048, 4096, 8192
@pytest.mark.parametrize("n,b", [(20, 32), (300, 32), (16384, 32), (16417, 32), (40003, 64), (131072, 32), (262143, 32)])
@pytest.mark.parametrize("prec", [0, 1])
def test_orders_and_widths_agree(hm, n, b, prec):
    import torch

    d, ell, tol = 2, 0.1, 1e-4
    pts = hm.generate_dataset(n, d, seed=n)
    tree = hm.construct_kdtree(pts, n, d, b)
    st = hm.construct_hmatrix_structure(tree, hm.BOX_CENTER, 1.0)
    H = hm.build_hmatrix(tree, st, pts, kernel=hm.K_EXP, ell=ell, tol=tol, max_rank=64, precision=prec)
    perm = tree.copy_out()["perm"]
    g = torch.Generator(device="cuda").manual_seed(1)
    Xo = torch.randn((40, n), device="cuda", generator=g).t()
    p = torch.from_numpy(perm).cuda().long()
    Xt = Xo.t()[:, p].contiguous().t()
    rows = np.unique(np.random.default_rng(2).integers(0, n, 48))
    one = H.matvec(Xt[:, :1])
    for nr in (1, 3, 8, 9, 16, 17, 32, 40):
        Yt = H.matvec(Xt[:, :nr])
        Yo = H.matvec(Xo[:, :nr], original_order=True)
        assert torch.equal(Yo.t()[:, p], Yt.t()), nr
        assert (Yt[:, 0] - one[:, 0]).abs().max() <= 1e-5 * one.abs().max(), nr
        ref = oracle.dense_rows_matvec(pts.cpu().numpy(), n, d, perm, oracle.K_EXP, ell, 0.0, rows,
                                       Xt[:, nr - 1].double().cpu().numpy())[0]
        got = Yt[:, nr - 1].double().cpu().numpy()[rows]
        assert np.linalg.norm(got - ref) <= 2 * tol * np.linalg.norm(ref), nr
