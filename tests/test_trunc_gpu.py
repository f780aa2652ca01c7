"""The truncation stage over the basis widths at which its kernels change
(32, 64, 128 columns; wider bases are kept as sampled) and over blocks whose
Gram matrix is summed in several row chunks (more than 2048 rows).

V = B W_r with W_r the leading eigenvectors of B^T B, so V's columns are
orthogonal and come in decreasing norm, U's are orthonormal, and the block
meets its tolerance.  In FP32 (u = 6e-8) an entry of V^T V is a sum over n rows
of products of sums of k <= 128 terms: off by at most 2 k u |V_1|^2 = 1.6e-5
|V_1|^2 by rounding; U^T U likewise."""
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


@pytest.mark.parametrize("n,d,b,kind,ell,tol,eta,prec", [
    (24007, 3, 64, 0, 0.05, 1e-5, 1.5, 0),   # ranks past 128, 3000-row blocks
    (20011, 2, 64, 1, 0.2, 1e-5, 1.0, 0),    # ranks within 32 and 64, 2501-row blocks
    (9001, 2, 32, 0, 0.1, 1e-6, 1.0, 0),     # FP64 working precision
])
def test_factors_are_singular_pairs(hm, n, d, b, kind, ell, tol, eta, prec):
    pts = hm.generate_dataset(n, d, seed=n)
    tree = hm.construct_kdtree(pts, n, d, b)
    st = hm.construct_hmatrix_structure(tree, hm.BOX_CENTER, eta)
    H = hm.build_hmatrix(tree, st, pts, kernel=kind, ell=ell, tol=tol, max_rank=256, precision=prec)
    perm, p = tree.copy_out()["perm"], pts.cpu().numpy()
    lr, _ = H.blocks()
    stored = np.flatnonzero((lr[:, 0] > lr[:, 2]) & (lr[:, 4] > 0))
    rng = np.random.default_rng(1)
    picks = []
    for lo, hi in ((1, 2), (2, 17), (17, 33), (33, 65), (65, 129), (129, 257)):  # by rank
        of = stored[(lr[stored, 4] >= lo) & (lr[stored, 4] < hi)]
        picks += list(rng.choice(of, min(4, len(of)), replace=False))
    picks += list(stored[np.argsort(lr[stored, 3])[-4:]])  # the tallest
    for i in picks:
        r0, m, c0, nn, k, _ = (int(v) for v in lr[i])
        U, V = H.block_factors(int(i))
        err = oracle.block_error(p, n, d, perm, kind, ell, 0.0, r0, m, c0, nn, U, V)
        assert err <= tol, (m, nn, k, err)
        assert np.abs(U.T @ U - np.eye(k)).max() < 1.6e-5, (m, k)
        if k > 128:
            continue  # kept as sampled
        G = V.T @ V
        s = np.diag(G)
        off = np.abs(G - np.diag(s)).max()
        assert off < 1.6e-5 * s[0], (m, nn, k, off / s[0])
        assert np.all(s[1:] <= s[:-1] * (1 + 1e-5) + 1.6e-5 * s[0]), (m, nn, k)
