"""The orthogonalisation stage of the compression over the heights at which
its kernel changes shape: one CTA up to 64, 128 and 256 rows, clusters of 2, 4
and 8 CTAs above, slices streamed instead of resident above 2048 rows (half of
these in FP64).  The heights are those of the levels of odd-sized clouds.

Every checked block meets its tolerance against the FP64 oracle, and its U is
orthonormal: Q has orthonormal columns to FP32 rounding (u = 6e-8 per entry)
and W_r is an orthogonal matrix in FP32, so an entry of U^T U - I is a sum of
at most k <= 64 products each off by a few u: below 64 * 2 u = 8e-6."""
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


# leaf heights 39-40 .. and 64-65 .. : levels of 39, 78, 156, 312, 625, 1250, 2500, 5000 rows, resp. 32.., 2080
@pytest.mark.parametrize("n,d,b,kind,ell,tol", [
    (40003, 2, 64, 0, 0.1, 1e-4),   # FP32 working precision
    (33300, 2, 64, 1, 0.3, 1e-5),   # 65 .. 2081 rows: just past the edges
    (16389, 2, 32, 0, 0.1, 1e-6),   # FP64 working precision
    (9001, 2, 32, 1, 0.3, 1e-6),
])
def test_blocks_of_every_height(hm, n, d, b, kind, ell, tol):
    pts = hm.generate_dataset(n, d, seed=n)
    tree = hm.construct_kdtree(pts, n, d, b)
    st = hm.construct_hmatrix_structure(tree, hm.BOX_CENTER, 1.0)
    H = hm.build_hmatrix(tree, st, pts, kernel=kind, ell=ell, tol=tol, max_rank=64)
    perm, p = tree.copy_out()["perm"], pts.cpu().numpy()
    lr, _ = H.blocks()
    lr_i = np.flatnonzero((lr[:, 0] > lr[:, 2]) & (lr[:, 4] > 0))
    rng = np.random.default_rng(0)
    heights = set()
    for level in np.unique(lr[lr_i, 5]):
        of = lr_i[lr[lr_i, 5] == level]
        for i in rng.choice(of, min(4, len(of)), replace=False):
            r0, m, c0, nn, k, _ = (int(v) for v in lr[i])
            heights.add(m)
            U, V = H.block_factors(int(i))
            err = oracle.block_error(p, n, d, perm, kind, ell, 0.0, r0, m, c0, nn, U, V)
            assert err <= tol, (m, nn, k, err)
            G = U.T @ U
            assert np.abs(G - np.eye(k)).max() < 8e-6, (m, k, np.abs(G - np.eye(k)).max())
    assert min(heights) <= 64 and max(heights) > (1024 if tol < 5e-6 else 2048) // (2 if n == 9001 else 1), heights
