"""The mixed form's dense blocks: one copy of each, read by the warp-level
kernels and by the tcgen05 kernels alike.

The products of matrices whose blocks are all dense are compared with the
kernel matrix in 64 bits, at leaf sizes around the 8- and 32-row pieces of a
tile and at every width class.  Bound per entry of Y, relative to |K| |X|: K
and X are each held as BF16 hi + lo (2^-17), the product of the two low parts
is left out (2^-16), and the FP32 entries and sums add less than 2^-18
together at these sizes: below 2^-15 in all."""
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


# (points, bucket): one leaf, two leaves, unequal leaves of many
@pytest.mark.parametrize("n,b", [(1, 32), (8, 32), (31, 32), (32, 32), (33, 64), (63, 32), (127, 64), (300, 32), (777, 200)])
def test_dense_products(hm, n, b):
    import torch

    rng = np.random.default_rng(n)
    p = rng.random((3, n)).astype(np.float32).astype(np.float64)
    pts = torch.from_numpy(np.ascontiguousarray(p.reshape(-1))).cuda()
    tree = hm.construct_kdtree(pts, n, 3, b)
    st = hm.construct_hmatrix_structure(tree, hm.BOX_CENTER, 1e-3)  # nothing is admissible above the leaves
    H = hm.build_hmatrix(tree, st, pts, kernel=hm.K_EXP, ell=0.2, nugget=0.5, tol=1e-12, max_rank=1, leaf_max_rank=1,
                         precision=hm.PREC_MIXED, diag_from_coords=0)
    assert H.stats()["num_lowrank"] == 0
    r = np.sqrt(((p[:, :, None] - p[:, None, :]) ** 2).sum(0))
    K = np.exp(-r / 0.2) + 0.5 * np.eye(n)
    X = rng.standard_normal((n, 130)).astype(np.float32)
    for nrhs in (1, 8, 16, 17, 33, 64, 65, 128, 130):
        Xg = torch.from_numpy(np.ascontiguousarray(X[:, :nrhs].T)).cuda().t()
        Y = H.matvec(Xg, original_order=True)
        H.check()
        err = np.abs(Y.cpu().numpy() - K @ X[:, :nrhs].astype(np.float64))
        assert (err <= 2.0**-15 * (np.abs(K) @ np.abs(X[:, :nrhs]))).all(), (nrhs, err.max())


def test_one_copy_of_the_dense_blocks(hm):
    n, b = 4096, 1024  # four diagonal blocks of whole tiles
    pts = hm.generate_dataset(n, 3, seed=1)
    tree = hm.construct_kdtree(pts, n, 3, b)
    st = hm.construct_hmatrix_structure(tree, hm.WEAK, 1.0)
    size = [
        hm.build_hmatrix(tree, st, pts, kernel=hm.K_MATERN32, ell=0.2, tol=1e-2, max_rank=128, leaf_max_rank=128,
                         precision=hm.PREC_MIXED, diag_from_coords=diag).stats()["device_bytes"] for diag in (0, 1)
    ]
    tiles = 4 * n * b  # hi and lo, 2 bytes each
    assert tiles <= size[0] - size[1] <= tiles + 4096
