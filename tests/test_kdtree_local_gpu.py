"""The on-chip part of the KD tree over the sizes at which it changes: subtrees
of less than a warp, of a power of two and one past it, odd splits at every
level, empty leaves (bucket 1), coordinates whose leading 32 bits agree, exact
ties and duplicate points, and the most points one CTA takes.  Permutation,
offsets, boxes and split dimensions equal the oracle's bit for bit."""
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


def _points(kind, n, d, rng):
    if kind == "uniform":
        return rng.random((d, n))
    if kind == "close":  # equal in their leading 32 bits
        return 0.5 + 1e-12 * rng.random((d, n))
    if kind == "lattice":  # exact ties in every dimension, duplicates
        return rng.integers(-3, 4, (d, n)).astype(np.float64) / 4
    return np.where(rng.random((d, n)) < 0.5, -0.0, 0.0) * np.ones((d, n))  # one point, both zeros


@pytest.mark.parametrize("kind", ["uniform", "close", "lattice", "zeros"])
@pytest.mark.parametrize("n,d,b", [(1, 1, 1), (3, 2, 1), (31, 3, 2), (33, 1, 1), (64, 2, 8), (65, 3, 1), (1000, 3, 7),
                                   (4097, 3, 64), (8191, 1, 4), (8192, 2, 32), (8193, 2, 32), (5000, 16, 16)])
def test_tree_equals_oracle(hm, kind, n, d, b):
    import torch

    p = np.ascontiguousarray(_points(kind, n, d, np.random.default_rng(n + d)))
    pts = torch.from_numpy(p.reshape(-1)).cuda()
    tree = hm.construct_kdtree(pts, n, d, b)
    got, ref = tree.copy_out(), oracle.kdtree(p.reshape(-1), n, d, b)
    assert tree.depth == ref["depth"]
    np.testing.assert_array_equal(got["perm"], ref["perm"])
    np.testing.assert_array_equal(got["offsets"], ref["offsets"])
    full = (np.diff(ref["offsets"]) > 0).all()
    for k in ("bmin", "bmax"):
        if full:  # an empty leaf has no box to compare
            np.testing.assert_array_equal(got[k][: len(ref[k])], ref[k])
