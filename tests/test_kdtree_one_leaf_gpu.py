"""Trees of a single leaf: nothing to sort, so a CTA's shared memory holds as
many points as their coordinates allow.  Up to 8192 points in 1 or 2
dimensions, 4096 up to 6, 2048 up to 13 and 1024 up to 16; one more point is
refused.  Permutation and box equal the oracle's bit for bit."""
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


@pytest.mark.parametrize("d,most", [(1, 8192), (2, 8192), (3, 4096), (6, 4096), (7, 2048), (13, 2048), (14, 1024), (16, 1024)])
def test_one_leaf(hm, d, most):
    import torch

    rng = np.random.default_rng(d)
    for n in (most, most // 2 + 1):
        p = rng.random((d, n))
        tree = hm.construct_kdtree(torch.from_numpy(p.reshape(-1)).cuda(), n, d, most)
        got, ref = tree.copy_out(), oracle.kdtree(p.reshape(-1), n, d, most)
        assert tree.depth == ref["depth"] == 0
        for k in ("perm", "offsets"):
            np.testing.assert_array_equal(got[k], ref[k])
        for k in ("bmin", "bmax"):
            np.testing.assert_array_equal(got[k][:d], ref[k][:d])
    n = most + 1
    with pytest.raises(hm.HMError):
        hm.construct_kdtree(torch.zeros(n * d, dtype=torch.float64, device="cuda"), n, d, n)
    torch.cuda.synchronize()  # the refusal leaves no error behind
