"""Boxes and split dimensions of every node that has points, trees with empty
leaves included, bit for bit against the oracle: subtrees whose segments share
the CTA's warps (several per segment, one each, several segments per warp),
the last step of a box when leaves are ragged, and ties between dimensions."""
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


@pytest.mark.parametrize("kind", ["uniform", "lattice", "cube"])
@pytest.mark.parametrize("n,d,b", [(3, 2, 1), (5, 1, 1), (33, 3, 1), (65, 3, 1), (100, 2, 3), (1000, 3, 7), (1001, 5, 1),
                                   (4097, 3, 64), (8191, 1, 4), (8193, 2, 32), (5000, 16, 16), (30001, 3, 2)])
def test_every_node(hm, kind, n, d, b):
    import torch

    rng = np.random.default_rng(7 * n + d)
    p = rng.random((d, n))
    if kind == "lattice":
        p = rng.integers(-3, 4, (d, n)).astype(np.float64) / 4
    elif kind == "cube":  # every dimension has the same extent: ties go to the first
        p = np.round(p * 8) / 8
        p[:, 0], p[:, 1] = 0.0, 1.0
    p = np.ascontiguousarray(p)
    tree = hm.construct_kdtree(torch.from_numpy(p.reshape(-1)).cuda(), n, d, b)
    got, ref = tree.copy_out(), oracle.kdtree(p.reshape(-1), n, d, b)
    depth = ref["depth"]
    assert tree.depth == depth
    np.testing.assert_array_equal(got["offsets"], ref["offsets"])
    offs = ref["offsets"].astype(np.int64)
    x = p[:, ref["perm"]]
    for level in range(depth + 1):
        nodes = 1 << level
        starts = offs[:: 1 << (depth - level)]
        first = nodes - 1
        some = np.flatnonzero(starts[1:] > starts[:-1])
        lo = np.stack([x[:, starts[a]:starts[a + 1]].min(1) for a in some])
        hi = np.stack([x[:, starts[a]:starts[a + 1]].max(1) for a in some])
        at = first + some
        for k, want in (("bmin", lo), ("bmax", hi)):
            np.testing.assert_array_equal(got[k].reshape(-1, d)[at], want)
            np.testing.assert_array_equal(ref[k].reshape(-1, d)[at], want)
        if level < depth:
            many = np.flatnonzero(starts[1:] - starts[:-1] > 0)
            np.testing.assert_array_equal(got["split_dim"][first + many], ref["split_dim"][first + many])
