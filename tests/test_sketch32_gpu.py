"""The FP32 sketches and projections (tolerances from 5e-6 up, up to three
dimensions) over what changes their kernel: blocks whose columns end inside a
16-column step, sample blocks that fill a part of the 2, 4 and 8 column tiles,
bases past 32, 64 and 128 columns, every kernel and its derivative.

Every checked block below its rank cap meets its tolerance against the FP64
oracle, and the product agrees with dense FP64 rows at the tolerance."""
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


@pytest.mark.parametrize("n,d,b,kind,ell,tol,bs,cap,deriv", [
    (5003, 1, 32, 0, 0.3, 1e-4, 16, 64, 0),
    (6007, 2, 32, 1, 0.2, 1e-3, 5, 64, 0),
    (6007, 2, 64, 0, 0.1, 1e-4, 32, 64, 1),
    (6007, 2, 64, 1, 0.1, 1e-4, 24, 64, 1),
    (4099, 3, 64, 2, 0.4, 2e-5, 16, 200, 0),   # first round of 64 columns
    (4099, 3, 64, 2, 0.4, 1e-4, 8, 64, 1),
    (8009, 3, 128, 0, 0.2, 2e-5, 32, 256, 0),  # bases past 64 and 128 columns
    (1501, 3, 16, 1, 3.0, 1e-3, 16, 64, 0),    # leaves of 11-12 rows
])
def test_blocks_and_product(hm, n, d, b, kind, ell, tol, bs, cap, deriv):
    import torch

    pts = hm.generate_dataset(n, d, seed=n)
    tree = hm.construct_kdtree(pts, n, d, b)
    st = hm.construct_hmatrix_structure(tree, hm.BOX_CENTER, 1.0)
    H = hm.build_hmatrix(tree, st, pts, kernel=kind, ell=ell, tol=tol, max_rank=cap, sample_block=bs, derivative=deriv)
    perm, p = tree.copy_out()["perm"], pts.cpu().numpy()
    lr, _ = H.blocks()
    stored = np.flatnonzero((lr[:, 0] > lr[:, 2]) & (lr[:, 4] > 0))
    rng = np.random.default_rng(0)
    picks = rng.choice(stored, min(24, len(stored)), replace=False)
    if len(stored):
        picks = np.append(picks, stored[np.argmax(lr[stored, 4])])
    for i in picks:
        r0, m, c0, nn, k, _ = (int(v) for v in lr[i])
        U, V = H.block_factors(int(i))
        err = oracle.block_error(p, n, d, perm, kind, ell, 0.0, r0, m, c0, nn, U, V, deriv=deriv)
        assert err <= tol or k == min(m, nn, cap), (m, nn, k, err)
    x = rng.standard_normal(n)
    y = H.matvec(torch.from_numpy(x.astype(np.float32)).cuda()[:, None]).cpu().numpy()[:, 0]
    rows = np.arange(0, n, 37)
    ref = oracle.dense_rows_matvec(p, n, d, perm, kind, ell, 0.0, rows, x.astype(np.float32).astype(np.float64),
                                   deriv=deriv)[0]
    assert np.linalg.norm(y[rows] - ref) <= 2 * tol * np.linalg.norm(ref)
