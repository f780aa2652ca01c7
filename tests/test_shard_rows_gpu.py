"""A block-row shard's product leaves the rows of Y that are not its own as they
are, in either order of the points, for every way in which Y is written: by
phase 2 itself, through a workspace and a scatter (more than 64 right-hand
sides, diagonal blocks from coordinates, the per-block kernels), and from
FP64 vectors.  Its own rows equal those of the product in tree order."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def hm():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import hmatrix

    return hmatrix


@pytest.mark.parametrize("mixed,diag,schedule,nrhs", [
    (1, 0, None, 5), (1, 0, None, 40), (1, 0, None, 65), (1, 0, None, 128), (1, 1, None, 5), (1, 1, None, 130),
    (0, 0, None, 5), (0, 1, None, 20), (0, 0, "fp32 p1_rows=256", 5),
])
@pytest.mark.parametrize("f64", [False, True])
def test_other_rows_stay(hm, mixed, diag, schedule, nrhs, f64):
    import torch

    n = 5003
    pts = hm.generate_dataset(n, 3, seed=2)
    tree = hm.construct_kdtree(pts, n, 3, 64)
    st = hm.construct_hmatrix_structure(tree, hm.BOX_CENTER, 1.0)
    t = tree.copy_out()
    offs, perm = t["offsets"], torch.from_numpy(t["perm"]).cuda().long()
    dtype = torch.float64 if f64 else torch.float32
    X = torch.randn((nrhs, n), device="cuda", dtype=dtype).t()
    Xt = X.t()[:, perm].contiguous().t()
    for lo, hi in ((0, 37), (37, 64), (64, len(offs) - 1)):
        H = hm.build_hmatrix(tree, st, pts, kernel=hm.K_MATERN32, ell=0.2, nugget=1e-3, tol=1e-4, max_rank=128,
                             precision=hm.PREC_MIXED if mixed else hm.PREC_FP32, diag_from_coords=diag, leaves=(lo, hi))
        if schedule:
            hm.schedule_set(H, schedule)
        call = H.matvec_f64 if f64 else H.matvec
        Yt = torch.full((nrhs, n), float("nan"), device="cuda", dtype=dtype).t()
        Yo = torch.full((nrhs, n), float("nan"), device="cuda", dtype=dtype).t()
        call(Xt, Y=Yt)
        call(X, Y=Yo, original_order=True)
        own = torch.zeros(n, dtype=torch.bool, device="cuda")
        own[int(offs[lo]):int(offs[hi])] = True
        Yo_tree = Yo.t()[:, perm].t()
        for Y in (Yt, Yo_tree):
            assert torch.isfinite(Y[own]).all()
            assert torch.isnan(Y[~own]).all()
        assert torch.equal(Yo_tree[own], Yt[own])
