"""Little device memory left: the library keeps at most 256 MB of what its
objects released, so that a program's other allocators can have the rest."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def hm():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import hmatrix

    return hmatrix


def test_little_is_kept_when_memory_is_short(hm):
    import torch

    n = 40000
    pts = hm.generate_dataset(n, 3, seed=1)

    def use():
        tree = hm.construct_kdtree(pts, n, 3, 64)
        st = hm.construct_hmatrix_structure(tree, hm.BOX_CENTER, 1.0)
        H = hm.build_hmatrix(tree, st, pts, kernel=hm.K_MATERN32, ell=0.2, nugget=1e-3, tol=1e-5, max_rank=128)
        b = torch.ones((n, 1), device="cuda")
        H.matvec(b)
        held = torch.cuda.mem_get_info()[0]
        H.free(), st.free(), tree.free()
        return held

    use()  # loads the kernels
    hm.release_memory()
    torch.cuda.empty_cache()
    hold = torch.empty(torch.cuda.mem_get_info()[0] - (6 << 30), dtype=torch.uint8, device="cuda")
    try:
        before = torch.cuda.mem_get_info()[0]
        assert before - use() > 1 << 30  # a matrix of some size
        torch.cuda.empty_cache()
        assert before - torch.cuda.mem_get_info()[0] <= (256 + 64) << 20
        rest = torch.empty(before - (512 << 20), dtype=torch.uint8, device="cuda")  # the rest of what was free
        del rest
    finally:
        del hold
        torch.cuda.empty_cache()
