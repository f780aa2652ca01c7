"""A build whose blocks all reach wide bases, with little more device memory
free than the finished matrix takes: what a batch of blocks needs while their
bases grow is kept within the memory there is, in smaller batches.

512 clouds of two 2048-point halves, one block pair each, sampled to 144
columns in rounds of 8 (wider than the truncation handles, so kept).  In FP32
words per row of a pair, N = 128: the finished matrix holds its factors and
their panels in both orders (6 * 144) and 65 words per point of vectors and
fragments (130), 7.77 N; one batch of all pairs holds the bases at 64, 128 and
256 columns and the sample (464), B, the packed basis and the factors (4 *
144), 8.13 N."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def hm():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import hmatrix

    return hmatrix


def test_batches_fit_the_memory_there_is(hm):
    import torch

    clouds, half = 512, 2048
    N = clouds * half * 128 * 4
    pts = hm.generate_dataset(2 * half, 3, seed=5)
    tree = hm.construct_kdtree(pts, 2 * half, 3, half)
    st = hm.construct_hmatrix_structure(tree, hm.WEAK, 1.0)

    def build(free):
        B = hm.Batch([tree] * clouds, [st] * clouds)
        torch.cuda.empty_cache()
        hm.release_memory()
        torch.cuda.synchronize()
        hold = None
        if free:
            hold = torch.empty(torch.cuda.mem_get_info()[0] - free, dtype=torch.uint8, device="cuda")
        try:
            B.build(kernel=hm.K_EXP, ell=0.2, tol=1.3e-2, max_rank=256, leaf_max_rank=256, sample_block=8,
                    diag_from_coords=1)
            H = B.hmatrix()
            s = H.stats()
            X = torch.ones((1, B.n), device="cuda").t()
            return s["num_lowrank"], s["rank_sum"], H.matvec(X).clone()
        finally:
            B.free()
            del hold
            torch.cuda.empty_cache()

    lr, ranks, Y = build(0)
    assert (lr, ranks) == (2 * clouds, 2 * clouds * 144)
    assert build(int(8.1 * N))[:2] == (lr, ranks)
    hm.release_memory()
