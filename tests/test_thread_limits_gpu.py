"""Builds on several threads at once whose kernels need different amounts of
shared memory: a kernel's shared-memory limit is the process's, so no thread
may set it to its own launch's size.  Trees of 1 to 16 dimensions, whose
on-chip part differs in size, and matrices whose rank caps put the
orthogonalisation of every height class at 32 to 256 basis columns."""
import threading

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def hm():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import hmatrix

    return hmatrix


def _run(works):
    errors = []

    def guard(work):
        try:
            work()
        except Exception as e:  # reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=guard, args=(w,)) for w in works]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


def test_trees_of_different_sizes_at_once(hm):
    import torch

    shapes = [(40, 1, 4), (8192, 2, 32), (300, 3, 8), (2000, 16, 16)]
    clouds = [torch.rand(n * d, dtype=torch.float64, device="cuda") for n, d, _ in shapes]
    torch.cuda.synchronize()

    def work(i):
        n, d, b = shapes[i]
        s = torch.cuda.Stream()
        for _ in range(300):
            hm.construct_kdtree(clouds[i], n, d, b, stream=s).free()

    _run([lambda i=i: work(i) for i in range(len(shapes))])


@pytest.mark.parametrize("tol", [1e-4, 1e-6])  # FP32 and FP64 sketches
def test_matrices_of_different_rank_caps_at_once(hm, tol):
    import torch

    caps = [16, 64, 128, 256]

    def work(cap):
        s = torch.cuda.Stream()
        n = 2500
        pts = hm.generate_dataset(n, 3, seed=cap, stream=s)
        tree = hm.construct_kdtree(pts, n, 3, 128, stream=s)
        st = hm.construct_hmatrix_structure(tree, hm.BOX_CENTER, 1.0, stream=s)
        for _ in range(60):
            hm.build_hmatrix(tree, st, pts, kernel=hm.K_EXP, ell=0.2, tol=tol, max_rank=cap, leaf_max_rank=cap,
                             stream=s).free()

    _run([lambda c=c: work(c) for c in caps])
