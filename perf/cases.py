"""The work that users of this engine have it do, as measurable cases.

Each case is one call, or one short sequence of calls, of the Python binding
(hmatrix.py) on seeded points: clustering, building, multiplying, gradients
with respect to the vectors and the length scale, batches of clouds, solving.
Sizes, kernels and tolerances are those of the benchmark's workloads and of
the tests, at the sizes between them too, odd ones included.

    listed()            the named cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) what the caller has in hand before the call
    run(state)          one pass
    work(case)          bytes and operations that a pass cannot do without
    exact(case, seed)   the result in 64 bits, from dense kernel matrices
"""
import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "kaust-hierarchical-matrices_b200"))

import hmatrix as hm  # noqa: E402

KERNELS = {"exp": hm.K_EXP, "matern32": hm.K_MATERN32, "gauss": hm.K_GAUSS}

# The families of operators: what stays fixed while the number of points goes
# over a range.  `stored`: bytes of factors and dense blocks per point, each
# value once in its stored type, at 2^17 points, and its growth per doubling
# (hm_hmatrix_stats of such matrices); `rank`: their mean block rank.
FAMILIES = {
    # the plain method at its small size (2-D, exponential kernel, tight tolerance)
    "plain": dict(points="uniform", d=2, bucket=32, kernel="exp", ell=0.1, nugget=0.0, eta=1.0, tol=1e-6,
                  max_rank=64, precision="fp32", stored=(3900, 250), rank=12),
    # the precision workload in either form
    "precision": dict(points="uniform", d=3, bucket=64, kernel="matern32", ell=0.2, nugget=1e-3, eta=1.0, tol=1e-4,
                      max_rank=128, precision="mixed", stored=(4800, 240), rank=9),
    "precision_fp32": dict(points="uniform", d=3, bucket=64, kernel="matern32", ell=0.2, nugget=1e-3, eta=1.0,
                           tol=1e-4, max_rank=128, precision="fp32", stored=(7300, 500), rank=9),
    # the differentiation workload's kernel
    "gauss": dict(points="uniform", d=3, bucket=64, kernel="gauss", ell=0.15, nugget=0.0, eta=1.0, tol=1e-5,
                  max_rank=128, precision="fp32", stored=(15000, 1200), rank=20),
    # the scale stress: unbalanced clouds, variable ranks up to a high cap
    "mixture": dict(points="mixture", d=3, bucket=64, kernel="exp", ell=0.05, nugget=0.0, eta=1.5, tol=1e-4,
                    max_rank=256, precision="mixed", stored=(5400, 900), rank=19),
    # the batch workload's clouds
    "clouds": dict(points="uniform", d=3, bucket=64, kernel="exp", ell=0.1, nugget=0.0, eta=1.0, tol=1e-5,
                   max_rank=64, precision="mixed", stored=(20000, 2000), rank=18),
    # a kernel ridge system: nugget of the kernel's own scale
    "ridge": dict(points="uniform", d=3, bucket=64, kernel="matern32", ell=0.2, nugget=1.0, eta=1.0, tol=1e-6,
                  max_rank=64, precision="fp32", stored=(14000, 1500), rank=22),
}


def listed():
    return [
        # a new cloud is clustered and its block structure asked for: the headline's number of points
        dict(name="tree_1m", do="tree", points="uniform", n=1 << 20, d=3, bucket=64, eta=1.0),
        # points to first product, the plain method's small size: a user's first program
        dict(name="build_plain_8k", do="build", family="plain", n=8192, nrhs=1),
        # points to first product, mixed precision, the headline's settings
        dict(name="build_precision_128k", do="build", family="precision", n=1 << 17, nrhs=16),
        # points to first product for an unbalanced cloud with high ranks, an odd number of points
        dict(name="build_mixture_60k", do="build", family="mixture", n=60001, nrhs=8),
        # one step of fitting the length scale: K and dK/dl on a kept structure, value, adjoint, derivative
        dict(name="grad_gauss_20k", do="grad", family="gauss", n=20000, nrhs=1),
        # an interactive product: small matrix, one vector, the points' own order
        dict(name="apply_plain_8k", do="apply", family="plain", n=8192, nrhs=1, original=True),
        # a few vectors on a matrix of ordinary size, FP32, odd sizes throughout
        dict(name="apply_fp32_100k", do="apply", family="precision_fp32", n=100003, nrhs=5, original=True),
        # the headline product: 2^20 points, 16 right-hand sides, tree order
        dict(name="apply_precision_1m", do="apply", family="precision", n=1 << 20, nrhs=16, original=False),
        # many right-hand sides in one pass, unbalanced cloud
        dict(name="apply_mixture_128k", do="apply", family="mixture", n=1 << 17, nrhs=128, original=True),
        # adjoint product with the derivative matrix, whose diagonal blocks come from the coordinates
        dict(name="adjoint_deriv_30k", do="adjoint", family="gauss", n=30011, nrhs=2, original=True),
        # a batch of clouds, one recorded graph per product
        dict(name="batch_12_clouds", do="batch", family="clouds", n=8192, clouds=12, nrhs=32),
        # kernel ridge regression: a few right-hand sides by conjugate gradients
        dict(name="solve_ridge_16k", do="solve", family="ridge", n=16384, nrhs=4, tol_cg=1e-6),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    do = rng.choice(["tree", "build", "build", "grad", "apply", "apply", "apply", "adjoint", "batch", "solve"])
    if do == "tree":
        return dict(do=do, points=rng.choice(["uniform", "mixture"]), n=_log_int(rng, 2000, 1 << 20),
                    d=rng.choice([2, 3]), bucket=rng.choice([32, 64]), eta=rng.choice([1.0, 1.5]))
    if do == "build":
        family = rng.choice(["plain", "precision", "precision_fp32", "mixture"])
        top = {"plain": 1 << 17, "mixture": 60001}.get(family, 1 << 17)
        return dict(do=do, family=family, n=_log_int(rng, 3000, top), nrhs=rng.randint(1, 16))
    if do == "grad":
        return dict(do=do, family="gauss", n=_log_int(rng, 3000, 20000), nrhs=rng.randint(1, 4))
    if do == "apply":
        family = rng.choice(["plain", "precision", "precision", "precision_fp32", "mixture"])
        top = {"plain": 1 << 17, "precision": 1 << 20, "precision_fp32": 1 << 18}.get(family, 1 << 17)
        nrhs = rng.choice([1, rng.randint(2, 15), 16, rng.randint(17, 64), 128])
        return dict(do=do, family=family, n=_log_int(rng, 3000, top), nrhs=nrhs, original=rng.random() < 0.7)
    if do == "adjoint":
        return dict(do=do, family="gauss", n=_log_int(rng, 3000, 30011), nrhs=rng.randint(1, 4), original=True)
    if do == "batch":
        return dict(do=do, family="clouds", n=_log_int(rng, 2500, 10000), clouds=rng.randint(3, 12),
                    nrhs=rng.choice([1, 16, 32]))
    return dict(do=do, family="ridge", n=_log_int(rng, 2000, 16384), nrhs=rng.randint(1, 8), tol_cg=1e-6)


# --- inputs ------------------------------------------------------------------


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _points(kind, n, d, g):
    """(d, n) float64: uniform in the unit cube, or a 16-component isotropic
    Gaussian mixture (sigma log-uniform in [0.01, 0.1], flat Dirichlet weights)."""
    if kind == "uniform":
        return torch.rand((d, n), dtype=torch.float64, device="cuda", generator=g)
    k = 16
    centres = torch.rand((d, k), dtype=torch.float64, device="cuda", generator=g)
    sigma = 0.01 * 10 ** torch.rand(k, dtype=torch.float64, device="cuda", generator=g)
    weights = -torch.log(1.0 - torch.rand(k, dtype=torch.float64, device="cuda", generator=g))
    of = torch.multinomial(weights, n, replacement=True, generator=g)
    noise = torch.randn((d, n), dtype=torch.float64, device="cuda", generator=g)
    return (centres[:, of] + sigma[of] * noise).contiguous()


def _vectors(n, nrhs, g):
    """(n, nrhs) float32, column-major as the engine takes it."""
    return torch.randn((nrhs, n), dtype=torch.float32, device="cuda", generator=g).t()


def _build(f, tree, structure, points, **more):
    kw = dict(kernel=KERNELS[f["kernel"]], ell=f["ell"], nugget=f["nugget"], tol=f["tol"], max_rank=f["max_rank"],
              precision=hm.PREC_MIXED if f["precision"] == "mixed" else hm.PREC_FP32)
    kw.update(more)
    return hm.build_hmatrix(tree, structure, points, **kw)


def _cloud_sizes(case):
    """Log-uniform within a factor of four below and above n, multiples of 32 of at least 2048."""
    r = random.Random(case["clouds"])
    return [max(2048, 32 * round(case["n"] * 4.0 ** r.uniform(-1, 1) / 32)) for _ in range(case["clouds"])]


def _block_room(case):
    """Room for the block list of each level: what a user who clusters clouds of one size keeps."""
    levels = max(0, math.ceil(math.log2(case["n"] / case["bucket"])))
    return [min(4 ** lv, 256 * 2 ** lv) for lv in range(1, levels + 1)]


def _inputs(case, seed):
    """The random part of a case: the same for prepare and exact."""
    g = _generator(seed)
    if case["do"] == "tree":
        return _points(case["points"], case["n"], case["d"], g), None
    f = FAMILIES[case["family"]]
    if case["do"] == "batch":
        clouds = [_points(f["points"], n, f["d"], g) for n in _cloud_sizes(case)]
        return clouds, _vectors(sum(p.shape[1] for p in clouds), case["nrhs"], g)
    p = _points(f["points"], case["n"], f["d"], g)
    x = _vectors(case["n"], case["nrhs"], g)
    if case["do"] == "grad":
        return p, (x, _vectors(case["n"], case["nrhs"], g))
    return p, x


def prepare(case, seed):
    points, x = _inputs(case, seed)
    state = dict(case=case, points=points, x=x)
    do = case["do"]
    if do == "tree":
        state["blocks"] = [np.full(room, -1, np.int32) for room in _block_room(case)]
    if do in ("tree", "build"):
        return state
    f = FAMILIES[case["family"]]
    if do == "batch":
        trees = [hm.construct_kdtree(p, p.shape[1], f["d"], f["bucket"]) for p in points]
        structures = [hm.construct_hmatrix_structure(t, hm.BOX_CENTER, f["eta"]) for t in trees]
        stream = torch.cuda.Stream()
        batch = hm.Batch(trees, structures)
        batch.build(kernel=KERNELS[f["kernel"]], ell=f["ell"], tol=f["tol"], max_rank=f["max_rank"],
                    precision=hm.PREC_MIXED)
        torch.cuda.synchronize()
        state.update(batch=batch, stream=stream, y=torch.empty_like(x.t()).t())
        return state
    tree = hm.construct_kdtree(points, case["n"], f["d"], f["bucket"])
    structure = hm.construct_hmatrix_structure(tree, hm.BOX_CENTER, f["eta"])
    state.update(tree=tree, structure=structure)
    if do == "apply":
        state["H"] = _build(f, tree, structure, points)
    elif do == "adjoint":
        state["H"] = _build(f, tree, structure, points, derivative=1)
    elif do == "solve":
        state["H"] = _build(f, tree, structure, points)
        perm = torch.from_numpy(tree.copy_out()["perm"]).cuda().long()
        state["b"] = x.t()[:, perm].contiguous().t()  # the solver works in tree order
        state["back"] = torch.argsort(perm)
    return state


# --- one pass ----------------------------------------------------------------


def run(state):
    case = state["case"]
    do = case["do"]
    if do == "tree":
        tree = hm.construct_kdtree(state["points"], case["n"], case["d"], case["bucket"])
        structure = hm.construct_hmatrix_structure(tree, hm.BOX_CENTER, case["eta"])
        for kept, tiles in zip(state["blocks"], structure.all_tiles()):
            kept[: len(tiles)] = tiles
        return dict(tree.copy_out(), counts=structure.counts, blocks=state["blocks"])
    if do == "apply":
        return state["H"].matvec(state["x"], original_order=case["original"])
    if do == "adjoint":
        return state["H"].matvec(state["x"], trans=1, original_order=case["original"])
    if do == "batch":
        state["stream"].wait_stream(torch.cuda.current_stream())
        y = state["batch"].matvec(state["x"], state["y"], state["stream"], original_order=True)
        torch.cuda.current_stream().wait_stream(state["stream"])
        return y
    if do == "solve":
        x, _, _ = hm.cg_solve(state["H"], state["b"], tol=case["tol_cg"], max_iter=1000)
        return x.t()[:, state["back"]].t()
    f = FAMILIES[case["family"]]
    if do == "build":
        tree = hm.construct_kdtree(state["points"], case["n"], f["d"], f["bucket"])
        structure = hm.construct_hmatrix_structure(tree, hm.BOX_CENTER, f["eta"])
        return _build(f, tree, structure, state["points"]).matvec(state["x"], original_order=True)
    # grad: y = H x, the adjoint H^T w and (dH/dl) x
    x, w = state["x"]
    H = _build(f, state["tree"], state["structure"], state["points"])
    D = _build(f, state["tree"], state["structure"], state["points"], derivative=1)
    return dict(y=H.matvec(x, original_order=True), gx=H.matvec(w, trans=1, original_order=True),
                dy=D.matvec(x, original_order=True))


# --- what a pass cannot do without ---------------------------------------------


def _stored(f, n):
    at, step = f["stored"]
    return n * max(at + step * (math.log2(n) - 17), 0.25 * at)


def work(case):
    """Bytes: points, stored factors and dense blocks, vectors, each once.
    Operations: a product's multiply-adds; a build's two passes over the
    kernel entries of one triangle (a sample and a projection, of the mean
    rank each, and about ten operations per entry)."""
    do, n = case["do"], case["n"]
    if do == "tree":
        levels = max(1, math.ceil(math.log2(n / case["bucket"])))
        boxes = 2 * 2 ** (levels + 1) * case["d"] * 8
        return dict(bytes=8 * case["d"] * n + 4 * n + boxes, flops=n * levels)
    f = FAMILIES[case["family"]]
    width = 2 if f["precision"] == "mixed" else 4
    vec = 8 * case["nrhs"]
    if do == "batch":
        sizes = _cloud_sizes(case)
        total = sum(sizes)
        stored = sum(_stored(f, m) for m in sizes)
        return dict(bytes=stored + total * vec, flops=4 * stored / width * case["nrhs"])
    stored = _stored(f, n)
    apply_flops = 4 * stored / width * case["nrhs"]
    build_flops = n * n * (2 * f["rank"] + 10)
    if do == "build":
        return dict(bytes=8 * f["d"] * n + stored + n * vec, flops=build_flops + apply_flops)
    if do == "grad":
        return dict(bytes=8 * f["d"] * n + 2 * stored + 2.5 * n * vec, flops=2 * build_flops + 3 * apply_flops)
    if do == "solve":
        return dict(bytes=20 * (stored + 3 * n * vec), flops=20 * apply_flops)  # about 20 iterations
    return dict(bytes=stored + n * vec, flops=apply_flops)


# --- in 64 bits ------------------------------------------------------------------


def _dense_rows(p, r0, r1, f, deriv=False):
    """Rows [r0, r1) of the kernel matrix of the points p (d, n), float64."""
    r = torch.cdist(p.t()[r0:r1], p.t(), compute_mode="donot_use_mm_for_euclid_dist")
    ell = f["ell"]
    if f["kernel"] == "gauss":
        q = r.square_().mul_(1.0 / (ell * ell))
        k = torch.exp(q * -0.5)
        return k.mul_(q).mul_(1.0 / ell) if deriv else k
    if f["kernel"] == "matern32":
        a = r.mul_(math.sqrt(3.0) / ell)
        k = torch.exp(-a)
        k = k.mul_(a.add_(1.0))
    else:
        k = torch.exp_(r.mul_(-1.0 / ell))
    if f["nugget"]:
        i = torch.arange(r0, r1, device=p.device)
        k[i - r0, i] += f["nugget"]
    return k


def _dense_apply(p, x, f, deriv=False):
    n = p.shape[1]
    y = torch.empty((n, x.shape[1]), dtype=torch.float64, device="cuda")
    step = max(1, (1 << 27) // n)
    for r0 in range(0, n, step):
        r1 = min(n, r0 + step)
        y[r0:r1] = _dense_rows(p, r0, r1, f, deriv) @ x
    return y


def exact(case, seed):
    if case["do"] == "tree":
        return None  # whole numbers, and boxes that are coordinates of the points
    if case["n"] > 300000 or (case["do"] == "apply" and not case["original"]):
        return None
    f = FAMILIES[case["family"]]
    p, x = _inputs(case, seed)
    if case["do"] == "batch":
        parts, at = [], 0
        for q in p:
            parts.append(_dense_apply(q, x[at:at + q.shape[1]].double(), f))
            at += q.shape[1]
        return torch.cat(parts)
    if case["do"] == "solve":
        return torch.linalg.solve(_dense_rows(p, 0, case["n"], f), x.double())
    if case["do"] == "grad":
        x, w = x
        return dict(y=_dense_apply(p, x.double(), f), gx=_dense_apply(p, w.double(), f),
                    dy=_dense_apply(p, x.double(), f, deriv=True))
    return _dense_apply(p, x.double(), f, deriv=case["do"] == "adjoint")
