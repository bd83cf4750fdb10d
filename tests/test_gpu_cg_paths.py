"""The paths of the CG solvers: vectors longer than a step of the vector
kernels' grid, products that set y (slices and chains serve every row) and
products that add onto it, rows of more than 256 elements in chains, and
solves that end at their start.  The residual is checked on the CPU from the
returned x; a solve does not depend on which kernels serve its products, so x is
also compared bitwise between them."""
import numpy as np
import pytest

from abhsf_b200 import AbhsfMatrix, cg, cg_mixed
from abhsf_b200 import workloads as W
from oracle import oracle

pytestmark = pytest.mark.gpu


def _residual(coo, b, x):
    ax = oracle.spmv_elements(coo.rows, coo.cols, coo.vals, x, np.zeros(coo.m))
    return np.linalg.norm(b - ax) / np.linalg.norm(b)


def _arrow(n, reach, dense=0):
    """Symmetric, diagonally dominant: a 1D Laplacian, a first row and column of
    `reach` elements, and `dense` leading 64 x 64 diagonal tiles half full."""
    rng = np.random.default_rng(3)
    i = np.arange(n - 1)
    j = np.sort(rng.choice(np.arange(2, n), reach, replace=False))
    v = rng.uniform(-0.01, 0.01, reach)
    rows, cols, vals = [i, i + 1, np.zeros(reach, np.int64), j], [i + 1, i, j, np.zeros(reach, np.int64)], \
        [np.full(n - 1, -1.0), np.full(n - 1, -1.0), v, v]
    for t in range(dense):
        p, q = np.nonzero(np.triu(rng.random((64, 64)) < 0.5, 2))
        keep = p + 64 * t > 0  # the first row is the arrow's
        p, q = p[keep] + 64 * t, q[keep] + 64 * t
        w = rng.uniform(-0.02, 0.02, p.size)
        rows, cols, vals = rows + [p, q], cols + [q, p], vals + [w, w]
    r, c, v = (np.concatenate(t) for t in (rows, cols, vals))
    d = np.zeros(n)
    np.add.at(d, r, np.abs(v))
    r, c, v = np.concatenate([r, np.arange(n)]), np.concatenate([c, np.arange(n)]), np.concatenate([v, d + 0.05])
    order = np.lexsort((c, r))
    return W.Coo(r[order].astype(np.int64), c[order].astype(np.int64), v[order], n, n)


def _build(coo, s=64, vt="f64", slices=True):
    return AbhsfMatrix.from_elements(coo.rows, coo.cols, coo.vals, coo.m, coo.n, block_size=s, value_type=vt,
                                     slice_tile_nnz=0 if slices else -1)


def _solve(coo, A, lo=None, rtol=1e-10, offset=0, **kw):
    import torch
    b = np.random.default_rng(7).uniform(-1, 1, coo.n)
    bd, xd = (torch.zeros(coo.n + 1, dtype=torch.float64, device="cuda")[offset:offset + coo.n] for _ in range(2))
    bd.copy_(torch.from_numpy(b))
    info = cg(A, bd, xd, rtol=rtol, **kw) if lo is None else cg_mixed(A, lo, bd, xd, rtol=rtol, **kw)
    return b, xd.cpu().numpy(), info


def _check(coo, b, x, info, rtol=1e-10):
    r = _residual(coo, b, x)
    assert info["converged"] and r <= rtol and abs(r - info["rel_residual"]) <= 1e-12


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("low", [None, "f32", "bf16"])
def test_more_unknowns_than_a_step_of_the_grid(gpu, low, offset):
    """87^3 = 658,503 unknowns, odd: three steps of 16-byte packs in FP64, two in
    f32; five of single elements (offset 1: 8 bytes off a 16-byte boundary)."""
    coo = W.laplacian_3d(87)
    A = _build(coo)
    lo = _build(coo, 32, low) if low else None
    _check(coo, *_solve(coo, A, lo, offset=offset))


@pytest.mark.parametrize("low", [None, "f32", "bf16"])
@pytest.mark.parametrize("s", [16, 32, 64, 128, 256])
def test_products_that_set_y_and_that_add(gpu, s, low):
    coo = W.laplacian_2d(61)
    rows = -(-coo.n // s)
    out = []
    for slices in (True, False):
        A = _build(coo, 64 if low else s, slices=slices)
        lo = _build(coo, s, low, slices) if low else None
        assert (lo or A).slices()["block_rows"] == (rows if slices else 0)
        b, x, info = _solve(coo, A, lo)
        _check(coo, b, x, info)
        out.append((x, info["iterations"], info["outer_iterations"]))
    assert np.array_equal(out[0][0], out[1][0]) and out[0][1:] == out[1][1:]


@pytest.mark.parametrize("low", [None, "f32", "bf16"])
@pytest.mark.parametrize("s", [16, 64, 256])
@pytest.mark.parametrize("dense", [0, 3])
def test_a_row_in_a_chain(gpu, dense, s, low):
    """dense = 0: chains and slices serve every row, and their product sets y;
    else bitmap tiles go to the ring or streaming kernel, which adds."""
    coo = _arrow(5001, 1500, dense)
    out = []
    for slices in (True, False):
        A = _build(coo, 64 if low else s, slices=slices)
        lo = _build(coo, s, low, slices) if low else None
        if slices and not dense:
            assert np.count_nonzero((lo or A).slices()["chain"]) == 1
        b, x, info = _solve(coo, A, lo)
        _check(coo, b, x, info)
        out.append((x, info["iterations"], info["outer_iterations"]))
    assert out[0][1] > 20
    assert np.array_equal(out[0][0], out[1][0]) and out[0][1:] == out[1][1:]


@pytest.mark.parametrize("slices", [True, False])
@pytest.mark.parametrize("most", [0, 1, 5, 8, 9, 24])
def test_iteration_limits(gpu, slices, most):
    coo = W.laplacian_2d(40)
    A = _build(coo, slices=slices)
    b, x, info = _solve(coo, A, max_iters=most)
    assert not info["converged"] and info["iterations"] == most
    assert (most == 0) == (not x.any())
    assert abs(_residual(coo, b, x) - info["rel_residual"]) <= 1e-12


@pytest.mark.parametrize("slices", [True, False])
def test_a_solve_that_is_done_at_its_start(gpu, slices):
    import torch
    coo = W.laplacian_2d(40)
    A = _build(coo, slices=slices)
    lo = _build(coo, 32, "f32", slices)
    z = torch.zeros(coo.n, dtype=torch.float64, device="cuda")
    for info in (cg(A, z, z.clone()), cg_mixed(A, lo, z, z.clone())):
        assert info["converged"] and info["iterations"] == 0
    x = torch.ones(coo.n, dtype=torch.float64, device="cuda")
    b = torch.zeros_like(x)
    A.spmv(x, b)
    info = cg(A, b, x)
    assert info["converged"] and info["iterations"] == 0 and bool((x == 1).all())
