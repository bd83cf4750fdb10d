"""The chains (rows of more than 256 elements, summed by a whole warp): y must
be bitwise the additions in turn, for sums that cross binades, end in ties,
overflow or cancel, and at lengths around the groups of 512 elements (the SpMM: 128)."""
import numpy as np
import pytest

from abhsf_b200 import AbhsfBatch, AbhsfMatrix
from oracle import oracle

pytestmark = pytest.mark.gpu

LENGTHS = (257, 296, 297, 303, 511, 512, 513, 769, 1000, 4099, 20000)


def _values(kind, z, rng):
    if kind == "normal":
        return rng.standard_normal(z)
    if kind == "positive":
        return np.abs(rng.standard_normal(z))
    if kind == "ones":
        return np.ones(z)
    if kind == "ties":  # small multiples of half a spacing of the sums reached (y starts at 700)
        return (rng.integers(-4, 5, z)) * 2.0 ** -44
    if kind == "powers":
        return np.ldexp(rng.choice([-1.0, 1.0], z), -rng.integers(0, 60, z))
    if kind == "wide":
        return rng.standard_normal(z) * np.exp(rng.uniform(-30, 30, z))
    if kind == "zeros":
        return rng.choice([0.0, -0.0], z)
    if kind == "tiny":
        return rng.standard_normal(z) * 2.0 ** -1070
    v = rng.standard_normal(z)  # "special": the sums overflow, then become NaN in some rows
    v[z // 2] = np.inf
    v[z - 3] = -np.inf if z % 2 else 1.0
    return v


def _matrix(kind, seed=3):
    """One long row per length and a few short ones, n = 20,480; x of ones for
    the kinds whose products must be the values themselves."""
    rng = np.random.default_rng(seed)
    n = 20480
    rows, cols, vals = [], [], []
    for i, z in enumerate(LENGTHS):
        rows.append(np.full(z, 67 * i + 5))
        cols.append(np.sort(rng.choice(n, z, replace=False)))
        vals.append(_values(kind, z, rng))
    m = 67 * len(LENGTHS) + 5
    for r in range(0, m, 67):
        rows.append(np.full(7, r))
        cols.append(np.sort(rng.choice(n, 7, replace=False)))
        vals.append(rng.standard_normal(7))
    r, c, v = (np.concatenate(t) for t in (rows, cols, vals))
    x = rng.uniform(-1, 1, n) if kind in ("normal", "wide") else np.ones(n)
    y0 = np.full(m, 700.0) if kind == "ties" else -np.zeros(m) if kind == "zeros" else rng.standard_normal(m)
    return r.astype(np.int64), c.astype(np.int64), v, m, n, x, y0


def _same(a, b):
    nan = np.isnan(a) & np.isnan(b)
    return np.array_equal(a.view(np.uint8).reshape(a.size, -1)[~nan], b.view(np.uint8).reshape(b.size, -1)[~nan]) \
        and np.array_equal(np.isnan(a), np.isnan(b))


KINDS = ["normal", "positive", "ones", "ties", "powers", "wide", "zeros", "tiny", "special"]


@pytest.mark.parametrize("s", [16, 64, 256])
@pytest.mark.parametrize("kind", KINDS)
def test_chains_in_turn(gpu, kind, s):
    import torch
    r, c, v, m, n, x, y0 = _matrix(kind)
    order = np.lexsort((c, r))
    ref = oracle.spmv_elements(r[order], c[order], v[order], x, y0.copy())
    A = AbhsfMatrix.from_elements(r, c, v, m, n, block_size=s)
    assert np.count_nonzero(A.slices()["chain"]) == len(LENGTHS)
    y = torch.from_numpy(y0.copy()).cuda()
    A.spmv(torch.from_numpy(x).cuda(), y)
    assert _same(y.cpu().numpy(), ref)
    if s == 64:  # the batched kernel, and columns 0 .. k-1 of the SpMM ones
        B = AbhsfBatch([A, A])
        xs = [torch.from_numpy(x).cuda()] * 2
        ys = [torch.from_numpy(y0.copy()).cuda() for _ in range(2)]
        B.spmv(xs, ys)
        assert all(_same(t.cpu().numpy(), ref) for t in ys)


@pytest.mark.parametrize("k", [2, 5, 16])
@pytest.mark.parametrize("kind", KINDS)
def test_chains_in_turn_columns(gpu, kind, k):
    import torch
    r, c, v, m, n, x, y0 = _matrix(kind)
    order = np.lexsort((c, r))
    A = AbhsfMatrix.from_elements(r, c, v, m, n, block_size=64)
    X = np.stack([x * 2.0 ** (j % 3) for j in range(k)], axis=1).copy()
    Y = torch.from_numpy(np.repeat(y0[:, None], k, axis=1).copy()).cuda()
    A.spmm(torch.from_numpy(X).cuda(), Y)
    out = Y.cpu().numpy()
    for j in range(k):
        ref = oracle.spmv_elements(r[order], c[order], v[order], X[:, j].copy(), y0.copy())
        assert _same(np.ascontiguousarray(out[:, j]), ref)


@pytest.mark.parametrize("vt", ["f32", "bf16"])
@pytest.mark.parametrize("kind", ["normal", "positive", "ones", "powers", "zeros", "special"])
def test_chains_in_turn_f32(gpu, kind, vt):
    """In f32 a tie is one addition in a few hundred."""
    import torch
    r, c, v, m, n, x, y0 = _matrix(kind)
    x32, y32 = x.astype(np.float32), y0.astype(np.float32)
    order = np.lexsort((c, r))
    stored = torch.from_numpy(v[order]).float()
    if vt == "bf16":
        stored = stored.bfloat16().float()
    ref = oracle.spmv_elements_f32(r[order], c[order], stored.numpy(), x32, y32.copy())
    A = AbhsfMatrix.from_elements(r, c, v, m, n, block_size=64, value_type=vt)
    y = torch.from_numpy(y32.copy()).cuda()
    A.spmv_f32(torch.from_numpy(x32).cuda(), y)
    assert _same(y.cpu().numpy(), ref)
