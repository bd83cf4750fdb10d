"""The builder's paths: input in row-major order (sorted by tile only) or in any
other (sorted whole), element counts around a CTA's chunk, every scheme; and
the slices of matrices whose sliced rows fall into several segments."""
import numpy as np
import pytest

from abhsf_b200 import AbhsfMatrix, capi
from oracle import oracle

pytestmark = pytest.mark.gpu

ARRAYS = ("brow_ptr", "tile_col", "tile_nnz", "tile_scheme", "tile_val_off", "tile_idx_off", "payload", "values")


def _elements(nnz, m, n, seed):
    rng = np.random.default_rng(seed)
    # dense, half-full and sparse corners, the rest anywhere
    at = [np.arange(min(nnz // 3, 40 * 300)) % 40 * n + np.arange(min(nnz // 3, 40 * 300)) // 40]
    at.append(rng.choice(m * n, nnz, replace=False))
    key = np.unique(np.concatenate(at))
    key = np.sort(rng.permutation(key)[:nnz])
    return key // n, key % n, rng.standard_normal(key.size)


def _order(kind, r, c, seed):
    if kind == "row":
        return np.lexsort((c, r))
    if kind == "column":
        return np.lexsort((r, c))
    return np.random.default_rng(seed).permutation(r.size)


@pytest.mark.parametrize("s", [16, 64, 256])
@pytest.mark.parametrize("kind", ["row", "column", "any"])
@pytest.mark.parametrize("nnz", [1, 2047, 2048, 2049, 30000])
def test_format_whatever_the_order(gpu, nnz, kind, s):
    m, n = 700, 900
    r, c, v = _elements(nnz, m, n, nnz)
    p = _order(kind, r, c, 5)
    A = AbhsfMatrix.from_elements(r[p], c[p], v[p], m, n, block_size=s)
    e, b = A.export(), oracle.build(r, c, v, m, n, s)
    for k in ARRAYS:
        np.testing.assert_array_equal(e[k], getattr(b, "idx" if k == "payload" else k), err_msg=k)
    st = A.stats()
    assert sum(st["tiles_per_scheme"].values()) == st["tiles"]
    assert sum(st["nnz_per_scheme"].values()) == st["nnz"] == r.size
    for i, name in enumerate(capi.SCHEME_NAMES):
        assert st["nnz_per_scheme"][name] == int(e["tile_nnz"][e["tile_scheme"] == i].sum())


@pytest.mark.parametrize("kind", ["row", "any"])
def test_duplicates_whatever_the_order(gpu, kind):
    r, c, v = _elements(3000, 700, 900, 9)
    r, c, v = np.append(r, r[1500]), np.append(c, c[1500]), np.append(v, 1.0)
    p = _order(kind, r, c, 6)
    with pytest.raises(capi.DuplicateEntry):
        AbhsfMatrix.from_elements(r[p], c[p], v[p], 700, 900, block_size=64)


@pytest.mark.parametrize("s", [16, 64])
def test_slices_of_several_segments(gpu, s):
    """Rows of 0, 1, ... 256 and more elements spread over the matrix: the
    segments' slices and chains, word for word the oracle's."""
    rng = np.random.default_rng(11)
    n, r, c = 5000, [], []
    for i in range(1500):
        z = int(rng.choice([0, 1, 2, 7, 40, 255, 256, 257, 400], p=[.2, .2, .2, .2, .1, .025, .025, .025, .025]))
        r.append(np.full(z, i))
        c.append(np.sort(rng.choice(n, z, replace=False)))
    r, c = np.concatenate(r).astype(np.int64), np.concatenate(c).astype(np.int64)
    v = rng.standard_normal(r.size)
    A = AbhsfMatrix.from_elements(r, c, v, 1500, n, block_size=s)
    b = oracle.build(r, c, v, 1500, n, s)
    got, want = A.slices(), b.slices(32.0)
    for k in ("base", "meta", "brow", "steps", "lanes", "chain", "lane", "words"):
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)
    held = want["vidx"] >= 0
    np.testing.assert_array_equal(got["values"][held], b.values[want["vidx"][held]])
