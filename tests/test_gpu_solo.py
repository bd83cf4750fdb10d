"""Small matrices whose SpMV is one launch of the ring kernel over every block
row, the sliced ones among them: which matrices that is, and y bitwise the
reference order's either way."""
import numpy as np
import pytest

from abhsf_b200 import AbhsfMatrix
from oracle import oracle

pytestmark = pytest.mark.gpu


def _matrix(s, dense, wide, z, seed):
    """`dense` diagonal tiles about 30% full (bitmaps), then a block row of
    `wide` tiles of z elements (COO, at the wide end z = 1), ragged at the end."""
    rng = np.random.default_rng(seed)
    nb = max(dense + 2, wide + 1)  # the last block row and column, cut by three, stay empty
    n = nb * s - 3
    rows, cols = [], []
    for d in range(dense):
        k = np.nonzero(rng.random(s * s) < 0.3)[0]
        rows.append(d * s + k // s)
        cols.append(d * s + k % s)
    for J in rng.choice(nb - 1, wide, replace=False):
        k = rng.choice(s * s, z, replace=False)
        rows.append(dense * s + k // s)
        cols.append(J * s + k % s)
    r, c = np.concatenate(rows), np.concatenate(cols)
    ok = (r < n) & (c < n)
    key = np.unique(r[ok].astype(np.int64) * n + c[ok])
    return key // n, key % n, rng.standard_normal(key.size), n


def _check(r, c, v, n, s, vt, kernels):
    import torch
    rng = np.random.default_rng(5)
    A = AbhsfMatrix.from_elements(r, c, v, n, n, block_size=s, value_type=vt)
    assert A.kernels() == kernels
    x, y0 = rng.uniform(-1, 1, n), rng.standard_normal(n)
    if vt == "f64":
        y = torch.from_numpy(y0.copy()).cuda()
        A.spmv(torch.from_numpy(x).cuda(), y)
        ref = oracle.spmv_elements(r, c, v, x, y0.copy())
    else:
        x, y0 = x.astype(np.float32), y0.astype(np.float32)
        stored = torch.from_numpy(v).float()
        if vt == "bf16":
            stored = stored.bfloat16().float()
        y = torch.from_numpy(y0.copy()).cuda()
        A.spmv_f32(torch.from_numpy(x).cuda(), y)
        ref = oracle.spmv_elements_f32(r, c, stored.numpy(), x, y0.copy())
    assert np.array_equal(y.cpu().numpy(), ref)
    return A


@pytest.mark.parametrize("vt", ["f64", "f32", "bf16"])
@pytest.mark.parametrize("s", [32, 64])
@pytest.mark.parametrize("wide,z,kernels", [(1, 30, 1), (5, 40, 1), (6, 40, 2), (13, 8, 1), (14, 8, 2), (23, 1, 1),
                                            (24, 1, 2), (300, 8, 2), (3000, 1, 2)])
def test_a_wide_sliced_block_row_keeps_its_slices(gpu, s, vt, wide, z, kernels):
    """One CTA of the ring sums a whole block row: a sliced one is walked there
    while its tiles at 8 and up to 32 elements each are no more than 208, a wider
    one stays with the slices."""
    r, c, v, n = _matrix(s, 30, wide, z, seed=wide)
    _check(r, c, v, n, s, vt, kernels)


@pytest.mark.parametrize("tiles,kernels", [(4096, 1), (4097, 2)])
def test_tiles_of_a_one_launch_matrix(gpu, tiles, kernels):
    r, c, v, n = _matrix(32, tiles - 2, 2, 20, seed=1)
    A = _check(r, c, v, n, 32, "f64", kernels)
    assert A.stats()["tiles"] == tiles


@pytest.mark.parametrize("wide", [4, 300])
def test_bytes_an_spmv_reads(gpu, wide):
    """One launch reads the format and no slice; else the block row of `wide`
    tiles is read as slices (word and value an element, 32 bytes a slice, a lane
    record a row) in place of its share of the format (row pointer, 25 bytes of
    header and 16 of COO keys a tile, 8 an element)."""
    r, c, v, n = _matrix(64, 9, wide, 8, seed=2)
    A = AbhsfMatrix.from_elements(r, c, v, n, n, block_size=64)
    st, sl = A.stats(), A.slices()
    assert sl["block_rows"] == 1
    if A.kernels() == 1:
        assert st["spmv_bytes"] == st["format_bytes"]
        return
    share = 8 + (st["tiles"] - 9) * (25 + 16) + 8 * sl["elements"]
    assert st["spmv_bytes"] == st["format_bytes"] - share + 12 * sl["elements"] + 32 * sl["slices"] + \
        4 * int(sl["lanes"].sum())
