"""SpMM over sliced rows: 16 columns by a quarter of a slice's rows where there
are many short slices, 4 columns by all 32 rows otherwise and for the columns past
the last 16.  Every column bitwise the SpMV of that column, which is the oracle's."""
import numpy as np
import pytest

from abhsf_b200 import AbhsfMatrix
from oracle import oracle

pytestmark = pytest.mark.gpu


def _matrix(m, longest, seed):
    """Rows of 0 .. longest elements, none in a chain; m odd, so that the last
    slices hold fewer than 32 rows."""
    rng = np.random.default_rng(seed)
    n = m + 37
    length = rng.integers(0, longest + 1, m)
    rows = np.repeat(np.arange(m), length)
    cols = (rows + rng.integers(-3000, 3000, rows.size)) % n
    key = np.unique(rows * n + cols)
    return key // n, key % n, rng.standard_normal(key.size), m, n


@pytest.mark.parametrize("s", [16, 64, 256])
@pytest.mark.parametrize("m,longest", [(150_001, 7), (20_003, 9), (4_001, 200), (33, 3)])
def test_units_of_columns_and_rows(gpu, m, longest, s):
    import torch
    r, c, v, m, n = _matrix(m, longest, seed=m)
    A = AbhsfMatrix.from_elements(r, c, v, m, n, block_size=s, slice_tile_nnz=1000)
    sl = A.slices()
    assert sl["elements"] == r.size and not sl["chain"].any()
    rng = np.random.default_rng(2)
    wide = 53
    X, Y0 = rng.uniform(-1, 1, (n, wide)), rng.standard_normal((m, wide))
    Xd = torch.from_numpy(X).cuda()
    want = torch.empty(m, wide, dtype=torch.float64, device="cuda")
    for j in range(wide):
        y = torch.from_numpy(Y0[:, j].copy()).cuda()
        A.spmv(Xd[:, j].contiguous(), y)
        want[:, j] = y
    assert np.array_equal(want[:, 7].cpu().numpy(), oracle.spmv_elements(r, c, v, X[:, 7].copy(), Y0[:, 7].copy()))
    for k in (2, 4, 15, 16, 17, 20, 31, 32, 33, 48, 50):
        for off in (0, 3):
            Y = torch.from_numpy(Y0.copy()).cuda()
            A.spmm(Xd[:, off:off + k], Y[:, off:off + k])
            out = torch.from_numpy(Y0.copy()).cuda()
            out[:, off:off + k] = want[:, off:off + k]
            assert torch.equal(Y, out), (k, off)
