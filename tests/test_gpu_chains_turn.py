"""Chains at the lengths and start values where a group of 512 products goes
from being added in turn to being summed by segments (more than 12 segments of 16 in
FP64, 19 in f32, and a sum 4 or 5 binades above the products): y bitwise the
additions in turn either way."""
import numpy as np
import pytest

from abhsf_b200 import AbhsfMatrix
from oracle import oracle
from test_gpu_chains import _same

pytestmark = pytest.mark.gpu

STARTS = [0.0, -0.0, 1e-40, 1.5, 12.0, 24.0, 31.9, 32.0, 48.0, -24.0, -48.0, 96.0, -96.0, 1e6, 1e30, np.inf, -np.inf,
          np.nan]


@pytest.mark.parametrize("vt", ["f64", "f32", "bf16"])
@pytest.mark.parametrize("segments", [12, 13, 19, 20, 31, 32])
@pytest.mark.parametrize("extra", [0, 1])
def test_groups_in_turn_and_by_segments(gpu, segments, extra, vt):
    """Rows of 512 + 16 (segments - 1) + (16 or 1) products in +-[1, 2), and of
    the last group alone where it is long enough to be a chain."""
    import torch
    rng = np.random.default_rng(segments)
    z = 16 * (segments - 1) + (16 if extra == 0 else 1)
    lengths = [512 + z] + ([z] if z > 256 else [])
    n, rows, cols, vals, start_of = 40960, [], [], [], {}
    for start in STARTS:
        for k in lengths:
            row = 67 * len(start_of) + 5  # apart: tiles of few elements
            rows.append(np.full(k, row))
            cols.append(np.sort(rng.choice(n, k, replace=False)))
            vals.append(rng.choice([-1.0, 1.0], k) * rng.uniform(1, 2, k))
            start_of[row] = start
    r, c, v = (np.concatenate(t) for t in (rows, cols, vals))
    m = 67 * len(start_of)
    y0 = np.zeros(m)
    y0[list(start_of)] = list(start_of.values())
    A = AbhsfMatrix.from_elements(r, c, v, m, n, block_size=64, value_type=vt)
    assert np.count_nonzero(A.slices()["chain"]) == len(start_of)
    if vt == "f64":
        x = np.ones(n)
        ref = oracle.spmv_elements(r, c, v, x, y0.copy())
        y = torch.from_numpy(y0.copy()).cuda()
        A.spmv(torch.from_numpy(x).cuda(), y)
    else:
        x, y0 = np.ones(n, np.float32), y0.astype(np.float32)
        stored = torch.from_numpy(v).float()
        if vt == "bf16":
            stored = stored.bfloat16().float()
        ref = oracle.spmv_elements_f32(r, c, stored.numpy(), x, y0.copy())
        y = torch.from_numpy(y0.copy()).cuda()
        A.spmv_f32(torch.from_numpy(x).cuda(), y)
    assert _same(y.cpu().numpy(), ref)
