"""Chains in f32 and bf16 on values made for f32's spacing: ties (a sum near
700 has a spacing of 2^-14), products of widely different size, subnormals.  y
must be bitwise the additions in turn."""
import numpy as np
import pytest

from abhsf_b200 import AbhsfMatrix
from oracle import oracle
from test_gpu_chains import LENGTHS, _same

pytestmark = pytest.mark.gpu


def _values(kind, z, rng):
    if kind == "ties":  # small multiples of half a spacing of the sums reached
        return rng.integers(-4, 5, z) * 2.0 ** -15
    if kind == "ties up":  # sums that climb through binades by ties and spacings
        return rng.integers(1, 4, z) * 2.0 ** -15
    if kind == "wide":
        return rng.standard_normal(z) * np.exp(rng.uniform(-30, 30, z))
    return rng.standard_normal(z) * 2.0 ** -138  # "tiny": subnormal


@pytest.mark.parametrize("s", [16, 64])
@pytest.mark.parametrize("vt", ["f32", "bf16"])
@pytest.mark.parametrize("kind", ["ties", "ties up", "wide", "tiny"])
def test_chains_at_the_scale_of_f32(gpu, kind, vt, s):
    import torch
    rng = np.random.default_rng(11)
    n, rows, cols, vals = 20480, [], [], []
    for i, z in enumerate(LENGTHS):
        rows.append(np.full(z, 67 * i + 5))
        cols.append(np.sort(rng.choice(n, z, replace=False)))
        vals.append(_values(kind, z, rng))
    r, c, v = (np.concatenate(t) for t in (rows, cols, vals))
    m = 67 * len(LENGTHS) + 5
    x = np.ones(n, np.float32)
    y0 = np.zeros(m, np.float32) if kind == "tiny" else np.full(m, 700.0, np.float32)
    stored = torch.from_numpy(v).float()
    if vt == "bf16":
        stored = stored.bfloat16().float()
    ref = oracle.spmv_elements_f32(r, c, stored.numpy(), x, y0.copy())
    A = AbhsfMatrix.from_elements(r, c, v, m, n, block_size=s, value_type=vt)
    assert np.count_nonzero(A.slices()["chain"]) == len(LENGTHS)
    y = torch.from_numpy(y0.copy()).cuda()
    A.spmv_f32(torch.from_numpy(x).cuda(), y)
    assert _same(y.cpu().numpy(), ref)
