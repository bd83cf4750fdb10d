"""The histograms of all 64 block sizes from one sort, against the oracle's
count of each size: tiles of one, two, up to 32 and more elements (each counted
its own way), full and ragged tiles, repeated elements."""
import numpy as np
import pytest

from abhsf_b200 import block_histograms_all, capi
from abhsf_b200 import workloads as W
from oracle import oracle

pytestmark = pytest.mark.gpu


def _tiles_of(counts, seed):
    """256 x 256 tiles on a diagonal, tile i with counts[i] distinct elements."""
    rng = np.random.default_rng(seed)
    r, c = [], []
    for i, z in enumerate(counts):
        at = rng.choice(65536, z, replace=False)
        r.append(256 * i + at // 256)
        c.append(256 * i + at % 256)
    r, c = np.concatenate(r), np.concatenate(c)
    p = rng.permutation(r.size)
    return r[p].astype(np.int64), c[p].astype(np.int64), 256 * len(counts)


CASES = {
    "ones_and_twos": lambda: _tiles_of([1, 2, 2, 1, 2, 2, 2], 1),
    "around_a_warp": lambda: _tiles_of([3, 31, 32, 33, 34, 64], 2),
    "large": lambda: _tiles_of([1000, 20000, 65536, 65535], 3),
    "two_in_a_cell": lambda: (np.array([0, 0, 300, 301, 511]), np.array([0, 1, 300, 300, 0]), 512),
    "one_element": lambda: (np.array([5]), np.array([7]), 9),
}


@pytest.mark.parametrize("where", ["host", "device"])
@pytest.mark.parametrize("case", list(CASES))
def test_all_sizes(gpu, case, where):
    import torch
    r, c, n = CASES[case]()
    r, c = r.astype(np.int64), c.astype(np.int64)
    got = block_histograms_all(*(torch.from_numpy(t).cuda() if where == "device" else t for t in (r, c)), n, n)
    for k in range(1, 9):
        for l in range(1, 9):
            assert got[f"{1 << k}x{1 << l}"] == oracle.block_histogram(r, c, k, l), (k, l)


@pytest.mark.parametrize("maker", [lambda: W.rmat(5000, 12, seed=4), lambda: W.banded(3000, 40, seed=5),
                                   lambda: W.random_blocky(1500, 2300, 64, 200, seed=6)])
def test_all_sizes_generated(gpu, maker):
    coo = maker()
    got = block_histograms_all(coo.rows, coo.cols, coo.m, coo.n)
    for k in range(1, 9):
        for l in range(1, 9):
            assert got[f"{1 << k}x{1 << l}"] == oracle.block_histogram(coo.rows, coo.cols, k, l), (k, l)


@pytest.mark.parametrize("others", [0, 10, 200])
def test_repeated_elements(gpu, others):
    """Repeats count; a block of more elements than positions is refused
    (five in one 2 x 2 block), whichever way its tile is counted."""
    rng = np.random.default_rng(7)
    at = rng.choice(60000, others, replace=False) + 5000
    for times in (4, 5):
        r = np.concatenate([np.full(times, 3), at // 256]).astype(np.int64)
        c = np.concatenate([np.full(times, 2), at % 256]).astype(np.int64)
        if times == 4:
            assert block_histograms_all(r, c, 256, 256)["2x2"].get(4, 0) >= 1
        else:
            with pytest.raises(capi.InvalidValue):
                block_histograms_all(r, c, 256, 256)
