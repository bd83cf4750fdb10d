"""Matrices built, used and released by several threads at once, each on a
stream of its own: their memory comes from one pool."""
import threading

import numpy as np
import pytest

from abhsf_b200 import AbhsfMatrix
from abhsf_b200 import workloads as W
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("s", [16, 64])
def test_threads_share_the_pool(gpu, s):
    import torch
    coos = [W.random_blocky(900 + 130 * i, 1100, 64, 90, seed=50 + i) for i in range(4)]
    xs = [W.rhs(c.n, 7) for c in coos]
    refs = []
    for c, x in zip(coos, xs):
        order = np.lexsort((c.cols, c.rows))
        refs.append(oracle.spmv_elements(c.rows[order], c.cols[order], c.vals[order], x, np.zeros(c.m)))
    bad = []

    def work(i):
        c, st = coos[i], torch.cuda.Stream()
        with torch.cuda.stream(st):
            x = torch.from_numpy(xs[i]).cuda()
            for _ in range(6):
                A = AbhsfMatrix.from_elements(c.rows, c.cols, c.vals, c.m, c.n, block_size=s)
                y = torch.zeros(c.m, dtype=torch.float64, device="cuda")
                A.spmv(x, y)
                A.release()  # the product may still be running
                if not np.array_equal(y.cpu().numpy(), refs[i]):
                    bad.append(i)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
