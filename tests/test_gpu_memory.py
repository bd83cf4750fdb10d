"""The library's device memory while other threads and streams use the GPU: a
handle's memory is not handed out again before the work that reads it is done,
and giving it back disturbs nobody's stream capture."""
import ctypes as C
import threading
import time

import numpy as np
import pytest

from abhsf_b200 import AbhsfMatrix, capi, cg, cg_mixed, trim_device_memory
from abhsf_b200 import workloads as W
from oracle import oracle

pytestmark = pytest.mark.gpu


def _reference(coo, x):
    order = np.lexsort((coo.cols, coo.rows))
    return oracle.spmv_elements(coo.rows[order], coo.cols[order], coo.vals[order], x, np.zeros(coo.m))


def test_solves_beside_builds_and_releases(gpu):
    """A solve captures its iterations into a graph.  Another thread's builds
    and releases must not undo that capture, nor get memory that is in use."""
    import torch
    lap = W.laplacian_2d(60)
    A = AbhsfMatrix.from_elements(lap.rows, lap.cols, lap.vals, lap.m, lap.n)
    lo = AbhsfMatrix.from_elements(lap.rows, lap.cols, lap.vals, lap.m, lap.n, value_type="f32")
    b = torch.from_numpy(np.random.default_rng(1).uniform(-1, 1, lap.n)).cuda()

    def solve(mixed):
        x = torch.zeros_like(b)
        info = cg_mixed(A, lo, b, x, rtol=1e-10) if mixed else cg(A, b, x, rtol=1e-10)
        assert info["converged"]
        return x.cpu().numpy()

    want = [solve(False), solve(True)]
    coos = [W.random_blocky(700 + 150 * i, 900, 64, 70, seed=60 + i) for i in range(3)]
    xs = [W.rhs(c.n, 8) for c in coos]
    refs = [_reference(c, x) for c, x in zip(coos, xs)]
    until = time.monotonic() + 6.0
    bad, counts = [], [0, 0]

    def solver(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            while time.monotonic() < until and not bad:
                try:
                    if not np.array_equal(solve(bool(i)), want[i]):
                        bad.append(("solve", i))
                except Exception as e:  # noqa: BLE001
                    bad.append(("solve", i, repr(e)))
                counts[0] += 1

    def builder(i):
        c = coos[i]
        with torch.cuda.stream(torch.cuda.Stream()):
            x = torch.from_numpy(xs[i]).cuda()
            while time.monotonic() < until and not bad:
                try:
                    M = AbhsfMatrix.from_elements(c.rows, c.cols, c.vals, c.m, c.n, block_size=(16, 32, 64)[i])
                    y = torch.zeros(c.m, dtype=torch.float64, device="cuda")
                    M.spmv(x, y)
                    M.release()  # the product may still be running
                    if not np.array_equal(y.cpu().numpy(), refs[i]):
                        bad.append(("product", i))
                except Exception as e:  # noqa: BLE001
                    bad.append(("build", i, repr(e)))
                counts[1] += 1

    threads = [threading.Thread(target=solver, args=(i,)) for i in range(2)]
    threads += [threading.Thread(target=builder, args=(i,)) for i in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad
    assert counts[0] > 4 and counts[1] > 4


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("s", [16, 64])
def test_release_waits_for_queued_products(gpu, s, graph):
    """Products queued by the caller (directly, or replayed from a graph the
    library knows nothing of) read the matrix after release() was called; the
    memory must not go to the next builds before."""
    import torch
    coo = W.random_blocky(20000, 20000, 64, 900, seed=71)
    x = W.rhs(coo.n, 9)
    times = 400
    xd = torch.from_numpy(x).cuda()
    ref = None
    for _ in range(3):
        A = AbhsfMatrix.from_elements(coo.rows, coo.cols, coo.vals, coo.m, coo.n, block_size=s)
        if ref is None:  # the same products, waited for
            y = torch.zeros(coo.m, dtype=torch.float64, device="cuda")
            A.spmv(xd, y)
            assert np.array_equal(y.cpu().numpy(), _reference(coo, x))
            for _ in range(times - 1):
                A.spmv(xd, y)
            ref = y.cpu().numpy()
        y = torch.zeros(coo.m, dtype=torch.float64, device="cuda")
        st = torch.cuda.Stream()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.stream(st):
            if graph:
                torch.cuda.synchronize()
                with torch.cuda.graph(g, stream=st):
                    A.spmv(xd, y)
                for _ in range(times):
                    g.replay()
            else:
                for _ in range(times):
                    A.spmv(xd, y)
        A.release()
        other = [AbhsfMatrix.from_elements(coo.cols, coo.rows, -coo.vals, coo.n, coo.m, block_size=s)
                 for _ in range(2)]
        torch.cuda.synchronize()
        assert np.array_equal(y.cpu().numpy(), ref)
        for o in other:
            o.release()
    assert capi.lib.abhsf_test_blocks_set_aside() == 0


def test_release_while_a_capture_forbids_waiting(gpu):
    """While this thread captures in global mode the device cannot be waited
    for: the memory of a handle released then is kept aside, and given back by
    the next release that can wait."""
    rt = C.CDLL("libcudart.so.12")
    coo = W.random_blocky(900, 900, 64, 80, seed=72)

    def build():
        return AbhsfMatrix.from_elements(coo.rows, coo.cols, coo.vals, coo.m, coo.n)

    A, B = build(), build()
    st, g = C.c_void_p(), C.c_void_p()
    assert rt.cudaStreamCreateWithFlags(C.byref(st), 1) == 0
    assert rt.cudaStreamBeginCapture(st, 0) == 0  # cudaStreamCaptureModeGlobal
    A.release()
    rt.cudaStreamEndCapture(st, C.byref(g))  # whether it is still a valid capture or not
    if g.value:
        rt.cudaGraphDestroy(g)
    rt.cudaGetLastError()
    assert rt.cudaStreamDestroy(st) == 0
    assert capi.lib.abhsf_test_blocks_set_aside() > 0
    B.release()
    assert capi.lib.abhsf_test_blocks_set_aside() == 0
    x = W.rhs(coo.n, 10)
    import torch
    y = torch.zeros(coo.m, dtype=torch.float64, device="cuda")
    build().spmv(torch.from_numpy(x).cuda(), y)
    assert np.array_equal(y.cpu().numpy(), _reference(coo, x))


def test_unused_memory_is_given_back(gpu):
    """What builds and releases leave is kept for the next call, and goes back
    to the device on request; a matrix in use stays as it is."""
    import torch
    coo = W.random_blocky(900, 900, 64, 80, seed=73)
    x = W.rhs(coo.n, 11)
    A = AbhsfMatrix.from_elements(coo.rows, coo.cols, coo.vals, coo.m, coo.n)
    big = W.random_uniform(400000, 400000, 6_000_000, seed=74)

    def build():
        AbhsfMatrix.from_elements(big.rows, big.cols, big.vals, big.m, big.n).release()

    build()  # the kernels' code and stacks are on the device from here on
    trim_device_memory()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    build()
    kept = free - torch.cuda.mem_get_info()[0]
    assert 0 < kept <= (2 << 30) + (64 << 20)
    back = trim_device_memory()
    assert back > 0.9 * kept - (64 << 20) and free - torch.cuda.mem_get_info()[0] <= 64 << 20
    y = torch.zeros(coo.m, dtype=torch.float64, device="cuda")
    A.spmv(torch.from_numpy(x).cuda(), y)
    assert np.array_equal(y.cpu().numpy(), _reference(coo, x))


def test_other_allocations_get_what_the_library_keeps(gpu):
    """Memory that the library keeps unused is there for the process's other
    allocations: one of more than what is reported free succeeds."""
    import torch
    big = W.random_uniform(400000, 400000, 6_000_000, seed=76)
    trim_device_memory()
    AbhsfMatrix.from_elements(big.rows, big.cols, big.vals, big.m, big.n).release()
    torch.cuda.empty_cache()
    try:
        t = torch.empty(torch.cuda.mem_get_info()[0] + (128 << 20), dtype=torch.uint8, device="cuda")
        assert t.data_ptr()
        del t
    finally:
        torch.cuda.empty_cache()


def test_scratch_of_block_rows_with_one_element(gpu):
    """200,000 block rows of 64 rows and one element each: the build's scratch
    is 20 bytes a row (counts, row starts, slots), what goes with the rows that
    hold elements comes on top (here 1/64 of them)."""
    k = 200_000
    rows = np.arange(k, dtype=np.int64) * 640 + 3
    cols = np.random.default_rng(1).integers(0, 1000, k)
    trim_device_memory()
    A = AbhsfMatrix.from_elements(rows, cols, np.ones(k), 640 * k, 1000, block_size=64)
    assert A.slices()["block_rows"] == k
    A.release()
    back = trim_device_memory()
    assert 20 * 64 * k <= back <= 30 * 64 * k
