"""What one SpMV puts on the stream: its kernels, and one memset where the
streaming kernel (block sizes 16, 128, 256) has block rows to hand out."""
import ctypes as C

import numpy as np
import pytest

from abhsf_b200 import AbhsfMatrix
from abhsf_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _nodes(run):
    rt = C.CDLL("libcudart.so.12")
    st, g, n = C.c_void_p(), C.c_void_p(), C.c_size_t()
    assert rt.cudaStreamCreateWithFlags(C.byref(st), 1) == 0
    assert rt.cudaStreamBeginCapture(st, 2) == 0  # cudaStreamCaptureModeRelaxed
    try:
        run(st.value)
    finally:
        assert rt.cudaStreamEndCapture(st, C.byref(g)) == 0
    assert rt.cudaGraphGetNodes(g, None, C.byref(n)) == 0
    rt.cudaGraphDestroy(g)
    rt.cudaStreamDestroy(st)
    return n.value


class _Stream:
    def __init__(self, ptr):
        self.cuda_stream = ptr


@pytest.mark.parametrize("vt", ["f64", "bf16"])
@pytest.mark.parametrize("s", [16, 64, 256])
@pytest.mark.parametrize("shape", ["laplacian", "blocky", "rmat"])
def test_nodes_of_a_captured_spmv(gpu, shape, s, vt):
    import torch
    coo = {"laplacian": lambda: W.laplacian_2d(90), "blocky": lambda: W.random_blocky(9000, 9000, 64, 300, seed=3),
           "rmat": lambda: W.rmat(1 << 14, 16, seed=3)}[shape]()
    A = AbhsfMatrix.from_elements(coo.rows, coo.cols, coo.vals, coo.m, coo.n, block_size=s, value_type=vt)
    dt = torch.float64 if vt == "f64" else torch.float32
    x, y = torch.ones(coo.n, dtype=dt, device="cuda"), torch.zeros(coo.m, dtype=dt, device="cuda")
    run = A.spmv if vt == "f64" else A.spmv_f32
    run(x, y)  # set up
    torch.cuda.synchronize()
    sl, tree = A.slices(), len({int(r) // s for r in coo.rows})
    streaming = s != 64 and sl["block_rows"] < tree
    if shape == "laplacian":
        assert not streaming and A.kernels() == 1
    assert _nodes(lambda st: run(x, y, stream=_Stream(st))) == A.kernels() + (1 if streaming else 0)
