"""A LUT gradient whose set-up fails (here: its allocations, refused while a stream is captured)
reports the error, and the next call sets up anew and returns the gradient."""
import ctypes

import numpy as np
import pytest
import torch

import golden_io as G
from test_smem_products_gpu import _problem

pytestmark = pytest.mark.gpu


def _cudart():
    """The CUDA runtime that torch has loaded."""
    path = next(l.split()[-1] for l in open('/proc/self/maps') if 'libcudart.so' in l)
    return ctypes.CDLL(path)


def test_call_after_a_failed_set_up():
    from commit_gb300._lib import CgbError
    from commit_gb300.autograd import lut_gradient
    from commit_gb300.operator import LinearOperator
    D, K = _problem(33, 300)
    A, B = LinearOperator(D, K, None), LinearOperator(D, K, None)
    rng = np.random.default_rng(0)
    x, g = torch.from_numpy(rng.normal(size=A.nCOLS)).cuda(), torch.from_numpy(rng.normal(size=A.nROWS)).cuda()
    ref = lut_gradient(B, x, g)
    torch.cuda.synchronize()
    rt, s = _cudart(), torch.cuda.Stream()
    st, graph = ctypes.c_void_p(s.cuda_stream), ctypes.c_void_p()
    outs = [torch.zeros_like(t) for t in ref]
    ptr = [ctypes.c_void_p(t.data_ptr()) for t in [x, g] + outs]
    torch.cuda.synchronize()
    from commit_gb300._lib import check, lib
    assert rt.cudaStreamBeginCapture(st, 1) == 0     # thread-local
    try:
        with pytest.raises(CgbError):
            check(lib().cgb_op_lut_grad(A.handle, *ptr, st))
    finally:
        rt.cudaStreamEndCapture(st, ctypes.byref(graph))
        rt.cudaGetLastError()
    got = lut_gradient(A, x, g)
    for a, b in zip(got, ref):
        assert torch.equal(a, b) and float(b.abs().max()) > 0
    assert G.rel(got[2].cpu().numpy()[0], x[-2 * D['ISO']['n']:][:D['ISO']['n']].cpu().numpy()
                 @ g.cpu().numpy().reshape(-1, 33)) <= 1e-12
