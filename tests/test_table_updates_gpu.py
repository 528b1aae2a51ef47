"""Products right after a table update, on streams that the legacy stream does not order: a
non-blocking stream, the pipelined host path's own streams, and the autograd function inside a
side stream.  The update has to be complete when it returns, so every product is bit for bit
that of an operator created with the new table (same kernels, same order)."""
import ctypes

import numpy as np
import pytest
import torch

from test_smem_products_gpu import _problem

pytestmark = pytest.mark.gpu


def _tables(K, n):
    rng = np.random.default_rng(n)
    for _ in range(n):
        yield dict(K, wmr=(K['wmr'] * rng.uniform(0.5, 1.0, K['wmr'].shape)).astype(np.float32))


def _set(A, K):
    from commit_gb300._lib import check, lib
    check(lib().cgb_op_set_lut(A.handle, K['wmr'].ctypes.data_as(ctypes.c_void_p), None, None))


def test_products_on_a_side_stream():
    from commit_gb300.operator import LinearOperator
    D, K = _problem(70, 6000, ndirs=500, nIC=3)
    A = LinearOperator(D, K, None)
    rng = np.random.default_rng(0)
    x, y = torch.from_numpy(rng.uniform(0, 1, A.nCOLS)).cuda(), torch.from_numpy(rng.uniform(0, 1, A.nROWS)).cuda()
    A.dot(x), A.T.dot(y)                                        # the layout exists
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    for K2 in _tables(K, 4):
        with torch.cuda.stream(s):
            _set(A, K2)
            ax, aty = A.dot(x), A.T.dot(y)
        s.synchronize()
        B = LinearOperator(D, K2, None)
        assert torch.equal(ax, B.dot(x)) and torch.equal(aty, B.T.dot(y))


def test_pipelined_host_products():
    from commit_gb300.operator import LinearOperator
    D, K = _problem(97, 30000, n_mask=44000, dim=(60, 60, 24))
    A = LinearOperator(D, K, None)
    assert A.nROWS >= 1 << 22
    rng = np.random.default_rng(1)
    x, y = rng.uniform(0, 1, A.nCOLS), rng.uniform(0, 1, A.nROWS)
    A.dot(x), A.T.dot(y)
    for K2 in _tables(K, 2):
        B = LinearOperator(D, K2, None)
        rx, ry = B.dot(x), B.T.dot(y)
        _set(A, K2)
        assert np.array_equal(A.dot(x), rx)
        _set(A, K)
        _set(A, K2)
        assert np.array_equal(A.T.dot(y), ry)


def test_autograd_on_a_side_stream():
    from commit_gb300.autograd import commit_apply
    from commit_gb300.operator import LinearOperator
    D, K = _problem(97, 6000)
    A = LinearOperator(D, K, None)
    rng = np.random.default_rng(2)
    x, y = torch.from_numpy(rng.uniform(0, 1, A.nCOLS)).cuda(), torch.from_numpy(rng.uniform(0, 1, A.nROWS)).cuda()
    A.dot(x), A.T.dot(y)
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    for K2 in _tables(K, 3):
        with torch.cuda.stream(s):
            lut = torch.from_numpy(K2['wmr']).cuda().requires_grad_(True)
            xs = x.clone().requires_grad_(True)
            pred = commit_apply(A, xs, lut)
            gx, = torch.autograd.grad((pred * y).sum(), xs)
        s.synchronize()
        B = LinearOperator(D, K2, None)
        assert torch.equal(pred.detach(), B.dot(x)) and torch.equal(gx, B.T.dot(y))
