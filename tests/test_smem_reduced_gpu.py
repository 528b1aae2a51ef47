"""FP32-vector products (FP16 / BF16 table and FP16 lengths, or both in FP32) of operators large enough for the
kernels that keep the table in shared memory, against the oracle.

The sizes sit at the edges of the kernels' quads of samples, chunks and ranges of responses.
Bound: the error of a row is measured against |A| |x|.  Two roundings to FP16 are off by at most
2^-11 each (BF16: 2^-8 for the table), together 1.0e-3 (4.4e-3); the FP32 sums of at most 500
terms add 500 * 2^-24 = 3e-5 (FP32 table: 850 terms and a rounding of the product each, 6e-5).
"""
import numpy as np
import pytest
import torch

import oracle as O
from test_smem_products_gpu import _problem

pytestmark = pytest.mark.gpu

TOL = {'fp16': 1.1e-3, 'bf16': 4.5e-3, 'f32': 6e-5}


@pytest.mark.parametrize('arith', ['fp16', 'bf16', 'f32'])
@pytest.mark.parametrize('nS,n_fibers,ndirs,nIC,nEC,nISO,slabs', [
    (17, 42000, 120, 1, 1, 2, 1), (32, 23000, 120, 1, 0, 0, 1), (33, 23000, 120, 1, 2, 0, 3), (97, 8000, 500, 2, 1, 1, 1),
    (128, 6000, 33, 1, 0, 3, 1), (130, 6000, 500, 1, 1, 2, 4), (192, 5000, 120, 2, 0, 1, 1), (193, 9000, 120, 1, 1, 0, 1),
    (288, 9000, 500, 2, 2, 2, 1), (160, 5000, 120, 3, 1, 1, 2)])
def test_products_match_the_oracle(arith, nS, n_fibers, ndirs, nIC, nEC, nISO, slabs):
    from commit_gb300.operator import LinearOperator
    D, K = _problem(nS, n_fibers, ndirs=ndirs, nIC=nIC, nEC=nEC, nISO=nISO, mask=nIC > 1)
    P = O.PortOperator(D, K, None, nthreads=8)
    A, B = LinearOperator(D, K, None), LinearOperator(D, K, None)
    B.ff_shape(0)  # the gathering kernels
    for M in (A, B):
        M.tensor_cores(1)  # off
    A.set_slabs(slabs)
    rng = np.random.default_rng(nS)
    for signed in (False, True):
        x = rng.uniform(0, 1, P.nCOLS).astype(np.float32)
        y = rng.uniform(0, 1, P.nROWS).astype(np.float32)
        ref = P.dot(x.astype(np.float64)), P.T.dot(y.astype(np.float64))
        if signed:
            x, y = x * rng.choice([-1, 1], x.size).astype(np.float32), y * rng.choice([-1, 1], y.size).astype(np.float32)
        got = []
        for M in (A, B):
            # an odd offset in a larger buffer: rows that are not 16-byte aligned
            buf = torch.zeros(P.nROWS + 1, device='cuda')
            ax = M.dot(torch.from_numpy(x).cuda(), out=buf[1:] if signed else None, arith=arith).cpu().numpy()
            got.append((ax, M.T.dot(torch.from_numpy(y).cuda(), arith=arith).cpu().numpy()))
        exact = P.dot(x.astype(np.float64)), P.T.dot(y.astype(np.float64))
        for g, e, scale in zip(got[0], exact, ref):
            assert np.all(np.abs(g - e) <= TOL[arith] * scale + 1e-30)
        if arith != 'f32' or ndirs * nIC <= 500:
            assert not np.array_equal(got[0][0], got[1][0])  # the kernels under test ran


@pytest.mark.parametrize('nS,nIC,n_fibers,dim,fwd,adj', [
    (128, 1, 3000, (14, 14, 14), True, True), (129, 1, 2500, (14, 14, 14), True, False),
    (129, 1, 16000, (14, 14, 14), True, True), (192, 1, 12000, (14, 14, 14), True, True),
    (193, 1, 12000, (14, 14, 14), False, False), (97, 2, 8000, (14, 14, 14), False, False)])
def test_bf16_choice_against_the_tensor_cores(nS, nIC, n_fibers, dim, fwd, adj):
    """The automatic choice is the shared-memory kernel (tensor cores off) or the tensor-core one
    (always on) by quads of samples x responses and segments per voxel."""
    from commit_gb300.operator import LinearOperator
    D, K = _problem(nS, n_fibers, n_mask=900, dim=dim, ndirs=120, nIC=nIC)
    rng = np.random.default_rng(1)
    got = []
    for mode in (0, 1, 2):
        A = LinearOperator(D, K, None)
        A.tensor_cores(mode)
        if mode == 0:
            assert A.tensor_cores() == 1
            x = torch.from_numpy(rng.uniform(0, 1, A.nCOLS).astype(np.float32)).cuda()
            y = torch.from_numpy(rng.uniform(0, 1, A.nROWS).astype(np.float32)).cuda()
        got.append((A.dot(x, arith='bf16'), A.T.dot(y, arith='bf16')))
    for k, smem in ((0, fwd), (1, adj)):
        assert torch.equal(got[0][k], got[1 if smem else 2][k])
        assert not torch.equal(got[1][k], got[2][k])
