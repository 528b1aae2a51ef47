"""The second pass of A' (column sums of the per-segment terms) with 8 lanes and with one
thread per column: average list lengths on both sides of the choice, lists that are empty,
of one term, and not a multiple of the lanes, a last warp that is partly empty, slabs.

Bound: a column is the FP64 sum of terms that are good to about 2^-45 each (float-float) or
2^-21 (FP32 products and sums over 8 samples), of one sign or both: the 2-norm is held to
1e-12 and 2e-5, the bounds of the products elsewhere in the tests."""
import numpy as np
import pytest
import torch

import golden_io as G
import oracle as O

pytestmark = pytest.mark.gpu


def _dictionary(nF, n, nIC, seed, nV=400, ndirs=20, nS=8):
    rng = np.random.default_rng(seed)
    v = np.sort(rng.integers(0, nV, n)).astype(np.uint32)
    f = rng.integers(0, nF, n)
    f[rng.uniform(size=n) < 0.1] = 0                    # one long list
    IC = {'str': f.astype(np.uint32), 'vox': v, 'dir': rng.integers(0, ndirs, n).astype(np.uint16),
          'len': rng.uniform(0, 1, n).astype(np.float32), 'n': n, 'nSTR': nF, 'nVOX': nV,
          'eval': rng.integers(0, 2, nF * nIC).astype(np.uint32)}
    z16, z32 = np.zeros(0, np.uint16), np.zeros(0, np.uint32)
    D = {'IC': IC, 'EC': {'vox': z32, 'dir': z16, 'n': 0}, 'ISO': {'vox': z32, 'n': 0}}
    K = {'wmr': rng.uniform(0, 1, (nIC, ndirs, nS)).astype(np.float32), 'wmh': np.zeros((0, ndirs, nS), np.float32),
         'iso': np.zeros((0, nS), np.float32)}
    return D, K


@pytest.mark.parametrize('nF,n,nIC', [(1, 500, 1), (33, 100, 1), (301, 1500, 2), (301, 900, 1), (5003, 90001, 1),
                                      (120001, 600000, 1), (40001, 900000, 3), (150001, 3200000, 1)])
def test_column_sums(nF, n, nIC):
    from commit_gb300.operator import LinearOperator
    D, K = _dictionary(nF, n, nIC, nF)
    A = LinearOperator(D, K, None)
    P = O.PortOperator(D, K, None, nthreads=8)
    y = np.random.default_rng(1).normal(size=A.nROWS)
    ref = P.T.dot(y)
    x = A.T.dot(torch.from_numpy(y).cuda()).cpu().numpy()
    assert G.rel(x, ref) <= 1e-12
    x32 = A.T.dot(torch.from_numpy(y).float().cuda(), arith='f32').double().cpu().numpy()
    assert G.rel(x32, ref) <= 2e-5
    B = LinearOperator(D, K, None)
    assert B.set_slabs(7) == 7
    assert np.array_equal(B.T.dot(torch.from_numpy(y).cuda()).cpu().numpy(), x)
