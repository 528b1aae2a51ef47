"""Accuracy of the shared-memory float-float products on tables whose rows differ much in size,
measured against each voxel's and each column's own size: the fast sums carry a bias taken from the largest
table value of a sample, which must not show where a voxel's own rows are small.

Bound: a voxel or column is a sum of at most N = 600 terms of one sign, each off by at most 3 units of 2^-48
of the partial sum it joins; the bias is at most 4 times a voxel's sum (A) and 8 times a dot product
(A'), which the biased sums add to the partial sums: 9 * 3 * 2^-48 * N = 6e-11 if every rounding had the
same sign.  They have either sign, so the deviation grows with the root of N: 2e-12 is held
per voxel and per column."""
import numpy as np
import pytest
import torch

import oracle as O
from test_smem_products_gpu import _problem

pytestmark = pytest.mark.gpu

TOL = 2e-12


def _table(D, K, kind):
    """The IC table with uneven rows, and rows y that make the unevenness show in A'."""
    w = K['wmr'].copy()
    used = np.bincount(D['IC']['dir'], minlength=w.shape[1])
    nV, nS = D['IC']['nVOX'], w.shape[2]
    y = np.random.default_rng(3).uniform(0.1, 1.0, (nV, nS))
    if kind.startswith('large'):                 # one row that few voxels use
        w[0, used.argmin()] *= float(kind[5:])
    elif kind.startswith('small'):               # half of the rows small: whole voxels of them
        w[0, ::2] *= 1.0 / float(kind[5:])
    elif kind == 'response':                     # one response much smaller than the other
        w[1] *= 1e-7
    elif kind == 'sample':                       # one sample far smaller in all rows but one, and y only there
        w[0, :, 40] *= 1e-6
        w[0, used.argmin(), 40] = 1.0
        y[:] = 0.0
        y[:, 40] = 1.0
    elif kind.startswith('faint'):               # the same, less extreme: an even table, but uneven dot products
        w[0, :, 40:42] *= float(kind[5:])
        w[0, used.argmin(), 40:42] = 1.0
        y[:, :40] = y[:, 42:] = 0.0
    elif kind == 'zero':                         # rows of zeros
        w[0, ::3] = 0.0
    return dict(K, wmr=w), y


@pytest.mark.parametrize('kind,nS,nIC', [('large1e6', 70, 1), ('large1e8', 97, 1), ('small1e6', 97, 1), ('small1e9', 288, 1),
                                         ('response', 70, 2), ('sample', 97, 1), ('faint1e-4', 97, 1), ('faint1e-6', 288, 1),
                                         ('zero', 97, 1)])
def test_rows_of_different_size(kind, nS, nIC):
    from commit_gb300.operator import LinearOperator
    D, K = _problem(nS, 6000, nIC=nIC, nEC=0, nISO=0)
    K, y = _table(D, K, kind)
    IC = D['IC']
    if kind.startswith('small'):                 # voxels whose segments all have small rows
        some = IC['vox'] % 2 == 0
        IC['dir'][some] -= IC['dir'][some] % 2
    A, P = LinearOperator(D, K, None), O.PortOperator(D, K, None, nthreads=8)
    x = np.random.default_rng(4).uniform(0.0, 1.0, A.nCOLS)
    if kind == 'response':
        x[:IC['nSTR']][::2] = 0.0
    ref = P.dot(x).reshape(-1, nS)
    err = np.linalg.norm(A.dot(torch.from_numpy(x).cuda()).cpu().numpy().reshape(-1, nS) - ref, axis=1)
    assert np.all(err <= TOL * np.linalg.norm(ref, axis=1))
    y = y.reshape(-1)
    ref = P.T.dot(y)
    got = A.T.dot(torch.from_numpy(y).cuda()).cpu().numpy()
    assert np.all(np.abs(got - ref) <= TOL * np.abs(ref))
    # negative weights and rows of both signs
    s = np.random.default_rng(5).choice([-1.0, 1.0], x.size)
    ref, scale = P.dot(x * s).reshape(-1, nS), P.dot(x).reshape(-1, nS)
    err = np.linalg.norm(A.dot(torch.from_numpy(x * s).cuda()).cpu().numpy().reshape(-1, nS) - ref, axis=1)
    assert np.all(err <= TOL * np.linalg.norm(scale, axis=1))
