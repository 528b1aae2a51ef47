"""LUT gradients over the layouts of the chunk kernel: samples below, at and above a round of
lanes x samples, several responses, voxels whose elements share an orientation, orientations
without elements, zero weights, chunks with a partly filled last batch.

Bound: FP64 sums of FP64 products of N <= 40000 terms, N * 2^-53 = 5e-12 in the worst case of
one-sided rounding; terms of either sign are held to 1e-12 in the 2-norm."""
import numpy as np
import pytest
import torch

import golden_io as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('nS,nIC,nEC,nISO', [(1, 1, 1, 1), (72, 1, 1, 2), (73, 2, 1, 1), (96, 1, 2, 1), (97, 1, 1, 1),
                                            (144, 1, 1, 0), (145, 1, 0, 1), (193, 3, 1, 1), (288, 1, 1, 2), (289, 1, 1, 1)])
def test_gradient_rows(nS, nIC, nEC, nISO):
    from commit_gb300.autograd import lut_gradient
    from commit_gb300.operator import LinearOperator
    rng = np.random.default_rng(nS)
    nV, nF, nd, n, nE = 301, 97, 23, 20011, 1501
    v = np.sort(rng.integers(0, nV, n)).astype(np.uint32)
    o = rng.integers(0, nd - 3, n).astype(np.uint16)               # the last orientations have no segment
    o[o == 5] = 6
    f = rng.integers(0, nF, n).astype(np.uint32)
    ln = rng.uniform(0, 1, n).astype(np.float32)
    ev = rng.integers(0, 3, nF * nIC).astype(np.uint32)
    ecv = np.sort(rng.integers(0, nV, nE)).astype(np.uint32)
    eco = rng.integers(0, 2, nE).astype(np.uint16) * 7              # few orientations: elements share them
    D = {'IC': {'str': f, 'vox': v, 'dir': o, 'len': ln, 'n': n, 'nSTR': nF, 'nVOX': nV, 'eval': ev},
         'EC': {'vox': ecv, 'dir': eco, 'n': nE}, 'ISO': {'vox': np.arange(nV, dtype=np.uint32), 'n': nV}}
    K = {'wmr': rng.uniform(0, 1, (nIC, nd, nS)).astype(np.float32), 'wmh': rng.uniform(0, 1, (nEC, nd, nS)).astype(np.float32),
         'iso': rng.uniform(0, 1, (nISO, nS)).astype(np.float32)}
    A = LinearOperator(D, K, None)
    x = rng.normal(size=A.nCOLS) * (rng.uniform(size=A.nCOLS) < 0.7)
    g = rng.normal(size=(nV, nS))
    got = lut_gradient(A, torch.from_numpy(x).cuda(), torch.from_numpy(g.reshape(-1)).cuda())
    for i in range(nIC):
        w = np.zeros((nd, nS))
        np.add.at(w, o, (ln.astype(np.float64) * x[i * nF + f] * ev[i * nF + f])[:, None] * g[v])
        assert G.rel(got[0][i].cpu().numpy(), w) <= 1e-12
    for i in range(nEC):
        w = np.zeros((nd, nS))
        np.add.at(w, eco, x[nF * nIC + i * nE:nF * nIC + (i + 1) * nE, None] * g[ecv])
        assert G.rel(got[1][i].cpu().numpy(), w) <= 1e-12
    for i in range(nISO):
        b = nF * nIC + nE * nEC + i * nV
        assert G.rel(got[2][i].cpu().numpy(), x[b:b + nV] @ g) <= 1e-12
