"""Float-float products of operators large and dense enough for the kernels that keep the
response table in shared memory (A and A' by sample chunks, A' also by orientation ranges).

The sizes sit at the kernels' edges: one sample below and above a chunk count and an even or
odd number of sample pairs, several responses (orientation ranges), voxels without segments,
more voxels than one sorting window, masks, inputs of one sign and of both, and inputs that
need the range guard.  Bound: an accumulator's error word is renormalised every 8 terms on
the fast sums and never holds more than one unit per term on the general ones, so N terms
are off by less than 3 N 2^-48 of the largest partial sum; N <= 500 gives 6e-12, and the 2-norm
of the rows is held to 1e-12 (the errors are rounding errors of either sign).
"""
import numpy as np
import pytest
import torch

import golden_io as G
import oracle as O

pytestmark = pytest.mark.gpu

TOL = 1e-12


def _problem(nS, n_fibers, n_mask=3000, dim=(20, 20, 16), ndirs=120, nIC=1, nEC=1, nISO=2, mask=False, seed=0):
    from commit_gb300 import synth
    spec = synth.ProblemSpec(dim=dim, n_mask=n_mask, n_fibers=n_fibers, ndirs=ndirs, n_b0=1, shells=[(1000.0, nS - 1)],
                             n_ic=nIC, d_perps=(0.51e-3, 0.9e-3)[:nEC], d_isos=(1.7e-3, 3.0e-3, 0.9e-3)[:nISO], seed=seed)
    D, K = synth.make_dictionary(spec)
    if mask:
        D['IC']['eval'] = np.random.default_rng(1).choice([0, 1, 1, 1, 2], D['IC']['nSTR'] * nIC).astype(np.uint32)
    return D, K


def _check(D, K, x, y, grows=True):
    from commit_gb300.operator import LinearOperator
    A = LinearOperator(D, K, None)
    P = O.PortOperator(D, K, None, nthreads=8)
    before = A.device_bytes()
    ax = A.dot(torch.from_numpy(x).cuda()).cpu().numpy()
    aty = A.T.dot(torch.from_numpy(y).cuda()).cpu().numpy()
    assert (A.device_bytes() > before) == grows  # the run layout was built: the kernels under test ran
    s, t = max(np.abs(x).max(), 1e-300), max(np.abs(y).max(), 1e-300)
    assert G.rel(ax / s, P.dot(x) / s) <= TOL
    assert G.rel(aty / t, P.T.dot(y) / t) <= TOL
    return A, ax, aty


# samples: chunks of 96, an odd and an even number of sample pairs per lane, one below and above
@pytest.mark.parametrize('nS,n_fibers', [(17, 21000), (32, 11500), (33, 11500), (65, 6000), (96, 4000), (97, 6000),
                                         (192, 3000), (193, 4500), (288, 4500), (289, 6000)])
def test_sample_counts(nS, n_fibers):
    D, K = _problem(nS, n_fibers)
    rng = np.random.default_rng(nS)
    n, m = D['IC']['nSTR'] + D['EC']['n'] + 2 * D['ISO']['n'], D['IC']['nVOX'] * nS
    _check(D, K, rng.uniform(0, 1, n), rng.uniform(0, 1, m))
    _check(D, K, rng.normal(size=n), rng.normal(size=m))


# responses: several orientation ranges of A' and a small chunk of A; compartments that are absent
@pytest.mark.parametrize('nIC,nEC,nISO,ndirs', [(1, 0, 0, 120), (2, 0, 1, 500), (3, 2, 3, 500), (1, 2, 0, 33), (4, 1, 1, 300)])
def test_compartments(nIC, nEC, nISO, ndirs):
    D, K = _problem(70, 6000, ndirs=ndirs, nIC=nIC, nEC=nEC, nISO=nISO, mask=True)
    rng = np.random.default_rng(nIC)
    n = D['IC']['nSTR'] * nIC + D['EC']['n'] * nEC + D['ISO']['n'] * nISO
    x = rng.uniform(0, 1, n) * (rng.uniform(size=n) < 0.6)      # many zero weights
    y = rng.normal(size=(D['IC']['nVOX'], 70))
    y[::2] = np.abs(y[::2])                                     # rows of one sign beside mixed ones
    y[::5, ::3] = 0.0
    _check(D, K, x, y.reshape(-1))


@pytest.mark.parametrize('scale', [1e-200, 1e-45, 1e45, 1e200])
def test_range_guard(scale):
    D, K = _problem(97, 6000)
    rng = np.random.default_rng(3)
    n, m = D['IC']['nSTR'] + D['EC']['n'] + 2 * D['ISO']['n'], D['IC']['nVOX'] * 97
    _check(D, K, scale * rng.uniform(0, 1, n), scale * rng.normal(size=m))


def test_windows_slabs_and_ranges_are_bitwise_the_one_launch():
    """More voxels than a sorting window, voxels without segments, unsorted input; slabs cut
    windows and the four voxels of a step, and every voxel's arithmetic stays its own."""
    from commit_gb300.operator import LinearOperator
    D, K = _problem(97, 12000, n_mask=9000, dim=(28, 28, 24), seed=2)
    IC = dict(D['IC'])
    keep = IC['vox'] % 7 != 3                                   # every seventh voxel loses its segments
    order = np.random.default_rng(0).permutation(int(keep.sum()))
    for k in ('str', 'vox', 'dir', 'len'):
        IC[k] = IC[k][keep][order]
    IC['n'] = int(keep.sum())
    D = dict(D, IC=IC)
    rng = np.random.default_rng(4)
    x = rng.uniform(0, 1, IC['nSTR'] + D['EC']['n'] + 2 * D['ISO']['n'])
    y = rng.normal(size=IC['nVOX'] * 97)
    A, ax, aty = _check(D, K, x, y)
    for s in (2, 5, 16):
        B = LinearOperator(D, K, None)
        assert B.set_slabs(s) == s
        assert np.array_equal(B.T.dot(torch.from_numpy(y).cuda()).cpu().numpy(), aty)
    assert np.array_equal(A.dot(torch.from_numpy(x).cuda()).cpu().numpy(), ax)


def test_table_signs_and_new_tables():
    """A table with a negative entry takes the general kernels, also when it is set later; a
    new table of one sign is used by the next product."""
    from commit_gb300._lib import check, lib
    from commit_gb300.operator import LinearOperator
    import ctypes
    D, K = _problem(97, 6000)
    rng = np.random.default_rng(5)
    x = rng.uniform(0, 1, D['IC']['nSTR'] + D['EC']['n'] + 2 * D['ISO']['n'])
    y = rng.uniform(0, 1, D['IC']['nVOX'] * 97)
    A, _, _ = _check(D, K, x, y)
    for sign in (1.0, -1.0, 1.0):
        K2 = dict(K, wmr=(K['wmr'] * rng.uniform(0.5, 1.0, K['wmr'].shape)).astype(np.float32))
        K2['wmr'][0, 0, 0] *= sign
        check(lib().cgb_op_set_lut(A.handle, K2['wmr'].ctypes.data_as(ctypes.c_void_p), None, None))
        P = O.PortOperator(D, K2, None, nthreads=8)
        assert G.rel(A.dot(x), P.dot(x)) <= TOL and G.rel(A.T.dot(y), P.T.dot(y)) <= TOL
        B = LinearOperator(D, K2, None)
        assert G.rel(B.dot(x), P.dot(x)) <= TOL and G.rel(B.T.dot(y), P.T.dot(y)) <= TOL


def test_captured_products_follow_the_table():
    """A caller's graph of A and A', captured before and after the layout exists, gives the
    products of the table in place when it is replayed, also one with other signs."""
    import ctypes
    from commit_gb300._lib import check, lib
    from commit_gb300.operator import LinearOperator
    D, K = _problem(97, 6000)
    A = LinearOperator(D, K, None)
    rng = np.random.default_rng(8)
    x, y = rng.uniform(0, 1, A.nCOLS), rng.uniform(0, 1, A.nROWS)
    xd, yd = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    graphs = []
    for _ in range(2):
        ax, aty = torch.empty_like(yd), torch.empty_like(xd)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            A.dot(xd, out=ax)
            A.T.dot(yd, out=aty)
        graphs.append((g, ax, aty))
        A.dot(xd), A.T.dot(yd)
    for sign in (1.0, -1.0):
        K2 = dict(K, wmr=(K['wmr'] * rng.uniform(0.5, 1.0, K['wmr'].shape)).astype(np.float32))
        K2['wmr'][0, 0::2] *= sign
        check(lib().cgb_op_set_lut(A.handle, K2['wmr'].ctypes.data_as(ctypes.c_void_p), None, None))
        P = O.PortOperator(D, K2, None, nthreads=8)
        rx, ry = P.dot(x), P.T.dot(y)
        for g, ax, aty in graphs:
            g.replay()
            torch.cuda.synchronize()
            assert G.rel(ax.cpu().numpy(), rx) <= TOL and G.rel(aty.cpu().numpy(), ry) <= TOL


@pytest.mark.parametrize('bad', [np.inf, -np.inf, np.nan])
def test_non_finite_input_stays_in_its_voxels(bad):
    D, K = _problem(97, 6000)
    from commit_gb300.operator import LinearOperator
    A = LinearOperator(D, K, None)
    rng = np.random.default_rng(6)
    y = rng.uniform(0, 1, (D['IC']['nVOX'], 97))
    x = rng.uniform(0, 1, A.nCOLS)
    x[5] = bad
    touched = np.unique(D['IC']['vox'][D['IC']['str'] == 5])
    r = A.dot(torch.from_numpy(x).cuda()).cpu().numpy().reshape(-1, 97)
    assert np.array_equal(np.flatnonzero(~np.isfinite(r).all(1)), touched)
    y[7, 3] = bad
    g = A.T.dot(torch.from_numpy(y.reshape(-1)).cuda()).cpu().numpy()
    hit = np.zeros(A.nCOLS, bool)
    hit[np.unique(D['IC']['str'][D['IC']['vox'] == 7])] = True
    e = D['IC']['nSTR'] + np.flatnonzero(D['EC']['vox'] == 7)
    hit[e] = True
    hit[D['IC']['nSTR'] + D['EC']['n'] + np.array([7, D['ISO']['n'] + 7])] = True
    assert np.array_equal(~np.isfinite(g), hit)


@pytest.mark.parametrize('table', ['wmh', 'iso'])
def test_non_finite_table_rows_stay_in_their_voxels(table):
    """A zero coefficient skips its row also where a neighbour's does not: an Inf in an EC or ISO
    row reaches only the voxels with a coefficient for it."""
    from commit_gb300.operator import LinearOperator
    D, K = _problem(97, 6000)
    K = dict(K, **{table: K[table].copy()})
    o = int(np.bincount(D['EC']['dir']).argmax())
    K[table].reshape(-1, 97)[o if table == 'wmh' else 0, 3] = np.inf
    A = LinearOperator(D, K, None)
    x = np.random.default_rng(7).uniform(0.1, 1, A.nCOLS)
    base, comp = (D['IC']['nSTR'], 'EC') if table == 'wmh' else (D['IC']['nSTR'] + D['EC']['n'], 'ISO')
    n = D[comp]['n']
    x[base:base + n:2] = 0.0
    rows = D[comp]['dir'] == o if comp == 'EC' else np.ones(n, bool)
    hit = np.unique(D[comp]['vox'][rows & (x[base:base + n] != 0)])
    r = A.dot(torch.from_numpy(x).cuda()).cpu().numpy().reshape(-1, 97)
    assert hit.size and np.array_equal(np.flatnonzero(~np.isfinite(r).all(1)), hit)


def test_fit_matches_the_oracle():
    """FISTA on the residual rows of the shared-memory gradient, host loop and graph."""
    from commit_gb300 import solvers, synth
    from commit_gb300.operator import LinearOperator
    D, K = _problem(97, 6000)
    P = O.PortOperator(D, K, None, nthreads=8)
    y = synth.make_signal(P.dot(synth.make_x(P.nCOLS, 1)), 2)
    rp = O.reg_params(D, K)
    kw = dict(tol_fun=0.0, tol_x=0.0, max_iter=12, verbose=0)
    conf = np.random.default_rng(2).uniform(0.5, 1.0, y.size)
    xo, _ = O.solve(y, P, P.T, regularisation=O.init_regularisation(dict(rp)), confidence_array=conf, **kw)
    A = LinearOperator(D, K, None)
    xs = [solvers.solve(y, A, A.T, regularisation=solvers.init_regularisation(dict(rp)), confidence_array=conf,
                        graph=g, **kw)[0] for g in (False, True)]
    assert G.rel(xs[0], xo) <= 1e-9
    assert np.array_equal(xs[0], xs[1])
