"""Which products take the kernels that keep the table in shared memory, and what the handle holds
for them."""
import ctypes

import numpy as np
import pytest
import torch

import golden_io as G
import oracle as O
from kernel_trace import ran
from test_smem_products_gpu import TOL, _problem

pytestmark = pytest.mark.gpu


# segments x responses per voxel below and above 4 per chunk of 96 samples (two chunks: 8), far below
# for three chunks (12), and between A' (two orientation ranges: 12) and A (three chunks for one: 20)
@pytest.mark.parametrize('nS,n_fibers,nIC,ndirs,fwd,adj', [
    (97, 3000, 1, 120, False, False), (97, 3800, 1, 120, True, True), (288, 2500, 1, 120, False, False),
    (70, 3000, 2, 500, False, True), (70, 5000, 2, 500, True, True)])
def test_layout_only_for_the_products_that_use_it(nS, n_fibers, nIC, ndirs, fwd, adj):
    """An operator too sparse for these kernels holds nothing for them; one dense enough for A' only
    holds no run coefficients."""
    from commit_gb300.operator import LinearOperator
    D, K = _problem(nS, n_fibers, n_mask=60000, dim=(60, 60, 40), ndirs=ndirs, nIC=nIC)
    IC = D['IC']
    per = IC['n'] * nIC / IC['nVOX']
    chunks = -(-nS // 96)
    low_a, low_at = (20.0, 12.0) if nIC == 2 else (4.0 * chunks,) * 2
    assert IC['n'] * nIC * nS >= 1e7 and (per >= low_a) == fwd and (per >= low_at) == adj
    A, P = LinearOperator(D, K, None), O.PortOperator(D, K, None, nthreads=8)
    rng = np.random.default_rng(0)
    x, y = rng.uniform(0, 1, A.nCOLS), rng.normal(size=A.nROWS)
    xd, yd = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    before = A.device_bytes()
    assert G.rel(A.dot(xd).cpu().numpy(), P.dot(x)) <= TOL
    assert G.rel(A.T.dot(yd).cpu().numpy(), P.T.dot(y)) <= TOL
    held = A.device_bytes() - before
    v, runs = IC['nVOX'], np.unique(IC['vox'].astype(np.int64) * ndirs + IC['dir']).size
    layout, coef, part = 8 * v + 6 * runs, 8 * nIC * runs, 8 * nIC * runs * chunks
    want = (layout + part + (coef if fwd else 0)) if adj else 0
    small = (2 << 20) + 4 * 4 * v                                # table images, orientation ranges, EC / ISO parts
    if chunks > 1:
        small += 8 * chunks * (D['EC']['n'] + 2 * D['ISO']['n'])
    assert want <= held <= want + (small if want else 0)
    assert fwd == adj or small < coef                            # the bound tells the coefficients apart
    assert ran(lambda: A.dot(xd), 'k_fwd_smem', 'k_forward_p') == [fwd, not fwd]
    assert ran(lambda: A.T.dot(yd), 'k_adj_smem', 'k_adjoint_p') == [adj, not adj]


def _set_table(A, K):
    from commit_gb300._lib import check, lib
    check(lib().cgb_op_set_lut(A.handle, K['wmr'].ctypes.data_as(ctypes.c_void_p), None, None))


def test_bytes_follow_the_layout():
    """A table with a negative entry releases the layout of the FP64 products and the next one builds it again:
    the handle's bytes do not grow with the changes."""
    from commit_gb300.operator import LinearOperator
    D, K = _problem(97, 6000)
    A = LinearOperator(D, K, None)
    x, y = torch.rand(A.nCOLS, dtype=torch.float64, device='cuda'), torch.rand(A.nROWS, dtype=torch.float64, device='cuda')
    neg = dict(K, wmr=K['wmr'].copy())
    neg['wmr'][0, 0, 0] *= -1
    start = A.device_bytes()
    A.dot(x), A.T.dot(y)
    full = A.device_bytes()
    for _ in range(3):
        _set_table(A, neg)
        A.dot(x), A.T.dot(y)
        assert start < A.device_bytes() < full
        _set_table(A, K)
        A.dot(x), A.T.dot(y)
        assert A.device_bytes() == full
    A.dot(x.float(), arith='f32'), A.T.dot(y.float(), arith='f32')
    assert A.device_bytes() > full


def test_set_builds_and_shapes_hold_their_own_products():
    """A register build that is set keeps the products of its kernel, and no others, from the shared-memory
    kernels; a shape keeps all; selecting the default family releases both."""
    from commit_gb300.operator import LinearOperator
    D, K = _problem(97, 6000)
    A = LinearOperator(D, K, None)
    A.tensor_cores(1)
    x, y = torch.rand(A.nCOLS, dtype=torch.float64, device='cuda'), torch.rand(A.nROWS, dtype=torch.float64, device='cuda')
    x32, y32 = x.float(), y.float()

    def shared():
        out = ran(lambda: A.dot(x), 'k_fwd_smem') + ran(lambda: A.T.dot(y), 'k_adj_smem')
        for ar in ('bf16', 'fp16', 'f32'):
            out += ran(lambda: A.dot(x32, arith=ar), 'k_fwd_mix_smem') + ran(lambda: A.T.dot(y32, arith=ar), 'k_adj_mix_smem')
        return out
    # FP64 A, A'; BF16 A, A'; FP16 A, A'; FP32 A, A'
    assert shared() == [True] * 8
    A.occupancy({'bf16_adjoint': 1})
    assert shared() == [True, True, True, False, True, True, True, True]
    A.occupancy({'ff_forward': 2, 'f32_forward': 0})
    assert shared() == [False, True, True, False, True, True, False, True]
    assert A.ff_kernels(1) == 1
    assert shared() == [True] * 8
    A.ff_shape(1)
    assert shared() == [False] * 8
    A.ff_kernels(1)
    assert shared() == [True] * 8


def test_products_on_reused_stream_handles():
    """Streams that come and go: a new stream may have the handle of a destroyed one and is still
    another stream, so its product waits for the last one before it writes the shared buffers."""
    from commit_gb300._lib import check, lib, DTYPE_F32, DTYPE_F64
    from commit_gb300.operator import LinearOperator
    path = next(l.split()[-1] for l in open('/proc/self/maps') if 'libcudart.so' in l)
    rt = ctypes.CDLL(path)
    D, K = _problem(97, 20000, n_mask=9000, dim=(28, 28, 24), ndirs=120)
    A = LinearOperator(D, K, None)
    xs = [torch.rand(A.nCOLS, dtype=torch.float64, device='cuda') for _ in range(4)]
    for dtype, num, arith in ((torch.float64, DTYPE_F64, 1), (torch.float32, DTYPE_F32, 3)):
        ins = [x.to(dtype) for x in xs]
        refs = [A.dot(v, arith='fp16' if num == DTYPE_F32 else None) for v in ins]
        outs = [torch.empty_like(r) for r in refs]
        torch.cuda.synchronize()
        for v, out in zip(ins, outs):
            st = ctypes.c_void_p()
            assert rt.cudaStreamCreateWithFlags(ctypes.byref(st), 1) == 0    # non-blocking
            check(lib().cgb_op_apply(A.handle, 0, ctypes.c_void_p(v.data_ptr()), v.numel(), ctypes.c_void_p(out.data_ptr()),
                                     out.numel(), num, arith, st))
            assert rt.cudaStreamDestroy(st) == 0                             # its work goes on
        torch.cuda.synchronize()
        for out, r in zip(outs, refs):
            assert torch.equal(out, r)
