"""Host waits of reduced-precision products: the preparation of the reduced tables waits for the
device once per 16-bit product, whichever kernels run it, and not at all with the FP32 table."""
import pytest
import torch

from kernel_trace import trace
from test_smem_products_gpu import _problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('arith', ['bf16', 'fp16', 'f32'])
@pytest.mark.parametrize('large,kernels', [(False, 'gathering'), (True, 'gathering'), (True, 'shared memory'),
                                           (True, 'tensor cores')])
def test_one_wait_per_product(arith, large, kernels):
    from commit_gb300.operator import LinearOperator
    D, K = _problem(97, 6000 if large else 300)
    A = LinearOperator(D, K, None)
    A.tensor_cores(2 if kernels == 'tensor cores' else 1)
    if kernels == 'gathering':
        A.occupancy({arith + '_forward': 1, arith + '_adjoint': 1})
    x, y = torch.rand(A.nCOLS, device='cuda'), torch.rand(A.nROWS, device='cuda')
    base = trace(lambda: A.dot(x.double())).get('cudaDeviceSynchronize', 0)   # the trace's own
    for f, v in ((A.dot, x), (A.T.dot, y)):
        t = trace(lambda: f(v, arith=arith))
        if kernels == 'tensor cores' and arith == 'bf16':
            assert any('_tc(' in k for k in t)
        assert t.get('cudaDeviceSynchronize', 0) - base == (0 if arith == 'f32' else 1)
