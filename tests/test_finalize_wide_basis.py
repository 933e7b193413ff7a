"""A basis of more columns than a thread block's shared memory holds floats
(cpab_finalize.cu keeps its share of dtheta there), with one CTA per theta and
with a cluster of them.  With an identity basis the same call returns dL/dA;
dtheta is its product with the basis to within the rounding of a 32-bit dot
product of D terms, 2 D 2^-24 sum |terms|.
"""
import pytest
import torch

from test_finalize import setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('mode', [0, 1])
@pytest.mark.parametrize('nc', [[2], [64], [2, 2]])
@pytest.mark.parametrize('d', [8191, 8192, 8193, 60000, 70001])
def test_wide_basis(cuda, nc, d, mode):
    from libcpab_gb300 import _native as N
    g = torch.Generator(device=cuda).manual_seed(d)
    A, E, pts, gout = setup(cuda, nc, 2, 300)
    D = A[0].numel()
    dA, _ = N.backward(nc, 20, mode, pts, A, E, torch.eye(D, device=cuda), gout)
    B = torch.randn(D, d, generator=g, device=cuda)
    dth, _ = N.backward(nc, 20, mode, pts, A, E, B, gout)
    ref = dA.double() @ B.double()
    bound = 2 * D * 2.0 ** -24 * (dA.abs().double() @ B.abs().double())
    assert ((dth.double() - ref).abs() <= bound).all()
