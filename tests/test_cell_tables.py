"""The cell-table kernel (cpab_tables.cu) at the edges of its tiles of cells, chunks
of basis columns and groups of thetas, against 64 bits."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('nc', [[1], [63], [130], [1, 1], [3, 3], [8, 8], [1, 1, 1], [2, 3, 4]])
@pytest.mark.parametrize('n_theta,d', [(1, 1), (1, 33), (9, 31), (40, 32), (200, 65), (1500, 3)])
def test_tables(cuda, nc, n_theta, d):
    """A = B theta in 32 bits is within (d + 1) 2^-24 sum |terms| of 64 bits; the
    exponential is a polynomial of degree ten in E (under 2^7 roundings) of a matrix
    of norm below one half."""
    from libcpab_gb300 import _native as N
    ndim, nC = len(nc), N.num_cells(nc)
    g = torch.Generator(device=cuda).manual_seed(n_theta + d)
    basis = torch.randn(nC * ndim * (ndim + 1), d, generator=g, device=cuda) / d ** 0.5
    theta = torch.randn(n_theta, d, generator=g, device=cuda)
    A, Tm, E = N.cell_tables(nc, 50, theta, basis, want_T=True)
    ref = theta.double() @ basis.double().T
    mag = theta.double().abs() @ basis.double().abs().T
    assert ((A.reshape(n_theta, -1).double() - ref).abs() <= (d + 1) * 2.0 ** -24 * mag).all()
    X = torch.zeros(n_theta, nC, ndim + 1, ndim + 1, dtype=torch.float64, device=cuda)
    X[:, :, :ndim] = A.double() * float(np.float32(1 / 50))
    want = (torch.matrix_exp(X) - torch.eye(ndim + 1, dtype=torch.float64, device=cuda))[:, :, :ndim]
    bound = 2.0 ** -17 * want.abs().amax((2, 3), keepdim=True) + 1e-30
    assert ((E.double() - want).abs() <= bound).all()
    eye = torch.eye(ndim, ndim + 1, device=cuda)
    assert torch.equal(Tm, E + eye)
    again = N.cell_tables(nc, 50, theta, basis, want_A=False)[2]
    assert torch.equal(again, E)
    assert torch.equal(N.cell_tables(nc, 50, theta[:1].contiguous(), basis)[0], A[:1])
