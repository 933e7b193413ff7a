"""dtheta's tail (cpab_finalize.cu): partial sums, cell map and basis
contraction split over the CTAs of a cluster.

The contraction is checked on synthetic bases of 1 .. 700 columns (fewer than,
exactly and more than the block's 512 threads) and cell counts that leave the
last CTA of a cluster a short or empty slice: with an identity basis the same
call returns dL/dA itself, and dtheta must be its product with the basis to
within the rounding of a 32-bit dot product of D terms, 2 D 2^-24 sum |terms|.
The partial sums are checked across cluster sizes: one theta (8 CTAs) against
the same theta in a batch of 700 (one CTA each), to the 1e-5 that other
summation orders are held to.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu


def setup(cuda, nc, n_theta, nP, seed=0):
    from libcpab_gb300 import _native as N
    g = torch.Generator(device=cuda).manual_seed(seed)
    nC, n = N.num_cells(nc), len(nc)
    theta = 0.3 * torch.randn(n_theta, 4, generator=g, device=cuda)
    smooth = torch.randn(nC * n * (n + 1), 4, generator=g, device=cuda)
    A, _, E = N.cell_tables(nc, 20, theta, smooth)
    pts = torch.rand(n, nP, generator=g, device=cuda)
    gout = torch.randn(n_theta, n, nP, generator=g, device=cuda)
    return A, E, pts, gout


@pytest.mark.parametrize('mode', [0, 1])
@pytest.mark.parametrize('nc', [[1], [31], [33], [130], [2, 2], [3, 3], [5, 7], [2, 2, 2]])
def test_contraction(cuda, nc, mode):
    from libcpab_gb300 import _native as N
    g = torch.Generator(device=cuda).manual_seed(1)
    for n_theta in (1, 90):
        A, E, pts, gout = setup(cuda, nc, n_theta, 500)
        D = A[0].numel()
        dA, _ = N.backward(nc, 20, mode, pts, A, E, torch.eye(D, device=cuda), gout)
        for d in (1, 3, 34, 511, 512, 513, 700):
            B = torch.randn(D, d, generator=g, device=cuda)
            dth, _ = N.backward(nc, 20, mode, pts, A, E, B, gout)
            ref = dA.double() @ B.double()
            bound = 2 * D * 2.0 ** -24 * (dA.abs().double() @ B.abs().double())
            assert ((dth.double() - ref).abs() <= bound).all()


@pytest.mark.parametrize('nc,nP', [([64], 7), ([64], 20000), ([4, 4], 1), ([4, 4], 30000),
                                   ([2, 2, 2], 3000)])
def test_cluster_sizes_agree(cuda, nc, nP):
    from libcpab_gb300 import _native as N
    A, E, pts, gout = setup(cuda, nc, 1, nP)
    eye = torch.eye(A[0].numel(), device=cuda)
    one, _ = N.backward(nc, 20, 0, pts, A, E, eye, gout)
    many, _ = N.backward(nc, 20, 0, pts, A.repeat(700, 1, 1, 1), E, eye, gout.repeat(700, 1, 1))
    assert (many - many[:1]).abs().max() == 0
    assert (one - many[:1]).norm() <= 1e-5 * one.norm()
