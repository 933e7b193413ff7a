"""The order in which the adjoint kernels take the points: patches of a
meshgrid (row lengths that give 8 x 4, 4 x 8 and 16 x 2 patches, that give
none, and that are longer than the kernel looks), against the same points in a
random order, which are taken as they come.  A point's own arithmetic does not
depend on the order: dpoints is bit-identical; dtheta agrees to the 1e-5 that
other summation orders are held to.  The fused image backward walks patches of
the output (whole, cut by the edge, or none) and is held to the unfused chain.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu


def mesh(cuda, size):
    axes = [torch.linspace(0, 1, s, device=cuda) for s in size]
    m = torch.meshgrid(*axes[::-1], indexing='ij')
    return torch.stack([a.reshape(-1) for a in m[::-1]]).contiguous()


@pytest.mark.parametrize('mode', [0, 1, 2])
@pytest.mark.parametrize('nc,size', [
    ([3, 3], (8, 8)), ([3, 3], (40, 12)), ([8, 8], (12, 24)), ([3, 3], (16, 6)), ([3, 3], (48, 2)),
    ([4, 4], (9, 32)), ([3, 3], (1024, 4)), ([3, 3], (1032, 4)), ([3, 3], (2, 512)),
    ([8, 8], (224, 224)), ([2, 2, 2], (8, 6, 10)), ([2, 2, 2], (20, 5, 7)), ([1, 1], (64, 1))])
def test_meshgrid_and_shuffled(cuda, nc, size, mode):
    from libcpab_gb300 import _native as N
    g = torch.Generator(device=cuda).manual_seed(sum(size))
    n, nC = len(nc), N.num_cells(nc)
    pts = mesh(cuda, size)
    nP = pts.shape[1]
    B = torch.randn(nC * n * (n + 1), 5, generator=g, device=cuda)
    for n_theta in (1, 3):
        theta = 0.2 * torch.randn(n_theta, 5, generator=g, device=cuda)
        gout = torch.randn(n_theta, n, nP, generator=g, device=cuda)
        A, _, E = N.cell_tables(nc, 50, theta, B)
        dth, dp = N.backward(nc, 50, mode, pts, A, E, B, gout, want_dpoints=True)
        perm = torch.randperm(nP, generator=g, device=cuda)
        dth2, dp2 = N.backward(nc, 50, mode, pts[:, perm].contiguous(), A, E, B,
                               gout[:, :, perm].contiguous(), want_dpoints=True)
        assert torch.equal(dp[:, :, perm], dp2)
        assert (dth - dth2).norm() <= 1e-5 * dth2.norm()
        # one grid per theta takes the same route
        dth3, dp3 = N.backward(nc, 50, mode, pts.expand(n_theta, n, nP).contiguous(), A, E, B,
                               gout, want_dpoints=True)
        assert torch.equal(dp3, dp) and torch.equal(dth3, dth)


@pytest.mark.parametrize('gradient', ['reference', 'exact'])
@pytest.mark.parametrize('nc,size,outsize', [
    ([3, 3], (20, 30), (32, 64)), ([3, 3], (33, 31), (33, 47)), ([4, 4], (16, 16), (5, 7)),
    ([3, 3], (9, 9), (4, 8)), ([8, 8], (64, 40), (70, 81)), ([2, 2, 2], (8, 9, 10), (6, 8, 16)),
    ([2, 2, 2], (8, 9, 10), (5, 7, 9)), ([7], (30,), (77,))])
def test_fused_backward_walks_every_point(cuda, tmp_path, nc, size, outsize, gradient):
    from libcpab_gb300 import Cpab
    T = Cpab(nc, backend='pytorch', device='gpu', basis_dir=str(tmp_path))
    T.set_solver_params(gradient=gradient)
    g = torch.Generator(device=cuda).manual_seed(len(size))
    theta = (0.3 * torch.randn(3, T.get_theta_dim(), generator=g, device=cuda)).requires_grad_(True)
    data = torch.rand(3, 2, *size, generator=g, device=cuda).requires_grad_(True)
    out = T.transform_data(data, theta, list(outsize))
    w = torch.randn(out.shape, generator=g, device=cuda)
    a = torch.autograd.grad(out, [theta, data], w)
    ref = T.interpolate(data, T.transform_grid(T.uniform_meshgrid(list(outsize)), theta),
                        list(outsize))
    b = torch.autograd.grad(ref, [theta, data], w)
    assert (a[0] - b[0]).norm() <= 1e-4 * b[0].norm()
    assert (a[1] - b[1]).norm() <= 1e-5 * b[1].norm()


@pytest.mark.parametrize('nc,size', [([3, 3], (40, 12)), ([3, 3], (9, 32)), ([8, 8], (64, 64)),
                                     ([2, 2, 2], (8, 6, 10)), ([7], (50,))])
def test_exact_flow_meshgrid_and_shuffled(cuda, nc, size):
    """The exact flow takes a meshgrid, and its image in the backward, in patches
    too; a point's flow does not depend on the points beside it."""
    from libcpab_gb300 import _native as N
    g = torch.Generator(device=cuda).manual_seed(sum(size))
    n = len(nc)
    pts = mesh(cuda, size)
    nP = pts.shape[1]
    B = torch.randn(N.num_cells(nc) * n * (n + 1), 5, generator=g, device=cuda)
    A, _, _ = N.cell_tables(nc, 50, 0.2 * torch.randn(2, 5, generator=g, device=cuda), B)
    gout = torch.randn(2, n, nP, generator=g, device=cuda)
    out = N.integrate_exact(nc, pts, A)
    dth, dp = N.backward_exact(nc, out, A, B, gout, want_dpoints=True)
    perm = torch.randperm(nP, generator=g, device=cuda)
    out2 = N.integrate_exact(nc, pts[:, perm].contiguous(), A)
    dth2, dp2 = N.backward_exact(nc, out2, A, B, gout[:, :, perm].contiguous(), want_dpoints=True)
    assert torch.equal(out[:, :, perm], out2) and torch.equal(dp[:, :, perm], dp2)
    assert (dth - dth2).norm() <= 1e-5 * dth2.norm()
    assert torch.equal(dth, N.backward_exact(nc, out, A, B, gout)[0])
    N.device_status()   # cleared: a trajectory may reach the step limit, in any order
