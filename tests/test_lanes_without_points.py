"""A warp's lanes without a point (sets whose size is not a multiple of 32, the end of
an image) bring nothing into dtheta, whatever the field does away from the call's own
points: a trajectory that overflows would, with a zero cotangent too (0 * inf is NaN).

The points lie in cells whose field is zero and all others expand by e^80 a step
(A = 4000 at 50 steps; the midpoint map by 3281): a trajectory from the domain's
centre, say, is infinite after a few steps.  The basis is the identity: dtheta is dL/dA.  It is
compared with the same points in full blocks of 256, filled up with more points of
the zero cells whose cotangent is zero: the same sums in another order (1e-5).
"""
import pytest
import torch

pytestmark = pytest.mark.gpu

BIG = 4000.0


def setup(cuda, nc, calm):
    """(A, E, basis): zero field in the cells `calm` of each theta, BIG elsewhere."""
    from libcpab_gb300 import _native as N
    n, nC = len(nc), N.num_cells(nc)
    A = torch.zeros(1, nC, n, n + 1, device=cuda)
    for j in range(n):
        A[:, :, j, j] = BIG
    A[:, calm] = 0.0
    basis = torch.eye(A[0].numel(), device=cuda)
    A, _, E = N.cell_tables(nc, 50, A.reshape(1, -1), basis)
    return A, E, basis


def calm_points(cuda, n, count, seed=0):
    """Points of the first cell / square / cube of a tessellation with three per axis."""
    g = torch.Generator(device=cuda).manual_seed(seed)
    return 0.02 + 0.28 * torch.rand(n, count, generator=g, device=cuda)


def first_cells(n):
    return list(range({1: 1, 2: 4, 3: 5}[n]))


def full_blocks(N, nc, mode, A, E, basis, pts, gout):
    n, count = pts.shape
    more = -count % 256
    p = torch.cat([pts, calm_points(pts.device, n, more, 9)], 1).contiguous()
    g = torch.cat([gout, torch.zeros(n, more, device=pts.device)], 1)[None].contiguous()
    return N.backward(nc, 50, mode, p, A, E, basis, g)[0]


def same(a, b):
    assert torch.isfinite(a).all() and b.norm() > 0
    assert (a - b).norm() <= 1e-5 * b.norm()


@pytest.mark.parametrize('mode', [0, 1, 2])
@pytest.mark.parametrize('count', [1, 31, 33])
@pytest.mark.parametrize('nc', [[3], [3, 3], [3, 3, 3]])
def test_points(cuda, nc, count, mode):
    from libcpab_gb300 import _native as N
    n = len(nc)
    A, E, basis = setup(cuda, nc, first_cells(n))
    pts = calm_points(cuda, n, count)
    g = torch.Generator(device=cuda).manual_seed(count)
    gout = torch.randn(n, count, generator=g, device=cuda)
    want = full_blocks(N, nc, mode, A, E, basis, pts, gout)
    assert torch.isfinite(want).all()
    same(N.backward(nc, 50, mode, pts, A, E, basis, gout[None].contiguous())[0], want)
    # three ragged sets of the same points
    off = torch.tensor([0, count, 2 * count, 3 * count], device=cuda)
    got, _ = N.ragged_points_backward(nc, 50, mode, A.repeat(3, 1, 1, 1), E.repeat(3, 1, 1, 1),
                                      off, pts.repeat(1, 3), basis, gout.repeat(1, 3))
    for s in range(3):
        same(got[s:s + 1], want)


@pytest.mark.parametrize('cells', [3, 151])
@pytest.mark.parametrize('mode', [0, 1, 2])
def test_series_of_one_value(cuda, cells, mode):
    """A series of one value lies at 0 and its position has no gradient."""
    from libcpab_gb300 import _native as N
    A, E, basis = setup(cuda, [cells], list(range((cells + 1) // 3)))
    off = torch.arange(6, device=cuda)
    values, gout = torch.randn(2, 5, device=cuda)
    five = A.repeat(5, 1, 1, 1), E.repeat(5, 1, 1, 1)
    dtheta, dvalues = N.ragged_backward([cells], 50, mode, *five, off, values, basis, gout)
    assert not dtheta.any() and torch.equal(dvalues, gout)
    res = N.ragged_mse([cells], 50, mode, *five, off, values, gout, basis)
    assert not res['dtheta'].any() and torch.equal(res['sse'], (values - gout) ** 2)


@pytest.mark.parametrize('mode', [0, 1, 2])
@pytest.mark.parametrize('nc,outsize', [([3], (1,)), ([3, 3], (1, 1)), ([3, 3], (1, 2)),
                                        ([3, 3], (2, 1)), ([3, 3, 3], (1, 1, 1)),
                                        ([3, 3, 3], (1, 1, 2))])
def test_image(cuda, nc, outsize, mode):
    """Output points in the domain's corners only."""
    from libcpab_gb300 import _native as N
    n = len(nc)
    per = {1: 1, 2: 4, 3: 5}[n]
    corner = [per * 2 * 3 ** j + k for j in range(n) for k in range(per)] if n > 1 else []
    A, E, basis = setup(cuda, nc, first_cells(n) + corner)
    g = torch.Generator(device=cuda).manual_seed(n)
    data = torch.rand(1, 2, *[5] * n, generator=g, device=cuda)
    lin = torch.cat([torch.linspace(0, 1, o, device=cuda) for o in outsize])
    out, grid = N.transform_data(nc, 50, lin, outsize, E, data, save_grid=True)
    gout = torch.randn(out.shape, generator=g, device=cuda)
    axes = [torch.linspace(0, 1, o, device=cuda) for o in outsize]
    pts = torch.stack([a.reshape(-1) for a in torch.meshgrid(*axes, indexing='ij')])
    _, dgrid = N.interpolate_backward(data, pts[None].contiguous(), outsize, gout)
    want = full_blocks(N, nc, mode, A, E, basis, pts, dgrid[0])
    _, dtheta = N.transform_data_backward(nc, 50, mode, lin, outsize, A, E, grid, data, basis, gout)
    same(dtheta, want)
