"""The ragged kernels hand out their tiles in chunks (cpab_ragged.cuh): totals
below, around and above one tile per warp, few long and many short sets, against
each set on its own, and against themselves.  The forward has the same bits; the
sums of dtheta are formed in another order: each is a sum of random signs of which
a lost or doubled chunk (there are at most 64 per SM) would be 1 % or more, while
rounding is below 1e-4 of it for up to 2^20 terms added in chains of under 2^10.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _sets(total, S):
    cuts = np.sort(np.random.RandomState(S).randint(0, total + 1, S - 1))
    return np.concatenate([[0], cuts, [total]]).astype(np.int64)


@pytest.mark.parametrize('nc', [[3, 3], [2, 2, 2], [20]])
@pytest.mark.parametrize('total,S', [(31, 2), (5000, 7), (120_000, 3), (120_000, 900),
                                     (700_000, 2), (700_000, 40)])
def test_points(cuda, nc, total, S):
    from libcpab_gb300 import Cpab, _native as N
    from libcpab_gb300.functions import basis_on
    T = Cpab(nc, backend='pytorch', device='gpu', zero_boundary=False)
    g = torch.Generator(device=cuda).manual_seed(total + S)
    off = _sets(total, S)
    pts = torch.rand(len(nc), total, generator=g, device=cuda)
    gout = torch.randn(len(nc), total, generator=g, device=cuda)
    theta = 0.5 * torch.randn(S, T.get_theta_dim(), generator=g, device=cuda)
    basis = basis_on(T.params, cuda)
    A, _, E = N.cell_tables(nc, 20, theta, basis)
    offd = torch.tensor(off, device=cuda)
    out = N.ragged_points_forward(nc, 20, E, offd, pts)
    runs = [N.ragged_points_backward(nc, 20, 0, A, E, offd, pts, basis, gout)[0] for _ in range(2)]
    assert torch.equal(runs[0], runs[1])
    for s in {0, S // 2, S - 1, int(np.argmax(np.diff(off)))}:
        a, b = int(off[s]), int(off[s + 1])
        if a == b:
            assert not runs[0][s].any()
            continue
        p = pts[:, a:b].contiguous()
        assert torch.equal(N.integrate(nc, 20, p, E[s:s + 1])[0], out[:, a:b])
        one = N.backward(nc, 20, 0, p, A[s:s + 1], E[s:s + 1], basis,
                         gout[None, :, a:b].contiguous())[0][0]
        assert (runs[0][s] - one).abs().max() <= 1e-4 * one.abs().max()


@pytest.mark.parametrize('cells', [1, 7, 8, 9, 100, 128, 129])
@pytest.mark.parametrize('total,S', [(33, 2), (20_000, 50), (700_000, 2), (700_000, 300)])
def test_series(cuda, cells, total, S):
    from libcpab_gb300 import Cpab, _native as N
    from libcpab_gb300.functions import basis_on
    T = Cpab([cells], backend='pytorch', device='gpu', zero_boundary=False)
    g = torch.Generator(device=cuda).manual_seed(total + S)
    off = _sets(total, S)
    values = torch.randn(total, generator=g, device=cuda)
    gout = torch.randn(total, generator=g, device=cuda)
    theta = 0.5 * torch.randn(S, T.get_theta_dim(), generator=g, device=cuda)
    basis = basis_on(T.params, cuda)
    A, _, E = N.cell_tables([cells], 20, theta, basis)
    offd = torch.tensor(off, device=cuda)
    runs = [N.ragged_backward([cells], 20, 0, A, E, offd, values, basis, gout)[0]
            for _ in range(2)]
    assert torch.equal(runs[0], runs[1])
    for s in {0, S // 2, S - 1, int(np.argmax(np.diff(off)))}:
        a, b = int(off[s]), int(off[s + 1])
        if b - a < 2:
            continue
        one = N.ragged_backward([cells], 20, 0, A[s:s + 1], E[s:s + 1],
                                torch.tensor([0, b - a], device=cuda), values[a:b].contiguous(),
                                basis, gout[a:b].contiguous())[0][0]
        assert (runs[0][s] - one).abs().max() <= 1e-4 * one.abs().max()
