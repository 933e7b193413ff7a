"""The sampler's backward channel by channel (5 and more channels in 2D, 3 and more in
3D) and the rows of tiles that the image's edge cuts, spread over a block's warps:
output rows from 1 to a few more than a tile's 32.  Held as the paths for few channels
are (test_interp_backward): d(data) to n 2^-23 sum |terms| of the sum in 64 bits,
d(grid) to 1e-5 of the oracle's largest value.
"""
import numpy as np
import pytest
import torch

from test_interp_backward import scatter

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('kind', ['smooth', 'random', 'outside'])
@pytest.mark.parametrize('size,outsize,C', [
    ((9, 8), (1, 33), 5), ((20, 30), (7, 40), 16), ((30, 20), (8, 5), 6), ((12, 40), (9, 64), 5),
    ((33, 33), (39, 31), 17), ((40, 40), (41, 33), 2), ((9, 8), (1, 3), 3), ((20, 20), (17, 32), 1),
    ((6, 7, 8), (1, 2, 33), 3), ((6, 7, 8), (9, 3, 31), 4), ((9, 5, 6), (40, 2, 8), 5),
    ((5, 5, 5), (33, 3, 34), 8), ((6, 7, 8), (8, 2, 40), 1), ((6, 7, 8), (41, 2, 9), 2)])
def test_backward(cuda, oracle, size, outsize, C, kind):
    from libcpab_gb300 import _native as N
    n, nb = len(size), 2
    g = torch.Generator(device=cuda).manual_seed(len(kind) + sum(outsize) + C)
    axes = [torch.linspace(0, 1, o, device=cuda) for o in outsize]
    mesh = torch.stack([m.reshape(-1) for m in
                        torch.meshgrid(*axes[::-1], indexing='ij')[::-1]])
    grid = mesh.expand(nb, *mesh.shape).clone()
    if kind == 'smooth':
        grid += 0.08 * torch.sin(5 * grid.roll(1, 1) + torch.arange(nb, device=cuda)[:, None, None])
    elif kind == 'random':
        grid = torch.rand(grid.shape, generator=g, device=cuda)
    else:
        grid = 2.2 * grid - 0.6
    data = torch.rand(nb, C, *size, generator=g, device=cuda)
    gout = torch.randn(nb, C, *outsize, generator=g, device=cuda)
    dd, dg = N.interpolate_backward(data, grid, outsize, gout)
    ref, mag, count = scatter(grid, gout, size, outsize)
    assert ((dd.double() - ref).abs() <= (count + 4) * 2.0 ** -23 * mag).all()
    _, dg_o = oracle.interpolate_backward(data.cpu().numpy(), grid.cpu().numpy(), list(outsize),
                                          gout.cpu().numpy())
    assert np.abs(dg.cpu().numpy() - dg_o).max() <= 1e-5 * max(1e-30, np.abs(dg_o).max())
    none, only = N.interpolate_backward(data, grid, outsize, gout, want_ddata=False)
    assert none is None and torch.equal(only, dg)
