"""The interpolation backward's shared reductions (cpab_interp.cu): output
sizes around the 32 x 32 tiles and the rows a warp takes, 1 to 5 channels,
several images, grids whose points sample the same, neighbouring, distant and
clamped pixels.  d(data) against the same sum in 64 bits: a sum of n terms in
32 bits, in any order, is within n 2^-23 sum |terms| of it (each term carries
two roundings more); d(grid) within 1e-5 of the C oracle's largest value.
"""
import itertools

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def scatter(grid, gout, size, outsize):
    """(sum, sum of |terms|, count) of the corner weights times gout, in 64 bits."""
    nb, n, nP = grid.shape
    C = gout.shape[1]
    last = torch.tensor([s - 1.0 for s in size], device=grid.device)
    x = grid.transpose(1, 2) * last                       # 32-bit, as the kernel forms it
    lo = torch.minimum(x.floor().clamp(min=0), last)
    hi = torch.minimum((x.floor() + 1).clamp(min=0), last)
    f = (x - lo).double()
    w = gout.permute(0, 1, *[n + 1 - j for j in range(n)]).reshape(nb, C, nP).double()
    out = [torch.zeros(nb, C, int(np.prod(size)), dtype=torch.float64, device=grid.device)
           for _ in range(3)]
    for bits in itertools.product((0, 1), repeat=n):
        idx, wt = 0, 1.0
        for j in range(n):
            idx = idx * size[j] + (hi if bits[j] else lo)[..., j].long()
            wt = wt * (f[..., j] if bits[j] else 1 - f[..., j])
        idx = idx[:, None].expand(nb, C, nP)
        for o, t in zip(out, (wt[:, None] * w, (wt[:, None] * w).abs(), torch.ones_like(w))):
            o.scatter_add_(2, idx, t)
    return [o.reshape(nb, C, *size) for o in out]


@pytest.mark.parametrize('kind', ['identity', 'smooth', 'random', 'constant', 'outside'])
@pytest.mark.parametrize('size,outsize,C', [
    ((40, 50), (32, 32), 3), ((40, 50), (33, 31), 1), ((33, 65), (65, 33), 2), ((7, 9), (5, 3), 4),
    ((64, 64), (36, 100), 5), ((1, 6), (8, 40), 3), ((10, 12, 14), (9, 3, 33), 1),
    ((6, 7, 8), (34, 2, 31), 2), ((6, 7, 8), (8, 8, 8), 3)])
def test_backward(cuda, oracle, size, outsize, C, kind):
    from libcpab_gb300 import _native as N
    n, nb = len(size), 3
    g = torch.Generator(device=cuda).manual_seed(len(kind) + sum(size))
    axes = [torch.linspace(0, 1, o, device=cuda) for o in outsize]
    mesh = torch.stack([m.reshape(-1) for m in
                        torch.meshgrid(*axes[::-1], indexing='ij')[::-1]])
    grid = mesh.expand(nb, *mesh.shape).clone()
    if kind == 'smooth':
        grid += 0.08 * torch.sin(5 * grid.roll(1, 1) + torch.arange(nb, device=cuda)[:, None, None])
    elif kind == 'random':
        grid = torch.rand(grid.shape, generator=g, device=cuda)
    elif kind == 'constant':
        grid = torch.full_like(grid, 0.4)
    elif kind == 'outside':
        grid = 2.2 * grid - 0.6
    data = torch.rand(nb, C, *size, generator=g, device=cuda)
    gout = torch.randn(nb, C, *outsize, generator=g, device=cuda)
    dd, dg = N.interpolate_backward(data, grid, outsize, gout)
    ref, mag, count = scatter(grid, gout, size, outsize)
    assert ((dd.double() - ref).abs() <= (count + 4) * 2.0 ** -23 * mag).all()
    _, dg_o = oracle.interpolate_backward(data.cpu().numpy(), grid.cpu().numpy(), list(outsize),
                                          gout.cpu().numpy())
    assert np.abs(dg.cpu().numpy() - dg_o).max() <= 1e-5 * max(1e-30, np.abs(dg_o).max())
    only, none = N.interpolate_backward(data, grid, outsize, gout, want_dgrid=False)
    assert none is None and ((only.double() - ref).abs() <= (count + 4) * 2.0 ** -23 * mag).all()
    none, only = N.interpolate_backward(data, grid, outsize, gout, want_ddata=False)
    assert none is None and torch.equal(only, dg)
