"""The squared error of the fused series loss: the sum of a series' chunk sums.

`out` comes back with it, so the sum is checked against 64 bits over the same
32-bit residuals.  A long series has up to 64 chunks per SM; its sum is a tree over
them.  A term meets fewer than 128 additions in all (up to 60 points of a lane, 32
lanes, 10,000 chunks over 512 threads, 16 warps): 128 * 2^-24 relative, all terms
being positive.  Equal residuals are the case in
which a serial chain over the chunks errs most (its roundings have one sign).
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('cells', [20, 150])
@pytest.mark.parametrize('lengths', [[4_000_000], [1, 31, 33, 3_000_000, 0, 500_000], [700] * 2000])
@pytest.mark.parametrize('residual', ['equal', 'random'])
def test_sum(cuda, cells, lengths, residual):
    from libcpab_gb300 import Cpab, _native as N
    from libcpab_gb300.functions import basis_on
    T = Cpab([cells], backend='pytorch', device='gpu')
    basis = basis_on(T.params, cuda)
    S, total = len(lengths), sum(lengths)
    off = torch.tensor(np.concatenate([[0], np.cumsum(lengths)]), device=cuda)
    g = torch.Generator(device=cuda).manual_seed(S)
    A, _, E = N.cell_tables([cells], 20, torch.zeros(S, T.get_theta_dim(), device=cuda), basis)
    values = torch.ones(total, device=cuda)
    target = torch.full((total,), 0.7, device=cuda) if residual == 'equal' else \
        torch.randn(total, generator=g, device=cuda)
    runs = [N.ragged_mse([cells], 20, 0, A, E, off, values, target, basis, want_out=True)
            for _ in range(2)]
    assert torch.equal(runs[0]['sse'], runs[1]['sse'])
    r2 = (runs[0]['out'] - target).double() ** 2
    sums = torch.cat([torch.zeros(1, device=cuda, dtype=torch.float64), r2.cumsum(0)])
    want = sums[off[1:]] - sums[off[:-1]]
    got = runs[0]['sse'].double()
    assert ((got - want).abs() <= 128 * 2.0 ** -24 * want).all()
