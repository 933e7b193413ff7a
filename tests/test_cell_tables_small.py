"""Cell tables of small bases are formed by one thread per (theta, cell), others on
tiles (cpab_tables.cu: small_basis).  Both add the terms of A in the order of the
columns and take the same exponential: the rows of a batch that goes one way equal,
bit for bit, the same thetas in a call that goes the other.  Sizes on both sides of
each line of the rule: 1024 and 2048 floats of basis, 50 loads a thread, 4096 thetas.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('nc,d', [([1], 1), ([1], 25), ([1], 26), ([2], 256), ([2], 257),
                                  ([21], 24), ([21], 25), ([1, 1], 8), ([1, 1], 9), ([1, 1], 42),
                                  ([1, 1], 43), ([1, 1], 85), ([1, 1], 86), ([2, 2], 10),
                                  ([2, 2], 11), ([1, 1, 1], 4), ([1, 1, 1], 17), ([1, 1, 1], 18),
                                  ([1, 1, 1], 34), ([1, 1, 1], 35)])
def test_both_ways(cuda, nc, d):
    from libcpab_gb300 import _native as N
    n = len(nc)
    g = torch.Generator(device=cuda).manual_seed(d)
    basis = torch.randn(N.num_cells(nc) * n * (n + 1), d, generator=g, device=cuda) / d ** 0.5
    theta = torch.randn(4097, d, generator=g, device=cuda)
    whole = N.cell_tables(nc, 50, theta, basis, want_T=True)
    for count in (1, 7, 4095, 4096):
        part = N.cell_tables(nc, 50, theta[:count].contiguous(), basis, want_T=True)
        for a, b in zip(whole, part):
            assert torch.equal(a[:count], b)
    # the same basis with unused columns (zeros) goes on tiles at any number of thetas
    wide = torch.cat([basis, torch.zeros(len(basis), 2100, device=cuda)], 1)
    more = torch.cat([theta, torch.zeros(len(theta), 2100, device=cuda)], 1)
    for a, b in zip(whole, N.cell_tables(nc, 50, more, wide, want_T=True)):
        assert torch.equal(a, b)
