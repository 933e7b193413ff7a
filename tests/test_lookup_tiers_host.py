"""The first tier of the 2D and 3D cell lookups (cell_2d_quick, cell_3d_quick)
at tessellations and points where its margins matter, compiled for the host:
single cells, oblong and fine tessellations (the 2D margin grows with the
square of the cell count), and points from one ulp to a few margins away from
every kind of line (interior lines, diagonals, domain edges, and the diagonals
continued outside the domain).  Wherever the FP32 tiers answer they equal the
FP64 replica, and on random points the replica is hardly ever needed.
"""
import numpy as np
import pytest

from test_lookup_host import adversarial, harness, run  # noqa: F401 (fixture)


def near_lines(nc, rng, m=60000):
    """Points at distance 2^-24 .. 2^-10 of a cell from a line, in and around
    the domain."""
    n = len(nc)
    u = np.stack([rng.uniform(-1.5, c + 1.5, m) for c in nc])       # in cells
    eps = rng.choice([-1.0, 1.0], m) * 2.0 ** -rng.uniform(10, 25, m)
    kind = rng.integers(0, 3, m)
    a = rng.integers(0, n, m)
    b = (a + 1) % n
    cols = np.arange(m)
    edge = np.where(rng.random(m) < 0.3, np.where(rng.random(m) < 0.5, 0, np.array(nc)[a]),
                    np.round(u[a, cols]))
    u[a, cols] = np.where(kind == 0, edge + eps, u[a, cols])
    if n > 1:
        fb = u[b, cols] - np.round(u[b, cols])
        u[a, cols] = np.where(kind == 1, np.round(u[a, cols]) + fb + eps, u[a, cols])
        u[a, cols] = np.where(kind == 2, np.round(u[a, cols]) - fb + eps, u[a, cols])
    return (u / np.array(nc)[:, None]).astype(np.float32)


@pytest.mark.parametrize('nc', [[1, 1], [1, 5], [20, 3], [13, 13], [16, 16], [31, 31], [49, 49],
                                [1, 1, 1], [4, 2, 1], [2, 4, 8], [8, 8, 8], [2, 2, 3], [1], [977]])
def test_first_tier(nc, harness, tmp_path):  # noqa: F811
    rng = np.random.default_rng(sum(nc) * 131 + len(nc))
    P = np.concatenate([adversarial(nc, rng, 120000), near_lines(nc, rng)], axis=1)
    if len(nc) == 1:
        P = P[:, np.abs(P[0]) < 1e6]
    fast, exact = run(harness, tmp_path, nc, P)
    bad = np.nonzero((fast >= 0) & (fast != exact))[0]
    assert bad.size == 0, 'FP32 tiers wrong at %s' % P[:, bad[:5]].T
    fast, _ = run(harness, tmp_path, nc, rng.random((len(nc), 100000)).astype(np.float32))
    assert (fast < 0).mean() < 1e-4
