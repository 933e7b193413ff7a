"""One sub-step of the exact flow and of its adjoint (csrc/cpab_flow.cuh), compiled
for the host, against 64 bits (Taylor series of 40 terms, 16 Gauss nodes).

  * the certificate: |A| dt <= 1, and over the sub-step the point moves no further
    than the distance to the nearest face plus the overshoot, both to 2^-20, with the
    root and the quotient of the rule off by 2^-22 either way (the GPU's approximate
    ones are within that), and with them rounded;
  * the flow's series: with u = 2^-24 its rounding is below 33 u |v| dt (11 terms of
    N products each, their sum), 5 u (|A| |p| + |a|) e dt for the velocity and u |p|
    for the last addition; the first term left out is 2e-9 of the step;
  * the adjoint's quadrature: both series at the nodes, their products and four
    additions are below 90 u e^2 |lambda| (|p| + 1 + |v| dt) dt beside the 1.5e-7
    that the node count leaves.
|A| dt runs over all magnitudes, the switch between the short and the full series
at 0.06 among them.
"""
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import REPO

NVCC = shutil.which('nvcc') or '/usr/local/cuda/bin/nvcc'
U = 2.0 ** -24


@pytest.fixture(scope='module', params=['0.f', '2.384185791015625e-07f',
                                        '-2.384185791015625e-07f'])
def harness(tmp_path_factory, request):
    if not os.path.exists(NVCC):
        pytest.skip('nvcc not available')
    out = str(tmp_path_factory.mktemp('flow') / 'flow_check')
    subprocess.check_call([NVCC, '-O2', '-std=c++17', '-Xcompiler', '-ffp-contract=off',
                           '-DCPAB_FLOW_ERROR=' + request.param, '-o', out,
                           os.path.join(REPO, 'tests', 'flow_check.cu')])
    return out


def run(harness, tmp_path, nc, A, p, lam, time):
    n = len(nc)
    fin, fout = str(tmp_path / 'in.bin'), str(tmp_path / 'out.bin')
    with open(fin, 'wb') as f:
        f.write(np.array([n] + list(nc) + [1] * (3 - n), dtype=np.int32).tobytes())
        f.write(np.int64(len(p)).tobytes())
        for x in (A, p, lam, time):
            f.write(np.ascontiguousarray(x, dtype=np.float32).tobytes())
    subprocess.check_call([harness, fin, fout])
    r = np.fromfile(fout, dtype=np.float32).astype(np.float64).reshape(len(p), -1)
    cuts = np.cumsum([1, 1, 1, 1, n, n, n])
    step, norm, reach, dt, end, start, lam0, grad = np.split(r, cuts, axis=1)
    return step[:, 0], norm[:, 0], reach[:, 0], dt[:, 0], end, start, lam0, \
        grad.reshape(-1, n, n + 1)


def flow(M, a, p, t):
    """p(t) of p' = M p + a, 40 terms of the series (|M| t <= 1)."""
    term = t[:, None] * (np.einsum('irk,ik->ir', M, p) + a)
    x = p + term
    for k in range(2, 40):
        term = t[:, None] / k * np.einsum('irk,ik->ir', M, term)
        x = x + term
    return x


def norm2(x):
    return np.sqrt((x * x).sum(-1))


@pytest.mark.parametrize('scale', [0.01, 1.0, 30.0])
@pytest.mark.parametrize('nc', [[1], [2], [50], [1, 1], [3, 3], [8, 5], [1, 1, 1], [2, 2, 2],
                                [3, 4, 2]])
def test_substep(harness, tmp_path, nc, scale):
    n, m = len(nc), 1500
    rng = np.random.default_rng(17 * n + sum(nc))
    A = (scale * rng.standard_normal((m, n, n + 1))).astype(np.float32)
    # a quarter of the fields have a velocity that vanishes near the point, as next to
    # a fixed point
    p = rng.uniform(-0.1, 1.1, (m, n)).astype(np.float32)
    A[: m // 4, :, n] = -np.einsum('irk,ik->ir', A[: m // 4, :, :n], p[: m // 4])
    lam = rng.standard_normal((m, n)).astype(np.float32)
    time = np.where(rng.random(m) < 0.3, 1.0, 10.0 ** rng.uniform(-6, 0, m)).astype(np.float32)
    step, norm, reach, dt, end, start, lam0, grad = run(harness, tmp_path, nc, A, p, lam, time)
    assert (dt > 0).all() and (dt <= time).all()

    M, a = A[:, :, :n].astype(np.float64), A[:, :, n].astype(np.float64)
    p, lam = p.astype(np.float64), lam.astype(np.float64)
    speed, Mn = norm2(np.einsum('irk,ik->ir', M, p) + a), np.sqrt((M * M).sum((1, 2)))
    assert (Mn * dt <= 1 + 2.0 ** -20).all()
    # the velocity's own rounding may carry the point on
    vel = 5 * U * (Mn * norm2(p) + norm2(a))
    for f in (0.25, 0.5, 1.0):
        moved = np.maximum(norm2(flow(M, a, p, f * dt) - p), norm2(flow(M, a, p, -f * dt) - p))
        assert (moved <= reach * (1 + 2.0 ** -20) + np.e * vel * dt).all()

    forth, back = flow(M, a, p, dt), flow(M, a, p, -dt)
    tol = (33 * U + 2e-9) * np.e * speed * dt + np.e * vel * dt + U * (norm2(p) + speed * dt)
    assert (norm2(end - forth) <= tol).all()
    assert (norm2(start - back) <= tol).all()

    zero = np.zeros_like(lam)
    Mt = M.transpose(0, 2, 1)
    ltol = (40 * U + 2e-9) * np.e * norm2(lam)
    assert (norm2(lam0 - flow(Mt, zero, lam, dt)) <= ltol).all()
    want = np.zeros_like(grad)
    x, w = np.polynomial.legendre.leggauss(16)
    for xi, wi in zip(0.5 * (x + 1), 0.5 * w):
        h = np.concatenate([flow(M, a, p, -xi * dt), np.ones((m, 1))], axis=1)
        want += (wi * dt)[:, None, None] * flow(Mt, zero, lam, xi * dt)[:, :, None] * h[:, None]
    size = norm2(lam) * (norm2(p) + 1 + speed * dt + vel * dt) * dt
    assert (np.sqrt(((grad - want) ** 2).sum((1, 2))) <= (90 * U + 1.5e-7) * np.e ** 2 * size).all()
