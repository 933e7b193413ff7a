"""The exact flow's gradient on a 1D tessellation of one cell: the flow is affine,
x(1) = e^a x + b (e^a - 1) / a, and no face bounds a sub-step, so that |a| times the
whole time may be well above 1.  Against 64-bit autograd of the closed form; the
backward integrates back from a 32-bit result, which costs e^|a| roundings of it
(55 * 2^-24 at |a| = 4), beside some 100 roundings of its own: 2e-5.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('a', [-4.0, -2.5, -0.3, 1.0, 2.5, 4.0])
@pytest.mark.parametrize('nP', [1, 33, 500])
def test_affine_flow(cuda, a, nP):
    from libcpab_gb300 import _native as N
    g = torch.Generator(device=cuda).manual_seed(nP)
    theta = torch.tensor([[a, 0.7]], device=cuda)
    pts = torch.rand(1, nP, generator=g, device=cuda)
    gout = torch.rand(1, 1, nP, generator=g, device=cuda) + 0.5
    basis = torch.eye(2, device=cuda)
    A, _, _ = N.cell_tables([1], 50, theta, basis)
    out = N.integrate_exact([1], pts, A)
    dtheta, dpoints = N.backward_exact([1], out, A, basis, gout, want_dpoints=True)
    t64 = theta.double().requires_grad_(True)
    p64 = pts.double().requires_grad_(True)
    ea = torch.exp(t64[0, 0])
    flow = ea * p64 + t64[0, 1] * (ea - 1) / t64[0, 0]
    assert (out.double() - flow).abs().max() <= 1e-6 * flow.abs().max()
    want, wantp = torch.autograd.grad((flow * gout[0].double()).sum(), [t64, p64])
    assert (dtheta.double() - want).abs().max() <= 2e-5 * want.abs().max()
    assert (dpoints.double() - wantp).abs().max() <= 2e-5 * wantp.abs().max()
