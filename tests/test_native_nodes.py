"""The native autograd nodes (csrc/torch_bind.cpp) against the Python classes
they stand in for: the same bits forward and for dtheta, and the same answers
at the edges of autograd -- missing cotangents, create_graph, retained and freed
graphs, in-place changes of saved tensors, saved-tensor hooks, settings changed
between forward and backward -- and the calls they leave to the Python classes.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture()
def python_only(monkeypatch):
    """Run a function with the native nodes out of the way."""
    def run(f):
        from libcpab_gb300 import functions
        with monkeypatch.context() as m:
            m.setattr(functions, 'native', lambda *t: False)
            return f()
    return run


def make(cuda, tmp_path, nc=(3, 3), **solver):
    from libcpab_gb300 import Cpab
    T = Cpab(list(nc), backend='pytorch', device='gpu', basis_dir=str(tmp_path))
    if solver:
        T.set_solver_params(**solver)
    g = torch.Generator(device=cuda).manual_seed(5)
    theta = (0.4 * torch.randn(3, T.get_theta_dim(), generator=g, device=cuda)).requires_grad_(True)
    return T, theta, g


def grads(out, inputs, w):
    return torch.autograd.grad(out, inputs, w, allow_unused=True)


@pytest.mark.parametrize('solver', [{}, {'gradient': 'exact'}, {'gradient': 'reference_map'},
                                    {'integration': 'exact'}, {'nstepsolver': 7},
                                    {'point_gradient': True},
                                    {'point_gradient': True, 'integration': 'exact'}])
@pytest.mark.parametrize('nc', [(7,), (3, 3), (2, 2, 2)])
def test_transform_grid(cuda, tmp_path, python_only, nc, solver):
    T, theta, g = make(cuda, tmp_path, nc, **solver)
    for shape in ((len(nc), 50), (3, len(nc), 50)):
        pts = torch.rand(*shape, generator=g, device=cuda)
        w = torch.randn(3, len(nc), 50, generator=g, device=cuda)

        def run():
            p = pts.clone().requires_grad_(True)
            out = T.transform_grid(p, theta)
            return (out.detach(),) + grads(out, [theta, p], w)

        got = run()
        for a, b in zip(got, python_only(run)):
            assert (a is None) == (b is None)
            assert a is None or torch.equal(a, b)
        with torch.no_grad():
            assert torch.equal(T.transform_grid(pts, theta), got[0])


@pytest.mark.parametrize('gradient', ['reference', 'exact', 'reference_map'])
@pytest.mark.parametrize('nc,size,outsize', [((7,), (30,), (20,)), ((3, 3), (16, 12), (9, 11)),
                                             ((2, 2, 2), (6, 7, 8), (5, 6, 7))])
def test_transform_data(cuda, tmp_path, python_only, nc, size, outsize, gradient):
    T, theta, g = make(cuda, tmp_path, nc, gradient=gradient)
    data = torch.rand(3, 2, *size, generator=g, device=cuda)
    w = torch.randn(3, 2, *outsize, generator=g, device=cuda)
    for want in ('theta', 'data', 'both'):
        def run():
            d = data.clone().requires_grad_(want != 'theta')
            t = theta.detach().clone().requires_grad_(want != 'data')
            out = T.transform_data(d, t, list(outsize))
            return (out.detach(),) + grads(out, [x for x in (d, t) if x.requires_grad], w)

        for a, b in zip(run(), python_only(run)):
            assert a.dtype == b.dtype and (a - b).abs().max() <= 1e-5 * b.abs().max()
    # other types and layouts
    odd = data.double().transpose(-1, -2).contiguous().transpose(-1, -2) if len(nc) > 1 \
        else data.double()
    out = T.transform_data(odd.requires_grad_(True), theta, list(outsize))
    d, = torch.autograd.grad(out, [odd], w)
    assert d.dtype == torch.float64 and torch.equal(out, T.transform_data(data, theta,
                                                                          list(outsize)))


@pytest.mark.parametrize('gradient', ['reference', 'exact'])
def test_transform_data_mixed(cuda, tmp_path, python_only, gradient):
    T, theta, g = make(cuda, tmp_path, gradient=gradient)
    ims = [torch.rand(2, *s, generator=g, device=cuda) for s in ((9, 14), (20, 5), (7, 7))]
    w = [torch.randn(i.shape, generator=g, device=cuda) for i in ims]

    def run(used=(0, 1, 2)):
        leaves = [i.clone().requires_grad_(True) for i in ims]
        outs = T.transform_data_mixed(leaves, theta)
        return [o.detach() for o in outs], grads([outs[k] for k in used], [theta] + leaves,
                                                 [w[k] for k in used])

    for used in ((0, 1, 2), (1,)):
        a, b = run(used), python_only(lambda: run(used))
        assert all(torch.equal(x, y) for x, y in zip(a[0], b[0]))
        for x, y in zip(a[1], b[1]):
            y = torch.zeros_like(x) if y is None else y
            assert (x - y).abs().max() <= 1e-5 * max(1.0, float(y.abs().max()))


def test_autograd_edges(cuda, tmp_path):
    T, theta, g = make(cuda, tmp_path)
    pts = torch.rand(2, 40, generator=g, device=cuda)
    data = torch.rand(3, 1, 8, 8, generator=g, device=cuda)
    w = torch.randn(3, 2, 40, generator=g, device=cuda)
    # twice through a retained graph, an error through a freed one
    out = T.transform_grid(pts, theta)
    a, = torch.autograd.grad(out, [theta], w, retain_graph=True)
    b, = torch.autograd.grad(out, [theta], w)
    assert torch.equal(a, b)
    with pytest.raises(RuntimeError):
        torch.autograd.grad(out, [theta], w)
    # differentiable once
    wg = w.clone().requires_grad_(True)
    a, = torch.autograd.grad(T.transform_grid(pts, theta), [theta], wg, create_graph=True)
    with pytest.raises(RuntimeError, match='once_differentiable'):
        a.sum().backward()
    # theta may change in place before the backward, saved points may not
    t = theta.detach().clone().requires_grad_(True)
    out = T.transform_grid(pts, t)
    with torch.no_grad():
        t.add_(1.0)
    assert torch.equal(torch.autograd.grad(out, [t], w)[0], b)
    p = pts.clone()
    out = T.transform_grid(p, theta)
    p.add_(1.0)
    with pytest.raises(RuntimeError):
        torch.autograd.grad(out, [theta], w)
    # the settings that count are those at the time of the backward
    out = T.transform_grid(pts, theta)
    T.set_solver_params(gradient='exact')
    late, = torch.autograd.grad(out, [theta], w)
    now, = torch.autograd.grad(T.transform_grid(pts, theta), [theta], w)
    T.set_solver_params(gradient='reference')
    assert torch.equal(late, now) and not torch.equal(late, b)
    # saved-tensor hooks see the saved tensors
    seen = []
    with torch.autograd.graph.saved_tensors_hooks(lambda x: seen.append(x.shape) or x,
                                                  lambda x: x):
        out = T.transform_data(data.requires_grad_(True), theta, [8, 8])
    assert len(seen) >= 4
    out.sum().backward()
    # an output that only feeds the points of a later call: zeros for theta
    t1 = theta.detach().clone().requires_grad_(True)
    T.transform_grid(T.transform_grid(pts, t1), theta).sum().backward()
    assert t1.grad is not None and not t1.grad.any()


def test_left_to_the_python_classes(cuda, tmp_path):
    """functorch transforms, forward-mode AD and subclasses are refused or served
    as before; errors carry the C ABI's message."""
    from libcpab_gb300 import _native as N
    T, theta, g = make(cuda, tmp_path)
    pts = torch.rand(2, 40, generator=g, device=cuda)
    with pytest.raises(RuntimeError):
        torch.func.vmap(lambda t: T.transform_grid(pts, t[None]))(theta.detach())
    with pytest.raises(RuntimeError):
        torch.func.grad(lambda t: T.transform_grid(pts, t).sum())(theta.detach())
    with torch.autograd.forward_ad.dual_level():
        dual = torch.autograd.forward_ad.make_dual(theta.detach(), torch.ones_like(theta))
        with pytest.raises(RuntimeError):
            T.transform_grid(pts, dual)

    class Sub(torch.Tensor):
        pass

    out = T.transform_grid(pts.as_subclass(Sub), theta)
    assert torch.equal(torch.as_tensor(out).as_subclass(torch.Tensor),
                       T.transform_grid(pts, theta))
    with pytest.raises(N.CpabError):
        T.transform_grid(pts, theta.detach().repeat(30000, 1))
