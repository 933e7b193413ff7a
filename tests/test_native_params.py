"""What a native node holds of the transformer: its params go with the last node and
transformer (they own the basis, meshgrid axes and image layouts on the GPU).
"""
import gc
import time
import weakref

import pytest
import torch


class Params:
    pass


def test_refused_call_keeps_nothing():
    """A basis of another tessellation is refused on the host, before any launch."""
    from libcpab_gb300 import _native as N
    theta = torch.zeros(2, 3, requires_grad=True)
    p = Params()
    alive = weakref.ref(p)
    settings = (50, 0, False, None, torch.zeros(5, 3))
    assert N.bind().transform_grid(torch.zeros(1, 4), theta, p, [3], settings, False) is None
    del p
    gc.collect()
    assert alive() is None


@pytest.mark.gpu
@pytest.mark.parametrize('backward', [False, True])
@pytest.mark.parametrize('which', ['grid', 'data', 'mixed'])
def test_params_are_released(cuda, tmp_path, which, backward):
    from libcpab_gb300 import Cpab
    T = Cpab([3, 3], backend='pytorch', device='gpu', basis_dir=str(tmp_path))
    theta = torch.zeros(2, T.get_theta_dim(), device=cuda, requires_grad=True)
    data = torch.rand(2, 1, 8, 8, device=cuda)
    out = {'grid': lambda: T.transform_grid(torch.rand(2, 9, device=cuda), theta),
           'data': lambda: T.transform_data(data, theta, [8, 8]),
           'mixed': lambda: T.transform_data_mixed(list(data), theta)[0]}[which]()
    if backward:
        out.sum().backward()
    alive = weakref.ref(T.params)
    del T, out
    gc.collect()
    deadline = time.time() + 5.0      # a node that died on the engine's thread hands its
    while alive() is not None and time.time() < deadline:     # reference to this one
        time.sleep(0.01)
    assert alive() is None
