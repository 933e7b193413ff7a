"""The torch extension is bound to one torch and Python: its file name says which,
the build makes it anew for another, and where it is missing or does not load the
Python classes take the calls, with one warning.
"""
import os
import warnings

import pytest
import torch


@pytest.fixture()
def unloaded(monkeypatch):
    """libcpab_gb300._native as before the first call."""
    from libcpab_gb300 import _native
    _native.load()
    monkeypatch.setattr(_native, '_bind', None)
    return _native


def test_built_for_this_torch():
    from libcpab_gb300 import _native, build
    assert torch.__version__ in os.path.basename(build.bind_path())
    assert os.path.exists(build.bind_path()) and _native.bind() is not None


@pytest.mark.parametrize('kind', ['missing', 'not a library'])
def test_without_extension(unloaded, monkeypatch, tmp_path, kind):
    from libcpab_gb300 import build, functions
    path = tmp_path / 'ext.so'
    if kind != 'missing':
        path.write_bytes(b'not a library')
    monkeypatch.setattr(build, 'bind_path', lambda: str(path))
    with pytest.warns(RuntimeWarning, match='torch extension'):
        assert unloaded.bind() is None
    with warnings.catch_warnings():
        warnings.simplefilter('error')
        assert unloaded.bind() is None

    # the calls reach the Python classes
    class Python:
        @staticmethod
        def apply(*args):
            return 'python'

    class Params:
        ndim, nc, numeric_grad, nstepsolver = 1, [3], False, 50
        domain_min, domain_max = [0.0], [1.0]

    for name in ('TransformGrid', 'TransformData'):
        monkeypatch.setattr(functions, name, Python)
    monkeypatch.setattr(functions, '_require_cuda', lambda *t: None)
    theta = torch.zeros(2, 4)
    assert functions.transformer(torch.zeros(1, 5), theta, Params()) == 'python'
    assert functions.transform_data(torch.zeros(2, 1, 5), theta, Params(), [5]) == 'python'


def test_another_torch_is_another_build(monkeypatch, tmp_path):
    from libcpab_gb300 import build
    before = build.bind_path()
    monkeypatch.setattr(build, 'HERE', str(tmp_path))
    monkeypatch.setattr(build, 'BUILD', str(tmp_path / 'obj'))
    made = []

    def compiled(src, obj):
        made.append(src)

    def linked(obj, path):
        made.append(path)
        open(path, 'w').close()

    def nvcc(*args):
        raise AssertionError('the C ABI library is up to date')

    monkeypatch.setattr(build, '_compile_bind', compiled)
    monkeypatch.setattr(build, '_link_bind', linked)
    monkeypatch.setattr(build, '_compile', nvcc)
    later = 2 * os.path.getmtime(build.__file__)
    lib = tmp_path / 'lib.so'
    lib.touch()
    os.utime(lib, (later, later))
    monkeypatch.setattr(build, 'LIB', str(lib))
    monkeypatch.setattr(torch, '__version__', '9.9.9+other')
    assert os.path.basename(build.bind_path()) != os.path.basename(before)
    build.build()
    assert [os.path.basename(m) for m in made] == ['torch_bind.cpp',
                                                   os.path.basename(build.bind_path())]
    build.build()
    assert len(made) == 2
