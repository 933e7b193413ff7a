"""Build the sm_103a shared library libcpab_gb300/libcpab_gb300.so and the
torch extension over it (_torch_bind: native autograd nodes).

The extension is bound to the torch and Python that it was compiled against, and
its file name carries both (bind_path): another torch finds no extension, never a
foreign one, and the next build makes its own.  Without torch the C ABI library is
built alone.

Each translation unit in csrc/ is compiled by nvcc in parallel
(-gencode arch=compute_103a,code=sm_103a) and linked into one shared library
whose exported symbols are the C ABI of include/cpab_gb300.h.  Objects go to
libcpab_gb300/_build/; both stay out of version control.

    python -m libcpab_gb300.build [-f] [-v]
"""
import concurrent.futures
import glob
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, 'csrc')
BUILD = os.path.join(HERE, '_build')
LIB = os.path.join(HERE, 'libcpab_gb300.so')
ARCH = ['-gencode', 'arch=compute_103a,code=sm_103a']


def nvcc_path():
    cand = [os.environ.get('NVCC'), shutil.which('nvcc'), '/usr/local/cuda/bin/nvcc']
    for c in cand:
        if c and os.path.exists(c):
            return c
    raise RuntimeError('nvcc not found')


def _compile(nvcc, src, obj, verbose):
    cmd = [nvcc, *ARCH, '-O3', '-lineinfo', '-std=c++17', '-Xcompiler', '-fPIC',
           '-Xcompiler', '-fvisibility=hidden', '-c', src, '-o', obj]
    if verbose:
        cmd.insert(1, '-Xptxas=-v')
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError('nvcc failed for %s:\n%s' % (src, r.stderr))
    return r.stderr


def bind_path():
    """File of the torch extension for the running Python and its torch."""
    import sysconfig
    import torch
    return os.path.join(HERE, '_torch_bind-torch%s-abi%d%s'
                        % (torch.__version__, int(torch._C._GLIBCXX_USE_CXX11_ABI),
                           sysconfig.get_config_var('EXT_SUFFIX')))


def _fresh(target, deps):
    if not os.path.exists(target):
        return False
    t = os.path.getmtime(target)
    return all(os.path.getmtime(d) <= t for d in deps if os.path.exists(d))


def _compile_bind(src, obj):
    """The native autograd nodes, against the installed torch (host code only)."""
    import sysconfig
    import torch
    root = os.path.join(os.path.dirname(torch.__file__), 'include')
    cuda = os.path.dirname(os.path.dirname(nvcc_path()))
    cmd = ['g++', '-O2', '-std=c++17', '-fPIC', '-fvisibility=hidden',
           '-D_GLIBCXX_USE_CXX11_ABI=%d' % int(torch._C._GLIBCXX_USE_CXX11_ABI)]
    for d in (root, os.path.join(root, 'torch', 'csrc', 'api', 'include'),
              sysconfig.get_paths()['include'], os.path.join(cuda, 'include')):
        cmd += ['-isystem', d]
    r = subprocess.run(cmd + ['-c', src, '-o', obj], capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError('g++ failed for %s:\n%s' % (src, r.stderr))


def _link_bind(obj, path):
    import torch
    lib = os.path.join(os.path.dirname(torch.__file__), 'lib')
    tmp = path + '.tmp%d' % os.getpid()
    # the C ABI library sits next to the extension and is found through $ORIGIN
    cmd = ['g++', '-shared', '-o', tmp, obj, '-L' + HERE, '-l:libcpab_gb300.so', '-L' + lib,
           '-ltorch_python', '-ltorch', '-ltorch_cpu', '-lc10', '-lc10_cuda',
           '-Wl,-rpath,$ORIGIN']
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError('link failed:\n' + r.stderr)
    os.replace(tmp, path)


def build(force=False, verbose=False):
    """Compile what is missing or older than its sources; returns the .so path of
    the C ABI."""
    srcs = sorted(glob.glob(os.path.join(CSRC, '*.cu')))
    bind_src = os.path.join(CSRC, 'torch_bind.cpp')
    header = os.path.join(os.path.dirname(HERE), 'include', 'cpab_gb300.h')
    deps = srcs + glob.glob(os.path.join(CSRC, '*.cuh')) + glob.glob(os.path.join(CSRC, '*.h')) + \
        [header, __file__]
    want_lib = force or not _fresh(LIB, deps)
    try:
        bind = bind_path()
    except ImportError:
        print('torch is not importable: building the C ABI library without the torch extension')
        bind = None
    want_bind = bind is not None and (force or not _fresh(bind, [bind_src, header, __file__]))
    os.makedirs(BUILD, exist_ok=True)
    objs = [os.path.join(BUILD, os.path.basename(s)[:-3] + '.o') for s in srcs]
    bind_obj = os.path.join(BUILD, 'torch_bind.o')
    with concurrent.futures.ThreadPoolExecutor(max_workers=min(9, len(srcs) + 1)) as ex:
        made = ex.submit(_compile_bind, bind_src, bind_obj) if want_bind else None
        if want_lib:
            nvcc = nvcc_path()
            logs = list(ex.map(lambda so: _compile(nvcc, so[0], so[1], verbose), zip(srcs, objs)))
            if verbose:
                for s, lg in zip(srcs, logs):
                    print('==', os.path.basename(s))
                    print(lg)
            tmp = LIB + '.tmp%d' % os.getpid()
            cmd = [nvcc, *ARCH, '-shared', '-o', tmp, *objs, '-lcudart']
            r = subprocess.run(cmd, capture_output=True, text=True)
            if r.returncode != 0:
                raise RuntimeError('link failed:\n' + r.stderr)
            os.replace(tmp, LIB)
        if made is not None:
            made.result()
            _link_bind(bind_obj, bind)
    return LIB


if __name__ == '__main__':
    print(build(force='-f' in sys.argv, verbose='-v' in sys.argv))
