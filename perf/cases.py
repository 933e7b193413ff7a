"""Workloads for timing this library and checking its results.

Each case is one call (or one forward and backward) through the public API of
``libcpab_gb300.Cpab``, as a training, registration or augmentation program
makes it.  ``listed`` names the standard ones, ``draw`` gives others of the
same ranges, ``prepare`` builds what a program holds before the call (inputs
and the transformer object), ``run`` makes the call, ``work`` counts the bytes
and operations that it cannot do without, and ``exact`` restates the result in
64-bit floating point with plain torch.
"""
import math

import torch

from libcpab_gb300 import Cpab

NSTEPS = 50

# The tessellations in use, by the names the cases carry:
# (cells per axis, zero_boundary, volume_perservation).
TESSELLATIONS = {
    '1d_50_zb': ([50], True, False),
    '1d_100_free': ([100], False, False),
    '2d_3x3_zb': ([3, 3], True, False),
    '2d_4x4_free': ([4, 4], False, False),
    '2d_8x8_free': ([8, 8], False, False),
    '3d_2x2x2_zb_vp': ([2, 2, 2], True, True),
    '3d_4x4x4_zb_vp': ([4, 4, 4], True, True),
}


def listed():
    return [
        # a handful of short signals warped once: the smallest call
        {'name': 'signals_small', 'kind': 'grid', 'tess': '1d_50_zb', 'batch': 16,
         'outsize': '1000', 'std': 1.0, 'grad': False},
        # one iteration of registering one image to another (d(theta) only)
        {'name': 'register_image', 'kind': 'image', 'tess': '2d_3x3_zb', 'batch': 1,
         'channels': 3, 'size': '224x224', 'outsize': '224x224', 'std': 0.5,
         'grad': 'theta', 'gradient': 'reference'},
        # data augmentation of one training batch (no gradient)
        {'name': 'augment_images', 'kind': 'image', 'tess': '2d_3x3_zb', 'batch': 64,
         'channels': 3, 'size': '224x224', 'outsize': '224x224', 'std': 0.5,
         'grad': 'none', 'gradient': 'reference'},
        # a transformer layer inside a network: d(theta) and d(images)
        {'name': 'train_images', 'kind': 'image', 'tess': '2d_3x3_zb', 'batch': 64,
         'channels': 3, 'size': '224x224', 'outsize': '224x224', 'std': 0.5,
         'grad': 'both', 'gradient': 'reference'},
        # the same with odd sizes, a free boundary, one channel and the exact
        # derivative of the forward map
        {'name': 'train_images_odd', 'kind': 'image', 'tess': '2d_4x4_free', 'batch': 13,
         'channels': 1, 'size': '179x241', 'outsize': '151x203', 'std': 0.5,
         'grad': 'both', 'gradient': 'exact'},
        # strong deformations on a fine tessellation: many cell crossings
        {'name': 'fine_tessellation_grid', 'kind': 'grid', 'tess': '2d_8x8_free', 'batch': 64,
         'outsize': '512x512', 'std': 3.0, 'grad': True},
        # volume registration / training
        {'name': 'train_volumes', 'kind': 'image', 'tess': '3d_4x4x4_zb_vp', 'batch': 8,
         'channels': 1, 'size': '128x128x128', 'outsize': '128x128x128', 'std': 1.0,
         'grad': 'both', 'gradient': 'reference'},
        # resampling images at a given grid, with both gradients
        {'name': 'resample_images', 'kind': 'interp', 'batch': 256, 'channels': 3,
         'size': '224x224', 'outsize': '224x224'},
        # time-series alignment: many series of uneven lengths, fused loss
        {'name': 'align_series', 'kind': 'series', 'tess': '1d_100_free', 'sets': 4096,
         'low': 16, 'high': 4096, 'std': 1.0},
        # point clouds of uneven sizes, d(theta)
        {'name': 'point_sets', 'kind': 'points', 'tess': '2d_3x3_zb', 'sets': 1024,
         'low': 256, 'high': 16384, 'std': 0.5},
        # a batch of images of mixed sizes, d(theta) and d(images)
        {'name': 'mixed_images', 'kind': 'mixed', 'tess': '2d_3x3_zb', 'sets': 24,
         'channels': 3, 'low': 128, 'high': 320, 'std': 0.5},
        # the true flow of the field instead of the fixed-step scheme
        {'name': 'exact_flow_grid', 'kind': 'flow', 'tess': '2d_3x3_zb', 'batch': 64,
         'outsize': '224x224', 'std': 0.5},
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(['grid1', 'grid2', 'image2', 'image2', 'image3', 'interp', 'series',
                       'points', 'mixed', 'flow'])
    if kind == 'grid1':
        return {'kind': 'grid', 'tess': rng.choice(['1d_50_zb', '1d_100_free']),
                'batch': _log_int(rng, 1, 512), 'outsize': str(_log_int(rng, 100, 16384)),
                'std': 1.0, 'grad': rng.random() < 0.7}
    if kind == 'grid2':
        side = [_log_int(rng, 32, 512) for _ in range(2)]
        return {'kind': 'grid', 'tess': rng.choice(['2d_3x3_zb', '2d_8x8_free']),
                'batch': _log_int(rng, 1, 64), 'outsize': '%dx%d' % tuple(side),
                'std': rng.choice([0.5, 3.0]), 'grad': rng.random() < 0.7}
    if kind == 'image2':
        side = [_log_int(rng, 32, 320) for _ in range(4)]
        return {'kind': 'image', 'tess': rng.choice(['2d_3x3_zb', '2d_4x4_free']),
                'batch': _log_int(rng, 1, 64), 'channels': rng.choice([1, 3]),
                'size': '%dx%d' % (side[0], side[1]), 'outsize': '%dx%d' % (side[2], side[3]),
                'std': 0.5, 'grad': rng.choice(['none', 'theta', 'both', 'both']),
                'gradient': rng.choice(['reference', 'reference', 'exact'])}
    if kind == 'image3':
        side = [_log_int(rng, 24, 128) for _ in range(3)]
        text = '%dx%dx%d' % tuple(side)
        return {'kind': 'image', 'tess': rng.choice(['3d_2x2x2_zb_vp', '3d_4x4x4_zb_vp']),
                'batch': _log_int(rng, 1, 8), 'channels': 1, 'size': text, 'outsize': text,
                'std': 1.0, 'grad': rng.choice(['none', 'both']), 'gradient': 'reference'}
    if kind == 'interp':
        side = [_log_int(rng, 32, 320) for _ in range(4)]
        return {'kind': 'interp', 'batch': _log_int(rng, 1, 128), 'channels': rng.choice([1, 3]),
                'size': '%dx%d' % (side[0], side[1]), 'outsize': '%dx%d' % (side[2], side[3])}
    if kind == 'series':
        return {'kind': 'series', 'tess': rng.choice(['1d_50_zb', '1d_100_free']),
                'sets': _log_int(rng, 32, 4096), 'low': 16, 'high': _log_int(rng, 64, 4096),
                'std': 1.0}
    if kind == 'points':
        return {'kind': 'points', 'tess': rng.choice(['2d_3x3_zb', '2d_4x4_free']),
                'sets': _log_int(rng, 8, 1024), 'low': 32, 'high': _log_int(rng, 256, 16384),
                'std': 0.5}
    if kind == 'mixed':
        return {'kind': 'mixed', 'tess': '2d_3x3_zb', 'sets': _log_int(rng, 2, 24),
                'channels': rng.choice([1, 3]), 'low': 48, 'high': _log_int(rng, 96, 320),
                'std': 0.5}
    side = [_log_int(rng, 32, 224) for _ in range(2)]
    return {'kind': 'flow', 'tess': '2d_3x3_zb', 'batch': _log_int(rng, 1, 64),
            'outsize': '%dx%d' % tuple(side), 'std': 0.5}


# --------------------------------- inputs ------------------------------------
def _size(text):
    return [int(x) for x in text.split('x')]


def _generator(seed, device='cuda'):
    return torch.Generator(device=device).manual_seed(seed)


def _transformer(case):
    nc, zero_boundary, volume = TESSELLATIONS[case['tess']]
    return Cpab(nc, backend='pytorch', device='gpu', zero_boundary=zero_boundary,
                volume_perservation=volume)


def _theta(T, n, case, gen):
    return case['std'] * torch.randn(n, T.get_theta_dim(), generator=gen, device='cuda')


def _images(n, channels, size, gen):
    """Box-filtered noise in 2D; in 3D the same (smooth, no flat regions)."""
    raw = torch.rand(n, channels, *size, generator=gen, device='cuda')
    pool = torch.nn.functional.avg_pool2d if len(size) == 2 else torch.nn.functional.avg_pool3d
    return pool(raw, kernel_size=5, stride=1, padding=2, count_include_pad=False).contiguous()


def _lengths(case, k=0):
    """Sizes of the sets: uneven, and the same for every seed of one case."""
    return torch.randint(case['low'], case['high'] + 1, (case['sets'],),
                         generator=_generator(1000 * k + case['sets'], 'cpu'))


def _offsets(lengths):
    return torch.cat([torch.zeros(1, dtype=torch.int64), torch.cumsum(lengths, 0)]).cuda()


def _smooth_warp(n, outsize, gen):
    """Meshgrids moved by a few smooth waves, some points outside [0, 1]."""
    mesh = torch.meshgrid(*[torch.linspace(0, 1, o, device='cuda') for o in outsize[::-1]],
                          indexing='ij')
    x, y = mesh[1].reshape(1, -1), mesh[0].reshape(1, -1)
    amp = 0.05 * torch.randn(n, 4, 1, generator=gen, device='cuda')
    gx = x + amp[:, 0] * torch.sin(6.0 * y) + amp[:, 1] * torch.cos(5.0 * x)
    gy = y + amp[:, 2] * torch.sin(4.0 * x) + amp[:, 3] * torch.cos(7.0 * y)
    return torch.stack([gx, gy], dim=1).contiguous()


def prepare(case, seed):
    gen = _generator(seed)
    randn = lambda *s: torch.randn(*s, generator=gen, device='cuda')
    kind = case['kind']
    st = {'case': case}
    if kind == 'interp':
        size, outsize = _size(case['size']), _size(case['outsize'])
        st['data'] = _images(case['batch'], case['channels'], size, gen).requires_grad_(True)
        st['grid'] = _smooth_warp(case['batch'], outsize, gen).requires_grad_(True)
        st['weight'] = randn(case['batch'], case['channels'], *outsize)
        st['outsize'] = outsize
        st['T'] = _transformer({'tess': '2d_3x3_zb'})
        return st
    T = st['T'] = _transformer(case)
    if kind in ('grid', 'flow'):
        outsize = _size(case['outsize'])
        st['theta'] = _theta(T, case['batch'], case, gen)
        st['grid'] = T.uniform_meshgrid(outsize)
        if kind == 'flow':
            T.set_solver_params(integration='exact')
        if kind == 'flow' or case['grad']:
            st['theta'].requires_grad_(True)
            st['weight'] = randn(case['batch'], *st['grid'].shape)
    elif kind == 'image':
        size, outsize = _size(case['size']), _size(case['outsize'])
        T.set_solver_params(gradient=case['gradient'])
        st['outsize'] = outsize
        st['theta'] = _theta(T, case['batch'], case, gen)
        st['data'] = _images(case['batch'], case['channels'], size, gen)
        if case['grad'] != 'none':
            st['theta'].requires_grad_(True)
            st['data'].requires_grad_(case['grad'] == 'both')
            st['weight'] = randn(case['batch'], case['channels'], *outsize)
    elif kind == 'series':
        lengths = _lengths(case)
        total = int(lengths.sum())
        st['offsets'] = _offsets(lengths)
        sid = torch.repeat_interleave(torch.arange(case['sets']), lengths).cuda()
        x = (torch.arange(total, device='cuda') - st['offsets'][sid]) \
            / (lengths.cuda()[sid] - 1).clamp(min=1)
        wave = torch.zeros(total, device='cuda')
        for _ in range(3):
            f = 1 + 9 * torch.rand(case['sets'], generator=gen, device='cuda')
            phase = 2 * math.pi * torch.rand(case['sets'], generator=gen, device='cuda')
            wave += torch.sin(2 * math.pi * f[sid] * x + phase[sid])
        st['values'] = wave + 0.1 * randn(total)
        st['target'] = wave.roll(3) + 0.1 * randn(total)
        st['theta'] = _theta(T, case['sets'], case, gen)
    elif kind == 'points':
        st['offsets'] = _offsets(_lengths(case))
        total = int(st['offsets'][-1])
        st['points'] = torch.rand(2, total, generator=gen, device='cuda')
        st['theta'] = _theta(T, case['sets'], case, gen).requires_grad_(True)
        st['weight'] = randn(2, total)
    else:
        sides = torch.stack([_lengths(case, 1), _lengths(case, 2)], 1).tolist()
        st['images'] = [_images(1, case['channels'], s, gen)[0].requires_grad_(True)
                        for s in sides]
        st['weights'] = [randn(case['channels'], *s) for s in sides]
        st['theta'] = _theta(T, case['sets'], case, gen).requires_grad_(True)
    return st


# ----------------------------------- run -------------------------------------
def run(st):
    case, T = st['case'], st['T']
    kind = case['kind']
    if kind in ('grid', 'flow'):
        out = T.transform_grid(st['grid'], st['theta'])
        if 'weight' not in st:
            return {'out': out}
        dtheta, = torch.autograd.grad(out, [st['theta']], st['weight'])
        return {'out': out.detach(), 'dtheta': dtheta}
    if kind == 'image':
        out = T.transform_data(st['data'], st['theta'], st['outsize'])
        if case['grad'] == 'none':
            return {'out': out}
        if case['grad'] == 'theta':
            dtheta, = torch.autograd.grad(out, [st['theta']], st['weight'])
            return {'out': out.detach(), 'dtheta': dtheta}
        dtheta, ddata = torch.autograd.grad(out, [st['theta'], st['data']], st['weight'])
        return {'out': out.detach(), 'dtheta': dtheta, 'ddata': ddata}
    if kind == 'interp':
        out = T.interpolate(st['data'], st['grid'], st['outsize'])
        ddata, dgrid = torch.autograd.grad(out, [st['data'], st['grid']], st['weight'])
        return {'out': out.detach(), 'ddata': ddata, 'dgrid': dgrid}
    if kind == 'series':
        res = T.ragged_mse(st['values'], st['target'], st['offsets'], st['theta'])
        return {k: res[k] for k in ('loss', 'sse', 'dtheta', 'dvalues')}
    if kind == 'points':
        out = T.transform_grid_ragged(st['points'], st['offsets'], st['theta'])
        dtheta, = torch.autograd.grad(out, [st['theta']], st['weight'])
        return {'out': out.detach(), 'dtheta': dtheta}
    outs = T.transform_data_mixed(st['images'], st['theta'])
    grads = torch.autograd.grad(outs, [st['theta']] + st['images'], st['weights'])
    return {'out': [o.detach() for o in outs], 'dtheta': grads[0], 'dimages': list(grads[1:])}


# ---------------------------------- work -------------------------------------
def _count(size):
    return math.prod(size)


def work(case):
    """Operations: per point and step one affine map (forward), and per step of
    a gradient that map again, one outer product and one transposed map; the
    true flow counts as ten in-cell steps.  Bytes: every input read once and
    every output written once, in 32-bit floats."""
    kind = case['kind']
    if kind == 'interp':
        out, data = _count(_size(case['outsize'])), _count(_size(case['size']))
        n, C = case['batch'], case['channels']
        return {'bytes': 4 * n * (2 * C * data + 2 * C * out + 4 * out),
                'flops': n * out * (12 + C * (9 + 8 + 12))}
    ndim = len(TESSELLATIONS[case['tess']][0])
    forward = {1: 5, 2: 17, 3: 37}[ndim]
    backward = forward + 2 * ndim * (ndim + 1) + 2 * ndim * ndim + forward
    steps = 10 if kind == 'flow' else NSTEPS
    if kind in ('grid', 'flow'):
        points = case['batch'] * _count(_size(case['outsize']))
        grad = kind == 'flow' or case['grad']
        return {'bytes': 4 * ndim * (points * (2 if grad else 1) + points // case['batch']),
                'flops': points * steps * (forward + (backward if grad else 0))}
    if kind == 'image':
        points = case['batch'] * _count(_size(case['outsize']))
        pixels = case['batch'] * _count(_size(case['size']))
        C = case['channels']
        values = C * (points + pixels)
        if case['grad'] != 'none':
            values += C * points + (C * pixels if case['grad'] == 'both' else 0)
        return {'bytes': 4 * values,
                'flops': points * (steps * (forward + (backward if case['grad'] != 'none' else 0))
                                   + 10 * C)}
    mean = (case['low'] + case['high']) / 2
    if kind == 'series':
        points = int(case['sets'] * mean)
        return {'bytes': 4 * 3 * points, 'flops': points * steps * (forward + backward)}
    if kind == 'points':
        points = int(case['sets'] * mean)
        return {'bytes': 4 * 6 * points, 'flops': points * steps * (forward + backward)}
    points = int(case['sets'] * mean * mean)
    return {'bytes': 4 * 4 * case['channels'] * points,
            'flops': points * steps * (forward + backward)}


# ---------------------------------- exact ------------------------------------
# The scheme in 64 bits.  Points are flat, p [P, n] with sid [P] the row of
# theta that moves each; tables are [rows * nC, n, n + 1].
def _cells(p, nc):
    """Cell of each point: the reference's rules (unit domain, cells of float
    width 1/nc, four triangles per square, five tetrahedra per cube)."""
    n = len(nc)
    inc = torch.tensor([1.0 / c for c in nc], dtype=torch.float32, device=p.device).double()
    if n == 1:
        return (p[:, 0] * nc[0]).floor().clamp(0, nc[0] - 1).long()
    if n == 2:
        u = p / inc
        top = torch.tensor([c - 1 for c in nc], dtype=torch.float64, device=p.device)
        sq = torch.minimum(u.floor().clamp(min=0), top)
        x, y = (u - sq).unbind(1)
        tri = (x + y > 1).long() ^ torch.where(x < y, 3, 0)
        return 4 * (sq[:, 0] + nc[0] * sq[:, 1]).long() + tri
    inside = ((p[:, :2] >= 0) & (p[:, :2] <= 1)).all(1, keepdim=True)
    q = p - 0.5
    a = q.abs()
    smallest = (a < a.roll(1, 1)) & (a < a.roll(2, 1))
    q = torch.where(a > 0.5, torch.copysign(0.5 - smallest * 0.5 * inc, q), q)
    limit = torch.tensor([float(nc[0] * inc[0]), float(nc[1] * inc[1]), float(nc[2] * inc[0])],
                         dtype=torch.float32, device=p.device).double()
    q = torch.minimum(torch.where(inside, p, q + 0.5).clamp(min=0), limit)
    top = torch.tensor([c - 1 for c in nc], dtype=torch.float64, device=p.device)
    whole = (q / inc).floor()
    x, y, z = (q / inc - whole).unbind(1)
    i, j, k = torch.minimum(whole, top).long().unbind(1)
    odd = (i + j + k) % 2 == 1
    x, y = torch.where(odd, y, x), torch.where(odd, 1 - x, y)
    sub = torch.where(z - x - y >= 0, 1, torch.where(
        x + y + z >= 2, 2, torch.where(y - x - z >= 0, 3, torch.where(x - y - z >= 0, 4, 0))))
    return 5 * (i + nc[0] * (j + nc[1] * k)) + sub


def _basis(T, device):
    return torch.as_tensor(T.get_basis(), dtype=torch.float64, device=device)


def _fields(T, theta):
    """Velocity maps A [rows, nC, n, n + 1]."""
    n = T.params.ndim
    return (theta.double() @ _basis(T, theta.device).t()).reshape(
        theta.shape[0], T.params.nC, n, n + 1)


def _exponential(A, t):
    """The top rows of expm(t [A; 0]), by its series on t A / 64, squared six
    times."""
    n = A.shape[-2]
    eye = torch.eye(n + 1, dtype=A.dtype, device=A.device)
    X = torch.cat([A * (t / 64), torch.zeros_like(A[..., :1, :])], -2)
    multiply = lambda P, Q: (P[..., :, :, None] * Q[..., None, :, :]).sum(-2)
    R = eye + X / 12
    for k in range(11, 0, -1):
        R = eye + multiply(X, R) / k
    for _ in range(6):
        R = multiply(R, R)
    return R[..., :n, :]


def _apply(M, p):
    return (M[..., :-1] * p[:, None, :]).sum(2) + M[..., -1]


def _transposed(M, v):
    """M_lin^T v."""
    return (M[..., :-1] * v[:, :, None]).sum(1)


def _integrate(nc, A, p, sid, log=None):
    nC = A.shape[1]
    T = _exponential(A, 1.0 / NSTEPS).flatten(0, 1)
    for _ in range(NSTEPS):
        c = sid * nC + _cells(p, nc)
        if log is not None:
            log.append((p, c))
        p = _apply(T[c], p)
    return p


def _add_rows(total, index, rows):
    """total[index] += rows, spread over copies of total to keep the additions
    to one address apart."""
    copies = 64
    wide = torch.zeros(total.shape[0] * copies, rows.shape[1], dtype=rows.dtype,
                       device=rows.device)
    lane = torch.arange(index.shape[0], device=index.device) % copies
    wide.index_add_(0, index * copies + lane, rows)
    total += wide.reshape(total.shape[0], copies, -1).sum(1)


def _one(p):
    return torch.cat([p, torch.ones_like(p[:, :1])], 1)


def _theta_gradient(T, A, p, sid, lam, gradient='reference'):
    """d(theta) of sum(lam * flow(p)): the midpoint-rule sensitivity along the
    midpoint trajectory ('reference') or the derivative of the step maps."""
    nc, nC, n = T.params.nc, A.shape[1], A.shape[2]
    total = torch.zeros(A.shape[0] * nC, n * (n + 1), dtype=A.dtype, device=A.device)
    h = 1.0 / NSTEPS
    if gradient == 'exact':
        leaf = A.detach().requires_grad_(True)
        with torch.enable_grad():
            maps = _exponential(leaf, h).flatten(0, 1)
        log = []
        _integrate(nc, A, p, sid, log)
        for q, c in reversed(log):
            _add_rows(total, c, (lam[:, :, None] * _one(q)[:, None, :]).flatten(1))
            lam = _transposed(maps.detach()[c], lam)
        dA, = torch.autograd.grad(maps, [leaf], total.reshape(maps.shape))
    else:
        flat, log = A.flatten(0, 1), []
        for _ in range(NSTEPS):
            c = sid * nC + _cells(p, nc)
            log.append((p, c))
            M = flat[c]
            p = p + h * _apply(M, p + 0.5 * h * _apply(M, p))
        for q, c in reversed(log):
            M = flat[c]
            middle = q + 0.5 * h * _apply(M, q)
            back = _transposed(M, lam)
            _add_rows(total, c, (h * lam[:, :, None] * _one(middle)[:, None, :]
                                 + 0.5 * h * h * back[:, :, None] * _one(q)[:, None, :]
                                 ).flatten(1))
            lam = lam + h * back + 0.5 * h * h * _transposed(M, back)
        dA = total
    return dA.reshape(A.shape[0], -1) @ _basis(T, A.device)


def _mesh(outsize, device):
    """[P, n] grid points, the first axis varying fastest."""
    axes = [torch.linspace(0, 1, o, dtype=torch.float64, device=device) for o in outsize]
    mesh = torch.meshgrid(*axes[::-1], indexing='ij')
    return torch.stack([m.reshape(-1) for m in mesh[::-1]], 1)


def _sample(data, p, outsize):
    """data [b, C, *size] at p [b, P, n] (meshgrid order): linear interpolation
    with the corners clamped to the image, [b, C, *outsize]."""
    b, C, size = data.shape[0], data.shape[1], data.shape[2:]
    n = len(size)
    last = torch.tensor([s - 1 for s in size], dtype=torch.float64, device=p.device)
    x = p * last
    low = torch.minimum(x.detach().floor().clamp(min=0), last)
    high = torch.minimum((x.detach().floor() + 1).clamp(min=0), last)
    f = x - low
    flat = data.reshape(b, C, -1)
    out = 0
    for corner in range(1 << n):
        index, weight = 0, 1
        for j in range(n):
            up = (corner >> j) & 1
            index = index * size[j] + (high if up else low)[..., j].long()
            weight = weight * (f[..., j] if up else 1 - f[..., j])
        out = out + weight[:, None] * flat.gather(2, index[:, None].expand(b, C, -1))
    axes = [0, 1] + [n + 1 - j for j in range(n)]
    return out.reshape(b, C, *outsize[::-1]).permute(*axes)


def _exact_image(T, case, data, theta, weight, outsize):
    """out, d(theta), d(data), one image at a time."""
    A = _fields(T, theta)
    outs, dthetas, ddatas = [], [], []
    for k in range(data.shape[0]):
        p0 = _mesh(outsize, data.device)
        sid = torch.zeros(p0.shape[0], dtype=torch.long, device=data.device)
        p = _integrate(T.params.nc, A[k:k + 1], p0, sid)
        if weight is None:
            outs.append(_sample(data[k:k + 1].double(), p[None], outsize))
            continue
        with torch.enable_grad():
            image = data[k:k + 1].detach().double().requires_grad_(True)
            grid = p[None].detach().requires_grad_(True)
            out = _sample(image, grid, outsize)
            ddata, lam = torch.autograd.grad(out, [image, grid], weight[k:k + 1].double())
        outs.append(out.detach())
        ddatas.append(ddata)
        dthetas.append(_theta_gradient(T, A[k:k + 1], p0, sid, lam[0], case['gradient']))
    return torch.cat(outs), torch.cat(dthetas) if dthetas else None, \
        torch.cat(ddatas) if ddatas else None


def _true_flow(nc, A, p, sid, lam=None):
    """The flow of the field for time 1: steps of the in-cell exponential, cut
    by bisection where a point leaves its cell (never below 1e-4, over which
    the fields of two neighbouring cells differ by 1e-8).  With lam, A is the
    field reversed in time and p the end points: the sweep goes back to the
    start and returns dL/dA, the integral of lam(t) [p(t); 1]^T over the time
    spent in each cell (Gauss-Legendre, three nodes a step)."""
    nC, n = A.shape[1], A.shape[2]
    flat = A.flatten(0, 1)
    total = torch.zeros(A.shape[0] * nC, n * (n + 1), dtype=A.dtype, device=A.device)
    left = torch.ones_like(p[:, 0])
    p = p.clone()
    todo = torch.arange(p.shape[0], device=p.device)
    nodes = [(0.5 - math.sqrt(0.15), 5 / 18), (0.5, 8 / 18), (0.5 + math.sqrt(0.15), 5 / 18)]
    while todo.numel():
        q, s = p[todo], sid[todo]
        own = _cells(q, nc)
        M = flat[s * nC + own]
        norm = M[..., :-1].flatten(1).norm(dim=1)
        dt = torch.minimum(left[todo], 0.2 / norm.clamp(min=0.2))
        end = _step(M, dt, q)
        other = _cells(end, nc)
        # a cell left by so little that the two fields agree is not left
        gap = _apply(flat[s * nC + other] - M, end).norm(dim=1) * dt
        out = ((other != own) & (gap > 1e-11)).nonzero()[:, 0]
        if out.numel():
            Mo, qo, co = M[out], q[out], own[out]
            low, high = torch.zeros_like(dt[out]), dt[out]
            for _ in range(40):
                mid = 0.5 * (low + high)
                past = _cells(_step(Mo, mid, qo), nc) != co
                low, high = torch.where(past, low, mid), torch.where(past, mid, high)
            dt[out] = torch.minimum(high.clamp(min=1e-4), dt[out])
        if lam is not None:
            mu, rows = lam[todo], 0
            for node, weight in nodes:
                rows = rows + (weight * dt)[:, None, None] * (
                    _carry(M, node * dt, mu)[:, :, None]
                    * _one(_step(M, node * dt, q))[:, None, :])
            _add_rows(total, s * nC + own, rows.flatten(1))
            lam[todo] = _carry(M, dt, mu)
        p[todo] = _step(M, dt, q)
        left[todo] -= dt
        todo = todo[left[todo] > 1e-15]
    return p if lam is None else total


def _step(M, dt, p):
    """expm(dt M~) [p; 1] for small dt |M|, by its series."""
    term = _apply(M, p) * dt[:, None]
    out = p + term
    for k in range(2, 13):
        term = (M[..., :-1] * term[:, None, :]).sum(2) * (dt / k)[:, None]
        out = out + term
    return out


def _carry(M, dt, mu):
    """The cotangent carried back over dt of the forward field -M:
    mu <- expm(dt (-M_lin)^T) mu."""
    term, out = mu, mu
    for k in range(1, 13):
        term = _transposed(M, term) * (-dt / k)[:, None]
        out = out + term
    return out


def _linspace_series(offsets):
    lengths = offsets[1:] - offsets[:-1]
    sid = torch.repeat_interleave(torch.arange(lengths.numel(), device=offsets.device), lengths)
    place = torch.arange(int(offsets[-1]), device=offsets.device) - offsets[sid]
    return sid, place, lengths


def _exact_series(T, st):
    offsets, values, target = st['offsets'], st['values'].double(), st['target'].double()
    sid, place, lengths = _linspace_series(offsets)
    last = (lengths - 1).double()[sid]
    p0 = (place / last.clamp(min=1))[:, None]
    A = _fields(T, st['theta'])
    p = _integrate(T.params.nc, A, p0, sid)[:, 0]
    x = p * last
    low = torch.minimum(x.floor().clamp(min=0), last)
    high = torch.minimum((x.floor() + 1).clamp(min=0), last)
    f = x - low
    i0, i1 = offsets[sid] + low.long(), offsets[sid] + high.long()
    r = values[i0] * (1 - f) + values[i1] * f - target
    sse = torch.zeros(lengths.numel(), dtype=torch.float64, device=x.device).index_add_(0, sid, r * r)
    g = 2.0 / values.numel() * r
    dvalues = torch.zeros_like(values).index_add_(0, i0, g * (1 - f)).index_add_(0, i1, g * f)
    lam = (g * (values[i1] - values[i0]) * last)[:, None]
    return {'loss': sse.sum() / values.numel(), 'sse': sse,
            'dtheta': _theta_gradient(T, A, p0, sid, lam), 'dvalues': dvalues}


@torch.no_grad()
def exact(case, seed):
    st = prepare(case, seed)
    T, kind = st['T'], case['kind']
    if kind == 'interp':
        outs, ddatas, dgrids = [], [], []
        for k in range(0, case['batch'], 16):
            with torch.enable_grad():
                data = st['data'][k:k + 16].detach().double().requires_grad_(True)
                grid = st['grid'][k:k + 16].detach().double().requires_grad_(True)
                out = _sample(data, grid.transpose(1, 2), st['outsize'])
                a, b = torch.autograd.grad(out, [data, grid], st['weight'][k:k + 16].double())
            outs.append(out.detach())
            ddatas.append(a)
            dgrids.append(b)
        return {'out': torch.cat(outs), 'ddata': torch.cat(ddatas), 'dgrid': torch.cat(dgrids)}
    if kind == 'series':
        return _exact_series(T, st)
    theta = st['theta'].detach()
    if kind == 'image':
        out, dtheta, ddata = _exact_image(T, case, st['data'].detach(), theta, st.get('weight'),
                                          st['outsize'])
        res = {'out': out}
        if dtheta is not None:
            res['dtheta'] = dtheta
        if case['grad'] == 'both':
            res['ddata'] = ddata
        return res
    if kind == 'mixed':
        outs, dthetas, dimages = [], [], []
        for k, image in enumerate(st['images']):
            out, dtheta, ddata = _exact_image(T, {'gradient': 'reference'}, image.detach()[None],
                                              theta[k:k + 1], st['weights'][k][None],
                                              list(image.shape[1:]))
            outs.append(out[0])
            dthetas.append(dtheta)
            dimages.append(ddata[0])
        return {'out': outs, 'dtheta': torch.cat(dthetas), 'dimages': dimages}
    A, nc = _fields(T, theta), T.params.nc
    if kind == 'points':
        sid, _, _ = _linspace_series(st['offsets'])
        p0 = st['points'].double().t().contiguous()
        out = _integrate(nc, A, p0, sid)
        lam = st['weight'].double().t().contiguous()
        return {'out': out.t().contiguous(), 'dtheta': _theta_gradient(T, A, p0, sid, lam)}
    start = st['grid'].double().t()
    if kind == 'flow':
        p0 = start.repeat(case['batch'], 1)
        sid = torch.arange(case['batch'], device=p0.device).repeat_interleave(start.shape[0])
        p = _true_flow(nc, A, p0, sid)
        lam = st['weight'].double().transpose(1, 2).reshape(-1, T.params.ndim).clone()
        dA = _true_flow(nc, -A, p, sid, lam)
        return {'out': p.reshape(case['batch'], -1, T.params.ndim).transpose(1, 2).contiguous(),
                'dtheta': dA.reshape(case['batch'], -1) @ _basis(T, p.device)}
    outs, dthetas = [], []
    for k in range(case['batch']):
        p0 = start.contiguous()
        sid = torch.zeros(p0.shape[0], dtype=torch.long, device=p0.device)
        outs.append(_integrate(nc, A[k:k + 1], p0, sid).t())
        if case['grad']:
            lam = st['weight'][k].double().t().contiguous()
            dthetas.append(_theta_gradient(T, A[k:k + 1], p0, sid, lam))
    res = {'out': torch.stack(outs)}
    if dthetas:
        res['dtheta'] = torch.cat(dthetas)
    return res
