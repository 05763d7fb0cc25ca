"""The work a program gives this framework, as a set of cases to time.

A case is a dict of plain values; `listed()` names the standing ones and
`draw(rng)` gives more of the same ranges.  `prepare` makes what a program
holds before the call (images or volumes on the GPU, the plan it keeps for
their size), `run` is one pass through the public entry points, `exact` is the
same result in 64 bits and `work` what the path cannot do without.

What is covered: the fused 2-D denoise of one image, of a batch of one size and
of a batch of several sizes; the separate operators (analysis, threshold,
synthesis), their adjoints, the pyramid on its own and the band re-weighting;
a training step with learnable thresholds; the 3-D denoise on both grids and
its gradient; the undecimated wavelets.  The points / curves separation is
covered through its building blocks (wavelets, TV step, re-weighting, denoise):
it iterates hard thresholds, so its parts are not a continuous function of the
input and two correct runs of it in another rounding differ visibly.
"""
import functools
import math

import numpy as np
import torch

import shearcuda_gb300 as sc

SIDES = (192, 256, 384, 512, 768, 1024, 2048)          # image sides in use (2^a and 3 * 2^a)
UNEVEN = ((256, 256), (384, 512), (512, 512), (768, 1024), (1024, 1024))
# name -> (dcomp, dsize): the demos' transform, the separation demo's long
# filters, and a shallow transform
TRANSFORMS = {
    'demo': ((3, 3, 4, 4), (32, 32, 16, 16)),
    'long': ((3, 3, 4, 4), (80, 80, 80, 80)),
    'shallow': ((3, 3), (32, 32)),
}
NUM_DIRS = {'v3': (2, 2, 4), 'demo': (8, 4, 4)}       # 3-D directions per level, finest first
# white-noise l2 norm of one pyramid level's bands together, finest level
# first: the noise table a program stores instead of estimating it per run
LEVEL_NORM = (0.872, 0.416, 0.206, 0.104, 0.052, 0.026)
LEVEL_NORM_3D = (0.9, 0.6, 0.6)
# The noise of rendered or frame-averaged data, a small fraction of a grey
# level, for the hard threshold (the only one in 3-D): here a coefficient that
# rounding carries across the threshold moves a value by less than 1e-3 of the
# data's scale.  Camera noise (10 to 40 grey levels) goes with the soft one.
FAINT = 0.02
# The training targets are the clean data at another exposure.
EXPOSURE = 60.0
MAX_PIXELS = 64 * 512 * 512


def listed():
    return [
        # one small image per call: an interactive denoise, all latency
        {'name': 'denoise_1x256', 'kind': 'denoise', 'H': 256, 'W': 256, 'n': 1, 'transform': 'demo', 'lpfilt': 'maxflat', 'soft': False, 'sigma': FAINT},
        # one photograph per call, the largest side
        {'name': 'denoise_1x2048', 'kind': 'denoise', 'H': 2048, 'W': 2048, 'n': 1, 'transform': 'demo', 'lpfilt': 'maxflat', 'soft': True, 'sigma': 20.0},
        # throughput: the headline batch
        {'name': 'denoise_64x512', 'kind': 'denoise', 'H': 512, 'W': 512, 'n': 64, 'transform': 'demo', 'lpfilt': 'maxflat', 'soft': True, 'sigma': 20.0},
        # throughput with images as they come: 64 of five sizes in one call
        {'name': 'uneven_64', 'kind': 'uneven', 'n': 64, 'soft': True, 'sizes_seed': 1},
        # the operators one by one, as a program that edits the coefficients does
        {'name': 'operators_384x512', 'kind': 'operators', 'H': 384, 'W': 512, 'transform': 'demo', 'lpfilt': 'maxflat', 'sigma': 20.0},
        # both adjoints: one step of an iterative inverse problem
        {'name': 'adjoints_512', 'kind': 'adjoints', 'H': 512, 'W': 512, 'transform': 'demo', 'lpfilt': 'maxflat'},
        # the pyramid alone, split and rebuilt, and its bands re-weighted; a ragged size
        {'name': 'pyramid_768x1024', 'kind': 'pyramid', 'H': 768, 'W': 1024, 'transform': 'demo', 'lpfilt': 'maxflat'},
        # a training step over the thresholds and the images
        {'name': 'train_16x512', 'kind': 'train', 'H': 512, 'W': 512, 'n': 16, 'transform': 'demo', 'sigma': 20.0},
        # four clips of a video in one call
        {'name': 'volume_4x128', 'kind': 'volume', 'n0': 128, 'n1': 128, 'n2': 128, 'n': 4, 'dirs': 'v3', 'grid': 'fast'},
        # one large ragged volume with the reference's own padding
        {'name': 'volume_192x125x186', 'kind': 'volume', 'n0': 192, 'n1': 125, 'n2': 186, 'n': 1, 'dirs': 'v3', 'grid': 'marshal'},
        # the gradient through the 3-D denoise
        {'name': 'volume_train_96', 'kind': 'volume_train', 'n0': 96, 'n1': 96, 'n2': 96, 'n': 1, 'dirs': 'v3', 'grid': 'fast'},
        # wavelet analysis, synthesis and TV step of the separation, its image size
        {'name': 'wavelet_32x256', 'kind': 'wavelet', 'H': 256, 'W': 256, 'n': 32, 'levels': 4, 'symmlet': 4},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _draw_size(rng, cap=MAX_PIXELS):
    while True:
        H, W = rng.choice(SIDES), rng.choice(SIDES)
        if H * W <= cap:
            return H, W


def _draw_transform(rng):
    return rng.choice(('demo', 'demo', 'demo', 'long', 'shallow'))


def _draw_lpfilt(rng):
    return rng.choice(('maxflat', 'maxflat', 'maxflat', '9-7', 'pyr', 'pyrexc'))


def draw(rng):
    kind = rng.choice(('denoise', 'denoise', 'denoise', 'uneven', 'operators', 'adjoints', 'pyramid', 'train',
                       'volume', 'volume', 'volume_train', 'wavelet'))
    if kind == 'denoise':
        H, W = _draw_size(rng)
        n = _log_int(rng, 1, min(64, MAX_PIXELS // (H * W)))
        soft = rng.random() < 0.6
        return {'kind': kind, 'H': H, 'W': W, 'n': n, 'transform': _draw_transform(rng), 'lpfilt': _draw_lpfilt(rng),
                'soft': soft, 'sigma': round(rng.uniform(10, 40), 1) if soft else FAINT}
    if kind == 'uneven':
        return {'kind': kind, 'n': _log_int(rng, 4, 64), 'soft': True, 'sizes_seed': rng.randrange(2, 1 << 20)}
    if kind in ('operators', 'adjoints', 'pyramid'):
        H, W = _draw_size(rng, 1 << 21)
        case = {'kind': kind, 'H': H, 'W': W, 'transform': _draw_transform(rng), 'lpfilt': _draw_lpfilt(rng)}
        return dict(case, sigma=round(rng.uniform(10, 40), 1)) if kind == 'operators' else case
    if kind == 'train':
        H, W = _draw_size(rng, 1 << 20)
        return {'kind': kind, 'H': H, 'W': W, 'n': _log_int(rng, 1, min(32, (1 << 22) // (H * W))),
                'transform': rng.choice(('demo', 'long')), 'sigma': round(rng.uniform(10, 40), 1)}
    if kind == 'wavelet':
        H, W = _draw_size(rng, 1 << 22)
        return {'kind': kind, 'H': H, 'W': W, 'n': _log_int(rng, 1, min(32, (1 << 22) // (H * W))),
                'levels': rng.randint(1, 5), 'symmlet': rng.randint(4, 10)}
    if kind == 'volume' and rng.random() < 0.4:  # the padded grids the reference's any-size demo meets here
        lo, hi = rng.choice(((84, 95), (120, 131), (132, 143), (180, 191), (192, 203)))
        n0, n1, n2 = (rng.randint(lo, hi) for _ in range(3))
        grid = 'marshal'
    else:
        n0, n1, n2 = (rng.randint(40, 192) for _ in range(3))
        grid = 'fast'
    if kind == 'volume_train':  # whole grids: at a padded volume's crop the cotangent, and what a kept coefficient carries, jumps
        n0, n1, n2 = (rng.choice((96, 96, 144, 192)) for _ in range(3))
    top = 4 if kind == 'volume' else 2
    return {'kind': kind, 'n0': n0, 'n1': n1, 'n2': n2, 'n': rng.randint(1, max(1, min(top, 4 * 128 ** 3 // (n0 * n1 * n2)))),
            'dirs': 'demo' if max(n0, n1, n2) <= 96 and rng.random() < 0.5 else 'v3', 'grid': grid}


# ---------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device='cuda').manual_seed(int(seed))


def _images(n, H, W, sigma, g):
    """n images (n, H, W): a gradient and ten filled ellipses each, plus noise."""
    u = torch.rand((n, 10, 6), generator=g, device='cuda')
    y = torch.arange(H, device='cuda', dtype=torch.float32)[None, :, None]
    x = torch.arange(W, device='cuda', dtype=torch.float32)[None, None, :]
    img = 40.0 + 80.0 * u[:, :1, :1] * (y / H) + 60.0 * u[:, :1, 1:2] * (x / W)
    for k in range(10):
        cy, cx, a, b, ang, val = (u[:, k, j, None, None] for j in range(6))
        a, b = (0.02 + 0.28 * a) * min(H, W), (0.02 + 0.28 * b) * min(H, W)
        c, s = torch.cos(math.pi * ang), torch.sin(math.pi * ang)
        dy, dx = y - cy * H, x - cx * W
        img = torch.where(((c * dx + s * dy) / a) ** 2 + ((c * dy - s * dx) / b) ** 2 <= 1.0, 255.0 * val, img)
    return (img + sigma * torch.randn((n, H, W), generator=g, device='cuda')).contiguous()


def _volumes(n, shape, sigma, g):
    """n volumes: eight ellipsoids each, moving along the last axis, plus noise."""
    u = torch.rand((n, 8, 8), generator=g, device='cuda')
    ax = [torch.arange(m, device='cuda', dtype=torch.float32) for m in shape]
    x, y, t = ax[0][None, :, None, None], ax[1][None, None, :, None], ax[2][None, None, None, :]
    vol = (40.0 + 60.0 * u[:, 0, 0])[:, None, None, None].expand(n, *shape)
    for k in range(8):
        c0, c1, c2, r0, r1, r2, v, val = (u[:, k, j, None, None, None] for j in range(8))
        r0, r1, r2 = ((0.08 + 0.25 * r) * min(shape) for r in (r0, r1, r2))
        t0 = t - c2 * shape[2]
        inside = ((x - c0 * shape[0] - (v - 0.5) * 0.6 * t) / r0) ** 2 + ((y - c1 * shape[1]) / r1) ** 2 + (t0 / r2) ** 2 <= 1.0
        vol = torch.where(inside, 255.0 * val, vol)
    return (vol + sigma * torch.randn((n,) + tuple(shape), generator=g, device='cuda')).contiguous()


def _scalars(transform):
    dcomp, _ = TRANSFORMS[transform]
    out = [LEVEL_NORM[len(dcomp) - 1] / 2]
    for level, c in enumerate(dcomp):
        out += [LEVEL_NORM[len(dcomp) - 1 - level] / math.sqrt(1 << c)] * (1 << c)
    return np.array(out)


def _scalars_3d(dirs):
    return np.concatenate([np.full(3 * d * d, LEVEL_NORM_3D[k] / math.sqrt(3 * d * d)) for k, d in enumerate(NUM_DIRS[dirs])])


def _K(transform):
    return [0.0] + [3.0] * (len(TRANSFORMS[transform][0]) - 1) + [4.0]


def _weights(transform):
    """Band weights: the separation demo's on its finest three levels, flat on shallower transforms."""
    return [0.1, 0.1, 1.5, 1.5] if len(TRANSFORMS[transform][0]) >= 3 else [0.1, 0.5, 1.5]


# A program keeps one plan per image or volume size and runs its inputs through it.
@functools.lru_cache(maxsize=6)
def _plan(transform, lpfilt, H, W, n):
    dcomp, dsize = TRANSFORMS[transform]
    plan = sc.prepare_shearing_filters_cuda(list(dcomp), list(dsize), H, W, lpfilt, batch=n)
    plan.set_scalars(_scalars(transform))
    return plan


@functools.lru_cache(maxsize=2)
def _volume_plan(dirs, grid, n0, n1, n2, n):
    plan = sc.VolumePlan(n0, n1, n2, num_dirs=NUM_DIRS[dirs], batch=n, grid=grid)
    plan.set_scalars(_scalars_3d(dirs))
    return plan


@functools.lru_cache(maxsize=1)
def _multi(sizes):
    """The plans of an uneven batch, one per size, and the object that runs them together."""
    return sc.MultiBatch([_plan('demo', 'maxflat', H, W, n) for (H, W), n in sizes])


def _uneven_sizes(case):
    r = np.random.default_rng(case['sizes_seed'])
    return [UNEVEN[int(i)] for i in r.integers(0, len(UNEVEN), case['n'])]


def prepare(case, seed):
    kind, g = case['kind'], _gen(seed)
    state = {'kind': kind, 'case': dict(case)}
    if kind == 'uneven':
        sizes = _uneven_sizes(case)
        r = np.random.default_rng(seed)
        state['sigmas'] = [float(s) for s in r.uniform(10, 40, len(sizes))]
        state['xs'] = [_images(1, H, W, s, g)[0].contiguous() for (H, W), s in zip(sizes, state['sigmas'])]
        state['multi'] = _multi(tuple(sorted((s, sizes.count(s)) for s in set(sizes))))
    elif kind in ('volume', 'volume_train'):
        shape = (case['n0'], case['n1'], case['n2'])
        state['plan'] = _volume_plan(case['dirs'], case['grid'], *shape, case['n'])
        state['x'] = _volumes(case['n'], shape, FAINT, g)
        if kind == 'volume_train':
            state['x'].requires_grad_(True)
            state['target'] = EXPOSURE + _volumes(case['n'], shape, 0.0, _gen(seed))
    elif kind == 'wavelet':
        state['x'] = _images(case['n'], case['H'], case['W'], 20.0, g)
        state['h'] = sc.MakeONFilter('Symmlet', case['symmlet'])
    else:
        state['plan'] = _plan(case['transform'], case.get('lpfilt', 'maxflat'), case['H'], case['W'], case.get('n', 1))
        x = _images(case.get('n', 1), case['H'], case['W'], case.get('sigma', 20.0), g)
        if kind == 'denoise':
            state['xs'] = [v.contiguous() for v in x]
        elif kind == 'train':
            state['target'] = EXPOSURE + _images(case['n'], case['H'], case['W'], 0.0, _gen(seed))
            state['x'] = x.requires_grad_(True)
            state['net'] = sc.NsstDenoiser(state['plan'], _scalars(case['transform']), case['sigma'], _K(case['transform']))
        elif kind == 'adjoints':
            state['x'] = x[0].contiguous()
            state['c'] = 20.0 * torch.randn((state['plan'].nbands, case['H'], case['W']), generator=g, device='cuda')
        else:
            state['x'] = x[0].contiguous()
    return state


# ----------------------------------------------------------------------- passes
def run(state):
    kind, case = state['kind'], state['case']
    if kind == 'denoise':
        mode = sc.THRESH_SOFT if case['soft'] else sc.THRESH_HARD
        if case['n'] == 1:
            return sc.nsst_denoise(state['xs'][0], state['plan'], case['sigma'], _K(case['transform']), mode=mode)
        return sc.nsst_denoise_batch(state['xs'], state['plan'], case['sigma'], _K(case['transform']), mode=mode)
    if kind == 'uneven':
        return state['multi'].denoise(state['xs'], state['sigmas'], _K('demo'),
                                      mode=sc.THRESH_SOFT if case['soft'] else sc.THRESH_HARD)
    if kind == 'operators':
        plan = state['plan']
        c = sc.shear_trans_cuda(state['x'], case['lpfilt'], plan)
        sc.softth_cuda(c, case['sigma'], _K(case['transform']), _scalars(case['transform']), plan)
        return c, sc.inverse_shear_cuda(c, case['lpfilt'], plan)
    if kind == 'adjoints':
        return sc.shear_trans_adjoint(state['c'], state['plan']), sc.inverse_shear_adjoint(state['x'], state['plan'])
    if kind == 'pyramid':
        y = sc.atrousdec(state['x'], state['plan'])
        return y, sc.atrousrec(y, state['plan']), sc.re_weight_band(state['x'], _weights(case['transform']), state['plan'])
    if kind == 'train':
        net, x = state['net'], state['x']
        net.tau.grad = x.grad = None
        out = net(x)
        (out - state['target']).square().mean().backward()
        return out.detach(), x.grad, net.tau.grad
    if kind == 'volume':
        return sc.denoise3(state['x'], state['plan'], FAINT)
    if kind == 'volume_train':
        x = state['x']
        x.grad = None
        out = sc.denoise3_diff(x, state['plan'], FAINT)
        (out - state['target']).square().mean().backward()
        return out.detach(), x.grad
    yl, yh = sc.mrdwt_cuda(state['x'], state['h'], case['levels'])
    return yl, yh, sc.mirdwt_cuda(yl, yh, state['h'], case['levels']), sc.tv_correction_cuda(state['x'], 3.0)


def work(case):
    """Bytes: every input, output and filter spectrum once.  Flops: the path's transforms."""
    kind = case['kind']

    def image(n, N, transform, fwd, inv):
        dcomp, _ = TRANSFORMS[transform]
        nb, L = sum(1 << c for c in dcomp), len(dcomp)
        return n * ((fwd + inv) * (nb + L + 1)) * 2.5 * N * math.log2(N), 4 * nb * N

    if kind == 'uneven':
        sizes = _uneven_sizes(case)
        flops = sum(image(1, H * W, 'demo', 1, 1)[0] for H, W in sizes)
        return {'bytes': sum(8 * H * W for H, W in sizes) + sum(image(1, H * W, 'demo', 1, 1)[1] for H, W in set(sizes)), 'flops': flops}
    if kind in ('volume', 'volume_train'):
        N = case['n0'] * case['n1'] * case['n2']
        d, flops, spec = NUM_DIRS[case['dirs']], 0.0, 0
        for k, m in enumerate((N, N / 1.5 ** 3, N / 3 ** 3)):
            flops += (3 * d[k] ** 2 + 3) * 2.5 * m * math.log2(m)
            spec += 4 * 3 * d[k] ** 2 * m
        t = 2 if kind == 'volume_train' else 1
        return {'bytes': t * (8 * N * case['n'] + spec), 'flops': t * case['n'] * flops}
    H, W, n = case['H'], case['W'], case.get('n', 1)
    N = H * W
    if kind == 'wavelet':
        L, taps = case['levels'], 2 * case['symmlet']
        return {'bytes': n * N * 4 * (2 * (3 * L + 1) + 4), 'flops': n * N * L * 2 * 12 * taps}
    if kind == 'pyramid':
        L = len(TRANSFORMS[case['transform']][0])
        return {'bytes': N * 4 * (2 * (L + 2) + 2), 'flops': (2 * L + 6) * 2.5 * N * math.log2(N)}
    flops, spec = image(n, N, case['transform'], 1, 1)
    nb = 1 + sum(1 << c for c in TRANSFORMS[case['transform']][0])
    if kind == 'denoise':
        return {'bytes': 8 * N * n + spec, 'flops': flops}
    if kind == 'train':
        return {'bytes': 20 * N * n + 2 * spec, 'flops': 2 * flops}
    if kind == 'adjoints':
        return {'bytes': 4 * N * (2 + 2 * nb) + 2 * spec, 'flops': flops}
    return {'bytes': 4 * N * (2 + 3 * nb) + 2 * spec, 'flops': flops}


# --------------------------------------------------------- the same in 64 bits
# The filter banks are the transforms' weights and are taken as the FP64 tables
# the package publishes; everything computed with them is plain torch.
def _ext(x):
    """Half-sample symmetric extension of (..., H, W) to (..., 2H, 2W)."""
    x = torch.cat([x, x.flip(-2)], -2)
    return torch.cat([x, x.flip(-1)], -1)


def _responses(lpfilt, L, H, W):
    """Per step the real responses (h0, h1, g0, g1) on the extension's half spectrum."""
    out = []
    for step in range(L):
        M, row = 1 << step, []
        for h in sc.pyramid_filters(lpfilt):
            h = torch.tensor(np.array(h), dtype=torch.float64, device='cuda')
            F = h.shape[0]
            off = M * (torch.arange(F, dtype=torch.float64, device='cuda') - F // 2)
            a = torch.cos(math.pi / H * torch.arange(2 * H, dtype=torch.float64, device='cuda')[:, None] * off)
            b = torch.cos(math.pi / W * torch.arange(W + 1, dtype=torch.float64, device='cuda')[:, None] * off)
            row.append(a @ h @ b.T)
        out.append(row)
    return out


def _filt(x, G):
    """x (..., H, W) filtered on its symmetric extension with the response G."""
    H, W = x.shape[-2:]
    return torch.fft.irfft2(torch.fft.rfft2(_ext(x)) * G, s=(2 * H, 2 * W))[..., :H, :W]


def _pyr_dec(x, R):
    """[lowpass, bands coarse to fine]."""
    bands = []
    for h0, h1, _, _ in R:
        bands.append(_filt(x, h1))
        x = _filt(x, h0)
    return [x] + bands[::-1]


def _pyr_rec(y, R):
    x = y[0]
    for i in range(len(R) - 1, -1, -1):
        x = _filt(x, R[i][2]) + _filt(y[len(R) - i], R[i][3])
    return x


def _spectra(transform, H, W):
    out = []
    for c, s in zip(*TRANSFORMS[transform]):
        F = torch.fft.rfft2(torch.tensor(sc.shearing_filters(s, c), dtype=torch.float64, device='cuda'), s=(H, W))
        out.append(F / F.abs().square().sum(0).sqrt())
    return out


def _dec(x, R, S):
    y = _pyr_dec(x, R)
    return [y[0][None]] + [torch.fft.irfft2(torch.fft.rfft2(b) * s, s=x.shape[-2:]) for b, s in zip(y[1:], S)]


def _rec(c, R, S):
    y = [c[0][0]] + [torch.fft.irfft2((torch.fft.rfft2(b) * s.conj()).sum(0), s=b.shape[-2:]) for b, s in zip(c[1:], S)]
    return _pyr_rec(y, R)


def _thresh(c, t, soft):
    keep = (c.abs() > t).to(c.dtype)
    return torch.sign(c) * keep * (c.abs() - t) if soft else c * keep


def _tau(transform, sigma):
    """Per-band thresholds, one (bands, 1, 1) tensor per level."""
    K, s, out, at = _K(transform), _scalars(transform), [], 0
    for level, nd in enumerate([1] + [1 << c for c in TRANSFORMS[transform][0]]):
        out.append(torch.tensor(K[level] * sigma * s[at:at + nd], device='cuda').float().double()[:, None, None])
        at += nd
    return out


def _denoise(x, R, S, tau, soft):
    return _rec([_thresh(c, t, soft) for c, t in zip(_dec(x, R, S), tau)], R, S)


def _window_1d(n, w, tbw):
    K = math.ceil(n / 2 * (w + tbw))
    k = torch.arange(K + 1, dtype=torch.float64, device='cuda')
    t = ((K - k) / (K - math.floor(n / 2 * (w - tbw)))).clamp(0, 1)
    v = torch.zeros(n, dtype=torch.float64, device='cuda')
    v[:K + 1] = (0.5 * (1 - torch.cos(math.pi * t))).sqrt()
    v[n - K:] = v[1:K + 1].flip(0)
    return v


def _lowpass_3d(shape, level):
    w, tbw = ((0.5, 1 / 7), (3 / 8, 1 / 9), (3 / 8, 1 / 9))[level]
    a, b, c = (_window_1d(n, w, tbw) for n in shape)
    return a[:, None, None] * b[None, :, None] * c[None, None, :]


def _resize_spectrum(X, shape):
    """The lower frequencies of a full spectrum on a smaller grid, or zero-extended to a larger one."""
    for axis, m in enumerate(shape):
        n, k = X.shape[axis], (min(X.shape[axis], m) - 1) // 2
        low, high = X.narrow(axis, 0, k + 1), X.narrow(axis, n - k, k)
        mid = list(X.shape)
        mid[axis] = m - 2 * k - 1
        X = torch.cat([low, torch.zeros(mid, dtype=X.dtype, device=X.device), high], axis)
    return X


def _denoise_3d(x, case):
    shape = x.shape
    if case['grid'] == 'marshal':
        grid = [n + 12 - n % 12 for n in shape]
    else:
        grid = [next(v for v in (96, 144, 192) if v >= n) for n in shape]
    for axis, (n, v) in enumerate(zip(shape, grid)):
        x = torch.cat([x, x.narrow(axis, n - 1, 1).expand(*[v - n if k == axis else x.shape[k] for k in range(3)])], axis)
    X, subs, D = torch.fft.fftn(x), [], (1.5, 2, 2)
    sizes = [tuple(grid)]
    for level in range(3):
        Lf = _lowpass_3d(sizes[level], level)
        subs.append(torch.fft.ifftn((1 - Lf ** 2).clamp_min(0).sqrt() * X).real)
        sizes.append(tuple(int(round(s / D[level])) for s in sizes[level]))
        X = _resize_spectrum(Lf * X, sizes[-1]) / D[level] ** 1.5
    filters = torch.tensor(np.array(sc.get_meyer_based_filter(NUM_DIRS[case['dirs']])), device='cuda')
    scal, T, at = _scalars_3d(case['dirs']), sc.DEMO_T, 0
    rec = []
    for level, d in enumerate(NUM_DIRS[case['dirs']]):
        full = [m + 23 for m in sizes[level]]
        B, total = torch.fft.rfftn(subs[level], s=full), 0
        for b in range(at, at + 3 * d * d):
            c = torch.fft.irfftn(B * torch.fft.rfftn(filters[b], s=full), s=full)
            c = c[tuple(slice(12, 12 + m) for m in sizes[level])]
            total = total + c * (c.abs() > float(np.float32(T[level] * FAINT * scal[b]))).to(c.dtype)
        at += 3 * d * d
        rec.append(total)
    for level in range(2, -1, -1):
        Lf = _lowpass_3d(sizes[level], level)
        X = (1 - Lf ** 2).clamp_min(0).sqrt() * torch.fft.fftn(rec[level]) + _resize_spectrum(X, sizes[level]) * Lf * D[level] ** 1.5
    return torch.fft.ifftn(X).real[:shape[0], :shape[1], :shape[2]]


def _roll_pair(x, lo, hi, step, axis):
    """Periodic filters along one axis: sum_j f[j] x[. + j step]."""
    a = b = 0
    for j in range(len(lo)):
        s = torch.roll(x, -j * step, axis)
        a, b = a + float(lo[j]) * s, b + float(hi[j]) * s
    return a, b


def _roll_sum(a, b, lo, hi, step, axis):
    return sum(torch.roll(a, j * step, axis) * float(lo[j]) + torch.roll(b, j * step, axis) * float(hi[j]) for j in range(len(lo)))


def _wavelet_pairs(h):
    sign = np.where(np.arange(len(h)) % 2 == 0, 1.0, -1.0)
    return (h, (-sign * h)[::-1]), (h / 2, sign * h[::-1] / 2)


def _mrdwt(x, h, L):
    (lo, hi), _ = _wavelet_pairs(h)
    yl, planes = x, []
    for level in range(L):
        a, b = _roll_pair(yl, lo, hi, 1 << level, -1)
        (yl, lh), (hl, hh) = _roll_pair(a, lo, hi, 1 << level, -2), _roll_pair(b, lo, hi, 1 << level, -2)
        planes += [lh, hl, hh]
    return yl, torch.stack(planes, -3)


def _mirdwt(yl, yh, h, L):
    _, (lo, hi) = _wavelet_pairs(h)
    for level in range(L - 1, -1, -1):
        lh, hl, hh = (yh[..., 3 * level + k, :, :] for k in range(3))
        yl = _roll_sum(_roll_sum(yl, lh, lo, hi, 1 << level, -2), _roll_sum(hl, hh, lo, hi, 1 << level, -2), lo, hi, 1 << level, -1)
    return yl


def exact(case, seed):
    state, kind = prepare(case, seed), case['kind']
    if kind == 'uneven':
        made = {}
        out = []
        for x, sigma in zip(state['xs'], state['sigmas']):
            H, W = x.shape
            if (H, W) not in made:
                made[H, W] = _responses('maxflat', 4, H, W), _spectra('demo', H, W)
            out.append(_denoise(x.double(), *made[H, W], _tau('demo', sigma), case['soft']))
        return out
    if kind == 'volume':
        return torch.stack([_denoise_3d(v.double(), case) for v in state['x']])
    if kind == 'volume_train':
        out, grad = [], []
        for v, target in zip(state['x'].detach(), state['target']):
            v = v.double().requires_grad_(True)
            y = _denoise_3d(v, case)
            ((y - target.double()).square().sum() / target.numel() / case['n']).backward()
            out.append(y.detach())
            grad.append(v.grad)
        return torch.stack(out), torch.stack(grad)
    if kind == 'wavelet':
        x, h = state['x'].double(), np.asarray(state['h'])
        yl, yh = _mrdwt(x, h, case['levels'])
        tl, th = _mrdwt(x, np.array([1.0, 1.0]) / math.sqrt(2), 1)
        tv = _mirdwt(tl, _thresh(th, 3.0, True), np.array([1.0, 1.0]) / math.sqrt(2), 1)
        return yl, yh, _mirdwt(yl, yh, h, case['levels']), tv
    H, W, name = case['H'], case['W'], case['transform']
    R, S = _responses(case.get('lpfilt', 'maxflat'), len(TRANSFORMS[name][0]), H, W), _spectra(name, H, W)
    if kind == 'denoise':
        out = [_denoise(x.double(), R, S, _tau(name, case['sigma']), case['soft']) for x in state['xs']]
        return out[0] if case['n'] == 1 else out
    if kind == 'operators':
        c = [_thresh(b, t, True) for b, t in zip(_dec(state['x'].double(), R, S), _tau(name, case['sigma']))]
        return torch.cat(c), _rec(c, R, S)
    if kind == 'pyramid':
        y = _pyr_dec(state['x'].double(), R)
        w = _weights(name)
        Rw = R[:len(w) - 1]
        return torch.stack(y), _pyr_rec(y, R), _pyr_rec([a * b for a, b in zip(_pyr_dec(state['x'].double(), Rw), w)], Rw)
    if kind == 'adjoints':  # the transposes, by differentiating the operators
        x = torch.zeros((H, W), dtype=torch.float64, device='cuda', requires_grad=True)
        (torch.cat(_dec(x, R, S)) * state['c'].double()).sum().backward()
        c = [torch.zeros((n, H, W), dtype=torch.float64, device='cuda', requires_grad=True) for n in [1] + [len(s) for s in S]]
        (_rec(c, R, S) * state['x'].double()).sum().backward()
        return x.grad, torch.cat([b.grad for b in c])
    # the soft threshold's derivative jumps at the threshold: the images' gradient has no one value
    # where a coefficient lies within rounding of it, and a few of the millions do
    tau = [t.detach().requires_grad_(True) for t in _tau(name, case['sigma'])]
    out = []
    for x, target in zip(state['x'].detach(), state['target']):
        y = _denoise(x.double(), R, S, tau, True)
        ((y - target.double()).square().sum() / target.numel() / case['n']).backward()
        out.append(y.detach())
    return torch.stack(out), None, torch.cat([t.grad.reshape(-1) for t in tau])
