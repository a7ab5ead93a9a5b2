"""The work that programs built on tractor_b200 have it do, as measurable cases.

Every case is one call (or the few calls that belong together) through public
entry points, at sizes from the repository's own workloads: galaxies through a
pixelized PSF (one, the 256 of the benchmark, thousands on ragged patches),
their vector-Jacobian product, whole scenes, batched blob fits, the blob
model's vector-Jacobian product, dense normal equations with their solve, EM
fits of PSF stamps, and a model image through the object API.  Patch
geometry follows from the case alone; every value follows from the seed.

`exact` restates each path in 64 bits with plain torch and numpy (the mixture
tables are read from the package's data file).
"""
import json
import math
import os

import numpy as np
import torch

import tractor_b200 as T
from tractor_b200 import _lib, batch, emfit, fit, grad, render

FLUX = 1000.
MAX_MASK = 253        # the largest square patch whose FFT size is 256


def listed():
    return [
        # one galaxy on a small patch, as a program that draws sources one by
        # one asks for it: launch and latency
        dict(name='fourier-one', kind='fourier', n=1, lo=32, hi=32, psf=63, mix='sersic'),
        # the benchmark's 256 galaxies on 128 x 128 patches, FFT size 256
        dict(name='fourier-256', kind='fourier', n=256, lo=128, hi=128, psf=63, mix='sersic'),
        # a catalog of galaxies of all profiles on ragged patches (FFT sizes
        # 64 to 256) through a smaller PSF: simulating or subtracting a field
        dict(name='fourier-ragged-2000', kind='fourier', n=2000, lo=25, hi=MAX_MASK, psf=45,
             mix='all'),
        # one gradient step of an optimizer over 256 galaxies on patches of
        # 64 to 253 px: model forward, vector-Jacobian product backward
        dict(name='fourier-grad-256', kind='fourier_grad', n=256, lo=64, hi=MAX_MASK, psf=63),
        # a small cutout of odd size with a few dozen sources
        dict(name='scene-cutout', kind='scene', n=150, w=501, h=397, kpsf=3),
        # the batched render's full field: 20,000 sources on 4096 x 4096
        dict(name='scene-field', kind='scene', n=20000, w=4096, h=4096, kpsf=3),
        # a handful of blobs, as fitted while a field is worked through
        dict(name='fit-4', kind='fit', blobs=4),
        # many blobs at once (192-512 px, 3 bands, about 6 sources each)
        dict(name='fit-300', kind='fit', blobs=300),
        # the blob model and its gradient for a caller's own optimizer
        dict(name='blob-grad-100', kind='blob_grad', blobs=100),
        # the least-squares step of 512 problems of 63 parameters
        dict(name='lsq-512x63', kind='lsq', n=512, p=63, rows=16384),
        # PSF stamps of a set of exposures, three Gaussians each
        dict(name='em-1024', kind='em', n=1024, side=25, k=3, steps=1000),
        # a small image through the object API, as the reference's callers do
        dict(name='model-image', kind='api', n=24, w=160, h=121),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['fourier', 'fourier', 'fourier_grad', 'scene', 'scene', 'fit', 'blob_grad',
                       'lsq', 'em', 'api'])
    if kind == 'fourier':
        lo = _log_int(rng, 24, MAX_MASK)
        return dict(kind=kind, n=_log_int(rng, 1, 2000), lo=lo, hi=rng.randint(lo, MAX_MASK),
                    psf=2 * rng.randint(10, 31) + 1, mix=rng.choice(['sersic', 'all']))
    if kind == 'fourier_grad':
        lo = _log_int(rng, 32, MAX_MASK)
        return dict(kind=kind, n=_log_int(rng, 1, 256), lo=lo, hi=rng.randint(lo, MAX_MASK),
                    psf=2 * rng.randint(10, 31) + 1)
    if kind == 'scene':
        side = _log_int(rng, 200, 4096)
        return dict(kind=kind, n=max(1, int(side * side * rng.uniform(2e-4, 1.2e-3))), w=side,
                    h=max(64, int(side * rng.uniform(0.5, 1.))), kpsf=rng.randint(1, 4))
    if kind == 'fit':
        return dict(kind=kind, blobs=_log_int(rng, 1, 300))
    if kind == 'blob_grad':
        return dict(kind=kind, blobs=_log_int(rng, 1, 100))
    if kind == 'lsq':
        p, rows = _log_int(rng, 4, 200), _log_int(rng, 1000, 16384)
        most = 512 * 64 * 16384 // ((p + 1) * rows)
        return dict(kind=kind, n=_log_int(rng, 1, max(1, min(2000, most))), p=p, rows=rows)
    if kind == 'em':
        return dict(kind=kind, n=_log_int(rng, 1, 1024), side=2 * rng.randint(7, 13) + 1,
                    k=rng.randint(1, 3), steps=1000)
    return dict(kind='api', n=rng.randint(1, 60), w=rng.randint(48, 256), h=rng.randint(48, 256))


def _numbers(case, seed=0):
    """A numpy generator of the case and a seed."""
    text = json.dumps({k: v for k, v in case.items() if k != 'name'}, sort_keys=True)
    return np.random.default_rng([int(seed)] + list(text.encode()))


def _device():
    return torch.device('cuda', torch.cuda.current_device())


def _on_device(rows):
    return torch.from_numpy(np.ascontiguousarray(rows).view(np.uint8).copy()).to(_device())


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _moffat(size, fwhm=4., beta=3.):
    alpha = fwhm / (2 * math.sqrt(2 ** (1 / beta) - 1))
    y, x = np.mgrid[:size, :size] - size // 2
    img = (1 + (x ** 2 + y ** 2) / alpha ** 2) ** (-beta)
    return (img / img.sum()).astype(np.float32)


def _ellipses(rng, n):
    """(r_e, e1, e2): r_e log-uniform in 0.5-8 px, axis ratio 0.2-1."""
    re = np.exp(rng.uniform(math.log(.5), math.log(8.), n))
    ab = 1. / rng.uniform(.2, 1., n)
    phi = rng.uniform(0., 180., n)
    e = (ab - 1) / (ab + 1)
    return re, e * np.cos(np.radians(-2 * phi)), e * np.sin(np.radians(-2 * phi))


def _patch_sizes(case):
    g = _numbers(case)
    size = lambda: np.round(np.exp(g.uniform(math.log(case['lo']), math.log(case['hi'] + .499),  # noqa: E731
                                             case['n']))).astype(np.int64)
    w = size()
    return w, np.clip(np.round(w * g.uniform(.8, 1.25, len(w))), case['lo'],
                      case['hi']).astype(np.int64) if case['hi'] > case['lo'] else w


def _galaxies(case, seed):
    """GALAXY_SRC records, each galaxy near the centre of its own patch."""
    n, rng = case['n'], _numbers(case, seed)
    w, h = _patch_sizes(case)
    s = np.zeros(n, batch.GALAXY_SRC)
    s['s0'], s['s1'], s['s2'] = _ellipses(rng, n)
    s['sersic_n'] = rng.uniform(.7, 6., n)
    s['px'] = w / 2 + rng.uniform(-.5, .5, n)
    s['py'] = h / 2 + rng.uniform(-.5, .5, n)
    s['counts'] = FLUX * np.exp(rng.uniform(-1., 1., n))
    s['profile'] = _lib.PROFILE_SERSIC if case.get('mix', 'sersic') == 'sersic' else rng.choice(
        [_lib.PROFILE_EXP, _lib.PROFILE_DEV, _lib.PROFILE_SERSIC], n)
    s['shape_type'] = _lib.SHAPE_ELLIPSE_E
    s['mw'], s['mh'] = w, h
    s['out_off'] = np.concatenate([[0], np.cumsum(w * h)[:-1]])
    return s, int((w * h).sum())


def _gradient_inputs(case, seed):
    """(records with single-precision parameters, pixels, upstream gradient)."""
    s, npix = _galaxies(case, seed)
    for name in ('px', 'py', 'counts', 's0', 's1', 's2', 'sersic_n'):
        s[name] = s[name].astype(np.float32)
    g = torch.Generator(device=_device()).manual_seed(seed)
    return s, npix, torch.randn(npix, generator=g, device=_device())


def _scene(case, seed):
    """SCENE_SRC records on one image and its PSF: 40 % points, 30 % exp,
    20 % deV, 10 % composites."""
    n, geo, rng = case['n'], _numbers(case), _numbers(case, seed)
    s = np.zeros(n, batch.SCENE_SRC)
    hw = np.round(np.exp(geo.uniform(math.log(7), math.log(127), n))).astype(np.int64)
    s['profile'] = rng.choice([_lib.PROFILE_POINT, _lib.PROFILE_EXP, _lib.PROFILE_DEV,
                               _lib.PROFILE_COMPOSITE], n, p=[.4, .3, .2, .1])
    s['px'], s['py'] = rng.uniform(0, case['w'], n), rng.uniform(0, case['h'], n)
    s['counts'] = np.exp(rng.uniform(math.log(10.), math.log(1e5), n))
    s['sa0'], s['sa1'], s['sa2'] = _ellipses(rng, n)
    s['sb0'], s['sb1'], s['sb2'] = _ellipses(rng, n)
    s['fdev'] = rng.uniform(0., 1., n)
    s['shape_type'] = _lib.SHAPE_ELLIPSE_E
    s['mx0'], s['my0'] = np.round(s['px']) - hw, np.round(s['py']) - hw
    s['mw'] = s['mh'] = 2 * hw + 1
    K = case['kpsf']
    sig = rng.uniform(.9, 1.6) * 1.8 ** np.arange(K)
    wt = .4 ** np.arange(K)
    return s, sig, wt / wt.sum()


def _blobs(case, seed):
    """The blob-fitting workload: 192-512 px images in three bands, about six
    Sersic galaxies each on a mask of its size, a three-Gaussian PSF and noise
    of its own per image; the truth and a start near it."""
    n, geo, rng = case['blobs'], _numbers(case), _numbers(case, seed)
    side, nsrc = geo.integers(192, 513, n), np.clip(geo.poisson(6, n), 1, 30)
    blob_of, m = np.repeat(np.arange(n), nsrc), int(nsrc.sum())
    sigma = rng.uniform(1., 2., (n, 3))
    truth = np.zeros((m, fit.NPAR))
    truth[:, 0], truth[:, 1] = rng.uniform(8, (side[blob_of] - 8)[None, :], (2, m))
    truth[:, 2:5] = np.exp(rng.uniform(math.log(500.), math.log(5e4), (m, 3)))
    re, e1, e2 = _ellipses(rng, m)
    e = np.hypot(e1, e2)
    truth[:, 5], truth[:, 6], truth[:, 7] = np.log(re), *(-np.log(1. - e) / e * np.stack([e1, e2]))
    truth[:, 8] = rng.uniform(.7, 6., m)
    start = truth.copy()
    start[:, 0:2] += rng.uniform(-.5, .5, (m, 2))
    start[:, 2:5] *= rng.uniform(.8, 1.25, (m, 3))
    start[:, 5] += rng.uniform(-.2, .2, m)
    start[:, 6:8] += rng.uniform(-.05, .05, (m, 2))
    start[:, 8] = np.clip(start[:, 8] + rng.uniform(-.5, .5, m), .5, 6.)
    hw = np.clip(np.round(6 * re + 12 * sigma.max(axis=1)[blob_of]), 8, 64).astype(np.int64)
    sources = np.zeros(m, _lib.FIT_SOURCE)
    sources['profile'] = _lib.PROFILE_SERSIC
    sources['x0'] = np.round(truth[:, 0]).astype(np.int64) - hw
    sources['y0'] = np.round(truth[:, 1]).astype(np.int64) - hw
    sources['w'] = sources['h'] = 2 * hw + 1
    psf = [[(np.array([.7, .2, .1]), np.zeros((3, 2)),
             np.eye(2) * (s * np.array([1., 2., 4.]))[:, None, None] ** 2) for s in row]
           for row in sigma]
    return dict(blob_src=np.concatenate([[0], np.cumsum(nsrc)]), sides=np.stack([side, side], 1),
                psf=psf, sources=sources, truth=truth, start=start, n_bands=3,
                noise=rng.uniform(1., 3., (n, 3)))


def _blob_images(w, seed):
    po = fit.pix_offsets(w['sides'], w['n_bands'])
    data = torch.zeros(int(po[-1]), dtype=torch.float32, device=_device())
    for at, patch in _blob_patches(w, torch.from_numpy(w['truth'])):
        data.as_strided(*at).add_(patch.float())
    sig = torch.from_numpy(np.repeat(w['noise'].reshape(-1), np.diff(po)).astype(np.float32))
    sig = sig.to(_device())
    g = torch.Generator(device=_device()).manual_seed(seed)
    data += sig * torch.randn(data.shape, generator=g, device=_device())
    return data, 1. / sig


def _fitter(w, data, inverr):
    return fit.BlobFitter(w['blob_src'], w['sides'], w['psf'], w['sources'], w['start'], data,
                          inverr, n_bands=w['n_bands'])


def _lsq_inputs(case, seed):
    n, p, rows = case['n'], case['p'], case['rows']
    g = torch.Generator(device=_device()).manual_seed(seed)
    A = torch.randn(n * p * rows, generator=g, device=_device())
    r = torch.randn(n * rows, generator=g, device=_device())
    return A, r


def _stamps(case, seed):
    """PSF stamps of two concentric Gaussians plus noise, as fromStamp
    normalises and clips them, and em_fit's usual start."""
    rng, n, side, K = _numbers(case, seed), case['n'], case['side'], case['k']
    y, x = np.mgrid[:side, :side] - float(side // 2)
    s = rng.uniform(1., 2., (n, 1, 1))
    cx, cy = rng.uniform(-.5, .5, (2, n, 1, 1))
    r2 = (x - cx) ** 2 + (y - cy) ** 2
    im = .7 * np.exp(-r2 / (2 * s * s)) + .3 * np.exp(-r2 / (2 * (2.5 * s) ** 2))
    im = im / im.sum(axis=(1, 2), keepdims=True) + rng.normal(0., 1e-5, im.shape)
    im = np.maximum(im / im.sum(axis=(1, 2), keepdims=True), 0.)
    return (im, np.full((n, K), 1. / K), np.zeros((n, K, 2)),
            np.broadcast_to(np.eye(2) * np.arange(1, K + 1)[:, None, None], (n, K, 2, 2)).copy())


API_SIGMAS, API_WEIGHTS = [1.5, 3.0], [.8, .2]


def _api_rows(case, seed):
    """Per source: profile, x, y, counts, ellipse, half-width of its mask."""
    n, geo, rng = case['n'], _numbers(case), _numbers(case, seed)
    kind = rng.choice([_lib.PROFILE_POINT, _lib.PROFILE_EXP, _lib.PROFILE_DEV,
                       _lib.PROFILE_SERSIC], n)
    ell = np.stack(_ellipses(rng, n), 1)
    return [dict(kind=int(kind[i]), x=rng.uniform(4, case['w'] - 4), y=rng.uniform(4, case['h'] - 4),
                 counts=math.exp(rng.uniform(math.log(100.), math.log(1e5))), ell=ell[i],
                 n=rng.uniform(.7, 6.), hw=int(geo.integers(8, 40))) for i in range(n)]


def _tractor(case, seed):
    w, h = case['w'], case['h']
    srcs, masks = [], {}
    for r in _api_rows(case, seed):
        pos, flux = T.PixPos(r['x'], r['y']), T.Flux(r['counts'])
        if r['kind'] == _lib.PROFILE_POINT:
            s = T.PointSource(pos, flux)
        elif r['kind'] == _lib.PROFILE_SERSIC:
            s = T.SersicGalaxy(pos, flux, T.EllipseE(*r['ell']), T.SersicIndex(r['n']))
        else:
            s = (T.ExpGalaxy if r['kind'] == _lib.PROFILE_EXP else T.DevGalaxy)(
                pos, flux, T.EllipseE(*r['ell']))
        x0, y0 = max(0, int(r['x']) - r['hw']), max(0, int(r['y']) - r['hw'])
        x1, y1 = min(w, int(r['x']) + r['hw'] + 1), min(h, int(r['y']) + r['hw'] + 1)
        masks[s] = T.ModelMask(x0, y0, x1 - x0, y1 - y0)
        srcs.append(s)
    tim = T.Image(data=np.zeros((h, w), np.float32), invvar=np.ones((h, w), np.float32),
                  psf=T.NCircularGaussianPSF(API_SIGMAS, API_WEIGHTS),
                  photocal=T.LinearPhotoCal(1.))
    tr = T.Tractor([tim], srcs)
    tr.setModelMasks([masks])
    return tr


# ---------------------------------------------------------------------------
# what a program holds, and one pass
# ---------------------------------------------------------------------------

def prepare(case, seed):
    kind = case['kind']
    if kind == 'fourier':
        s, npix = _galaxies(case, seed)
        return dict(kind=kind, n=case['n'], src=_on_device(s),
                    renderer=batch.FourierGalaxyRenderer(_moffat(case['psf'])),
                    out=torch.empty(npix, dtype=torch.float32, device=_device()))
    if kind == 'fourier_grad':
        s, npix, up = _gradient_inputs(case, seed)
        theta = s.view(np.float64).reshape(case['n'], -1)[:, :grad.NPARAM].astype(np.float32)
        return dict(kind=kind, npix=npix, up=up, template=_on_device(s),
                    renderer=batch.FourierGalaxyRenderer(_moffat(case['psf'])),
                    theta=torch.from_numpy(theta).to(_device()).requires_grad_())
    if kind == 'scene':
        s, sig, wt = _scene(case, seed)
        r = batch.SceneRenderer([batch.SceneImage.circular(case['w'], case['h'], sig, wt)])
        return dict(kind=kind, n=case['n'], renderer=r, src=_on_device(s),
                    pairs=r.max_pairs(s, r.tile_h),
                    out=torch.empty(r.npix, dtype=torch.float32, device=_device()))
    if kind == 'fit':
        w = _blobs(case, seed)
        return dict(kind=kind, start=w['start'], fitter=_fitter(w, *_blob_images(w, seed)))
    if kind == 'blob_grad':
        w = _blobs(case, seed)
        npix = int(fit.pix_offsets(w['sides'], w['n_bands'])[-1])
        none = torch.zeros(npix, dtype=torch.float32, device=_device())
        g = torch.Generator(device=_device()).manual_seed(seed)
        return dict(kind=kind, model=grad.BlobModel(_fitter(w, none, none)),
                    theta=torch.from_numpy(w['start']).to(_device()).requires_grad_(),
                    up=torch.randn(npix, generator=g, device=_device()))
    if kind == 'lsq':
        n, p, rows = case['n'], case['p'], case['rows']
        A, r = _lsq_inputs(case, seed)
        i = np.arange(n, dtype=np.int64)
        return dict(kind=kind, A=A, r=r, P=np.full(n, p, np.int32), a_off=i * p * rows,
                    r_off=i * rows, rows=np.full(n, rows, np.int32))
    if kind == 'em':
        return dict(kind=kind, steps=case['steps'], stamps=_stamps(case, seed))
    return dict(kind=kind, tractor=_tractor(case, seed))


def run(st):
    kind = st['kind']
    if kind == 'fourier':
        st['renderer'].render_device(st['src'], st['n'], st['out'])
        return st['out']
    if kind == 'fourier_grad':
        # single-precision parameters, as an optimizer of torch holds them
        model, _ = grad.RenderGalaxies.apply(st['theta'].double(), st['renderer'],
                                             st['template'], st['npix'])
        g, = torch.autograd.grad(model, st['theta'], st['up'])
        return model, g
    if kind == 'scene':
        st['renderer'].render_device(st['src'], st['n'], st['out'], st['pairs'])
        return st['out']
    if kind == 'fit':
        st['fitter'].fit(params0=st['start'])
        return st['fitter'].result().astype(np.float32)   # a catalog's columns
    if kind == 'blob_grad':
        model = grad.RenderBlobs.apply(st['theta'], st['model'])
        g, = torch.autograd.grad(model, st['theta'], st['up'])
        return model, g
    if kind == 'lsq':
        AtA, Atr, ao, ro = render.normal_equations(st['A'], st['r'], st['a_off'], st['r_off'],
                                                   st['rows'], st['P'], st['rows'])
        X, info, _ = render.solve_update(AtA, Atr, ao, ro, st['P'])
        # stored in single precision, as the columns they come from
        return AtA.float(), Atr.float(), X.float(), info
    if kind == 'em':
        img, amp, mean, var = st['stamps']
        return emfit.em_fit_2d_batch(img, amp, mean, var, steps=st['steps'])
    return st['tractor'].getModelImage(0)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def _fft_size(w, h, psf):
    hs = max(w / 2 + 1.5, h / 2 + 1.5, psf / 2)
    return 1 << max(0, math.ceil(math.log2(2 * math.ceil(hs))))


def work(case):
    kind = case['kind']
    if kind in ('fourier', 'fourier_grad'):
        w, h = _patch_sizes(case)
        npix = int((w * h).sum())
        flops = 0.
        for a, b in zip(w, h):
            sz = _fft_size(a, b, case['psf'])
            # 8 components of a spectrum (half of it by Hermitian symmetry),
            # the product, a real inverse FFT
            flops += sz * (sz / 2 + 1) * (8 * 8 + 6) + 2.5 * sz * sz * math.log2(sz * sz)
        if kind == 'fourier':
            return dict(bytes=4 * npix + 88 * case['n'], flops=flops)
        # the model, and the transform of the gradient against the spectrum's
        # derivatives
        return dict(bytes=8 * npix + 2 * 56 * case['n'], flops=3 * flops)
    if kind == 'scene':
        hw = np.round(np.exp(_numbers(case).uniform(math.log(7), math.log(127), case['n'])))
        px = float(((2 * hw + 1) ** 2).sum()) * min(1., .9)     # masks cut by the image's edge
        comps = case['kpsf'] * (.4 * 1 + .3 * 6 + .2 * 9 + .1 * 15)
        return dict(bytes=4 * case['w'] * case['h'] + 128 * case['n'], flops=px * comps * 10)
    if kind in ('fit', 'blob_grad'):
        n, npix = case['blobs'], case['blobs'] * 3 * 352. ** 2
        px = n * 6 * 3 * 70. ** 2                               # (source, band) mask pixels
        if kind == 'blob_grad':
            return dict(bytes=8 * npix, flops=px * 27 * (10 + 50))
        # ten iterations: model, derivatives and normal equations each time
        return dict(bytes=8 * npix, flops=10 * px * (27 * 50 + 8 * 8))
    if kind == 'lsq':
        n, p, rows = case['n'], case['p'], case['rows']
        return dict(bytes=4. * n * (p + 1) * rows + 8. * n * p * (p + 1),
                    flops=1. * n * rows * p * (p + 3))
    if kind == 'em':
        px = case['n'] * case['side'] ** 2
        return dict(bytes=8 * px, flops=1. * px * case['k'] * case['steps'] * 40)
    return dict(bytes=4 * case['w'] * case['h'], flops=case['n'] * 50. ** 2 * 12 * 10)


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------

_TABLES = []


def _tables():
    if not _TABLES:
        with open(os.path.join(os.path.dirname(T.__file__), 'data', 'profile_tables.json')) as f:
            _TABLES.append(json.load(f))
    return _TABLES[0]


def _spline(sp, x):
    """A B-spline by de Boor's recursion (x complex: its derivative too)."""
    t, c, k = sp['t'], sp['c'], sp['k']
    m = max(j for j in range(k, len(t) - k - 1) if j == k or t[j] <= x.real)
    d = [complex(v) for v in c[m - k:m + 1]]
    for r in range(1, k + 1):
        for j in range(k, r - 1, -1):
            lo, hi = t[j + m - k], t[j + 1 + m - r]
            a = (x - lo) / (hi - lo)
            d[j] = (1 - a) * d[j - 1] + a * d[j]
    return d[k]


def _profile(kind, n):
    """(amp, d amp / dn, var, d var / dn) of a profile's mixture."""
    t, zero = _tables(), lambda v: np.zeros(len(v))  # noqa: E731
    if kind == _lib.PROFILE_POINT:
        return np.ones(1), np.zeros(1), np.zeros(1), np.zeros(1)
    if kind != _lib.PROFILE_SERSIC:
        m = t['exp'] if kind == _lib.PROFILE_EXP else t['dev']
        return np.array(m['amp']), zero(m['amp']), np.array(m['var']), zero(m['var'])
    S, step = t['sersic'], 1e-30
    x = complex(min(max(n, S['lowest']), S['highest']), step)
    R = next((r for r in S['ranges'] if r['lo'] <= x.real < r['hi']), S['ranges'][-1])
    a = np.array([_spline(sp, x) for sp in R['amp_splines']])
    v = np.exp(np.array([_spline(sp, x) for sp in R['logvar_splines']]))
    a = a / a.sum()
    if x.real > 1.:
        core = _spline(S['core_spline'], x)
        a, v = np.append(a * (1 - core), core), np.append(v, 0j)
    return a.real, a.imag / step, v.real, v.imag / step


def _profiles(kinds, ns):
    """_profile of many sources, padded with components of no amplitude."""
    got = [_profile(int(k), float(n)) for k, n in zip(kinds, ns)]
    out = np.zeros((4, len(got), max(len(g[0]) for g in got)))
    for i, g in enumerate(got):
        for j in range(4):
            out[j, i, :len(g[0])] = g[j]
    return out


def _covariance(re, e1, e2):
    """(xx, xy, yy) of a unit-variance component of an EllipseE shape."""
    th, e = torch.atan2(e2, e1) / 2, torch.sqrt(e1 * e1 + e2 * e2)
    ba, c, s = (1 - e) / (1 + e), torch.cos(th), torch.sin(th)
    return (re * re * (c * c * ba * ba + s * s), re * re * c * s * (1 - ba * ba),
            re * re * (s * s * ba * ba + c * c))


def _soft(logre, ee1, ee2):
    """EllipseESoft -> EllipseE."""
    ee = torch.sqrt(ee1 * ee1 + ee2 * ee2)
    f = (1 - torch.exp(-ee)) / ee
    return torch.exp(logre), ee1 * f, ee2 * f


def _taps(d):
    """Normalised Lanczos-3 taps (n, 7) of shifts d (n,)."""
    i = torch.arange(7, dtype=torch.float64, device=d.device)
    p = math.pi * (i[None, :] - 3 + d[:, None])
    use = torch.where(d[:, None] > 0, i[None, :] < 6, i[None, :] > 0) & (d[:, None] != 0)
    safe = torch.where(p.abs() < 1e-300, torch.ones_like(p), p)
    t = torch.where(use, 3 * torch.sin(safe) * torch.sin(safe / 3) / (safe * safe),
                    torch.zeros_like(p))
    t = torch.where((d == 0)[:, None], (i == 3).double()[None, :], t)
    return t / t.sum(1, keepdim=True)


def _fourier64(rows, psf, npix, up=None):
    """The galaxies' patches, and with `up` the gradient of sum(up * patches)
    in (x, y, counts, shape, Sersic index)."""
    dev = _device()
    names = ('px', 'py', 'counts', 's0', 's1', 's2', 'sersic_n')
    theta = torch.from_numpy(np.stack([rows[k] for k in names], 1)).to(dev)
    theta.requires_grad_(up is not None)
    a0, da, v0, dv = (torch.from_numpy(q).to(dev) for q in _profiles(rows['profile'],
                                                                     rows['sersic_n']))
    out = torch.zeros(npix, dtype=torch.float64, device=dev)
    ph, pw = psf.shape
    sizes = np.array([_fft_size_at(r, psf.shape) for r in rows])
    for sz in np.unique(sizes):
        pad = np.zeros((sz, sz))
        oy, ox = (sz - ph) // 2, (sz - pw) // 2
        pad[oy:oy + ph, ox:ox + pw] = psf
        spec = torch.fft.rfft2(torch.from_numpy(pad).to(dev))
        V = torch.fft.rfftfreq(int(sz), device=dev, dtype=torch.float64)[None, None, None, :]
        W = torch.fft.fftfreq(int(sz), device=dev, dtype=torch.float64)[None, None, :, None]
        at = np.nonzero(sizes == sz)[0]
        step = 8 if up is not None else 48
        for q in range(0, len(at), step):
            idx = at[q:q + step]
            ti = torch.from_numpy(idx).to(dev)
            th = theta[ti]
            dn = (th[:, 6] - th[:, 6].detach())[:, None]
            a, v = a0[ti] + da[ti] * dn, v0[ti] + dv[ti] * dn
            cxx, cxy, cyy = (c[:, None] * v for c in _covariance(th[:, 3], th[:, 4], th[:, 5]))
            ex = lambda c: c[:, :, None, None]  # noqa: E731
            F = (ex(a) * torch.exp(-2 * math.pi ** 2 * (ex(cxx) * V * V + 2 * ex(cxy) * V * W +
                                                        ex(cyy) * W * W))).sum(1)
            G = torch.fft.irfft2(F * spec, s=(int(sz), int(sz)))
            mux = th[:, 0] - (ox + pw // 2) - torch.from_numpy(rows['mx0'][idx].astype(float)).to(dev)
            muy = th[:, 1] - (oy + ph // 2) - torch.from_numpy(rows['my0'][idx].astype(float)).to(dev)
            sx, sy = torch.round(mux.detach()), torch.round(muy.detach())
            fx, fy = _taps(mux - sx), _taps(muy - sy)
            P = torch.nn.functional.pad(G, (3, 3, 0, 0))
            G = sum(fx[:, j, None, None] * P[:, :, j:j + int(sz)] for j in range(7))
            P = torch.nn.functional.pad(G, (0, 0, 3, 3))
            G = sum(fy[:, j, None, None] * P[:, j:j + int(sz), :] for j in range(7))
            G = G * th[:, 2, None, None]
            total = 0.
            for j, i in enumerate(idx):
                w, h, o = int(rows['mw'][i]), int(rows['mh'][i]), int(rows['out_off'][i])
                dx, dy = int(sx[j]), int(sy[j])
                y0, y1, x0, x1 = max(0, -dy), min(int(sz), h - dy), max(0, -dx), min(int(sz), w - dx)
                if y1 <= y0 or x1 <= x0:
                    continue
                patch = G[j, y0:y1, x0:x1]
                out[o:o + w * h].view(h, w)[y0 + dy:y1 + dy, x0 + dx:x1 + dx] = patch.detach()
                if up is not None:
                    u = up[o:o + w * h].view(h, w)[y0 + dy:y1 + dy, x0 + dx:x1 + dx]
                    total = total + (patch * u.double()).sum()
            if up is not None and torch.is_tensor(total):
                total.backward()
    return out, theta.grad


def _fft_size_at(r, psf_shape):
    x1, y1 = r['mx0'] + r['mw'], r['my0'] + r['mh']
    hs = max(r['mh'] / 2, r['mw'] / 2, 1 + r['px'] - r['mx0'], 1 + x1 - r['px'],
             1 + r['py'] - r['my0'], 1 + y1 - r['py'], psf_shape[0] / 2, psf_shape[1] / 2)
    sz = 1
    while sz < 2 * math.ceil(hs):
        sz *= 2
    return sz


def _gaussians(box, amp, x, y, cxx, cxy, cyy):
    """A mixture (K,) on the pixels of box = (x0, x1, y0, y1)."""
    dev = amp.device
    dx = torch.arange(box[0], box[1], dtype=torch.float64, device=dev)[None, None, :] - x[:, None, None]
    dy = torch.arange(box[2], box[3], dtype=torch.float64, device=dev)[None, :, None] - y[:, None, None]
    det = cxx * cyy - cxy * cxy
    a = amp / (2 * math.pi * torch.sqrt(det))
    q = ((cyy / det)[:, None, None] * dx * dx - (2 * cxy / det)[:, None, None] * dx * dy +
         (cxx / det)[:, None, None] * dy * dy)
    return (a[:, None, None] * torch.exp(-.5 * q)).sum(0)


def _with_psf(amp, cov, wt, psf_cov):
    """Components (K,) convolved with centred PSF components (P,)."""
    a = (wt[:, None] * amp[None, :]).reshape(-1)
    return (a,) + tuple((p[:, None] + c[None, :]).reshape(-1) for p, c in zip(psf_cov, cov))


def _scene64(rows, w, h, sig, wt):
    dev = _device()
    out = torch.zeros((h, w), dtype=torch.float64, device=dev)
    d = lambda q: torch.from_numpy(np.ascontiguousarray(q, np.float64)).to(dev)  # noqa: E731
    wt, s2 = d(wt), d(np.asarray(sig) ** 2)
    psf_cov = (s2, torch.zeros_like(s2), s2)
    A = torch.stack(_covariance(d(rows['sa0']), d(rows['sa1']), d(rows['sa2'])))
    B = torch.stack(_covariance(d(rows['sb0']), d(rows['sb1']), d(rows['sb2'])))
    ea, _, ev, _ = (d(q) for q in _profile(_lib.PROFILE_EXP, 1.))
    va, _, vv, _ = (d(q) for q in _profile(_lib.PROFILE_DEV, 1.))
    px, py, counts = d(rows['px']), d(rows['py']), d(rows['counts'])
    for i, r in enumerate(rows):
        x0, y0 = max(0, int(r['mx0'])), max(0, int(r['my0']))
        x1, y1 = min(w, int(r['mx0'] + r['mw'])), min(h, int(r['my0'] + r['mh']))
        if x1 <= x0 or y1 <= y0:
            continue
        k = r['profile']
        if k == _lib.PROFILE_POINT:
            a, cov = torch.ones(1, dtype=torch.float64, device=dev), torch.zeros((3, 1), device=dev)
        elif k == _lib.PROFILE_EXP:
            a, cov = ea, A[:, i, None] * ev
        elif k == _lib.PROFILE_DEV:
            a, cov = va, A[:, i, None] * vv
        elif k == _lib.PROFILE_SERSIC:
            q = _profile(k, float(r['sersic_n']))
            a, cov = d(q[0]), A[:, i, None] * d(q[2])
        else:
            f = float(min(1., max(0., r['fdev'])))
            a = torch.cat([f * va, (1 - f) * ea])
            cov = torch.cat([B[:, i, None] * vv, A[:, i, None] * ev], 1)
        m = _with_psf(a, cov, wt, psf_cov)
        K = len(m[0])
        out[y0:y1, x0:x1] += counts[i] * _gaussians((x0, x1, y0, y1), m[0], px[i].expand(K),
                                                    py[i].expand(K), *m[1:])
    return out


def _blob_patches(w, theta):
    """Yields (strided view of the packed images, model patch) for every
    source and band; differentiable in theta (n, 9)."""
    dev = _device()
    theta = theta.to(dev)
    po = fit.pix_offsets(w['sides'], w['n_bands'])
    n = len(w['sources'])
    host = theta.detach().cpu().numpy()
    prof = torch.from_numpy(_profiles([_lib.PROFILE_SERSIC] * n, host[:, 8])).to(dev)
    psf = torch.from_numpy(np.array([[[m[0], m[2][:, 0, 0], m[2][:, 0, 1], m[2][:, 1, 1]]
                                      for m in row] for row in w['psf']])).to(dev)
    blob_of = np.repeat(np.arange(len(w['sides'])), np.diff(w['blob_src']))
    for s, r in enumerate(w['sources']):
        b = int(blob_of[s])
        W, H = (int(q) for q in w['sides'][b])
        x0, y0 = max(0, int(r['x0'])), max(0, int(r['y0']))
        x1, y1 = min(W, int(r['x0'] + r['w'])), min(H, int(r['y0'] + r['h']))
        if x1 <= x0 or y1 <= y0:
            continue
        th = theta[s]
        dn = th[8] - th[8].detach()
        a, v = prof[0, s] + prof[1, s] * dn, prof[2, s] + prof[3, s] * dn
        cov = [c * v for c in _covariance(*_soft(th[5], th[6], th[7]))]
        for k in range(w['n_bands']):
            m = _with_psf(a, cov, psf[b, k, 0], tuple(psf[b, k, 1:]))
            K = len(m[0])
            patch = th[2 + k] * _gaussians((x0, x1, y0, y1), m[0], th[0].expand(K),
                                           th[1].expand(K), *m[1:])
            yield ((y1 - y0, x1 - x0), (W, 1), int(po[b * w['n_bands'] + k]) + y0 * W + x0), patch


def _em64(case, seed):
    dev = _device()
    img, amp, mean, var = (torch.from_numpy(q).to(dev) for q in _stamps(case, seed))
    n, side, K = case['n'], case['side'], case['k']
    g = torch.arange(side, dtype=torch.float64, device=dev) - side // 2
    y, x = (q.reshape(1, 1, -1) for q in torch.meshgrid(g, g, indexing='ij'))
    I = img.reshape(n, 1, -1)
    cxx, cxy, cyy = var[:, :, 0, 0, None], var[:, :, 0, 1, None], var[:, :, 1, 1, None]
    amp, mx, my = amp[:, :, None], mean[:, :, 0, None], mean[:, :, 1, None]
    for _ in range(case['steps']):
        det = cxx * cyy - cxy * cxy
        dx, dy = x - mx, y - my
        q = (cyy * dx * dx - 2 * cxy * dx * dy + cxx * dy * dy) / det
        z = torch.where(q >= 100, 0., amp / (2 * math.pi * torch.sqrt(det)) * torch.exp(-.5 * q))
        s = z.sum(1, keepdim=True)
        wgt = I * z / torch.where(s != 0, s, 1.)
        amp = wgt.sum(2, keepdim=True)
        mx, my = (wgt * x).sum(2, keepdim=True) / amp, (wgt * y).sum(2, keepdim=True) / amp
        dx, dy = x - mx, y - my
        cxx, cxy, cyy = ((wgt * u * t).sum(2, keepdim=True) / amp
                         for u, t in ((dx, dx), (dx, dy), (dy, dy)))
    V = torch.cat([cxx, cxy, cxy, cyy], 2).reshape(n, K, 2, 2)
    return amp[:, :, 0], torch.cat([mx, my], 2), V, None


def exact(case, seed):
    kind = case['kind']
    if kind == 'fourier':
        s, npix = _galaxies(case, seed)
        return _fourier64(s, _moffat(case['psf']), npix)[0]
    if kind == 'fourier_grad':
        s, npix, up = _gradient_inputs(case, seed)
        return _fourier64(s, _moffat(case['psf']), npix, up)
    if kind == 'scene':
        s, sig, wt = _scene(case, seed)
        return _scene64(s, case['w'], case['h'], sig, wt).reshape(-1)
    if kind == 'blob_grad':
        w = _blobs(case, seed)
        theta = torch.from_numpy(w['start']).to(_device()).requires_grad_()
        npix = int(fit.pix_offsets(w['sides'], w['n_bands'])[-1])
        g = torch.Generator(device=_device()).manual_seed(seed)
        up = torch.randn(npix, generator=g, device=_device())
        model = torch.zeros(npix, dtype=torch.float64, device=_device())
        total, count = 0., 0
        for at, patch in _blob_patches(w, theta):
            model.as_strided(*at).add_(patch.detach())
            total, count = total + (patch * up.as_strided(*at).double()).sum(), count + 1
            if count % 3 == 0:      # a source's bands together
                total.backward()
                total = 0.
        return model, theta.grad
    if kind == 'lsq':
        n, p, rows = case['n'], case['p'], case['rows']
        A, r = _lsq_inputs(case, seed)
        AtA = torch.empty((n, p, p), dtype=torch.float64, device=_device())
        Atr = torch.empty((n, p), dtype=torch.float64, device=_device())
        for i in range(n):
            a = A[i * p * rows:(i + 1) * p * rows].view(p, rows).double()
            AtA[i], Atr[i] = a @ a.T, a @ r[i * rows:(i + 1) * rows].double()
        X = torch.linalg.solve(AtA, Atr[:, :, None])
        return AtA.reshape(-1), Atr.reshape(-1), X.reshape(-1), None
    if kind == 'em':
        return _em64(case, seed)
    if kind == 'api':
        rows = _api_rows(case, seed)
        s = np.zeros(len(rows), batch.SCENE_SRC)
        for q, r in zip(s, rows):
            q['profile'], q['sersic_n'], q['counts'] = r['kind'], r['n'], r['counts']
            q['px'], q['py'] = r['x'], r['y']
            q['sa0'], q['sa1'], q['sa2'] = r['ell']
            q['sb0'] = 1.
            q['mx0'], q['my0'] = int(r['x']) - r['hw'], int(r['y']) - r['hw']
            q['mw'] = q['mh'] = 2 * r['hw'] + 1
        return _scene64(s, case['w'], case['h'], API_SIGMAS, API_WEIGHTS)
    return None     # a whole fit: its path has no value of its own in 64 bits
