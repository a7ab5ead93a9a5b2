"""Batched blob fitting (tb_fit_prep / tb_fit_pass / tb_fit_step) against the
oracle's FP64 blob model, its central-difference normal equations and its
tightly converged FP64 fit.

Tolerances: A^T A and A^T r within 1e-4 of their natural scales
(sqrt(H_ii H_jj), sqrt(H_ii chi^2)); chi^2 within 1e-5 relative; fitted
parameters within 1e-3 sigma of the FP64 optimum (sigma from the FP64
inverse Fisher matrix)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _small_blobs(oracle, seed, n_blobs=3, flux=(300., 4000.)):
    from tractor_b200 import fit, _lib
    rng = np.random.default_rng(seed)
    w = fit.blob_workload(n_blobs, rng, side_range=(40, 64), mean_src=2, max_src=3,
                          flux_range=flux)
    # Sersic indices in the middle of the spline ranges (central differences
    # in the oracle must not straddle a range edge)
    ns = np.array([0.8, 1.2, 2.2, 4.5, 5.5])
    w['truth'][:, 8] = ns[rng.integers(0, len(ns), len(w['truth']))]
    w['start'][:, 8] = w['truth'][:, 8] + rng.uniform(-0.05, 0.05, len(w['truth']))
    datas, inverrs = [], []
    for b in range(n_blobs):
        s0, s1 = w['blob_src'][b], w['blob_src'][b + 1]
        W, H = w['sides'][b]
        rects = [tuple(int(v) for v in (r['x0'], r['y0'], r['w'], r['h']))
                 for r in w['sources'][s0:s1]]
        mod = oracle.blob_model(w['truth'][s0:s1], rects, W, H, w['psf'][b], 3)
        sig = w['noise'][b][:, None, None]
        datas.append((mod + sig * rng.normal(size=mod.shape)).astype(np.float32))
        inverrs.append(np.broadcast_to(1. / sig, mod.shape).astype(np.float32))
    return w, datas, inverrs


def _fitter(w, datas, inverrs):
    import torch
    from tractor_b200 import fit
    data = torch.from_numpy(np.concatenate([d.ravel() for d in datas])).cuda()
    inv = torch.from_numpy(np.concatenate([d.ravel() for d in inverrs])).cuda()
    return fit.BlobFitter(w['blob_src'], w['sides'], w['psf'], w['sources'], w['start'], data,
                          inv)


def _blob_args(w, b):
    s0, s1 = w['blob_src'][b], w['blob_src'][b + 1]
    W, H = (int(v) for v in w['sides'][b])
    rects = [tuple(int(v) for v in (r['x0'], r['y0'], r['w'], r['h']))
             for r in w['sources'][s0:s1]]
    return s0, s1, W, H, rects


def test_normal_equations_match_oracle(tb, oracle):
    """One pass at the starting parameters: the analytic FP32 derivative
    columns reproduce the FP64 central-difference A^T A, A^T r, chi^2."""
    w, datas, inverrs = _small_blobs(oracle, 1)
    f = _fitter(w, datas, inverrs)
    f.fit(max_iter=1, check_every=1, graph=False, refine=False)
    st = f.states()
    for b in range(len(datas)):
        s0, s1, W, H, rects = _blob_args(w, b)
        Ho, go, c2o = oracle.blob_normal_equations(w['start'][s0:s1], rects, W, H, w['psf'][b], 3,
                                                   datas[b].astype(np.float64),
                                                   inverrs[b].astype(np.float64))
        Hg, gg = f.normal_equations(b)
        d = np.sqrt(np.diag(Ho))
        scale = np.outer(d, d)
        live = scale > 0
        assert np.all(np.abs(Hg - Ho)[live] <= 1e-4 * scale[live]), b
        assert np.all(Hg[~live] == 0)
        assert np.all(np.abs(gg - go) <= 1e-4 * d * np.sqrt(c2o) + 1e-9), b
        assert abs(st['chi2'][b] - c2o) <= 1e-5 * c2o, b


def test_refine_normal_equations_match_oracle(tb, oracle):
    """The FP64 evaluation of the final iterations (tb_fit_refine) at the
    starting parameters: its A^T A and A^T r against the oracle's FP64
    central differences within 1e-6 of their natural scales (the
    differences' own error), chi^2 within 1e-9 relative."""
    w, datas, inverrs = _small_blobs(oracle, 1)
    f = _fitter(w, datas, inverrs)
    f.reset(w['start'], 1e-9)
    f._iteration(0.0, 100, precise=True)
    st = f.states()
    for b in range(len(datas)):
        s0, s1, W, H, rects = _blob_args(w, b)
        Ho, go, c2o = oracle.blob_normal_equations(w['start'][s0:s1], rects, W, H, w['psf'][b], 3,
                                                   datas[b].astype(np.float64),
                                                   inverrs[b].astype(np.float64))
        Hg, gg = f.normal_equations(b)
        d = np.sqrt(np.diag(Ho))
        scale = np.outer(d, d)
        live = scale > 0
        assert np.all(np.abs(Hg - Ho)[live] <= 1e-6 * scale[live]), b
        assert np.all(Hg[~live] == 0)
        assert np.all(np.abs(gg - go) <= 1e-6 * d * np.sqrt(c2o) + 1e-9), b
        assert abs(st['chi2'][b] - c2o) <= 1e-9 * c2o, (b, st['chi2'][b], c2o)


@pytest.mark.parametrize('n_src', [1, 2, 4, 5, 7, 8])
def test_refine_crowded_tiles_match_oracle(tb, oracle, n_src):
    """tb_fit_refine where n_src masks of odd sizes share tiles, cut by the
    edges of an odd-sized image: up to four sources in one evaluation, more in
    groups of three.  Tolerances as test_refine_normal_equations_match_oracle."""
    w, datas, inverrs = _small_blobs(oracle, 11, n_blobs=1)
    rng = np.random.default_rng(100 + n_src)
    W, H = 45, 37
    pick = rng.integers(0, len(w['truth']), n_src)
    for k in ('truth', 'start'):
        w[k] = w[k][pick].copy()
        w[k][:, 0], w[k][:, 1] = np.linspace(9., W - 7.3, n_src), np.linspace(H - 6.2, 5., n_src)
    w['start'] += rng.uniform(-0.02, 0.02, w['start'].shape)
    src = np.zeros(n_src, w['sources'].dtype)
    src['profile'] = w['sources']['profile'][0]
    hw = rng.integers(9, 18, n_src)
    src['x0'], src['y0'] = w['truth'][:, 0].astype(int) - hw, w['truth'][:, 1].astype(int) - hw
    src['w'], src['h'] = 2 * hw + 1, 2 * hw
    w.update(sources=src, blob_src=np.array([0, n_src]), sides=np.array([[W, H]]))
    data = rng.normal(2., 1., (3, H, W)).astype(np.float32)
    inv = rng.uniform(0.3, 1., (3, H, W)).astype(np.float32)
    f = _fitter(w, [data], [inv])
    f.reset(w['start'], 1e-9)
    f._iteration(0.0, 100, precise=True)
    _, _, _, _, rects = _blob_args(w, 0)
    Ho, go, c2o = oracle.blob_normal_equations(w['start'], rects, W, H, w['psf'][0], 3,
                                               data.astype(np.float64), inv.astype(np.float64))
    Hg, gg = f.normal_equations(0)
    d = np.sqrt(np.diag(Ho))
    assert np.all(np.abs(Hg - Ho) <= 1e-6 * np.outer(d, d))
    assert np.all(np.abs(gg - go) <= 1e-6 * d * np.sqrt(c2o) + 1e-9)
    assert abs(f.states()['chi2'][0] - c2o) <= 1e-9 * c2o


@pytest.mark.parametrize('n_src', [1, 3, 14, 15, 32])
def test_step_solves_the_damped_equations(tb, oracle, n_src):
    """tb_fit_step against numpy on the H and g it assembled: 9 to 288
    parameters (padded, in shared memory up to 128, in global memory above).
    With damping 0.3 the scaled matrix's condition number is at most
    P / 0.3, so FP64 leaves 1e3 x 1e-16 x P: 1e-10 of the largest step."""
    from tractor_b200 import fit
    w = fit.blob_workload(1, np.random.default_rng(31), side_range=(150, 150), mean_src=40,
                          max_src=n_src)
    assert len(w['truth']) == n_src
    data, inv = fit.render_blobs(w, w['truth'], seed=3)
    f = fit.BlobFitter(w['blob_src'], w['sides'], w['psf'], w['sources'], w['start'], data, inv)
    f.reset(w['start'], 1.0)
    f._iteration(0.0, 100, precise=True)
    H, g = f.normal_equations(0)
    assert np.array_equal(H, H.T) and f.states()['accepted'][0] == 1
    lam = f.states()['lambda'][0]
    assert lam == 0.3
    p = w['start'].ravel()
    d = np.sqrt(np.diag(H))
    assert np.all(d > 0)
    x = np.linalg.solve(H / np.outer(d, d) + lam * np.eye(len(d)), g / d) / d
    most = np.tile([1., 1., 0., 0., 0., 1., 0.1, 0.1, 0.1], n_src)
    big = (most > 0) & (np.abs(x) > most)
    lim = min([1.] + list(most[big] / np.abs(x[big])))
    for i in range(8, len(p), 9):
        if not 0.29 <= p[i] + x[i] <= 6.3:
            lim = min(lim, ((6.3 if x[i] > 0 else 0.29) - p[i]) / x[i])
    got = f.trial.cpu().numpy() - p
    assert np.all(np.abs(got - lim * x) * d <= 1e-10 * np.max(np.abs(lim * x) * d))


def test_fit_converges_to_fp64_optimum(tb, oracle):
    """From the same perturbed start, the batched FP32 fitter and the FP64
    oracle fitter reach the same optimum within 1e-3 sigma."""
    w, datas, inverrs = _small_blobs(oracle, 2)
    f = _fitter(w, datas, inverrs)
    f.fit(tol=1e-7, max_iter=80, check_every=4)
    st = f.states()
    assert np.all(st['status'] != 0), st['status']
    got = f.result()
    for b in range(len(datas)):
        s0, s1, W, H, rects = _blob_args(w, b)
        p, Hf, held = oracle.blob_fit(w['start'][s0:s1], rects, W, H, w['psf'][b], 3,
                                      datas[b].astype(np.float64),
                                      inverrs[b].astype(np.float64))
        # sigma from the Fisher matrix of the free parameters; a parameter
        # held at a bound must sit at the same bound
        free = ~held & (np.diag(Hf) > 0)
        sig = np.full(p.size, np.inf)
        sig[free] = np.sqrt(np.diag(np.linalg.inv(Hf[np.ix_(free, free)])))
        sig = sig.reshape(p.shape)
        assert np.array_equal(got[s0:s1].ravel()[held], p.ravel()[held]), b
        err = np.abs(got[s0:s1] - p) / sig
        assert err.max() < 1e-3, (b, err.max(), np.unravel_index(err.argmax(), err.shape))


def test_graph_and_eager_iterations_agree(tb, oracle):
    """CUDA-graph replays of the iteration give the same result as eager
    launches (same kernels, same order)."""
    w, datas, inverrs = _small_blobs(oracle, 3)
    f = _fitter(w, datas, inverrs)
    f.fit(tol=1e-3, max_iter=24, check_every=4, graph=True, params0=w['start'])
    a, sa = f.result().copy(), f.states().copy()
    f.fit(tol=1e-3, max_iter=24, check_every=4, graph=False, params0=w['start'])
    b, sb = f.result(), f.states()
    assert np.array_equal(a, b)
    assert np.array_equal(sa['iters'], sb['iters'])


def test_many_blobs_fit_at_least_as_well_as_truth(tb):
    """200 blobs of the full-size distribution (sides 192-512, Poisson(6)
    sources, 3 bands): every blob stops, and the fitted chi^2 is no worse
    than the chi^2 of the true parameters for nearly all of them."""
    from tractor_b200 import fit
    rng = np.random.default_rng(7)
    w = fit.blob_workload(200, rng)
    data, inv = fit.render_blobs(w, w['truth'], seed=11)
    f = fit.BlobFitter(w['blob_src'], w['sides'], w['psf'], w['sources'], w['start'], data, inv)
    f.fit(tol=1e-3, max_iter=60, check_every=4)
    st = f.states()
    assert np.all(st['status'] != 0)
    assert np.mean(st['status'] == 1) > 0.95, np.bincount(st['status'])
    fitted = st['chi2'].copy()
    f.fit(max_iter=1, check_every=1, graph=False, params0=w['truth'], refine=False)
    truth = f.states()['chi2']
    npix = np.diff(fit.pix_offsets(w['sides'], 3)).reshape(-1, 3).sum(axis=1)
    assert np.all(np.abs(truth / npix - 1) < 0.05)          # noise model sanity
    ok = fitted <= truth + 1.0
    assert np.mean(ok) > 0.95, np.sort(fitted - truth)[-10:]


def _tractors(w, datas, inverrs):
    """The blobs as reference-style Tractor objects (SersicGalaxy, NanoMaggies
    in g, r, z, EllipseESoft, SersicIndex, model masks)."""
    import tractor_b200 as T
    bands = ['g', 'r', 'z']
    tractors = []
    for b in range(len(datas)):
        s0, s1, W, H, rects = _blob_args(w, b)
        tims = []
        for k in range(3):
            amp, mean, var = w['psf'][b][k]
            tims.append(T.Image(data=datas[b][k], inverr=inverrs[b][k],
                                psf=T.GaussianMixturePSF(amp, mean, var),
                                photocal=T.LinearPhotoCal(1., band=bands[k])))
        srcs, masks = [], {}
        for i in range(s0, s1):
            th = w['start'][i]
            src = T.SersicGalaxy(T.PixPos(th[0], th[1]),
                                 T.NanoMaggies(g=th[2], r=th[3], z=th[4]),
                                 T.EllipseESoft(th[5], th[6], th[7]), T.SersicIndex(th[8]))
            srcs.append(src)
            masks[src] = T.ModelMask(*rects[i - s0])
        tr = T.Tractor(tims, srcs)
        tr.setModelMasks([masks] * 3)
        tractors.append(tr)
    return tractors


def _params_of(tr):
    return np.array([[s.pos.x, s.pos.y, s.brightness.getFlux('g'), s.brightness.getFlux('r'),
                      s.brightness.getFlux('z'), s.shape.logre, s.shape.ee1, s.shape.ee2,
                      s.sersicindex.val] for s in tr.catalog])


def _check_optimum(got, p, Hf, held, frozen, what, tol=None):
    """got within 1e-3 sigma (or the per-parameter `tol`) of the FP64 optimum
    p (sigma from the Fisher matrix of the parameters neither held at a
    bound nor frozen)."""
    free = ~held & ~frozen.ravel() & (np.diag(Hf) > 0)
    sig = np.full(p.size, np.inf)
    sig[free] = np.sqrt(np.diag(np.linalg.inv(Hf[np.ix_(free, free)])))
    err = np.abs(got - p).ravel() / sig
    t = np.full(p.size, 1e-3) if tol is None else tol.ravel()
    assert np.all(err < t), (what, err.max(), err)


def test_fit_tractors_through_the_object_api(tb, oracle):
    """fit.fit_tractors: the same blobs given as reference-style Tractor
    objects reach the FP64 optimum within 1e-3 sigma, and the parameters are
    written back into the objects."""
    from tractor_b200 import fit
    w, datas, inverrs = _small_blobs(oracle, 2)
    tractors = _tractors(w, datas, inverrs)
    st = fit.fit_tractors(tractors, tol=1e-7, max_iter=80)
    assert np.all(st['status'] != 0)
    for b, tr in enumerate(tractors):
        s0, s1, W, H, rects = _blob_args(w, b)
        p, Hf, held = oracle.blob_fit(w['start'][s0:s1], rects, W, H, w['psf'][b], 3,
                                      datas[b].astype(np.float64),
                                      inverrs[b].astype(np.float64))
        _check_optimum(_params_of(tr), p, Hf, held, np.zeros(p.shape, bool), b)


def test_fit_tractors_keeps_frozen_parameters(tb, oracle):
    """Frozen parameters (a source's whole shape, another's y position and r
    flux, a Sersic index), set to their true values, keep them exactly; the
    thawed ones reach the FP64 optimum of the restricted problem: the
    fitted chi^2 (evaluated in FP64) within 1e-4 of the optimum's, and the
    parameters within 1e-3 sigma, a source whose shape is frozen included
    (its Sersic index is then nearly unconstrained, sigma_n ~ 8 for the
    single-source blob here; the fit's FP64 phase takes the last steps on
    FP64 normal equations, so float32 cancellation in the index column no
    longer moves the end point).  (Frozen at wrong values the model misfits, and the FP32 derivatives'
    error, multiplied by the residuals, moves the stationary point by about
    1e-6 sqrt(chi^2) sigma.)"""
    from tractor_b200 import fit
    w, datas, inverrs = _small_blobs(oracle, 2)
    w = dict(w)
    w['start'] = w['start'].copy()
    fzall = np.zeros(w['start'].shape, bool)
    for i in range(len(fzall)):
        cols = [[5, 6, 7], [1, 3], [8]][i % 3]
        fzall[i, cols] = True
        w['start'][i, cols] = w['truth'][i, cols]
    tractors = _tractors(w, datas, inverrs)
    frozen = []
    for b, tr in enumerate(tractors):
        s0 = w['blob_src'][b]
        for i, src in enumerate(tr.catalog):
            if (s0 + i) % 3 == 0:
                src.freezeParam('shape')
            elif (s0 + i) % 3 == 1:
                src.getPosition().freezeParam('y')
                src.getBrightness().freezeParam('r')
            else:
                src.freezeParam('sersicindex')
        frozen.append(fzall[s0:w['blob_src'][b + 1]])
    before = [_params_of(tr) for tr in tractors]
    st = fit.fit_tractors(tractors, tol=1e-7, max_iter=80)
    assert np.all(st['status'] != 0)
    for b, tr in enumerate(tractors):
        s0, s1, W, H, rects = _blob_args(w, b)
        got = _params_of(tr)
        assert np.array_equal(got[frozen[b]], before[b][frozen[b]]), b
        assert np.any(got[~frozen[b]] != before[b][~frozen[b]]), b
        p, Hf, held = oracle.blob_fit(w['start'][s0:s1], rects, W, H, w['psf'][b], 3,
                                      datas[b].astype(np.float64),
                                      inverrs[b].astype(np.float64), frozen=frozen[b])
        tol = np.full(p.shape, 1e-3)
        _check_optimum(got, p, Hf, held, frozen[b], b, tol)
        args = (rects, W, H, w['psf'][b], 3, datas[b].astype(np.float64),
                inverrs[b].astype(np.float64))
        c2_got = oracle.blob_normal_equations(got, *args)[2]
        c2_opt = oracle.blob_normal_equations(p, *args)[2]
        assert c2_got - c2_opt < 1e-4, (b, c2_got - c2_opt)


def test_c5_blobs_reach_the_fp64_optimum(tb, oracle):
    """120 blobs drawn from the full-size blob-fitting distribution (sides
    192-512 px, Poisson(6) Sersic sources, 3 bands, per-band MoG PSFs and
    noise): the batched fit (FP32 iterations, then FP64 normal equations)
    ends within 1e-3 sigma of the FP64 optimum for every blob whose Sersic
    indices stay clear of the profile tables' range edges, and every blob
    stops.  The optimum is the FP64 fitter's
    (tractor_b200.plain.BlobFitFP64: model and analytic Jacobian in FP64 on
    the device, Levenberg-Marquardt to a predicted gain of 1e-10) started
    from the batched result; sigma from its FP64 Fisher matrix.  A blob
    whose optimum puts an index on a range edge (the mixture is a separate
    fit on each side, so the model jumps there and neither fitter has a
    stationary point to converge to), or along whose flattest direction the
    FP64 fitter itself does not converge within 100 iterations from the
    batched result, is held to 0.1 sigma.  The FP64 fitter's normal equations are first
    checked against the oracle's central differences on a small blob."""
    import torch
    from tractor_b200 import fit, plain
    dev = torch.device('cuda')
    # the FP64 fitter's A^T A and A^T r against the oracle's, on a small blob
    ws, datas, inverrs = _small_blobs(oracle, 5, n_blobs=1)
    s0, s1, W, H, rects = _blob_args(ws, 0)
    pf = plain.BlobFitFP64(datas[0].astype(np.float64), inverrs[0].astype(np.float64),
                           ws['psf'][0], rects, dev)
    th = ws['start'][s0:s1]
    Ho, go, c2o = oracle.blob_normal_equations(th, rects, W, H, ws['psf'][0], 3,
                                             datas[0].astype(np.float64),
                                             inverrs[0].astype(np.float64))
    model, J = pf.model_jacobian(th)
    A = (J * pf.w[None]).reshape(J.shape[0], -1)
    r = ((pf.data - model) * pf.w).reshape(-1)
    Hp, gp = (A @ A.T).cpu().numpy(), (A @ r).cpu().numpy()
    d = np.sqrt(np.diag(Ho))
    live = np.outer(d, d) > 0
    assert np.all(np.abs(Hp - Ho)[live] <= 1e-6 * np.outer(d, d)[live])
    assert np.all(np.abs(gp - go) <= 1e-6 * d * np.sqrt(c2o) + 1e-9)
    # the full-size blobs
    rng = np.random.default_rng(17)
    w = fit.blob_workload(120, rng)
    data, inv = fit.render_blobs(w, w['truth'], seed=18)
    f = fit.BlobFitter(w['blob_src'], w['sides'], w['psf'], w['sources'], w['start'], data, inv)
    f.fit(tol=1e-3, max_iter=200)
    st = f.states()
    # every blob stops by convergence or by rejections at the optimum, none
    # at the iteration limit; all of them are compared
    assert np.all((st['status'] == 1) | (st['status'] == 2)), np.bincount(st['status'])
    res = plain.optimum_distance(w, data, inv, f.result(), st['status'],
                                 np.arange(len(st)), dev)
    assert len(res) == 120, len(res)
    # blobs with a well-defined optimum: no index on a range edge, and the
    # FP64 fitter converges from the batched result
    inner = sorted([r for r in res if not r[3] and r[4]], reverse=True)
    other = sorted([r for r in res if r[3] or not r[4]], reverse=True)
    assert len(inner) >= 110 and len(other) <= 5, (len(inner), other)
    assert inner[0][0] < 1e-3, inner[:5]
    assert not other or other[0][0] < 0.1, other


def test_blob_without_sources_keeps_to_its_own_slices(tb, oracle):
    """A blob table entry with n_src = 0 (P = 0, slices of no elements) through
    the passes of both precisions and the step: nothing outside its slices is
    written (the word before them is its neighbour's accepted gradient), its
    chi^2 is its weighted data's, and it stops at once."""
    import torch
    w, datas, inverrs = _small_blobs(oracle, 3, n_blobs=2)
    f = _fitter(w, datas, inverrs)
    f.blobs_np['n_src'][1] = f.blobs_np['P'][1] = 0
    f.d_blobs.copy_(torch.from_numpy(f.blobs_np.view(np.uint8).copy()))
    f.reset(w['start'])
    ns, g0, u0 = (int(f.blobs_np[k][1]) for k in ('n_slices', 'g_off', 'unit0'))
    chi2 = float(((datas[1].astype(np.float64) * inverrs[1]) ** 2).sum())
    for refine in (False, True):
        f.gbuf.fill_(-7.)
        f._prep()
        f._refine_pass() if refine else f._pass(0)
        got = f.gbuf.cpu().numpy()
        assert got[g0 - 1] == -7. and np.all(got[g0:] == -7.), refine
        assert abs(float(f.chi2_part[u0:u0 + ns].sum()) - chi2) <= 1e-5 * chi2
    f.reset(w['start'])
    f._iteration(1e-3, 100)
    st = f.states()
    assert st['status'][1] == 1 and abs(st['chi2'][1] - chi2) <= 1e-5 * chi2


def test_blobs_with_an_undetermined_parameter_do_not_crawl(tb):
    """Two of 2,000 blobs, from where the FP32 iterations left them
    (golden/slow_blobs.npz): each holds a source whose shape is all but
    undetermined, and its step, beyond its limit by up to 1e5, scaled the steps
    of all the others; the FP64 iterations took 97 and more than 100 (4.9 sigma
    from the optimum).  Within 80 they converge to less than 1e-3 sigma from
    the FP64 optimum, as every other blob."""
    import os
    import torch
    from tractor_b200 import fit, plain
    z = np.load(os.path.join(os.path.dirname(__file__), 'golden', 'slow_blobs.npz'))
    w = fit.blob_workload(2000, np.random.default_rng(3000))
    data, inv = fit.render_blobs(w, w['truth'], seed=3001)
    po = fit.pix_offsets(w['sides'], 3)
    cut = [slice(int(po[3 * b]), int(po[3 * b + 3])) for b in z['blobs']]
    data, inv = (torch.cat([a[c] for c in cut]) for a in (data, inv))
    w = fit.subset_workload(w, z['blobs'])
    f = fit.BlobFitter(w['blob_src'], w['sides'], w['psf'], w['sources'], z['start'], data, inv)
    f.fit(params0=z['start'], max_iter=0, graph=False, refine_iter=80)
    st = f.states()
    assert np.all(st['status'] == 1), (st['status'], st['iters'])
    for sigma, b, _, _, converged in plain.optimum_distance(w, data, inv, f.result(), st['status'],
                                                            [0, 1], f.dev):
        assert converged and sigma < 1e-3, (b, sigma)


@pytest.mark.parametrize('unit_tiles', [1, 3, 64, 100])
def test_unit_tiles_are_the_callers(tb, unit_tiles):
    """A caller's unit_tiles is the size of the pass units, whatever the fitter
    would choose: ceil(active tiles / unit_tiles) units per image."""
    from tractor_b200 import fit
    w = fit.blob_workload(2, np.random.default_rng(41), side_range=(300, 400))
    data, inv = fit.render_blobs(w, w['truth'], seed=5)
    f = fit.BlobFitter(w['blob_src'], w['sides'], w['psf'], w['sources'], w['start'], data, inv,
                       unit_tiles=unit_tiles)
    assert np.all(f.blobs_np['n_active'] > 64)
    assert np.array_equal(f.blobs_np['n_slices'], 3 * -(-f.blobs_np['n_active'] // unit_tiles))


@pytest.mark.parametrize('unit_tiles', [1, None])
@pytest.mark.parametrize('n_bands', [1, 2, 3])
@pytest.mark.parametrize('precise', [False, True])
def test_mixed_profiles_crowd_tiles(tb, oracle, precise, n_bands, unit_tiles):
    """Both precisions of the pass where six point, exponential, de Vaucouleurs
    and Sersic sources share tiles in ever other sets, also in units of one tile
    whose slices hold different sources: the assembled A^T A and A^T r against
    FP64 central differences of the oracle's model (1e-4 of their scales in
    FP32, 1e-6 in FP64: the differences' own error), chi^2 to 1e-5 and 1e-9;
    parameters that a profile or a band does not have hold zeros."""
    import torch
    from tractor_b200 import fit, _lib
    rng = np.random.default_rng(51)
    W, H, n = 75, 61, 6
    w = fit.blob_workload(1, rng, side_range=(64, 64), n_bands=n_bands)
    prof = np.array([_lib.PROFILE_POINT, _lib.PROFILE_EXP, _lib.PROFILE_DEV, _lib.PROFILE_SERSIC,
                     _lib.PROFILE_SERSIC, _lib.PROFILE_POINT])
    p = np.zeros((n, 9))
    p[:, 0], p[:, 1] = np.linspace(12., W - 14.3, n), np.linspace(H - 9.2, 11., n)
    p[:, 2:2 + n_bands] = rng.uniform(500., 3000., (n, n_bands))
    gal = prof != _lib.PROFILE_POINT
    p[gal, 5], p[gal, 6:8] = rng.uniform(0., 1., gal.sum()), rng.uniform(-.3, .3, (gal.sum(), 2))
    p[3:5, 8] = 1.3, 4.4
    src = np.zeros(n, w['sources'].dtype)
    src['profile'] = prof
    hw = rng.integers(9, 18, n)
    src['x0'], src['y0'] = p[:, 0].astype(int) - hw, p[:, 1].astype(int) - hw
    src['w'], src['h'] = 2 * hw + 1, 2 * hw
    data = rng.normal(2., 1., (n_bands, H, W)).astype(np.float32)
    inv = rng.uniform(.3, 1., (n_bands, H, W)).astype(np.float32)
    f = fit.BlobFitter(np.array([0, n]), np.array([[W, H]]), w['psf'], src, p,
                       torch.from_numpy(data.ravel()).cuda(), torch.from_numpy(inv.ravel()).cuda(),
                       n_bands=n_bands, unit_tiles=unit_tiles)
    f.reset(p, 1e-9)
    f._iteration(0., 100, precise=precise)

    def model(q):
        """The oracle's model; exp and deV sources through their own mixtures."""
        out = np.zeros((n_bands, H, W))
        for k in range(n_bands):
            pamp, pmean, pvar = w['psf'][0][k]
            for th, pr, r in zip(q, prof, src):
                X0, Y0 = max(r['x0'], 0), max(r['y0'], 0)
                X1, Y1 = min(r['x0'] + r['w'], W), min(r['y0'] + r['h'], H)
                if pr == _lib.PROFILE_SERSIC:
                    a, v = oracle.sersic_profile(th[8])
                elif pr == _lib.PROFILE_POINT:
                    a, v = np.ones(1), np.zeros(1)
                else:
                    a, v = (oracle.exp_profile if pr == _lib.PROFILE_EXP else
                            oracle.dev_profile)()
                T = oracle.nullwcs_cdinv() @ oracle.ellipseE_basis(
                    *oracle.ellipseESoft_to_E(*th[5:8]))
                M = np.zeros((2, 2)) if pr == _lib.PROFILE_POINT else T @ T.T
                amp = (pamp[:, None] * a).ravel()
                mean = np.repeat(pmean, len(a), 0)
                var = (pvar[:, None] + v[None, :, None, None] * M).reshape(-1, 2, 2)
                out[k, Y0:Y1, X0:X1] += th[2 + k] * oracle.mog_grid(X0, X1, Y0, Y1, th[0], th[1],
                                                                    amp, mean, var)
        return out

    step = np.tile([1e-5, 1e-5, 1., 1., 1., 1e-5, 1e-5, 1e-5, 1e-5], (n, 1))
    has = np.ones((n, 9), bool)
    has[:, 2 + n_bands:5] = False
    has[~gal, 5:] = False
    has[prof != _lib.PROFILE_SERSIC, 8] = False
    A = np.zeros((n * 9, data.size))
    for i in np.flatnonzero(has):
        hi, lo = p.copy(), p.copy()
        hi.flat[i] += step.flat[i]
        lo.flat[i] -= step.flat[i]
        A[i] = ((model(hi) - model(lo)) / (2 * step.flat[i]) * inv).ravel()
    r = ((data - model(p)) * inv).ravel()
    Ho, go, c2 = A @ A.T, A @ r, float(r @ r)
    Hg, gg = f.normal_equations(0)
    tol, ctol = (1e-6, 1e-9) if precise else (1e-4, 1e-5)
    d = np.sqrt(np.diag(Ho))
    assert np.all(np.abs(Hg - Ho) <= tol * np.outer(d, d))
    assert np.all(np.abs(gg - go) <= tol * d * np.sqrt(c2))
    assert abs(f.states()['chi2'][0] - c2) <= ctol * c2
